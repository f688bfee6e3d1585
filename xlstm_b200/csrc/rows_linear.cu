// y = x W^T for a few rows of x (decoding: one row per stream): bf16 operands, fp32 accumulation.
//
// The whole cost is the stream of W from HBM, so W is the 128-row side of the products and the rows of x the narrow one
// (D^T [128 features x MB] = W [128 x K] x^T), and the kernel is built around bytes in flight: ~100 KB of TMA stages per
// block, two blocks per SM, the contraction of a 128-feature tile split over the blocks of a cluster (as many as fill the
// machine), which add their partial tiles through distributed shared memory in rank order.  For a caller who knows that the
// kernel in front does not write W (xl_rows_linear_ahead), W's first stages are requested before the wait for that kernel: the
// stream does not stop between the layers.  xl_rows_linear waits first.
// Eight rows, cold W, a small norm in front of every call, against the library GEMM (us): 4096 x 4096 9.3 / 13.0, 4096 x 10944
// 18.4 / 27.9, 2048 x 4096 7.5 / 12.1, 2048 x 5504 8.4 / 14.7, 50304 x 4096 67 / 72 (the bytes alone: 5.1, 13.7, 2.6, 3.4, 63).
// Where 33 to 255 tiles fill the machine unevenly the library is as fast or faster (12304 x 4096: 21.2 / 21.0, 6160 x 2048:
// 8.9 / 8.4), below 4 MB of W both take a launch (1552 x 512: 4.7 / 4.5), and from 32 rows on the tiles of x cost more than
// the split gains (4096 x 4096, 64 rows: 13.5 / 11.5): `LargeModel._linear` draws the lines there.
#include <cuda.h>

#include "common.cuh"

namespace xl {

constexpr int RL_THREADS = 192;        // warp 0 TMA, warp 1 UMMA, warps 2-5 epilogue
constexpr int RL_TILE = 128;           // features per cluster (UMMA M)
constexpr int RL_KB = 64;              // contraction per stage (128 bytes of a row)
constexpr int RL_W_BYTES = RL_TILE * 128;
constexpr int RL_ROWS = 16;            // most rows of x (the narrowest UMMA)
constexpr int RL_BLOCKS = 296;         // two blocks on each of 148 SMs

struct RlMaps {
  CUtensorMap w, x;
};

struct RlLayout {
  static constexpr int X_BYTES = RL_ROWS * 128, STAGE_BYTES = RL_W_BYTES + X_BYTES;
  static constexpr int STAGES = (108 * 1024) / STAGE_BYTES;
  static constexpr int OFF_BAR = STAGES * STAGE_BYTES;   // full, empty per stage, done
  static constexpr int OFF_TMEM = OFF_BAR + (2 * STAGES + 1) * 8;
  static constexpr int DYN_SMEM = OFF_TMEM + 8 + 1024;
  static constexpr uint32_t TMEM_COLS = 32;
  static_assert(RL_ROWS * RL_TILE * 4 <= STAGES * STAGE_BYTES, "the partial tile lies over the stages");
};

__device__ __forceinline__ void rl_load(uint32_t dst_smem, const void* tmap, uint32_t bar, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst_smem),
               "l"(tmap), "r"(bar), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ float rl_ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

__global__ void __launch_bounds__(RL_THREADS) rows_linear_kernel(const __grid_constant__ RlMaps maps, const xl_rows_linear_params p, int ahead) {
  using LY = RlLayout;
  constexpr int STAGES = LY::STAGES;
  extern __shared__ unsigned char rl_smem_raw[];
  unsigned char* smem = rl_smem_raw + ((1024u - (smem_u32(rl_smem_raw) & 1023u)) & 1023u);
  const uint32_t sbase = smem_u32(smem), bar0 = sbase + LY::OFF_BAR;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + LY::OFF_TMEM);
  const int part = blockIdx.x, parts = gridDim.x, n0 = blockIdx.y * RL_TILE;   // a cluster is one row of the grid
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int kb = (p.K + RL_KB - 1) / RL_KB;
  const int first = (int)((long long)kb * part / parts), count = (int)((long long)kb * (part + 1) / parts) - first;

  auto load_first_w = [&]() {   // one thread: W's part of the first stages (what x adds to a stage is announced here as well)
    for (int c = 0; c < STAGES && c < count; ++c) {
      mbar_expect_tx(bar0 + 8u * c, LY::STAGE_BYTES);
      rl_load(sbase + c * LY::STAGE_BYTES, &maps.w, bar0 + 8u * c, (first + c) * RL_KB, n0);
    }
  };
  if (tid == 0) {
    for (int s = 0; s < 2 * STAGES + 1; ++s) mbar_init(bar0 + 8u * s, 1);
    fence_barrier_init();
    if (ahead) load_first_w();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(s_tmem), LY::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  grid_dependency_wait();
  grid_dependents_launch();   // behind the wait, so that whatever the next kernel requests ahead of its own wait is complete

  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      if (!ahead) load_first_w();
      for (int c = 0; c < STAGES && c < count; ++c)
        rl_load(sbase + c * LY::STAGE_BYTES + RL_W_BYTES, &maps.x, bar0 + 8u * c, (first + c) * RL_KB, 0);
      int st = 0;
      uint32_t par = 0;
      for (int c = STAGES; c < count; ++c) {
        if (!mbar_wait(bar0 + 8u * (STAGES + st), par)) { ok = false; break; }
        const uint32_t bar = bar0 + 8u * st, dst = sbase + st * LY::STAGE_BYTES;
        mbar_expect_tx(bar, LY::STAGE_BYTES);
        rl_load(dst, &maps.w, bar, (first + c) * RL_KB, n0);
        rl_load(dst + RL_W_BYTES, &maps.x, bar, (first + c) * RL_KB, 0);
        if (++st == STAGES) { st = 0; par ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // warp-uniform issue code, descriptors from broadcast bases (see mlstm_chunkwise.cu)
    constexpr uint32_t IDESC = umma_idesc_bf16(RL_TILE, RL_ROWS, 0, 0);
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0), sbase_u = __shfl_sync(0xffffffffu, sbase, 0) & 0x3FFFFu;
    const uint32_t bar_u = __shfl_sync(0xffffffffu, bar0, 0);
    const int count_u = __shfl_sync(0xffffffffu, count, 0);
    bool okm = true;
    int st = 0;
    uint32_t par = 0;
#pragma unroll 1
    for (int c = 0; c < count_u; ++c) {
      okm &= okm ? mbar_wait(bar_u + 8u * st, par) : false;
      tc_fence_after();
      const uint32_t sw = sbase_u + st * LY::STAGE_BYTES, sx = sw + RL_W_BYTES;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) umma_ss_lo(tmem_u, umma_desc_lo(sw + kk * 32, 0), umma_desc_lo(sx + kk * 32, 0), IDESC, (c | kk) != 0);
      umma_commit_elect(bar_u + 8u * (STAGES + st));
      if (++st == STAGES) { st = 0; par ^= 1u; }
    }
    umma_commit_elect(bar_u + 16u * STAGES);
    ok = okm;
  } else {
    // lane = feature, tensor-memory column = row of x
    if (!mbar_wait(bar0 + 16u * STAGES, 0u)) ok = false;
    tc_fence_after();
    const int f = (warp & 3) * 32 + lane;
    __nv_bfloat16* y = static_cast<__nv_bfloat16*>(p.y) + n0 + f;
    float* s_part = reinterpret_cast<float*>(smem);   // [row][feature]; every stage has been read
    uint32_t r[16];
    tmem_ld_x16(tmem + ((uint32_t)((warp & 3) * 32) << 16), r);
    tc_wait_ld();
#pragma unroll
    for (int m = 0; m < RL_ROWS; ++m)
      if (m < p.rows) {
        if (parts > 1) s_part[m * RL_TILE + f] = __uint_as_float(r[m]);
        else if (n0 + f < p.N) y[(long long)m * p.N] = __float2bfloat16_rn(__uint_as_float(r[m]));
      }
  }
  if (!ok && p.status) atomicExch(p.status, 1);
  tc_fence_before();
  if (parts > 1) {
    __syncwarp();
    cluster_sync_all();   // (a barrier of the block, too)
    for (int e = part * RL_THREADS + tid; e < p.rows * RL_TILE; e += parts * RL_THREADS) {
      const int f = e & (RL_TILE - 1), m = e / RL_TILE;
      float sum = 0.f;
      for (int r = 0; r < parts; ++r) sum += rl_ld_cluster(mapa_u32(sbase + (uint32_t)e * 4, (uint32_t)r));
      if (n0 + f < p.N) static_cast<__nv_bfloat16*>(p.y)[(long long)m * p.N + n0 + f] = __float2bfloat16_rn(sum);
    }
    __syncwarp();
    cluster_sync_all();   // nobody leaves while its tile is read
  } else {
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, LY::TMEM_COLS);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
typedef CUresult (*rl_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// row-major bf16 matrix [rows x K] -> 2-D map, box = 64 columns x box_rows rows; what lies outside reads zero
static int rl_make_map(CUtensorMap* m, const void* base, int64_t rows, int64_t K, int64_t row_stride, int box_rows) {
  static const rl_encode_fn encode = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    const bool found = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess;
    return found ? reinterpret_cast<rl_encode_fn>(sym) : nullptr;
  }();
  if (!encode) {
    set_last_cuda_error(cudaErrorSymbolNotFound, "cudaGetDriverEntryPoint(cuTensorMapEncodeTiled)");
    return XL_ERR_CUDA;
  }
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)row_stride * 2};
  const cuuint32_t box[2] = {RL_KB, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  const CUresult r = encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled rejected the matrix layout");
    return XL_ERR_BAD_STRIDE;
  }
  return XL_OK;
}

static int launch_rows_linear(const xl_rows_linear_params* p, bool ahead, cudaStream_t st) {
  using LY = RlLayout;
  RlMaps maps;
  int rc = rl_make_map(&maps.w, p->w, p->N, p->K, p->w_sr, RL_TILE);
  if (rc != XL_OK) return rc;
  rc = rl_make_map(&maps.x, p->x, p->rows, p->K, p->x_sr, RL_ROWS);
  if (rc != XL_OK) return rc;
  auto kern = rows_linear_kernel;
  XL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LY::DYN_SMEM));
  // blocks per tile: a power of two (clusters of three, five or six pack badly: 6160 x 2048 9.0 us with four, 11.4 with six), no
  // more than give every SM its two blocks, none with fewer than two stages of work
  const int tiles = (p->N + RL_TILE - 1) / RL_TILE, kb = (p->K + RL_KB - 1) / RL_KB;
  int parts = 1;
  while (parts < 8 && 2 * parts * tiles <= RL_BLOCKS && 4 * parts <= kb) parts *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(parts, tiles);
  cfg.blockDim = dim3(RL_THREADS);
  cfg.dynamicSmemBytes = LY::DYN_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = parts; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  XL_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, maps, *p, ahead ? 1 : 0));
  return check_launch("xl_rows_linear");
}

static int rows_linear(const xl_rows_linear_params* p, bool ahead, void* cuda_stream) {
  if (!p || !p->x || !p->w || !p->y) return XL_ERR_NULL_POINTER;
  if (p->dtype != XL_BF16) return XL_ERR_BAD_DTYPE;
  if (p->rows <= 0 || p->N <= 0 || p->K <= 0) return XL_ERR_BAD_SHAPE;
  if (p->rows > RL_ROWS || p->N > 65535 * RL_TILE) return XL_ERR_TOO_LARGE;
  if (p->x_sr < p->K || p->w_sr < p->K || p->x_sr % 8 || p->w_sr % 8) return XL_ERR_BAD_STRIDE;
  if (!aligned16(p->x) || !aligned16(p->w) || (reinterpret_cast<uintptr_t>(p->y) & 1u)) return XL_ERR_BAD_ALIGNMENT;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  return launch_rows_linear(p, ahead, st);
}

}  // namespace xl

extern "C" int xl_rows_linear(const xl_rows_linear_params* p, void* cuda_stream) { return xl::rows_linear(p, false, cuda_stream); }
extern "C" int xl_rows_linear_ahead(const xl_rows_linear_params* p, void* cuda_stream) { return xl::rows_linear(p, true, cuda_stream); }
