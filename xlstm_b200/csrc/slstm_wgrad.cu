// Gradients of the sLSTM's recurrent matrix and bias from the backward kernel's dWx (slstm_bwd.cu):
//
//   dR[n, k, g, u]  = sum_{b, t >= 1} h[b, n, t-1, k] dWx[b, t, g, n, u]   ( + sum_b h0[b, n, k] dWx[b, 0, g, n, u] )
//   dbias[n, g, u]  = sum_{b, t} dWx[b, t, g, n, u]
//
// One pass over dWx and h as they lie: both are MN-major operands of a product over tokens, so tiles of 64 tokens come by
// TMA (128-byte swizzle) straight from the caller's layouts -- h at token t0, dWx at t0 + 1, which is the shift by one step --
// and no transposed or shifted copy exists.  A thread block owns 256 of a head's 4 DH (gate, unit) columns, all DH input
// features and a range of the tokens: two 128 x DH accumulators in tensor memory (all 512 columns at DH = 256), four
// UMMAs each per 64 tokens.  Four warps add up the columns of the dWx tile for dbias while the tensor core reads it.
// What bounds it is the stream of dWx and h from HBM; tokens are split over as many blocks as the machine has SMs, and a
// second kernel adds the blocks' partial sums in order (run-to-run identical) with what step 0 contributes.
// B = 16, S = 2048, 4 x 256: 62 + 9 us (335 MB: 5.4 TB/s), where copies of the operands in GEMM layout, a batched library GEMM
// and a column sum took 0.63 ms.  4 x 128: 52 us (345 before), 4 x 64: 40 us (224), one 64-token row: 17 us (81), both kernels
// and a cold L2.  dR is 4 to 20 times closer to 64 bits than before on long sums (a split accumulates fewer terms).
#include <cuda.h>

#include "common.cuh"

namespace xl {

constexpr int WG_THREADS = 192;            // warp 0 TMA, warp 1 UMMA, warps 2-5 column sums and epilogue
constexpr int WG_COLS = 256;               // (gate, unit) columns per block
constexpr int WG_TOKENS = 64;              // tokens per stage
constexpr int WG_BOX_BYTES = WG_TOKENS * 128;
constexpr int WG_SMS = 148;

struct WgMaps {
  CUtensorMap dwx, h;   // dWx (4 NH DH, S, B); h (DH, S - 1, B NH): rows past either end are zero on both sides at once
};

template <int DH>
struct WgLayout {
  static constexpr int W_BYTES = WG_COLS / 64 * WG_BOX_BYTES, H_BYTES = DH / 64 * WG_BOX_BYTES;
  static constexpr int STAGE_BYTES = W_BYTES + H_BYTES;
  static constexpr int STAGES = DH == 256 ? 3 : DH == 128 ? 4 : 5;
  static constexpr int OFF_BAR = STAGES * STAGE_BYTES;   // full, empty per stage, done
  static constexpr int OFF_TMEM = OFF_BAR + (2 * STAGES + 1) * 8;
  static constexpr int DYN_SMEM = OFF_TMEM + 8 + 1024;
  static constexpr uint32_t TMEM_COLS = 2 * DH;
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst_smem, const void* tmap, uint32_t bar, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst_smem),
               "l"(tmap), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}

template <int DH>
__global__ void __launch_bounds__(WG_THREADS, 1) slstm_weight_grads_kernel(const __grid_constant__ WgMaps maps, const xl_slstm_wgrad_params p, int chunks) {
  using LY = WgLayout<DH>;
  constexpr int STAGES = LY::STAGES;
  extern __shared__ unsigned char wg_smem_raw[];
  unsigned char* smem = wg_smem_raw + ((1024u - (smem_u32(wg_smem_raw) & 1023u)) & 1023u);
  const uint32_t sbase = smem_u32(smem), bar0 = sbase + LY::OFF_BAR;
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + LY::OFF_TMEM);
  const int split = blockIdx.x, slice = blockIdx.y, head = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int row_chunks = (p.S - 1 + WG_TOKENS - 1) / WG_TOKENS;
  const int first = (int)((long long)chunks * split / gridDim.x), count = (int)((long long)chunks * (split + 1) / gridDim.x) - first;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar0 + 8u * s, 1);
      mbar_init(bar0 + 8u * (STAGES + s), 5);   // the UMMAs' commit and one arrival of each summing warp
    }
    mbar_init(bar0 + 16u * STAGES, 1);
    fence_barrier_init();
    tma_prefetch_desc(&maps.dwx);
    tma_prefetch_desc(&maps.h);
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

  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      int c_w[4];   // first feature of each 64-column box in dWx: gate, head, unit
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int col = slice * WG_COLS + j * 64;
        c_w[j] = ((col / DH) * p.NH + head) * DH + col % DH;
      }
      int b = first / row_chunks, tc = first - b * row_chunks, st = 0;
      uint32_t par = 1;
      for (int c = 0; c < count; ++c) {
        if (!mbar_wait(bar0 + 8u * (STAGES + st), par)) { ok = false; break; }
        const uint32_t bar = bar0 + 8u * st, dst = sbase + st * LY::STAGE_BYTES;
        mbar_expect_tx(bar, LY::STAGE_BYTES);
#pragma unroll
        for (int j = 0; j < 4; ++j) tma_load_3d(dst + j * WG_BOX_BYTES, &maps.dwx, bar, c_w[j], tc * WG_TOKENS + 1, b);
#pragma unroll
        for (int j = 0; j < DH / 64; ++j) tma_load_3d(dst + LY::W_BYTES + j * WG_BOX_BYTES, &maps.h, bar, j * 64, tc * WG_TOKENS, b * p.NH + head);
        if (++tc == row_chunks) { tc = 0; ++b; }
        if (++st == STAGES) { st = 0; par ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // warp-uniform issue code, descriptors from broadcast bases (see mlstm_chunkwise.cu)
    constexpr uint32_t IDESC = umma_idesc_bf16(128, DH, 1, 1), LBO_MN = ((uint32_t)WG_BOX_BYTES >> 4) << 16;
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
      const uint32_t sw = sbase_u + st * LY::STAGE_BYTES, sh = sw + LY::W_BYTES;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          umma_ss_lo(tmem_u + i * DH, LBO_MN + ((sw + i * 2 * WG_BOX_BYTES + kk * 2048) >> 4), LBO_MN + ((sh + kk * 2048) >> 4), IDESC, (c | kk) != 0);
      umma_commit_elect(bar_u + 8u * (STAGES + st));
      if (++st == STAGES) { st = 0; par ^= 1u; }
    }
    umma_commit_elect(bar_u + 16u * STAGES);
    ok = okm;
  } else {
    // ---- column sums of the dWx tile: a warp takes one 64-column box, the lane two neighbouring columns
    const int box = warp - 2;
    float bx = 0.f, by = 0.f;
    int st = 0;
    uint32_t par = 0;
#pragma unroll 1
    for (int c = 0; c < count; ++c) {
      if (!mbar_wait(bar0 + 8u * st, par)) { ok = false; break; }
      const unsigned char* t = smem + st * LY::STAGE_BYTES + box * WG_BOX_BYTES;
      float sx[4] = {0.f, 0.f, 0.f, 0.f}, sy[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 16
      for (int r = 0; r < WG_TOKENS; ++r) {
        const float2 v = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(t + r * 128 + ((((lane >> 2) ^ (r & 7)) << 4) | ((lane & 3) << 2))));
        sx[r & 3] += v.x;
        sy[r & 3] += v.y;
      }
      bx += (sx[0] + sx[1]) + (sx[2] + sx[3]);
      by += (sy[0] + sy[1]) + (sy[2] + sy[3]);
      __syncwarp();
      if (lane == 0) mbar_arrive(bar0 + 8u * (STAGES + st));
      if (++st == STAGES) { st = 0; par ^= 1u; }
    }
    const size_t cols = (size_t)p.NH * 4 * DH, col0 = (size_t)head * 4 * DH + slice * WG_COLS;
    float* part = static_cast<float*>(p.scratch);
    float* bsum = part + (size_t)gridDim.x * cols * DH + split * cols + col0 + box * 64 + 2 * lane;
    *reinterpret_cast<float2*>(bsum) = make_float2(bx, by);
    // ---- partial product out of tensor memory: lane = (gate, unit) column, tensor-memory column = input feature
    if (ok && !mbar_wait(bar0 + 16u * STAGES, 0u)) ok = false;
    if (ok) {
      tc_fence_after();
      const int quarter = warp & 3;
#pragma unroll 1
      for (int i = 0; i < 2; ++i) {
        float* out = part + ((size_t)split * p.NH + head) * DH * 4 * DH + slice * WG_COLS + i * 128 + quarter * 32 + lane;
#pragma unroll 1
        for (int kb = 0; kb < DH; kb += 32) {
          uint32_t r[32];
          tmem_ld_x32(tmem + i * DH + kb + ((uint32_t)(quarter * 32) << 16), r);
          tc_wait_ld();
#pragma unroll
          for (int k = 0; k < 32; ++k) out[(size_t)(kb + k) * 4 * DH] = __uint_as_float(r[k]);
        }
      }
    }
  }
  if (!ok && p.status) atomicExch(p.status, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, LY::TMEM_COLS);
}

// Adds the splits' partial sums in order, and step 0: h0 (x) dWx_0 to dR, dWx_0 to dbias.  A thread owns four neighbouring
// (gate, unit) columns of one input feature; the threads of feature 0 form the bias as well.
constexpr int WG_SUM_THREADS = 256;
__global__ void __launch_bounds__(WG_SUM_THREADS) slstm_weight_grads_sum_kernel(const xl_slstm_wgrad_params p, int splits) {
  const int DH = p.DH, W = 4 * DH;
  const long long cols = (long long)p.NH * W, total = cols * DH;
  grid_dependency_wait();
  const long long e = ((long long)blockIdx.x * WG_SUM_THREADS + threadIdx.x) * 4;
  if (e >= total) return;
  const int col = (int)(e % W), k = (int)(e / W % DH), head = (int)(e / W / DH);
  const float* part = static_cast<const float*>(p.scratch);
  const __nv_bfloat16* w0 = static_cast<const __nv_bfloat16*>(p.dwx) + ((long long)(col / DH) * p.NH + head) * DH + col % DH;   // + b S 4 NH DH
  const long long w_sb = (long long)p.S * 4 * p.NH * DH;
  auto add = [](float4& a, const float4& b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; };
  auto row0 = [&](int b) {
    const uint2 raw = __ldg(reinterpret_cast<const uint2*>(w0 + b * w_sb));
    const float2 x = unpack_bf16x2(raw.x), y = unpack_bf16x2(raw.y);
    return make_float4(x.x, x.y, y.x, y.y);
  };
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int s = 0; s < splits; ++s) add(acc, __ldcg(reinterpret_cast<const float4*>(part + s * total + e)));
  if (p.h0) {
    const __nv_bfloat16* h0 = static_cast<const __nv_bfloat16*>(p.h0) + (long long)head * DH + k;
#pragma unroll 4
    for (int b = 0; b < p.B; ++b) {
      const float hv = to_float(h0[(long long)b * p.NH * DH]);
      const float4 w = row0(b);
      acc.x = fmaf(hv, w.x, acc.x); acc.y = fmaf(hv, w.y, acc.y); acc.z = fmaf(hv, w.z, acc.z); acc.w = fmaf(hv, w.w, acc.w);
    }
  }
  *reinterpret_cast<float4*>(p.dR + e) = acc;
  if (k == 0) {
    const long long c = (long long)head * W + col;
    float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int s = 0; s < splits; ++s) add(s4, __ldcg(reinterpret_cast<const float4*>(part + splits * total + s * cols + c)));
#pragma unroll 8
    for (int b = 0; b < p.B; ++b) add(s4, row0(b));
    *reinterpret_cast<float4*>(p.dbias + c) = s4;
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
static int wg_chunks(int B, int S) { return B * ((S - 1 + WG_TOKENS - 1) / WG_TOKENS); }

// Blocks that share a (head, column slice): as many as fill the machine, each with so many 64-token tiles that its operands
// outweigh the partial sums it writes and the second kernel reads (at DH = 256: 64 KB a tile against 512 KB).
static int wg_splits(int B, int S, int NH, int DH) {
  const int chunks = wg_chunks(B, S), units = NH * (4 * DH / WG_COLS);
  if (chunks == 0) return 0;
  int splits = units < WG_SMS ? WG_SMS / units : 1;
  const int worth = (chunks + DH / 32 - 1) / (DH / 32);
  return splits < worth ? splits : worth;
}

typedef CUresult (*wg_encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// [outer][rows][features] bf16, features contiguous -> 3-D map, box = 64 features x 64 rows
static int wg_make_map(CUtensorMap* m, const void* base, int64_t features, int64_t rows, int64_t outer, int64_t row_stride, int64_t outer_stride) {
  static const wg_encode_fn encode = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    const bool found = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess;
    return found ? reinterpret_cast<wg_encode_fn>(sym) : nullptr;
  }();
  if (!encode) {
    set_last_cuda_error(cudaErrorSymbolNotFound, "cudaGetDriverEntryPoint(cuTensorMapEncodeTiled)");
    return XL_ERR_CUDA;
  }
  const cuuint64_t dims[3] = {(cuuint64_t)features, (cuuint64_t)rows, (cuuint64_t)outer};
  const cuuint64_t strides[2] = {(cuuint64_t)row_stride * 2, (cuuint64_t)outer_stride * 2};
  const cuuint32_t box[3] = {64, WG_TOKENS, 1}, estr[3] = {1, 1, 1};
  const CUresult r = encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_last_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled rejected the matrix layout");
    return XL_ERR_BAD_STRIDE;
  }
  return XL_OK;
}

template <int DH>
static int launch_weight_grads(const xl_slstm_wgrad_params* p, int splits, cudaStream_t st) {
  using LY = WgLayout<DH>;
  static_assert(LY::DYN_SMEM <= 227 * 1024, "shared memory budget");
  if (splits > 0) {
    WgMaps maps;
    const int64_t H = (int64_t)p->NH * DH;
    int rc = wg_make_map(&maps.dwx, p->dwx, 4 * H, p->S, p->B, 4 * H, p->S * 4 * H);
    if (rc != XL_OK) return rc;
    rc = wg_make_map(&maps.h, p->h, DH, p->S - 1, (int64_t)p->B * p->NH, DH, (int64_t)p->S * DH);
    if (rc != XL_OK) return rc;
    auto kern = slstm_weight_grads_kernel<DH>;
    XL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LY::DYN_SMEM));
    XL_CUDA_TRY(launch_dependent(kern, dim3(splits, 4 * DH / WG_COLS, p->NH), dim3(WG_THREADS), LY::DYN_SMEM, st, maps, *p, wg_chunks(p->B, p->S)));
  }
  const int64_t threads = (int64_t)p->NH * DH * DH;
  XL_CUDA_TRY(launch_dependent(slstm_weight_grads_sum_kernel, dim3((unsigned)((threads + WG_SUM_THREADS - 1) / WG_SUM_THREADS)), dim3(WG_SUM_THREADS), 0, st, *p, splits));
  return check_launch("xl_slstm_weight_grads");
}

}  // namespace xl

extern "C" int64_t xl_slstm_weight_grads_scratch_bytes(int32_t B, int32_t S, int32_t NH, int32_t DH) {
  if (B <= 0 || S <= 0 || NH <= 0 || !(DH == 64 || DH == 128 || DH == 256)) return 0;
  return xl::wg_splits(B, S, NH, DH) * (int64_t)NH * 4 * DH * (DH + 1) * (int64_t)sizeof(float);
}

extern "C" int xl_slstm_weight_grads(const xl_slstm_wgrad_params* p, void* cuda_stream) {
  using namespace xl;
  if (!p || !p->dwx || !p->h || !p->dR || !p->dbias) return XL_ERR_NULL_POINTER;
  if (p->B <= 0 || p->S <= 0 || p->NH <= 0) return XL_ERR_BAD_SHAPE;
  if (p->dtype != XL_BF16) return XL_ERR_BAD_DTYPE;
  if (!(p->DH == 64 || p->DH == 128 || p->DH == 256)) return XL_ERR_UNSUPPORTED;
  if (p->NH > 4096 || (int64_t)p->B * ((p->S + WG_TOKENS - 1) / WG_TOKENS) > 0x7fffffff || (int64_t)p->B * p->NH > 0x7fffffff) return XL_ERR_TOO_LARGE;
  if (!aligned16(p->dwx) || !aligned16(p->h) || !aligned16(p->dR) || !aligned16(p->dbias) || !aligned16(p->scratch)) return XL_ERR_BAD_ALIGNMENT;
  const int splits = wg_splits(p->B, p->S, p->NH, p->DH);
  if (p->scratch_bytes < xl_slstm_weight_grads_scratch_bytes(p->B, p->S, p->NH, p->DH)) return XL_ERR_TOO_LARGE;
  if (splits > 0 && !p->scratch) return XL_ERR_NULL_POINTER;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  switch (p->DH) {
    case 64: return launch_weight_grads<64>(p, splits, st);
    case 128: return launch_weight_grads<128>(p, splits, st);
    default: return launch_weight_grads<256>(p, splits, st);
  }
}
