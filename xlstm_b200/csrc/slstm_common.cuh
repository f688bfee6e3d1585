// Shared by the sLSTM forward and backward kernels: the thread mapping constants, the layout of the training
// cache and the small device helpers both use.
#pragma once
#include "common.cuh"

namespace xl {

constexpr int SL_THREADS = 128;         // 4 warps; warp w owns units [8w, 8w+8) of the CTA's 32
constexpr int SL_UNITS = 32;            // hidden units per CTA
constexpr int SL_ROWS = 16;             // batch rows per cluster (mma M)
constexpr int SL_RING = 8;              // Wx prefetch depth in time steps
constexpr int SL_WX_ROW_BYTES = 4 * SL_UNITS * 2 + 16;  // 4 gates x 32 units bf16 + 16 B pad (bank spread)
constexpr int SL_WX_STEP_BYTES = SL_ROWS * SL_WX_ROW_BYTES;
// Training cache: one record per (step, thread): 4 x bf16x2 gates of batch row a (i', raw f, tanh z, sigmoid o), the same
// for row b, h' of rows a and b (bf16x2 each) + 8 B pad, then c'[4], n'[4], m'[4] in fp32 for the thread's four
// (row, unit) pairs.  Records of a CTA are contiguous: [cluster][CTA][step][thread].
constexpr int SL_REC_BYTES = 96;

// The eight-row kernels (the batch rows are the N = 8 side of the products, see slstm_fwd.cu): one cluster per (head, 8
// batch rows).  A thread owns one unit and two adjacent rows; its record is 48 bytes in three planes of 16 bytes per thread,
// so that a warp stores and loads each of them as 512 contiguous bytes: i', raw f, tanh z, sigmoid o as bf16 pairs over the
// rows | h' as such a pair, 4 B pad, c' | n', m' (fp32, two each).
constexpr int SL8_ROWS = 8;
constexpr int SL8_REC_PLANE = SL_THREADS * 16;
constexpr int SL8_REC_STEP = 3 * SL8_REC_PLANE;

// Whether a batch of B rows runs on the eight-row kernels: where all their clusters are resident at once.  Eight rows take
// half the products, half the gate arithmetic and half the exchange of a sixteen-row step, on twice the SMs; with more
// clusters than fit, a second round would cost more than that saves.  The training forward and the backward share the
// answer, because it decides the layout of the cache between them.
bool slstm_rows8(int B, int NH, int DH, bool train);
int slstm_max_clusters_fwd8(int DH, bool train);
int slstm_max_clusters_bwd8(int DH);

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// Bounded wait without back-off: this wait is the per-step latency chain, a sleep would land on it in full.
__device__ __forceinline__ bool sl_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t it = 0; it < (1u << 26); ++it)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
// 4-byte store into (another) CTA's shared memory that adds its 4 bytes to the transaction count of an mbarrier there
__device__ __forceinline__ void st_async_u32(uint32_t addr, uint32_t v, uint32_t remote_bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(remote_bar)
               : "memory");
}
// 16-byte version of the same store
__device__ __forceinline__ void st_async_v4(uint32_t addr, const uint32_t (&v)[4], uint32_t remote_bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(remote_bar)
               : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// ... each 8 x 8 matrix transposed: thread t receives elements (rows 2 (t%4) and + 1, column t/4)
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// transposes an 8 x 8 matrix of 16-bit elements held as an accumulator-like fragment (row t/4, columns 2 (t%4) and + 1)
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                               uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float fast_logsigmoid(float x) { return fminf(x, 0.f) - __logf(1.f + __expf(-fabsf(x))); }


// Number of clusters of DH/32 blocks of `kern` that can be resident at once (0 if that cannot be found out).
template <typename K>
static int slstm_resident_clusters(K kern, int ncta, int threads, size_t smem) {
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncta);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ncta;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
  return n;
}

// One cluster of `ncta` blocks per (head, batch group); the launch may overlap the tail of the kernel in front of it.
template <typename K, typename P>
static cudaError_t slstm_launch(K kern, const P& p, int ncta, int groups, int threads, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ncta, p.NH, groups);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ncta;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

}  // namespace xl
