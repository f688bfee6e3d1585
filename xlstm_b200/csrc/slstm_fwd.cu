// sLSTM forward over a whole sequence in ONE persistent kernel.
//
// Per time step (reference: slstm_pointwise.cu:60-115 / vanilla/slstm.py:19-37):
//   raw_g = Wx_g + (h_{t-1} R)_g + b_g ,  g in {i,f,z,o}
//   m' = (n == 0) ? i : max(i, m + logsig(f));  i' = min(1, e^{i-m'});  f' = min(1, e^{m + logsig(f) - m'})
//   c' = f' c + i' tanh(z);  n' = f' n + i';  h' = sigmoid(o) c' / n'
//
// Mapping.  One thread-block CLUSTER of DH/32 CTAs serves one (head, 16-row batch group); heads and batch
// groups never exchange data.  CTA r of the cluster owns hidden units [32r, 32r+32) and all four of their
// gates: its slice of the recurrent matrix (DH x 128 bf16) is read once and stays in REGISTERS as
// mma.sync B-fragments (a warp = 8 units x 4 gates = four n8 tiles x DH/16 k-steps).  The batch rows are
// the M=16 side of m16n8k16.  Each thread ends a step holding all four gate pre-activations of its four
// (row, unit) pairs in its accumulators, so the pointwise update runs in registers with c, n, m kept in
// fp32 registers for the whole sequence.  The new h (bf16) is pushed into the double-buffered h tile of
// EVERY CTA of the cluster with asynchronous distributed-shared-memory stores that count their bytes on the
// destination's mbarrier: a CTA starts step t+1 the moment all of h_t has landed in ITS tile -- no cluster-wide
// barrier and no release/acquire fence on the per-step chain (that barrier was 2/3 of the step time).  The data
// dependency itself orders buffer reuse: whoever pushes h_{t+1} into a tile has consumed h_t, which every CTA
// pushed only after its last read of h_{t-1}, the previous content of that buffer.
// A CTA takes in distributed shared memory in 32-byte sectors (~32 B per cycle), so the tile is laid out in 16-byte
// granules -- eight units of one batch row, what one ldmatrix row reads -- with rows r and r+8 of a unit group in one
// sector, and the pushes are whole granules gathered from the quad that computed them: the lanes of one store fill
// full sectors (8 KB of h per step = 256 sectors; 4-byte stores per row pair arrived as 512 half-filled ones).
// Gate arithmetic: one of i', f' is exp(0), the other exp(-|m + logsig(f) - i|); tanh and the sigmoid run on the
// hardware tanh (six special-function instructions per (row, unit) instead of nine).
// Wx is streamed through an 8-step cp.async ring so that HBM latency is off the dependency chain.
// A document boundary (cu_seqlens) zeroes h, c, n, m of that batch row inside the kernel.
//
// Training variant (TRAIN): every thread also writes one 96-byte record per step -- its activated gates
// (i', raw f, tanh z, sigmoid o as bf16 pairs), its h' and its c', n', m' in fp32 -- into a cache that the backward
// kernel (slstm_bwd.cu) reads back by the same (warp, lane) index (the counterpart of the reference's `states` and
// gate caches, slstm.cc:88-101).  The 12 KB of a step are staged in shared memory and leave as one bulk copy.
#include <atomic>

#include "common.cuh"
#include "slstm_common.cuh"

namespace xl {

constexpr int SL_REC_SLOTS = 3;                          // staging slots of the training cache (one step's records each)
constexpr int SL_REC_STEP = SL_THREADS * SL_REC_BYTES;   // bytes of one step's records of a CTA

// bulk copy of this CTA's shared memory to global memory (bulk-group completion)
__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
template <int N> __device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory"); }

// Advance `idx` past every boundary at or before time index `t_now` of batch row `gb`; return the time index
// of the next boundary inside the row, or INT_MAX.  Repeated offsets (empty documents) are skipped.
__device__ __forceinline__ int next_boundary(const xl_slstm_params& p, int gb, int t_now, int& idx) {
  const long long row0 = (long long)gb * p.S;
  while (idx <= p.num_docs && (long long)p.cu_seqlens[idx] <= row0 + t_now) ++idx;
  if (idx > p.num_docs) return 0x7fffffff;
  const long long pos = p.cu_seqlens[idx];
  return pos < row0 + p.S ? (int)(pos - row0) : 0x7fffffff;
}

// index of the first offset beyond the start of batch row gb
__device__ __forceinline__ int first_boundary_after(const xl_slstm_params& p, int gb) {
  const long long row0 = (long long)gb * p.S;
  int lo = 0, hi = p.num_docs + 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if ((long long)p.cu_seqlens[mid] > row0) hi = mid; else lo = mid + 1;
  }
  return lo;
}

template <int DH, bool TRAIN>
__global__ void __launch_bounds__(SL_THREADS, 1) slstm_forward_kernel(const xl_slstm_params p) {
  constexpr int KSTEPS = DH / 16;
  // h tile: 16-byte granules (eight consecutive units of one batch row, what one ldmatrix row reads), laid out so that
  // the granules of rows r and r + 8 of one unit group share a 32-byte sector: a warp's push then fills whole sectors of
  // the destination CTA, which takes in distributed shared memory sector by sector (~32 B per cycle), where separate
  // 4-byte stores per row pair arrived as twice as many half-filled ones.  Which half of its sector a granule takes
  // flips with bit 2 of the row, which keeps the eight rows of an ldmatrix matrix on distinct banks.
  constexpr int H_TILE = SL_ROWS * DH;   // bf16 elements of one tile (dense)
  auto granule_off = [](int row, int kgroup) -> uint32_t {   // byte offset of granule (batch row, unit / 8) in a tile
    return (uint32_t)(kgroup * 256 + (row & 7) * 32 + ((((row >> 3) ^ (row >> 2)) & 1) * 16));
  };
  extern __shared__ __align__(16) unsigned char sl_smem[];
  __nv_bfloat16* s_h = reinterpret_cast<__nv_bfloat16*>(sl_smem);                    // 2 x H_TILE
  unsigned char* s_wx = sl_smem + 2 * H_TILE * sizeof(__nv_bfloat16);                // SL_RING x SL_WX_STEP_BYTES
  const uint32_t s_bar = smem_u32(s_wx + SL_RING * SL_WX_STEP_BYTES);                // 2 mbarriers: h tile 0 / 1 complete
  constexpr uint32_t H_TILE_BYTES = SL_ROWS * DH * 2;                                // what one step delivers to a CTA
  unsigned char* s_recst = s_wx + SL_RING * SL_WX_STEP_BYTES + 16;                   // TRAIN: SL_REC_SLOTS x SL_REC_STEP

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = cluster_ctarank();       // which 32-unit slice of the head
  constexpr int NCTA = DH / SL_UNITS;
  const int head = blockIdx.y, bgroup = blockIdx.z;
  const int B = p.B, S = p.S, NH = p.NH, H = NH * DH;
  const int row_a = lane >> 2, row_b = row_a + 8;             // the two batch rows (within the group) of this thread
  const int unit_l = warp * 8 + (lane & 3) * 2;               // first of two adjacent units within the CTA
  const int unit_h = (int)rank * SL_UNITS + unit_l;           // ... within the head
  const int gb_a = bgroup * SL_ROWS + row_a, gb_b = bgroup * SL_ROWS + row_b;  // global batch rows
  const bool ok_a = gb_a < B, ok_b = gb_b < B;

  grid_dependency_wait();
  // ---- recurrent matrix slice -> registers (B fragments).  R is (NH, DH_in, 4, DH_out).
  uint32_t rfrag[KSTEPS][4][2];
  {
    const __nv_bfloat16* R = reinterpret_cast<const __nv_bfloat16*>(p.R) + (size_t)head * DH * 4 * DH;
    const int n_unit = (int)rank * SL_UNITS + warp * 8 + (lane >> 2);  // column n = lane/4 of every tile
    const int k0 = (lane & 3) * 2;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks)
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const __nv_bfloat16* base = R + ((size_t)(ks * 16 + k0) * 4 + g) * DH + n_unit;
        const uint16_t e0 = *reinterpret_cast<const uint16_t*>(base);
        const uint16_t e1 = *reinterpret_cast<const uint16_t*>(base + 4 * DH);
        const uint16_t e8 = *reinterpret_cast<const uint16_t*>(base + 8 * 4 * DH);
        const uint16_t e9 = *reinterpret_cast<const uint16_t*>(base + 9 * 4 * DH);
        rfrag[ks][g][0] = (uint32_t)e0 | ((uint32_t)e1 << 16);
        rfrag[ks][g][1] = (uint32_t)e8 | ((uint32_t)e9 << 16);
      }
  }
  // ---- bias for this thread's two units, four gates
  float bias[4][2];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    bias[g][0] = p.bias[((size_t)head * 4 + g) * DH + unit_h];
    bias[g][1] = p.bias[((size_t)head * 4 + g) * DH + unit_h + 1];
  }

  // ---- state registers: [pair] with pair = (row_a,u0), (row_a,u1), (row_b,u0), (row_b,u1)
  float c_[4], n_[4], m_[4], hlast[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gb = (i < 2) ? gb_a : gb_b;
    const bool ok = (i < 2) ? ok_a : ok_b;
    const size_t off = (size_t)gb * H + (size_t)head * DH + unit_h + (i & 1);
    const bool have = p.state0 != nullptr && ok;
    hlast[i] = have ? p.state0[0 * (size_t)B * H + off] : 0.f;
    c_[i] = have ? p.state0[1 * (size_t)B * H + off] : 0.f;
    n_[i] = have ? p.state0[2 * (size_t)B * H + off] : 0.f;
    m_[i] = have ? p.state0[3 * (size_t)B * H + off] : 0.f;
  }

  // ---- next document boundary (as a time index within the row) for the two batch rows
  int nxt_idx[2] = {0, 0};
  int nxt_t[2] = {0x7fffffff, 0x7fffffff};
  if (p.cu_seqlens) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int gb = r == 0 ? gb_a : gb_b;
      const bool ok = r == 0 ? ok_a : ok_b;
      if (!ok) continue;
      nxt_idx[r] = first_boundary_after(p, gb);
      nxt_t[r] = next_boundary(p, gb, 0, nxt_idx[r]);
    }
  }

  // ---- h tile (both buffers) of this CTA: buffer 0 holds h_{-1}; every CTA fills its own copy completely
  for (int i = tid; i < 2 * H_TILE; i += SL_THREADS) s_h[i] = __float2bfloat16_rn(0.f);
  if (tid == 0) {
    mbar_init(s_bar, 1);      // one arrival per phase: the local expect_tx
    mbar_init(s_bar + 8, 1);
    fence_barrier_init();
  }
  __syncthreads();
  if (p.state0) {
    for (int i = tid; i < SL_ROWS * DH; i += SL_THREADS) {
      const int r = i / DH, d = i % DH;
      const int gb = bgroup * SL_ROWS + r;
      if (gb < B) s_h[granule_off(r, d >> 3) / 2 + (d & 7)] = __float2bfloat16_rn(p.state0[(size_t)gb * H + (size_t)head * DH + d]);
    }
  }

  // ---- Wx ring: each thread copies two 16-byte granules per step
  const __nv_bfloat16* wx = reinterpret_cast<const __nv_bfloat16*>(p.wx);
  const uint32_t s_wx_u32 = smem_u32(s_wx);
  auto issue_wx = [&](int t) {
    if (t < S) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int gidx = tid + j * SL_THREADS;            // 0..255
        const int r = gidx >> 4, g = (gidx >> 2) & 3, part = gidx & 3;
        int gb = bgroup * SL_ROWS + r;
        gb = gb < B ? gb : B - 1;                          // padded rows re-read a valid row (result unused)
        const __nv_bfloat16* src = wx + (((size_t)gb * S + t) * 4 + g) * H + (size_t)head * DH + rank * SL_UNITS + part * 8;
        const uint32_t dst = s_wx_u32 + (t % SL_RING) * SL_WX_STEP_BYTES + r * SL_WX_ROW_BYTES + g * (SL_UNITS * 2) + part * 16;
        cp_async16(dst, src);
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int t = 0; t < SL_RING - 1; ++t) issue_wx(t);
  cp_async_wait<SL_RING - 2>();   // step 0 has landed (this thread's part)
  cluster_barrier();              // all CTAs of the cluster initialised; also a CTA-wide barrier

  // remote addresses of this thread's four h slots in every CTA of the cluster
  const uint32_t s_h_u32 = smem_u32(s_h);
  // Pushes: lanes 0..15 of a warp send the granule of batch row `lane` (gathered from the quad that computed it) to one
  // CTA, lanes 16..31 the same granules to the next CTA: four 16-byte stores per lane reach all eight CTAs.
  const int prow = lane & 15;
  const uint32_t pslot = granule_off(prow, unit_h >> 3 /* same for the whole warp */);
  const int psrc = 4 * (prow & 7);   // first lane of the quad that holds row prow (in pa if prow < 8, else in pb)
  // ldmatrix source row/column for this lane
  const uint32_t ldm_off = granule_off(lane & 15, lane >> 4);   // + 512 B per k-step (two unit groups)

  __nv_bfloat16* hout = reinterpret_cast<__nv_bfloat16*>(p.h_out);
  // training cache: [cluster][CTA][step][thread] records of SL_REC_BYTES.  The records of a step are staged in shared
  // memory and leave as ONE 12 KB bulk copy (six 16-byte global stores per thread and step cost 350 cycles of a step)
  unsigned char* rec = nullptr;
  if constexpr (TRAIN)
    rec = reinterpret_cast<unsigned char*>(p.train_cache) + (((size_t)bgroup * NH + head) * NCTA + rank) * (size_t)S * SL_REC_STEP;

  bool ok = true;
  for (int t = 0; t < S; ++t) {
    issue_wx(t + SL_RING - 1);
    const int cur = t & 1, nxt = cur ^ 1;
    // this step's h_t will land in tile `nxt` of this CTA: announce its size on that tile's barrier
    if (tid == 0) mbar_expect_tx(s_bar + 8u * nxt, H_TILE_BYTES);
    // h_{t-1} complete in tile `cur` (tile 0 holds the initial state at t = 0: nothing to wait for; its barrier's
    // first phase therefore belongs to t = 2)
    // (an expired wait does not leave the loop here: the decision to stop is taken by the whole CTA at the end of
    // the step, so that no thread is left behind in the barrier there)
    if (t >= 1 && !sl_wait(s_bar + 8u * cur, (uint32_t)((t >> 1) - (cur == 0 ? 1 : 0)) & 1u)) ok = false;

    // accumulators start from Wx + bias
    float acc[4][4];
    {
      const unsigned char* wrow_a = s_wx + (t % SL_RING) * SL_WX_STEP_BYTES + row_a * SL_WX_ROW_BYTES + unit_l * 2;
      const unsigned char* wrow_b = s_wx + (t % SL_RING) * SL_WX_STEP_BYTES + row_b * SL_WX_ROW_BYTES + unit_l * 2;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const float2 wa = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(wrow_a + g * (SL_UNITS * 2)));
        const float2 wb = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(wrow_b + g * (SL_UNITS * 2)));
        acc[g][0] = wa.x + bias[g][0];
        acc[g][1] = wa.y + bias[g][1];
        acc[g][2] = wb.x + bias[g][0];
        acc[g][3] = wb.y + bias[g][1];
      }
    }
    // h_{t-1} (16 x DH) times the register-resident R slice
    const uint32_t hbase = s_h_u32 + cur * (H_TILE * 2) + ldm_off;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) {
      uint32_t a0, a1, a2, a3;
      ldmatrix_x4(hbase + ks * 512, a0, a1, a2, a3);
#pragma unroll
      for (int g = 0; g < 4; ++g) mma_bf16_16816(acc[g], a0, a1, a2, a3, rfrag[ks][g][0], rfrag[ks][g][1]);
    }
    // pointwise update in registers
    const bool reset_next_a = (t + 1) == nxt_t[0], reset_next_b = (t + 1) == nxt_t[1];
    float hn[4];
    [[maybe_unused]] float gi[4], gz[4], go[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float ir = acc[0][i], fr = acc[1][i], zr = acc[2][i], orr = acc[3][i];
      const float lfm = m_[i] + fast_logsigmoid(fr);
      // One of the two stabilised gates is exp(0): with d = lfm - i, the other one is exp(-|d|) (a fresh unit, n == 0,
      // takes m' = i: its input gate is 1 and its forget gate min(1, e^d)).  One exponential instead of two.
      const bool fresh = n_[i] == 0.f;
      const float d = lfm - ir;
      const float mn = (fresh || d <= 0.f) ? ir : lfm;
      const float e = __expf(-fabsf(d));
      const float ig = (d > 0.f && !fresh) ? e : 1.f;
      const float fg = (d <= 0.f) ? e : 1.f;
      // tanh and the sigmoid (0.5 tanh(x/2) + 0.5) on the hardware tanh: one special-function instruction each
      const float zt = tanh_approx(zr), os = fmaf(0.5f, tanh_approx(0.5f * orr), 0.5f);
      c_[i] = fmaf(fg, c_[i], ig * zt);
      n_[i] = fmaf(fg, n_[i], ig);
      m_[i] = mn;
      hn[i] = __fdividef(c_[i], n_[i]) * os;
      if constexpr (TRAIN) { gi[i] = ig; gz[i] = zt; go[i] = os; }
    }
    const uint32_t pa = pack_bf16x2(hn[0], hn[1]), pb = pack_bf16x2(hn[2], hn[3]);
    // a row whose next token opens a new document restarts from the zero state
    uint32_t push_a = pa, push_b = pb;
    if (reset_next_a) {
      push_a = 0u;
      c_[0] = c_[1] = n_[0] = n_[1] = m_[0] = m_[1] = 0.f;
      nxt_t[0] = next_boundary(p, gb_a, t + 1, nxt_idx[0]);
    }
    if (reset_next_b) {
      push_b = 0u;
      c_[2] = c_[3] = n_[2] = n_[3] = m_[2] = m_[3] = 0.f;
      nxt_t[1] = next_boundary(p, gb_b, t + 1, nxt_idx[1]);
    }
    // broadcast h_t into buffer `nxt` of every CTA in the cluster
    const uint32_t nb = s_h_u32 + nxt * (H_TILE * 2);
    {
      uint32_t gr[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t va = __shfl_sync(0xffffffffu, push_a, psrc + i), vb = __shfl_sync(0xffffffffu, push_b, psrc + i);
        gr[i] = prow < 8 ? va : vb;
      }
      if constexpr (NCTA >= 2) {
#pragma unroll
        for (int r = 0; r < NCTA; r += 2) {
          const uint32_t dst = (uint32_t)(r + (lane >> 4));
          st_async_v4(map_to_cta(nb + pslot, dst), gr, map_to_cta(s_bar + 8u * nxt, dst));
        }
      } else {
        if (lane < 16) st_async_v4(map_to_cta(nb + pslot, 0), gr, map_to_cta(s_bar + 8u * nxt, 0));
      }
    }
    if constexpr (TRAIN) {
      // the record of this step (states after the update; the training path takes no document offsets, so nothing was
      // reset above) into this step's staging slot, behind the pushes like the output below
      uint4* r = reinterpret_cast<uint4*>(s_recst + (t % SL_REC_SLOTS) * SL_REC_STEP + tid * SL_REC_BYTES);
      r[0] = make_uint4(pack_bf16x2(gi[0], gi[1]), pack_bf16x2(acc[1][0], acc[1][1]), pack_bf16x2(gz[0], gz[1]), pack_bf16x2(go[0], go[1]));
      r[1] = make_uint4(pack_bf16x2(gi[2], gi[3]), pack_bf16x2(acc[1][2], acc[1][3]), pack_bf16x2(gz[2], gz[3]), pack_bf16x2(go[2], go[3]));
      r[2] = make_uint4(pa, pb, 0u, 0u);
      r[3] = make_uint4(__float_as_uint(c_[0]), __float_as_uint(c_[1]), __float_as_uint(c_[2]), __float_as_uint(c_[3]));
      r[4] = make_uint4(__float_as_uint(n_[0]), __float_as_uint(n_[1]), __float_as_uint(n_[2]), __float_as_uint(n_[3]));
      r[5] = make_uint4(__float_as_uint(m_[0]), __float_as_uint(m_[1]), __float_as_uint(m_[2]), __float_as_uint(m_[3]));
      fence_proxy_async_smem();
    }
    // output h_t, (B, NH, S, DH) -- after the pushes: they are on the step-to-step chain, this store is not
    if (ok_a) *reinterpret_cast<uint32_t*>(hout + (((size_t)gb_a * NH + head) * S + t) * DH + unit_h) = pa;
    if (ok_b) *reinterpret_cast<uint32_t*>(hout + (((size_t)gb_b * NH + head) * S + t) * DH + unit_h) = pb;
#pragma unroll
    for (int i = 0; i < 4; ++i) hlast[i] = hn[i];
    cp_async_wait<SL_RING - 2>();  // this thread's part of step t+1 has landed
    // ... and everybody else's (CTA-wide only); the same barrier tells every thread whether any wait expired
    if (__syncthreads_or(ok ? 0 : 1)) { ok = false; break; }
    if constexpr (TRAIN) {
      if (tid == 0) {
        bulk_store(rec + (size_t)t * SL_REC_STEP, smem_u32(s_recst) + (t % SL_REC_SLOTS) * SL_REC_STEP, SL_REC_STEP);
        bulk_commit();
        bulk_wait_read<1>();   // the copy of step t-1 has read its slot: step t+2, which reuses it, may stage (behind the next barrier)
      }
    }
  }
  if constexpr (TRAIN) {
    if (tid == 0) bulk_wait<0>();
  }
  // The pushes of h_{S-1} are still on their way into tile S & 1 of every CTA; their completion is signalled on that
  // tile's mbarrier only, so it is waited for (bounded) before anybody may leave: a CTA that exits while a peer's
  // asynchronous store into its shared memory is in flight is undefined behaviour.
  if (ok) {
    const int last = S & 1;
    if (!sl_wait(s_bar + 8u * last, (uint32_t)((S >> 1) - (last == 0 ? 1 : 0)) & 1u)) ok = false;
  }
  if (!ok && p.status) atomicExch(p.status, 1);
  cluster_barrier();  // nobody leaves while a peer may still push into its tile

  // final state (4, B, H): h, c, n, m
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gb = (i < 2) ? gb_a : gb_b;
    const bool ok = (i < 2) ? ok_a : ok_b;
    if (!ok) continue;
    const size_t off = (size_t)gb * H + (size_t)head * DH + unit_h + (i & 1);
    p.state_out[0 * (size_t)B * H + off] = hlast[i];
    p.state_out[1 * (size_t)B * H + off] = c_[i];
    p.state_out[2 * (size_t)B * H + off] = n_[i];
    p.state_out[3 * (size_t)B * H + off] = m_[i];
  }
}

// ---------------------------------------------------------------------------------------------
// The same recurrence for clusters of EIGHT batch rows: the rows are the N = 8 side of m16n8k16 and the recurrent matrix the
// A operand, so that a step costs 32 products per warp instead of 64, two (row, unit) pairs of gate arithmetic per thread
// instead of four, and 4 KB of h per CTA instead of 8.  The step chain is what the kernel is bound by, and a batch of 16 rows
// now uses 64 SMs where it used 32: 1.90 -> 1.13 ms at B = 16, S = 2048, 4 x 256.
//
// Rows of an A tile are (gate, unit): tile 0 = input gate of the warp's eight units, then their forget gate; tile 1 = z, o.
// A thread's accumulators are then all four gates of unit lane/4 for batch rows 2 (lane%4) and + 1.  Tiles in shared memory
// are 16-byte granules chosen so that every access is one conflict-free ldmatrix:
//   h   [unit group][row]                 granule = eight units of one row: B operand as it lies; a push fills whole sectors
//   Wx  [gate][unit group][row]           transposed by the load into the accumulators' layout
//   R   [warp][gate][k] (set-up only)     transposed by the load into A fragments; read coalesced, where the direct
//                                         fragment loads were 256 two-byte loads per thread (what a one-token call waited for)
// h' leaves the accumulator layout through one movmatrix: a thread then holds two units of row lane/4.
template <int DH, bool TRAIN>
struct Sl8Layout {
  static constexpr int H_TILE = SL8_ROWS * DH * 2;                      // bytes
  static constexpr int WX_STEP = SL8_ROWS * 4 * SL_UNITS * 2;
  static constexpr int OFF_WX = 2 * H_TILE;
  static constexpr int OFF_BAR = OFF_WX + SL_RING * WX_STEP;            // 2 mbarriers: h tile 0 / 1 complete
  static constexpr int OFF_R = OFF_BAR + 16;
  static constexpr int TOTAL = OFF_R + DH * 4 * SL_UNITS * 2;
};

template <int DH, bool TRAIN>
__global__ void __launch_bounds__(SL_THREADS, 1) slstm_forward_rows8_kernel(const xl_slstm_params p) {
  using LY = Sl8Layout<DH, TRAIN>;
  constexpr int KSTEPS = DH / 16, NCTA = DH / SL_UNITS;
  extern __shared__ __align__(16) unsigned char sl_smem[];
  const uint32_t s_h = smem_u32(sl_smem), s_wx = s_h + LY::OFF_WX, s_bar = s_h + LY::OFF_BAR, s_r = s_h + LY::OFF_R;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = cluster_ctarank();       // which 32-unit slice of the head
  const int head = blockIdx.y, bgroup = blockIdx.z;
  const int B = p.B, S = p.S, NH = p.NH, H = NH * DH;
  const int unit_h = (int)rank * SL_UNITS + warp * 8 + (lane >> 2);                 // this thread's unit within the head
  const int gb0 = bgroup * SL8_ROWS + 2 * (lane & 3);                               // its two batch rows: gb0, gb0 + 1
  const bool ok_row[2] = {gb0 < B, gb0 + 1 < B};

  if (tid == 0) {
    mbar_init(s_bar, 1);      // one arrival per phase: the local expect_tx
    mbar_init(s_bar + 8, 1);
    fence_barrier_init();
  }
  for (int i = tid; i < 2 * LY::H_TILE / 16; i += SL_THREADS) reinterpret_cast<uint4*>(sl_smem)[i] = make_uint4(0u, 0u, 0u, 0u);
  grid_dependency_wait();

  // ---- this CTA's slice of R, (NH, DH_in, 4, DH_out), into shared memory; then the first Wx steps behind it
  {
    // (the contract asks nothing of R's address: a view into a flat parameter buffer may start anywhere.  All pieces have
    // the alignment of the base, so one test decides; off a 16-byte boundary they come element by element.)
    const __nv_bfloat16* R = reinterpret_cast<const __nv_bfloat16*>(p.R) + (size_t)head * DH * 4 * DH + rank * SL_UNITS;
    const bool whole_pieces = (reinterpret_cast<uintptr_t>(p.R) & 15u) == 0;
    if (whole_pieces) {
#pragma unroll 8
      for (int i = tid; i < DH * 16; i += SL_THREADS) {
        const int w = i & 3, g = (i >> 2) & 3, k = i >> 4;
        cp_async16(s_r + ((w * 4 + g) * DH + k) * 16, R + ((size_t)k * 4 + g) * DH + w * 8);
      }
    } else {
      uint16_t* dst = reinterpret_cast<uint16_t*>(sl_smem + LY::OFF_R);
#pragma unroll 8
      for (int i = tid; i < DH * 4 * SL_UNITS; i += SL_THREADS) {   // neighbouring threads: neighbouring elements of a piece row
        const int u = i & (SL_UNITS - 1), g = (i >> 5) & 3, k = i >> 7;
        dst[(((u >> 3) * 4 + g) * DH + k) * 8 + (u & 7)] = *reinterpret_cast<const uint16_t*>(R + ((size_t)k * 4 + g) * DH + u);
      }
    }
    cp_async_commit();
  }
  // ---- Wx ring: one 16-byte granule (row, gate, eight units) per thread and step
  const int wrow = tid >> 4, wgate = (tid >> 2) & 3, wpart = tid & 3;
  const __nv_bfloat16* wx_src;
  {
    int gb = bgroup * SL8_ROWS + wrow;
    gb = gb < B ? gb : B - 1;                          // padded rows re-read a valid row (result unused)
    wx_src = reinterpret_cast<const __nv_bfloat16*>(p.wx) + ((size_t)gb * S * 4 + wgate) * H + (size_t)head * DH + rank * SL_UNITS + wpart * 8;
  }
  const uint32_t wx_dst = s_wx + ((wgate * 4 + wpart) * SL8_ROWS + wrow) * 16;
  auto issue_wx = [&](int t) {
    if (t < S) cp_async16(wx_dst + (t % SL_RING) * LY::WX_STEP, wx_src + (size_t)t * 4 * H);
    cp_async_commit();
  };
#pragma unroll
  for (int t = 0; t < SL_RING - 1; ++t) issue_wx(t);

  // ---- bias, state and document boundaries of this thread's unit and rows
  float bias[4];
#pragma unroll
  for (int g = 0; g < 4; ++g) bias[g] = p.bias[((size_t)head * 4 + g) * DH + unit_h];
  float c_[2], n_[2], m_[2], hlast[2];
  int nxt_idx[2] = {0, 0}, nxt_t[2] = {0x7fffffff, 0x7fffffff};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const size_t off = (size_t)(gb0 + i) * H + (size_t)head * DH + unit_h;
    const bool have = p.state0 != nullptr && ok_row[i];
    hlast[i] = have ? p.state0[0 * (size_t)B * H + off] : 0.f;
    c_[i] = have ? p.state0[1 * (size_t)B * H + off] : 0.f;
    n_[i] = have ? p.state0[2 * (size_t)B * H + off] : 0.f;
    m_[i] = have ? p.state0[3 * (size_t)B * H + off] : 0.f;
    if (p.cu_seqlens && ok_row[i]) {
      nxt_idx[i] = first_boundary_after(p, gb0 + i);
      nxt_t[i] = next_boundary(p, gb0 + i, 0, nxt_idx[i]);
    }
  }
  __syncthreads();   // (the zeroed h tiles)
  if (p.state0) {    // tile 0 holds h_{-1}; every CTA fills its own copy completely
    for (int i = tid; i < SL8_ROWS * DH; i += SL_THREADS) {
      const int r = i / DH, d = i % DH, gb = bgroup * SL8_ROWS + r;
      if (gb < B) reinterpret_cast<__nv_bfloat16*>(sl_smem)[(d >> 3) * 64 + r * 8 + (d & 7)] = __float2bfloat16_rn(p.state0[(size_t)gb * H + (size_t)head * DH + d]);
    }
  }

  // ---- R -> A fragments: [k-step][gate][k half], a register = (unit lane/4; k = 2 (lane%4) and + 1)
  cp_async_wait<SL_RING - 1>();
  __syncthreads();
  uint32_t rfrag[KSTEPS][4][2];
  {
    // lanes 0-7, 8-15: the two k halves of one gate; 16-23, 24-31: those of the next
    const uint32_t src = s_r + ((warp * 4 + (lane >> 4)) * DH + ((lane >> 3) & 1) * 8 + (lane & 7)) * 16;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks)
#pragma unroll
      for (int g = 0; g < 4; g += 2)
        ldmatrix_x4_trans(src + (g * DH + ks * 16) * 16, rfrag[ks][g][0], rfrag[ks][g][1], rfrag[ks][g + 1][0], rfrag[ks][g + 1][1]);
  }
  cp_async_wait<SL_RING - 2>();   // step 0 has landed (this thread's part)
  cluster_barrier();              // all CTAs of the cluster initialised; also a CTA-wide barrier

  // Pushes: eight lanes send the warp's eight granules (one batch row each) to one CTA, so a store reaches four CTAs.
  const int prow = lane & 7;
  const uint32_t pslot = (uint32_t)((((int)rank * 4 + warp) * SL8_ROWS + prow) * 16);
  const uint32_t ldm_h = s_h + (uint32_t)lane * 16;                                            // + 512 B per pair of k-steps
  const uint32_t ldm_wx = s_wx + (uint32_t)((((lane >> 3) * 4 + warp) * SL8_ROWS + (lane & 7)) * 16);   // matrix = gate

  // output: row lane/4, two units
  const int orow = bgroup * SL8_ROWS + (lane >> 2);
  uint32_t* hout = reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(p.h_out) +
                                               ((size_t)(orow < B ? orow : 0) * NH + head) * (size_t)S * DH + rank * SL_UNITS + warp * 8 + 2 * (lane & 3));
  unsigned char* rec = nullptr;
  if constexpr (TRAIN)
    rec = reinterpret_cast<unsigned char*>(p.train_cache) + (((size_t)bgroup * NH + head) * NCTA + rank) * (size_t)S * SL8_REC_STEP + tid * 16;

  bool ok = true;
  for (int t = 0; t < S; ++t) {
    issue_wx(t + SL_RING - 1);
    const int cur = t & 1, nxt = cur ^ 1;
    // this step's h_t will land in tile `nxt` of this CTA: announce its size on that tile's barrier
    if (tid == 0) mbar_expect_tx(s_bar + 8u * nxt, LY::H_TILE);
    // accumulators start from Wx + bias; the second set takes every other k-step (a chain of dependent products runs at
    // its latency, not at its issue rate)
    float acc[2][4], acb[2][4];
    {
      uint32_t w[4];
      ldmatrix_x4_trans(ldm_wx + (t % SL_RING) * LY::WX_STEP, w[0], w[1], w[2], w[3]);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const float2 v = unpack_bf16x2(w[g]);
        acc[g >> 1][2 * (g & 1)] = v.x + bias[g];
        acc[g >> 1][2 * (g & 1) + 1] = v.y + bias[g];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) acb[0][i] = acb[1][i] = 0.f;
    }
    // h_{t-1} complete in tile `cur` (phases as in the sixteen-row kernel; an expired wait is acted on at the step's barrier)
    if (t >= 1 && !sl_wait(s_bar + 8u * cur, (uint32_t)((t >> 1) - (cur == 0 ? 1 : 0)) & 1u)) ok = false;
    const uint32_t hbase = ldm_h + cur * LY::H_TILE;
#pragma unroll
    for (int kp = 0; kp < KSTEPS / 2; ++kp) {
      uint32_t b0, b1, b2, b3;
      ldmatrix_x4(hbase + kp * 512, b0, b1, b2, b3);
      mma_bf16_16816(acc[0], rfrag[2 * kp][0][0], rfrag[2 * kp][1][0], rfrag[2 * kp][0][1], rfrag[2 * kp][1][1], b0, b1);
      mma_bf16_16816(acc[1], rfrag[2 * kp][2][0], rfrag[2 * kp][3][0], rfrag[2 * kp][2][1], rfrag[2 * kp][3][1], b0, b1);
      mma_bf16_16816(acb[0], rfrag[2 * kp + 1][0][0], rfrag[2 * kp + 1][1][0], rfrag[2 * kp + 1][0][1], rfrag[2 * kp + 1][1][1], b2, b3);
      mma_bf16_16816(acb[1], rfrag[2 * kp + 1][2][0], rfrag[2 * kp + 1][3][0], rfrag[2 * kp + 1][2][1], rfrag[2 * kp + 1][3][1], b2, b3);
    }
    float hn[2];
    [[maybe_unused]] float gi[2], gf[2], gz[2], go[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float ir = acc[0][i] + acb[0][i], fr = acc[0][2 + i] + acb[0][2 + i], zr = acc[1][i] + acb[1][i], orr = acc[1][2 + i] + acb[1][2 + i];
      const float lfm = m_[i] + fast_logsigmoid(fr);
      const bool fresh = n_[i] == 0.f;
      const float d = lfm - ir;
      const float mn = (fresh || d <= 0.f) ? ir : lfm;
      const float e = __expf(-fabsf(d));
      const float ig = (d > 0.f && !fresh) ? e : 1.f;
      const float fg = (d <= 0.f) ? e : 1.f;
      const float zt = tanh_approx(zr), os = fmaf(0.5f, tanh_approx(0.5f * orr), 0.5f);
      c_[i] = fmaf(fg, c_[i], ig * zt);
      n_[i] = fmaf(fg, n_[i], ig);
      m_[i] = mn;
      hn[i] = __fdividef(c_[i], n_[i]) * os;
      if constexpr (TRAIN) { gi[i] = ig; gf[i] = fr; gz[i] = zt; go[i] = os; }
    }
    const uint32_t hp = pack_bf16x2(hn[0], hn[1]);
    // a row whose next token opens a new document restarts from the zero state
    uint32_t push = hp;
    if (p.cu_seqlens) {
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (t + 1 == nxt_t[i]) {
          push &= i == 0 ? 0xffff0000u : 0x0000ffffu;
          c_[i] = n_[i] = m_[i] = 0.f;
          nxt_t[i] = next_boundary(p, gb0 + i, t + 1, nxt_idx[i]);
        }
    }
    // broadcast h_t into tile `nxt` of every CTA in the cluster
    const uint32_t pw = movmatrix_trans(push);
    {
      uint32_t gr[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) gr[i] = __shfl_sync(0xffffffffu, pw, 4 * prow + i);
      const uint32_t dst_tile = s_h + nxt * LY::H_TILE + pslot;
#pragma unroll
      for (int r = 0; r < NCTA; r += 4) {
        const uint32_t dst = (uint32_t)(r + (lane >> 3));
        if (NCTA >= 4 || dst < (uint32_t)NCTA) st_async_v4(map_to_cta(dst_tile, dst), gr, map_to_cta(s_bar + 8u * nxt, dst));
      }
    }
    if constexpr (TRAIN) {
      // straight to global memory, a plane at a time: staged in shared memory and sent as one bulk copy, the records cost a
      // proxy fence on every step's chain (1.47 -> 1.38 ms at B = 16, S = 2048, 4 x 256)
      uint4* r = reinterpret_cast<uint4*>(rec + (size_t)t * SL8_REC_STEP);
      __stcs(r, make_uint4(pack_bf16x2(gi[0], gi[1]), pack_bf16x2(gf[0], gf[1]), pack_bf16x2(gz[0], gz[1]), pack_bf16x2(go[0], go[1])));
      __stcs(r + SL_THREADS, make_uint4(hp, 0u, __float_as_uint(c_[0]), __float_as_uint(c_[1])));
      __stcs(r + 2 * SL_THREADS, make_uint4(__float_as_uint(n_[0]), __float_as_uint(n_[1]), __float_as_uint(m_[0]), __float_as_uint(m_[1])));
    }
    // output h_t, (B, NH, S, DH) -- after the pushes: they are on the step-to-step chain, this store is not
    {
      const uint32_t ow = p.cu_seqlens ? movmatrix_trans(hp) : pw;
      if (orow < B) hout[(size_t)t * (DH / 2)] = ow;
    }
    hlast[0] = hn[0];
    hlast[1] = hn[1];
    cp_async_wait<SL_RING - 2>();  // this thread's part of step t+1 has landed
    // ... and everybody else's (CTA-wide only); the same barrier tells every thread whether any wait expired
    if (__syncthreads_or(ok ? 0 : 1)) { ok = false; break; }
  }
  // the pushes of h_{S-1} are waited for before anybody may leave (see the sixteen-row kernel)
  if (ok) {
    const int last = S & 1;
    if (!sl_wait(s_bar + 8u * last, (uint32_t)((S >> 1) - (last == 0 ? 1 : 0)) & 1u)) ok = false;
  }
  if (!ok && p.status) atomicExch(p.status, 1);
  cluster_barrier();  // nobody leaves while a peer may still push into its tile

  // final state (4, B, H): h, c, n, m
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (!ok_row[i]) continue;
    const size_t off = (size_t)(gb0 + i) * H + (size_t)head * DH + unit_h;
    p.state_out[0 * (size_t)B * H + off] = hlast[i];
    p.state_out[1 * (size_t)B * H + off] = c_[i];
    p.state_out[2 * (size_t)B * H + off] = n_[i];
    p.state_out[3 * (size_t)B * H + off] = m_[i];
  }
}

template <int DH, bool TRAIN>
static constexpr size_t slstm_smem() {
  return 2 * SL_ROWS * DH * 2 + (size_t)SL_RING * SL_WX_STEP_BYTES + 16 +  // + 2 mbarriers
         (TRAIN ? (size_t)SL_REC_SLOTS * SL_REC_STEP : 0);
}

template <int DH, bool TRAIN>
static int launch_slstm(const xl_slstm_params* p, cudaStream_t st) {
  constexpr int NCTA = DH / SL_UNITS;
  if (slstm_rows8(p->B, p->NH, DH, TRAIN)) {
    constexpr size_t smem = Sl8Layout<DH, TRAIN>::TOTAL;
    auto kern = slstm_forward_rows8_kernel<DH, TRAIN>;
    XL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    XL_CUDA_TRY(slstm_launch(kern, *p, NCTA, (p->B + SL8_ROWS - 1) / SL8_ROWS, SL_THREADS, smem, st));
  } else {
    constexpr size_t smem = slstm_smem<DH, TRAIN>();
    auto kern = slstm_forward_kernel<DH, TRAIN>;
    XL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    XL_CUDA_TRY(slstm_launch(kern, *p, NCTA, (p->B + SL_ROWS - 1) / SL_ROWS, SL_THREADS, smem, st));
  }
  return check_launch("xl_slstm_forward");
}

template <int DH>
static int max_clusters_fwd8(bool train) {
  return train ? slstm_resident_clusters(slstm_forward_rows8_kernel<DH, true>, DH / SL_UNITS, SL_THREADS, Sl8Layout<DH, true>::TOTAL)
               : slstm_resident_clusters(slstm_forward_rows8_kernel<DH, false>, DH / SL_UNITS, SL_THREADS, Sl8Layout<DH, false>::TOTAL);
}
int slstm_max_clusters_fwd8(int DH, bool train) {
  return DH == 64 ? max_clusters_fwd8<64>(train) : DH == 128 ? max_clusters_fwd8<128>(train) : max_clusters_fwd8<256>(train);
}

bool slstm_rows8(int B, int NH, int DH, bool train) {
  // residency per device and head size, asked for once: [device][DH][train]
  static std::atomic<int> limits[64][3][2];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { (void)cudaGetLastError(); return false; }
  std::atomic<int>& slot = limits[dev][DH == 64 ? 0 : DH == 128 ? 1 : 2][train];
  int limit = slot.load(std::memory_order_relaxed);   // 1 + clusters; 0: not asked yet
  if (limit == 0) {
    limit = slstm_max_clusters_fwd8(DH, train);
    if (train) {
      const int bwd = slstm_max_clusters_bwd8(DH);
      limit = bwd < limit ? bwd : limit;
    }
    slot.store(++limit, std::memory_order_relaxed);
  }
  return (long long)((B + SL8_ROWS - 1) / SL8_ROWS) * NH < limit;
}

}  // namespace xl

extern "C" int xl_slstm_forward(const xl_slstm_params* p, void* cuda_stream) {
  using namespace xl;
  if (!p || !p->wx || !p->R || !p->bias || !p->h_out || !p->state_out) return XL_ERR_NULL_POINTER;
  if (p->B <= 0 || p->S <= 0 || p->NH <= 0) return XL_ERR_BAD_SHAPE;
  if (p->dtype != XL_BF16) return XL_ERR_BAD_DTYPE;
  if (p->cu_seqlens && p->num_docs <= 0) return XL_ERR_BAD_SHAPE;
  if (p->NH > 65535 || (p->B + SL_ROWS - 1) / SL_ROWS > 65535) return XL_ERR_TOO_LARGE;
  if (!aligned16(p->wx) || (reinterpret_cast<uintptr_t>(p->h_out) & 3u)) return XL_ERR_BAD_ALIGNMENT;
  if (p->state0 && p->state0 == p->state_out) return XL_ERR_ALIASING;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  if (p->train_cache) {
    if (p->cu_seqlens) return XL_ERR_UNSUPPORTED;  // the backward pass takes no document offsets
    if (!aligned16(p->train_cache)) return XL_ERR_BAD_ALIGNMENT;
    switch (p->DH) {
      case 64: return launch_slstm<64, true>(p, st);
      case 128: return launch_slstm<128, true>(p, st);
      case 256: return launch_slstm<256, true>(p, st);
      default: return XL_ERR_UNSUPPORTED;
    }
  }
  switch (p->DH) {
    case 64: return launch_slstm<64, false>(p, st);
    case 128: return launch_slstm<128, false>(p, st);
    case 256: return launch_slstm<256, false>(p, st);
    default: return XL_ERR_UNSUPPORTED;
  }
}

extern "C" int64_t xl_slstm_cache_bytes(int32_t B, int32_t S, int32_t NH, int32_t DH) {
  if (B <= 0 || S <= 0 || NH <= 0 || DH <= 0 || DH % xl::SL_UNITS) return 0;
  const int64_t groups = (B + xl::SL_ROWS - 1) / xl::SL_ROWS;
  return groups * NH * (DH / xl::SL_UNITS) * (int64_t)S * xl::SL_THREADS * xl::SL_REC_BYTES;
}
