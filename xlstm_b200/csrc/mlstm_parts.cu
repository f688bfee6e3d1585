// Splitting long documents for the chunkwise kernel: the choice of the split (host), the plan of a packed batch, and the
// state every part of a document adds on its own.
//
// One sequence of 8 192 tokens with 8 heads of 256 x 512 is 32 chains of 128 chunks -- 32 of 148 SMs, 234 us; in four parts
// 112 us.  Four heads of 128 x 256: 199 -> 36 us, of 64 x 128: 181 -> 26 us.
//
// The part states are a plain product, C_loc^T [128 x DHQK] = (w V)^T K over the tokens of a part, because the gates of the
// whole part are scanned first: w_l = exp(a_l - mu) with the part's own stabiliser mu, so there is one frame and nothing is
// rescaled on the way.  Per 64-token chunk that is the four widest UMMAs of the chunkwise kernel (520 cycles of ~3 400), the
// scaling of v (in place in its TMA stage) and n_loc on the scaling threads, in fp32.  A value slice forms the 64-feature
// blocks of n_loc whose index is congruent to its own.
#include "mlstm_chunkwise.cuh"

namespace xl {

// warp 0 TMA, warp 1 UMMA, warps 4-7 and 8-11 scale v and form n, chunk by chunk in turn (a chunk's pass is ~1 500 cycles of
// mostly latency, three times what its UMMAs take); all scan the gates
constexpr int PS_THREADS = 384;
constexpr int PS_GROUPS = 2;
constexpr int PS_STAGES = 4;
// A stage is always scaled by the same group.  If two groups took turns on a stage, a group's parity wait could look at a
// phase its own last visit says nothing about -- one or two phases back -- and be satisfied too early or never.
static_assert(PS_STAGES % PS_GROUPS == 0, "a stage belongs to one scaling group");

template <int DHQK>
struct PsLayout {
  static constexpr int NKB = DHQK / 64;
  static constexpr int K_BYTES = NKB * CW_BOX_BYTES, V_BYTES = 2 * CW_BOX_BYTES;
  static constexpr int STAGE_BYTES = K_BYTES + V_BYTES;
  static constexpr int OFF_RED = 0;                                    // [8][DHQK] partial n_loc of the scaling warps, over the stages at the end
  static constexpr int OFF_BAR = PS_STAGES * STAGE_BYTES;              // full, scaled, empty per stage, done, tensor-memory base
  static constexpr int OFF_W = OFF_BAR + (3 * PS_STAGES + 2) * 8 + 8;  // w of every token of the part, fp32
  static constexpr int bytes(int chunks) { return OFF_W + chunks * CW_L * 4 + 1024; }
  static constexpr uint32_t TMEM_COLS = DHQK;
};

template <int DHQK>
__global__ void __launch_bounds__(PS_THREADS, 1)
mlstm_part_state_kernel(const __grid_constant__ CwMaps maps, const xl_mlstm_seq_params p, const CwSplit split) {
  using LY = PsLayout<DHQK>;
  constexpr int NKB = LY::NKB;
  const int slot = blockIdx.z, head = blockIdx.y, slice = blockIdx.x, nslices = gridDim.x;
  grid_dependency_wait();
  int doc, first_chunk, chunks;
  if (split.counts) {
    if (slot >= split.counts[1]) return;
    const CwItem it = split.slots[slot];
    doc = it.doc; first_chunk = it.first_chunk; chunks = it.chunks;
  } else {
    doc = slot / (split.parts - 1);
    first_chunk = (slot - doc * (split.parts - 1)) * split.part_chunks;
    chunks = split.part_chunks;
  }
  int b;
  long long tok0, doc_len;
  cw_document(p, doc, b, tok0, doc_len);
  tok0 += (long long)first_chunk * CW_L;   // (every token of a part with a slot is inside the document)

  extern __shared__ unsigned char ps_smem_raw[];
  unsigned char* smem = ps_smem_raw + ((1024u - (smem_u32(ps_smem_raw) & 1023u)) & 1023u);
  const uint32_t sbase = smem_u32(smem), bar0 = sbase + LY::OFF_BAR;
  float* s_w = reinterpret_cast<float*>(smem + LY::OFF_W);
  float* s_red = reinterpret_cast<float*>(smem + LY::OFF_RED);
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + LY::OFF_BAR + (3 * PS_STAGES + 2) * 8);
  __shared__ float s_part[PS_THREADS / 32], s_max[PS_THREADS / 32];
  auto full = [&](int st) { return bar0 + 8u * st; };
  auto scaled = [&](int st) { return bar0 + 8u * (PS_STAGES + st); };
  auto empty = [&](int st) { return bar0 + 8u * (2 * PS_STAGES + st); };
  const uint32_t done = bar0 + 8u * (3 * PS_STAGES);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  if (tid == 0) {
    for (int st = 0; st < PS_STAGES; ++st) {
      mbar_init(full(st), 1);
      mbar_init(scaled(st), 128);
      mbar_init(empty(st), 1);
    }
    mbar_init(done, 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(s_tmem), LY::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *s_tmem;
  // Parts that need no state in front of them may start beside this kernel -- not before this block holds its tensor memory:
  // a block of the chunkwise kernel takes all of an SM's, and may wait for this kernel while it holds it.
  grid_dependents_launch();
  const int col0 = slice * CW_DV;

  auto load_stage = [&](int chunk) {   // one thread
    const int st = chunk % PS_STAGES;
    const uint32_t dst = sbase + st * LY::STAGE_BYTES, bar = full(st);
    const int tk = (int)(tok0 + (long long)chunk * CW_L);
    mbar_expect_tx(bar, LY::STAGE_BYTES);
    auto at = [&](int t, int i) { return cw_coord(maps, t, i, tk, head, b); };
#pragma unroll
    for (int kb = 0; kb < NKB; ++kb) tma_load_4d(dst + kb * CW_BOX_BYTES, &maps.k, bar, kb * 64, at(1, 1), at(1, 2), at(1, 3));
#pragma unroll
    for (int vb = 0; vb < 2; ++vb) tma_load_4d(dst + LY::K_BYTES + vb * CW_BOX_BYTES, &maps.v, bar, col0 + vb * 64, at(2, 1), at(2, 2), at(2, 3));
  };
  if (tid == 0)
    for (int c = 0; c < PS_STAGES && c < chunks; ++c) load_stage(c);   // under the scan

  // ---- gates of the whole part: every thread owns `per` consecutive tokens.  a_l = i_l + (sum of log f over the tokens behind
  // l in the part), summed from the part's end: the tokens that matter are those with small sums, and nothing is a difference.
  // (As i_l minus the sum up to l, the weights of a strongly forgetting part of 2048 tokens and the part's stabiliser were off
  // by 1e-3; this way the error is that of a chunk's own scan.)
  {
    const int per = (chunks * CW_L + PS_THREADS - 1) / PS_THREADS, t0 = tid * per, t1 = min(t0 + per, chunks * CW_L);
    const float* ig = p.igate + b * p.g_sb + head * p.g_sh + tok0 * p.g_st;
    const float* fg = p.fgate + b * p.g_sb + head * p.g_sh + tok0 * p.g_st;
    float sum = 0.f;
#pragma unroll 4
    for (int t = t1 - 1; t >= t0; --t) {   // s_w[t] <- i_t + (sum of log f behind t up to this thread's last token)
      s_w[t] = ig[t * p.g_st] + sum;
      sum += fast_log_sigmoid(fg[t * p.g_st]);
    }
    float from = sum;   // this thread's tokens and those of the lanes behind it
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float x = __shfl_down_sync(0xffffffffu, from, o);
      if (lane + o < 32) from += x;
    }
    if (lane == 0) s_part[warp] = from;
    float behind = __shfl_down_sync(0xffffffffu, from, 1);
    if (lane == 31) behind = 0.f;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int w = PS_THREADS / 32 - 1; w >= 0; --w) {
      if (w > warp) behind += s_part[w];
      total += s_part[w];
    }
    float mx = -INFINITY;
    for (int t = t0; t < t1; ++t) {
      const float al = s_w[t] + behind;
      s_w[t] = al;
      mx = fmaxf(mx, al);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) s_max[warp] = mx;
    __syncthreads();
    float mu = s_max[0];
#pragma unroll
    for (int w = 1; w < PS_THREADS / 32; ++w) mu = fmaxf(mu, s_max[w]);
    // (input gates of -inf throughout, a caller's mask: the part adds nothing, its weights are 0 and its stabiliser is -inf)
    const float frame = mu == -INFINITY ? 0.f : mu;
    for (int t = t0; t < t1; ++t) s_w[t] = __expf(s_w[t] - frame);
    if (slice == 0 && tid == 0) split.gm[(long long)slot * p.NH + head] = make_float2(total, mu);
    __syncthreads();
  }

  bool ok = true;
  if (warp == 0) {
    if (lane == 0)
      for (int c = PS_STAGES; ok && c < chunks; ++c) {
        if (!mbar_wait(empty(c % PS_STAGES), ((uint32_t)(c / PS_STAGES) & 1u) ^ 1u)) { ok = false; break; }
        load_stage(c);
      }
    __syncwarp();
  } else if (warp == 1) {
    // warp-uniform issue code, descriptors from broadcast bases (see mlstm_chunkwise.cu)
    constexpr uint32_t IDESC = umma_idesc_bf16(128, DHQK, 1, 1), LBO_MN = ((uint32_t)CW_BOX_BYTES >> 4) << 16;
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0), sbase_u = __shfl_sync(0xffffffffu, sbase, 0) & 0x3FFFFu;
    const uint32_t bar_u = __shfl_sync(0xffffffffu, bar0, 0);
    const int chunks_u = __shfl_sync(0xffffffffu, chunks, 0);
    bool okm = true;
    int st = 0;
    uint32_t par = 0;
#pragma unroll 1
    for (int c = 0; c < chunks_u; ++c) {
      okm &= okm ? mbar_wait(bar_u + 8u * (uint32_t)(PS_STAGES + st), par) : false;
      tc_fence_after();
      const uint32_t sk = sbase_u + st * LY::STAGE_BYTES, sv = sk + LY::K_BYTES;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_ss_lo(tmem_u, LBO_MN + ((sv + kk * 2048) >> 4), LBO_MN + ((sk + kk * 2048) >> 4), IDESC, (c | kk) != 0);
      umma_commit_elect(bar_u + 8u * (uint32_t)(2 * PS_STAGES + st));
      if (++st == PS_STAGES) { st = 0; par ^= 1u; }
    }
    umma_commit_elect(bar_u + 8u * (uint32_t)(3 * PS_STAGES));
    ok = okm;
  } else if (warp >= 4) {
    const int grp = (warp - 4) >> 2, t = (tid - 128) & 127, l = t >> 1, half = t & 1;
    // n_loc: this warp takes 16 tokens of every chunk, the lane two neighbouring features of each of the slice's blocks
    const int l0 = (warp & 3) * 16;
    float nx[NKB], ny[NKB];
#pragma unroll
    for (int j = 0; j < NKB; ++j) nx[j] = ny[j] = 0.f;
#pragma unroll 1
    for (int c = grp; c < chunks; c += PS_GROUPS) {
      const int st = c % PS_STAGES;
      if (!mbar_wait(full(st), (uint32_t)(c / PS_STAGES) & 1u)) { ok = false; break; }
      const float* w = s_w + c * CW_L;
      const __nv_bfloat162 ww = __float2bfloat162_rn(w[l]);
      unsigned char* vt = smem + st * LY::STAGE_BYTES + LY::K_BYTES + half * CW_BOX_BYTES + l * 128;
      uint4 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = *reinterpret_cast<const uint4*>(vt + ((i ^ (half << 2) ^ (l & 7)) << 4));
#pragma unroll
      for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(vt + ((i ^ (half << 2) ^ (l & 7)) << 4)) = scale_bf16x8(v[i], ww);
      fence_proxy_async_smem();
#pragma unroll
      for (int j = 0; j < NKB; ++j) {
        const int kb = slice + j * nslices;
        if (kb < NKB) {
          const unsigned char* kt = smem + st * LY::STAGE_BYTES + kb * CW_BOX_BYTES;
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int r = l0 + i;
            const float2 kv = unpack_bf16x2(*reinterpret_cast<const uint32_t*>(kt + r * 128 + ((((lane >> 2) ^ (r & 7)) << 4) | ((lane & 3) << 2))));
            nx[j] = fmaf(w[r], kv.x, nx[j]);
            ny[j] = fmaf(w[r], kv.y, ny[j]);
          }
        }
      }
      mbar_arrive(scaled(st));
    }
    // every load has landed and every UMMA has read its operands: the stages are free
    if (ok && !mbar_wait(done, 0u)) ok = false;
#pragma unroll
    for (int j = 0; j < NKB; ++j) {
      const int kb = slice + j * nslices;
      if (kb < NKB) {
        s_red[(warp - 4) * DHQK + kb * 64 + 2 * lane] = nx[j];
        s_red[(warp - 4) * DHQK + kb * 64 + 2 * lane + 1] = ny[j];
      }
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    for (int d = tid - 128; d < DHQK; d += 128 * PS_GROUPS)
      if ((d >> 6) % nslices == slice) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < 4 * PS_GROUPS; ++w) sum += s_red[w * DHQK + d];
        split.n_loc[((long long)slot * p.NH + head) * DHQK + d] = sum;
      }
    // the product out of tensor memory: lane = value column
    if (ok) {
      tc_fence_after();
      const uint32_t tc = tmem + ((uint32_t)((warp & 3) * 32) << 16);
      uint4* out = reinterpret_cast<uint4*>(split.c_loc) + cw_c_loc_offset<DHQK>(p, slot, head, slice) + (warp & 3) * 32 + lane;
#pragma unroll 1
      for (int cb = grp; cb < DHQK / 32; cb += PS_GROUPS) {
        uint32_t r[32];
        tmem_ld_x32(tc + cb * 32, r);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) out[(cb * 8 + i) * CW_DV] = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
      }
    }
  }
  if (!ok && p.status) atomicExch(p.status, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, LY::TMEM_COLS);
}

// ---------------------------------------------------------------------------------------------
// Plan of a packed batch: every document in parts of at most `cap` chunks (equal but for the last), the parts listed
// longest first -- blocks are dispatched in that order, so the short ones fill in at the end -- and a slot for every part
// that is not its document's last.  One block; counting sort by length.
// ---------------------------------------------------------------------------------------------
constexpr int PLAN_THREADS = 256;

__device__ __forceinline__ void plan_parts(const xl_mlstm_seq_params& p, int doc, int cap, int& n, int& parts, int& pc) {
  n = (int)(((long long)p.cu_seqlens[doc + 1] - p.cu_seqlens[doc] + CW_L - 1) / CW_L);
  n = n < 0 ? 0 : n;
  parts = n <= cap ? 1 : min((n + cap - 1) / cap, CW_MAX_PARTS);
  pc = (n + parts - 1) / parts;
  if (pc > 0) parts = (n + pc - 1) / pc;
}

__global__ void __launch_bounds__(PLAN_THREADS)
mlstm_plan_kernel(const xl_mlstm_seq_params p, int cap, int max_items, int max_slots, int* counts, CwItem* items, CwItem* slots) {
  __shared__ int s_hist[CW_MAX_PART_CHUNKS + 1], s_base[CW_MAX_PART_CHUNKS + 1], s_slots, s_total;
  const int tid = threadIdx.x;
  grid_dependents_launch();
  grid_dependency_wait();
  for (int i = tid; i <= CW_MAX_PART_CHUNKS; i += PLAN_THREADS) s_hist[i] = 0;
  if (tid == 0) s_slots = 0;
  __syncthreads();
  for (int doc = tid; doc < p.num_docs; doc += PLAN_THREADS) {
    int n, parts, pc;
    plan_parts(p, doc, cap, n, parts, pc);
    atomicAdd(&s_hist[min(n - (parts - 1) * pc, CW_MAX_PART_CHUNKS)], 1);
    if (parts > 1) atomicAdd(&s_hist[min(pc, CW_MAX_PART_CHUNKS)], parts - 1);
  }
  __syncthreads();
  for (int i = tid; i <= CW_MAX_PART_CHUNKS; i += PLAN_THREADS) {
    int before = 0;
    for (int j = CW_MAX_PART_CHUNKS; j > i; --j) before += s_hist[j];
    s_base[i] = before;
    if (i == 0) s_total = before + s_hist[0];
  }
  __syncthreads();
  for (int doc = tid; doc < p.num_docs; doc += PLAN_THREADS) {
    int n, parts, pc;
    plan_parts(p, doc, cap, n, parts, pc);
    const int slot0 = parts > 1 ? atomicAdd(&s_slots, parts - 1) : 0;
    for (int j = 0; j < parts; ++j) {
      CwItem it;
      it.doc = doc; it.part = j; it.parts = parts; it.first_chunk = j * pc;
      it.chunks = j + 1 < parts ? pc : n - j * pc;
      it.slot0 = slot0;
      const int at = atomicAdd(&s_base[min(it.chunks, CW_MAX_PART_CHUNKS)], 1);
      if (at < max_items) items[at] = it;
      if (j + 1 < parts && slot0 + j < max_slots) slots[slot0 + j] = it;
    }
  }
  __syncthreads();
  if (tid == 0) {
    counts[0] = min(s_total, max_items);
    counts[1] = min(s_slots, max_slots);
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
struct CwChoice {
  bool split;           // false: one block per (document, head, slice), in document order
  int parts, chunks;    // equal rows: parts per row and chunks per part; packed: longest part (chunks)
  int64_t items, slots; // most items / slots there can be
};

// The split that the model below expects to be fastest.  Its times (us) are fitted to measurements on B200 with all SMs at
// work, heads of 64, 128 and 256 features: a chunk of the chunkwise kernel, a chunk of a part state, what a thread block of
// either costs beside its chunks, folding in the state of one part, the second launch.
static CwChoice choose_split(const xl_mlstm_seq_params* p) {
  const double w = p->DHQK / 256.;
  const double T_CHUNK = 0.9 + w, T_STATE = 0.35 + 0.5 * w, T_BLOCK = 4. + 2. * w, T_STATE_BLOCK = 4. + 3. * w, T_FOLD = 0.8 * w, T_LAUNCH = 2.;
  constexpr int SMS = 148;
  constexpr int64_t MAX_STATE_BYTES = 1ll << 30;
  CwChoice no = {false, 1, 0, 0, 0};
  const int64_t per_doc = (int64_t)p->NH * (p->DHV / CW_DV), row_chunks = (p->S + CW_L - 1) / CW_L;
  const int64_t state_bytes = (int64_t)p->NH * p->DHQK * p->DHV * 4;
  if (p->c0 && p->c0 == p->c_out) return no;   // a document's last part may finish before another has read c0
  if (row_chunks > (int64_t)CW_MAX_PARTS * CW_MAX_PART_CHUNKS) return no;
  if (!p->cu_seqlens) {
    auto waves = [](int64_t blocks) { return (double)((blocks + SMS - 1) / SMS); };
    const int64_t chains = p->B * per_doc;
    CwChoice best = no;
    const double whole = waves(chains) * (row_chunks * T_CHUNK + T_BLOCK);
    double best_t = 0.93 * whole;   // (a split that only just pays is not worth its memory)
    for (int64_t k = 2; k <= CW_MAX_PARTS && k <= row_chunks; ++k) {
      const int64_t pc = (row_chunks + k - 1) / k, parts = (row_chunks + pc - 1) / pc;
      if (parts != k || pc > CW_MAX_PART_CHUNKS || p->B * (parts - 1) * state_bytes > MAX_STATE_BYTES || p->B * parts > 65535) continue;
      const double t = waves(chains * parts) * (pc * T_CHUNK + T_BLOCK) + (parts - 1) * T_FOLD + waves(chains * (parts - 1)) * (pc * T_STATE + T_STATE_BLOCK) + T_LAUNCH;
      if (t < best_t) {
        best_t = t;
        best = {true, (int)parts, (int)pc, p->B * parts, p->B * (parts - 1)};
      }
    }
    return best;
  }
  // Packed documents: their lengths are on the device.  Half an SM's share of all chunks bounds a part: the longest parts
  // start first, so what is left at the end is short.
  const int64_t all_chunks = (int64_t)p->B * p->S / CW_L, docs = p->num_docs;
  const double share = (double)all_chunks * per_doc / SMS;
  int64_t cap = (int64_t)(0.5 * share) + 1;
  cap = cap < 8 ? 8 : (cap > CW_MAX_PART_CHUNKS ? CW_MAX_PART_CHUNKS : cap);
  const int64_t least = (row_chunks + CW_MAX_PARTS - 1) / CW_MAX_PARTS;
  if (cap < least) cap = least;
  // Nothing to gain where all blocks run at once anyway and no document can be longer than a part
  if (row_chunks <= cap && docs * per_doc <= SMS) return no;
  const int64_t slots = all_chunks / cap;
  if (slots * state_bytes > MAX_STATE_BYTES || docs + slots > 65535) return no;
  return {true, 0, (int)cap, docs + slots, slots};
}

struct SplitScratch { int64_t counts, items, slots, gm, n_loc, c_loc, total; };
static SplitScratch scratch_layout(const xl_mlstm_seq_params* p, const CwChoice& c) {
  auto up = [](int64_t x) { return (x + 255) / 256 * 256; };
  SplitScratch s;
  const bool packed = p->cu_seqlens != nullptr;
  s.counts = 0;
  s.items = packed ? 256 : 0;
  s.slots = s.items + (packed ? up(c.items * (int64_t)sizeof(CwItem)) : 0);
  s.gm = s.slots + (packed ? up(c.slots * (int64_t)sizeof(CwItem)) : 0);
  s.n_loc = s.gm + up(c.slots * p->NH * (int64_t)sizeof(float2));
  s.c_loc = s.n_loc + up(c.slots * p->NH * (int64_t)p->DHQK * 4);
  s.total = s.c_loc + up(c.slots * p->NH * (int64_t)p->DHQK * p->DHV * 4);
  return s;
}

int64_t cw_split_scratch_bytes(const xl_mlstm_seq_params* p) {
  if (p->B <= 0 || p->NH <= 0 || p->S <= 0 || p->DHQK <= 0 || p->DHV < CW_DV || p->num_docs < 0) return 0;
  const CwChoice c = choose_split(p);
  return c.split ? scratch_layout(p, c).total : 0;
}

template <int DHQK>
static int launch_part_state(const CwMaps& maps, const xl_mlstm_seq_params* p, const CwSplit& split, int chunks, int64_t slots, cudaStream_t st) {
  using LY = PsLayout<DHQK>;
  static_assert(LY::bytes(CW_MAX_PART_CHUNKS) <= 227 * 1024, "shared memory budget");
  auto kern = mlstm_part_state_kernel<DHQK>;
  XL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LY::bytes(CW_MAX_PART_CHUNKS)));
  XL_CUDA_TRY(launch_dependent(kern, dim3(p->DHV / CW_DV, p->NH, (unsigned)slots), dim3(PS_THREADS), LY::bytes(chunks), st, maps, *p, split));
  return check_launch("xl_mlstm_chunkwise");
}

int cw_prepare_split(const CwMaps& maps, const xl_mlstm_seq_params* p, void* scratch, int64_t scratch_bytes, CwSplit* split, unsigned* grid_z,
                     cudaStream_t st) {
  const CwChoice c = choose_split(p);
  const SplitScratch s = scratch_layout(p, c);
  if (scratch_bytes < s.total) return XL_ERR_TOO_LARGE;
  unsigned char* base = static_cast<unsigned char*>(scratch);
  split->gm = reinterpret_cast<float2*>(base + s.gm);
  split->n_loc = reinterpret_cast<float*>(base + s.n_loc);
  split->c_loc = reinterpret_cast<float*>(base + s.c_loc);
  *grid_z = (unsigned)c.items;
  if (p->cu_seqlens) {
    int* counts = reinterpret_cast<int*>(base + s.counts);
    CwItem *items = reinterpret_cast<CwItem*>(base + s.items), *slots = reinterpret_cast<CwItem*>(base + s.slots);
    split->counts = counts;
    split->items = items;
    split->slots = slots;
    XL_CUDA_TRY(launch_dependent(mlstm_plan_kernel, dim3(1), dim3(PLAN_THREADS), 0, st, *p, c.chunks, (int)c.items, (int)c.slots, counts, items, slots));
  } else {
    split->parts = c.parts;
    split->part_chunks = c.chunks;
  }
  split->after_states = c.slots > 0;
  if (c.slots == 0) return XL_OK;
  switch (p->DHQK) {
    case 64: return launch_part_state<64>(maps, p, *split, c.chunks, c.slots, st);
    case 128: return launch_part_state<128>(maps, p, *split, c.chunks, c.slots, st);
    default: return launch_part_state<256>(maps, p, *split, c.chunks, c.slots, st);
  }
}

}  // namespace xl
