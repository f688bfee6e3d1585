// mLSTM over a sequence in fp32 arithmetic throughout (operands, products, accumulation, state).
//
// It serves (a) fp32 models, where the tensor-core chunkwise kernel's bf16 operands would break the 1e-4
// tolerance, (b) head sizes the chunkwise kernel does not cover, and it is the on-device cross-check for
// the chunkwise kernel in the tests.
//
// One CTA owns a 32-column slice of one document's C matrix, keeps it transposed in shared memory for the whole document
// and walks the document in chunks of 32 tokens -- one warp's width, so every warp forms the gate recurrence of a chunk with
// shuffles, lane = token.  With b_j the in-chunk cumulative log forget gate, a_l = i_l - b_l, mu_j = max(m_prev, max_{l<=j} a_l):
//   [S | QC] = Q [K ; C^T]^T      P_jl = S_jl / sqrt(d) exp(a_l - mu_j) (l <= j)      r_j = exp(m_prev - mu_j) / sqrt(d)
//   h_j = (r_j QC_j + sum_l P_jl v_l) / (max(|r_j q_j.n + sum_l P_jl|, exp(-(b_j + mu_j))) + eps)
//   C <- exp(m_prev - mu_31) C + sum_l w_l k_l v_l^T,  n likewise,  w_l = exp(a_l - mu_31),  m <- b_31 + mu_31
// The gate recurrence alone is formed in 64 bits: a_l - mu_j is a difference of sums over the chunk, and its rounding would be
// the largest error of h.
// Token by token the kernel was a chain of two CTA barriers and a column reduction per token, 1.6 us each; a chunk
// is two barriers for 32 tokens, and the products run from registers at 2 x 5 outputs per thread (seven 16-byte
// shared-memory loads per 40 FMAs).  3 x 4 heads x 256 tokens, 64 x 128: 274 us token by token, 58 in chunks, 39 with q.n and n
// without shuffles and the head size compiled in; 1 x 8 x 203, 256 x 512: 451 -> 87 us.  h against 64 bits: 3.3e-7 (token by token
// 3.8e-7), with the gate sums and single chains in fp32 6.5e-7.  Chunks of 64 would double the redundant part of the work (S, formed by every slice).
#include "common.cuh"

namespace xl {

constexpr int REC_THREADS = 256;
constexpr int REC_L = 32;                         // tokens per chunk
constexpr int REC_COLS = 32;                      // C columns per CTA
constexpr int REC_LP = REC_L + 4;                 // padded row of the token-indexed tiles (floats)
constexpr float REC_HARD = -1e6f;                 // log f below which a chunk's gates are formed without differences of their
                                                  // sums: above it, 32 of them cost a 64-bit difference 1e-8 at most

__device__ __forceinline__ void rec_cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void rec_cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void fma4(float4& acc, const float4& a, const float4& b) {
  acc.x = fmaf(a.x, b.x, acc.x);
  acc.y = fmaf(a.y, b.y, acc.y);
  acc.z = fmaf(a.z, b.z, acc.z);
  acc.w = fmaf(a.w, b.w, acc.w);
}
__device__ __forceinline__ float sum4(const float4& v) { return (v.x + v.y) + (v.z + v.w); }

// shared memory (floats); rows of DP = DHQK rounded up to 4, plus 4: eight rows' 16-byte pieces then lie on distinct banks
struct RecLayout {
  int DQ4, DP, nbuf;
  size_t q, k, vt, vw, c, pm, n, w, total;
  __host__ __device__ explicit RecLayout(int DHQK) {
    DQ4 = (DHQK + 3) / 4;
    DP = 4 * DQ4 + 4;
    nbuf = DHQK <= 256 ? 2 : 1;                   // two chunks in flight where they fit
    q = 0;
    k = q + (size_t)nbuf * REC_L * DP;
    vt = k + (size_t)nbuf * REC_L * DP;           // v transposed [column][token]
    vw = vt + (size_t)nbuf * REC_COLS * REC_LP;   // the same times w_l
    c = vw + (size_t)REC_COLS * REC_LP;           // C^T [column][feature]
    pm = c + (size_t)REC_COLS * DP;               // P [row][token]
    n = pm + (size_t)REC_L * REC_LP;
    w = n + (size_t)DP;                           // w_l
    total = w + REC_L;
  }
};

// D: DHQK where it is known at compile time (addresses and trip counts of the inner loops are constants then), 0: any
template <typename T, int D>
__global__ void __launch_bounds__(REC_THREADS, 1) mlstm_recurrent_kernel(const xl_mlstm_seq_params p, int vec) {
  extern __shared__ __align__(16) float smem[];
  const RecLayout ly(D ? D : p.DHQK);
  const int DHQK = D ? D : p.DHQK, DHV = p.DHV, DQ4 = ly.DQ4, DP = ly.DP;
  float* s_c = smem + ly.c;
  float* s_n = smem + ly.n;
  float* s_p = smem + ly.pm;
  float* s_vw = smem + ly.vw;
  float* s_w = smem + ly.w;

  const int doc = blockIdx.z, head = blockIdx.y, col0 = blockIdx.x * REC_COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  // document -> (batch row, first token, length)
  int64_t tok0, len;
  int b;
  if (p.cu_seqlens) {
    const int64_t s = p.cu_seqlens[doc], e = p.cu_seqlens[doc + 1];
    b = (int)(s / p.S);
    tok0 = s - (int64_t)b * p.S;
    len = e - s;
  } else {
    b = doc; tok0 = 0; len = p.S;
  }
  const T* q = reinterpret_cast<const T*>(p.q) + b * p.q_sb + head * p.q_sh + tok0 * p.q_st;
  const T* k = reinterpret_cast<const T*>(p.k) + b * p.k_sb + head * p.k_sh + tok0 * p.k_st;
  const T* v = reinterpret_cast<const T*>(p.v) + b * p.v_sb + head * p.v_sh + tok0 * p.v_st;
  T* h = reinterpret_cast<T*>(p.h) + b * p.h_sb + head * p.h_sh + tok0 * p.h_st;
  const float* ig = p.igate + b * p.g_sb + head * p.g_sh + tok0 * p.g_st;
  const float* fg = p.fgate + b * p.g_sb + head * p.g_sh + tok0 * p.g_st;
  const int64_t sidx = (int64_t)doc * p.NH + head;
  const float qscale = rsqrtf((float)DHQK);
  const int nchunks = (int)((len + REC_L - 1) / REC_L);

  // q, k, v of a chunk into buffer `buf`; rows past the document, features past DHQK and columns past DHV are zero.  The
  // pieces a thread loads are the same for all tiles of a shape: 16-byte copies where rows are aligned (`vec`).
  const int r_first = tid / DQ4, d_first = tid - r_first * DQ4, r_step = REC_THREADS / DQ4, d_step = REC_THREADS - r_step * DQ4;
  auto load_chunk = [&](int chunk, int buf) {
    float* tq = smem + ly.q + (size_t)buf * REC_L * DP;
    float* tk = smem + ly.k + (size_t)buf * REC_L * DP;
    float* tv = smem + ly.vt + (size_t)buf * REC_COLS * REC_LP;
    const int64_t t0 = (int64_t)chunk * REC_L;
    const int rows = (int)(len - t0 < REC_L ? len - t0 : REC_L);
    if (sizeof(T) == 4 && vec) {
      const T *qc = q + t0 * p.q_st, *kc = k + t0 * p.k_st;
      int r = r_first, d4 = d_first;
      while (r < REC_L) {
        const int d = 4 * d4;
        if (r < rows) {
          rec_cp_async16(smem_u32(tq + r * DP + d), qc + r * p.q_st + d);
          rec_cp_async16(smem_u32(tk + r * DP + d), kc + r * p.k_st + d);
        } else {
          *reinterpret_cast<float4*>(tq + r * DP + d) = make_float4(0.f, 0.f, 0.f, 0.f);
          *reinterpret_cast<float4*>(tk + r * DP + d) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        r += r_step;
        d4 += d_step;
        if (d4 >= DQ4) { d4 -= DQ4; ++r; }
      }
    } else {
      const int W = 4 * DQ4;
#pragma unroll 4
      for (int u = tid; u < REC_L * W; u += REC_THREADS) {
        const int r = u / W, d = u - r * W;
        const bool in = r < rows && d < DHQK;
        tq[r * DP + d] = in ? to_float(q[(t0 + r) * p.q_st + d]) : 0.f;
        tk[r * DP + d] = in ? to_float(k[(t0 + r) * p.k_st + d]) : 0.f;
      }
    }
    const T* vc = v + (t0 + warp) * p.v_st + col0 + lane;   // a warp takes one token's columns
#pragma unroll
    for (int i = 0; i < REC_L / 8; ++i) {
      const int r = warp + 8 * i;
      const bool in = r < rows && col0 + lane < DHV;
      const T* src = vc + 8 * i * p.v_st;
      if (sizeof(T) == 4 && in) rec_cp_async4(smem_u32(tv + lane * REC_LP + r), src);
      else tv[lane * REC_LP + r] = in ? to_float(*src) : 0.f;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // initial state
  for (int u = tid; u < REC_COLS * 4 * DQ4; u += REC_THREADS) {
    const int d = u / REC_COLS, c = u % REC_COLS;
    s_c[c * DP + d] = (p.c0 && d < DHQK && col0 + c < DHV) ? p.c0[(sidx * DHQK + d) * DHV + col0 + c] : 0.f;
  }
  for (int d = tid; d < 4 * DQ4; d += REC_THREADS) s_n[d] = (p.n0 && d < DHQK) ? p.n0[sidx * DHQK + d] : 0.f;
  double m_prev = p.m0 ? p.m0[sidx] : 0.f;

  // output tile of a thread: rows j0, j0 + 16; S columns / value columns c0, c0 + 16
  const int j0 = (warp & 3) * 4 + (lane >> 3), c0 = (warp >> 2) * 8 + (lane & 7);

  if (nchunks > 0) load_chunk(0, 0);
  float gi = lane < len ? ig[lane * p.g_st] : 0.f, gf = lane < len ? fg[lane * p.g_st] : 0.f;
  for (int chunk = 0; chunk < nchunks; ++chunk) {
    const int buf = chunk % ly.nbuf;
    const float* tq = smem + ly.q + (size_t)buf * REC_L * DP;
    const float* tk = smem + ly.k + (size_t)buf * REC_L * DP;
    const float* tv = smem + ly.vt + (size_t)buf * REC_COLS * REC_LP;
    const int64_t t0 = (int64_t)chunk * REC_L;
    // ---- gate recurrence of the chunk, lane = token; every warp forms it for itself
    const bool live = t0 + lane < len;
    const float lf = live ? log_sigmoid(gf) : 0.f, iv = live ? gi : -INFINITY;
    {
      const int64_t tn = t0 + REC_L + lane;   // the next chunk's gates
      gi = tn < len ? ig[tn * p.g_st] : 0.f;
      gf = tn < len ? fg[tn * p.g_st] : 0.f;
    }
    double bcum = lf;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(0xffffffffu, bcum, o);
      if (lane >= o) bcum += t;
    }
    double al = iv - bcum, mu = fmax(al, m_prev);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double t = __shfl_up_sync(0xffffffffu, mu, o);
      if (lane >= o) mu = fmax(mu, t);
    }
    const double mu_last = __shfl_sync(0xffffffffu, mu, 31), b_last = __shfl_sync(0xffffffffu, bcum, 31);
    float r_tok = expf((float)(m_prev - mu)) * qscale, lower = expf((float)-(bcum + mu)), w_tok = expf((float)(al - mu_last));
    float decay = expf((float)(m_prev - mu_last));
    double m_next = b_last + mu_last;
    const bool hard = __any_sync(0xffffffffu, lf < REC_HARD);
    if (hard) {
      // A forget gate that resets the state (the same for every warp).  b reaches -inf, or a size beside which the input
      // gates are lost, so nothing may be a difference of its values: the stabilisers m_j themselves by a scan over
      // (sum of log f, max) pairs, sums in front of and behind a token on their own.  al and mu are i and m here; what lies
      // between two tokens is added below, where P is formed.
      double g = lf, x = iv, behind = 0.;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double tg = __shfl_up_sync(0xffffffffu, g, o), tx = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) {
          x = fmax(x, tx + g);
          g += tg;
        }
      }
#pragma unroll 1
      for (int t = 1; t < 32; ++t) {
        const float ft = __shfl_sync(0xffffffffu, lf, t);
        if (t > lane) behind += ft;
      }
      al = iv;
      mu = fmax(m_prev + g, x);
      m_next = __shfl_sync(0xffffffffu, mu, 31);
      r_tok = expf((float)(m_prev + g - mu)) * qscale;
      lower = expf((float)-mu);
      w_tok = expf((float)(iv + behind - m_next));
      decay = expf((float)(m_prev + __shfl_sync(0xffffffffu, g, 31) - m_next));
    }
    m_prev = m_next;

    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // the chunk is in shared memory; C and n of the previous chunk are complete
    if (ly.nbuf == 2 && chunk + 1 < nchunks) load_chunk(chunk + 1, buf ^ 1);

    // ---- [S | QC | q.n] = Q [K ; C^T ; n]^T, 2 x (2 + 2 + 1) outputs per thread: the eight threads of a row pair form the
    // same q.n, which costs less than the shuffles that would share the work.  Four chains per sum, one per component of the
    // 16-byte pieces: a quarter of the roundings in a row, no more instructions.
    float s[2][2], qc[2][2], qn0, qn1;
    {
      const float *q0 = tq + j0 * DP, *q1 = q0 + 16 * DP, *k0 = tk + c0 * DP, *k1 = k0 + 16 * DP, *x0 = s_c + c0 * DP, *x1 = x0 + 16 * DP;
      float4 acc[2][5] = {};
#pragma unroll 4
      for (int d = 0; d < 4 * DQ4; d += 4) {
        const float4 a0 = *reinterpret_cast<const float4*>(q0 + d), a1 = *reinterpret_cast<const float4*>(q1 + d);
        const float4 b[5] = {*reinterpret_cast<const float4*>(k0 + d), *reinterpret_cast<const float4*>(k1 + d), *reinterpret_cast<const float4*>(x0 + d),
                             *reinterpret_cast<const float4*>(x1 + d), *reinterpret_cast<const float4*>(s_n + d)};
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          fma4(acc[0][i], a0, b[i]);
          fma4(acc[1][i], a1, b[i]);
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        s[j][0] = sum4(acc[j][0]); s[j][1] = sum4(acc[j][1]);
        qc[j][0] = sum4(acc[j][2]); qc[j][1] = sum4(acc[j][3]);
      }
      qn0 = sum4(acc[0][4]);
      qn1 = sum4(acc[1][4]);
    }
    // ---- P and the w-scaled v
    const double mu0 = __shfl_sync(0xffffffffu, mu, j0), mu1 = __shfl_sync(0xffffffffu, mu, j0 + 16);
    const double al0 = __shfl_sync(0xffffffffu, al, c0), al1 = __shfl_sync(0xffffffffu, al, c0 + 16);
    float e00 = (float)(al0 - mu0), e10 = (float)(al0 - mu1), e11 = (float)(al1 - mu1);
    if (hard) {   // the sums of log f over the tokens behind l up to j
      double d00 = 0., d10 = 0., d11 = 0.;
#pragma unroll 1
      for (int t = 1; t < 32; ++t) {
        const float ft = __shfl_sync(0xffffffffu, lf, t);
        if (t > c0 && t <= j0) d00 += ft;
        if (t > c0 && t <= j0 + 16) d10 += ft;
        if (t > c0 + 16 && t <= j0 + 16) d11 += ft;
      }
      e00 = (float)(al0 + d00 - mu0);
      e10 = (float)(al0 + d10 - mu1);
      e11 = (float)(al1 + d11 - mu1);
    }
    s_p[j0 * REC_LP + c0] = c0 <= j0 ? s[0][0] * qscale * expf(e00) : 0.f;
    s_p[j0 * REC_LP + c0 + 16] = 0.f;                                     // (c0 + 16 > j0)
    s_p[(j0 + 16) * REC_LP + c0] = s[1][0] * qscale * expf(e10);          // (c0 < j0 + 16)
    s_p[(j0 + 16) * REC_LP + c0 + 16] = c0 <= j0 ? s[1][1] * qscale * expf(e11) : 0.f;
    bool odd_v = false;
#pragma unroll
    for (int i = 0; i < REC_COLS / 8; ++i) {
      const int at = (warp * (REC_COLS / 8) + i) * REC_LP + lane;
      const float x = tv[at];
      odd_v |= !(fabsf(x) < INFINITY);
      s_vw[at] = x * w_tok;
    }
    if (warp == 0) s_w[lane] = w_tok;
    // P, the scaled v and w are complete, C and n are read; and whether an infinity or a NaN is among the chunk's values
    const bool any_odd_v = __syncthreads_or(odd_v);

    // ---- h = (r QC + P V) / den
    {
      float4 oa[2][2] = {}, ra[2] = {};
      const float *p0 = s_p + j0 * REC_LP, *p1 = p0 + 16 * REC_LP, *v0 = tv + c0 * REC_LP, *v1 = v0 + 16 * REC_LP;
      const float4 one = make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
      for (int l = 0; l < REC_L; l += 4) {
        const float4 b0 = *reinterpret_cast<const float4*>(v0 + l), b1 = *reinterpret_cast<const float4*>(v1 + l);
        const float4 a1 = *reinterpret_cast<const float4*>(p1 + l);
        if (l < 16) {   // row j0 < 16 has no later tokens
          const float4 a0 = *reinterpret_cast<const float4*>(p0 + l);
          fma4(oa[0][0], a0, b0); fma4(oa[0][1], a0, b1);
          fma4(ra[0], a0, one);
        }
        fma4(oa[1][0], a1, b0); fma4(oa[1][1], a1, b1);
        fma4(ra[1], a1, one);
      }
      float o[2][2] = {{sum4(oa[0][0]), sum4(oa[0][1])}, {sum4(oa[1][0]), sum4(oa[1][1])}};
      const float rs0 = sum4(ra[0]), rs1 = sum4(ra[1]);
      if (any_odd_v) {   // 0 x inf: the zeros of P right of the diagonal must not meet the values of later tokens
        o[0][0] = o[0][1] = o[1][0] = o[1][1] = 0.f;
#pragma unroll 1
        for (int l = 0; l <= j0 + 16; ++l) {
          if (l <= j0) {
            o[0][0] = fmaf(p0[l], v0[l], o[0][0]);
            o[0][1] = fmaf(p0[l], v1[l], o[0][1]);
          }
          o[1][0] = fmaf(p1[l], v0[l], o[1][0]);
          o[1][1] = fmaf(p1[l], v1[l], o[1][1]);
        }
      }
      const float r0 = __shfl_sync(0xffffffffu, r_tok, j0), r1 = __shfl_sync(0xffffffffu, r_tok, j0 + 16);
      const float lo0 = __shfl_sync(0xffffffffu, lower, j0), lo1 = __shfl_sync(0xffffffffu, lower, j0 + 16);
      const float den0 = fmaxf(fabsf(fmaf(r0, qn0, rs0)), lo0) + p.eps, den1 = fmaxf(fabsf(fmaf(r1, qn1, rs1)), lo1) + p.eps;
      T* h0 = h + (t0 + j0) * p.h_st + col0 + c0;
      T* h1 = h0 + 16 * p.h_st;
      const bool ok0 = col0 + c0 < DHV, ok1 = col0 + c0 + 16 < DHV;
      if (t0 + j0 < len) {
        if (ok0) h0[0] = from_float<T>(fmaf(r0, qc[0][0], o[0][0]) / den0);
        if (ok1) h0[16] = from_float<T>(fmaf(r0, qc[0][1], o[0][1]) / den0);
      }
      if (t0 + j0 + 16 < len) {
        if (ok0) h1[0] = from_float<T>(fmaf(r1, qc[1][0], o[1][0]) / den1);
        if (ok1) h1[16] = from_float<T>(fmaf(r1, qc[1][1], o[1][1]) / den1);
      }
    }
    // ---- C^T <- decay C^T + (w v)^T K: units of two columns x four features
    for (int u = tid; u < (REC_COLS / 2) * DQ4; u += REC_THREADS) {
      const int cp = u / DQ4, d = 4 * (u - cp * DQ4);
      float4* x0 = reinterpret_cast<float4*>(s_c + cp * DP + d);
      float4* x1 = reinterpret_cast<float4*>(s_c + (cp + 16) * DP + d);
      float4 a = *x0, e = *x1;
      a.x *= decay; a.y *= decay; a.z *= decay; a.w *= decay;
      e.x *= decay; e.y *= decay; e.z *= decay; e.w *= decay;
#pragma unroll
      for (int l = 0; l < REC_L; l += 4) {
        const float4 wa = *reinterpret_cast<const float4*>(s_vw + cp * REC_LP + l), we = *reinterpret_cast<const float4*>(s_vw + (cp + 16) * REC_LP + l);
        const float ca[4] = {wa.x, wa.y, wa.z, wa.w}, ce[4] = {we.x, we.y, we.z, we.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 kk = *reinterpret_cast<const float4*>(tk + (l + i) * DP + d);
          a.x = fmaf(ca[i], kk.x, a.x); a.y = fmaf(ca[i], kk.y, a.y); a.z = fmaf(ca[i], kk.z, a.z); a.w = fmaf(ca[i], kk.w, a.w);
          e.x = fmaf(ce[i], kk.x, e.x); e.y = fmaf(ce[i], kk.y, e.y); e.z = fmaf(ce[i], kk.z, e.z); e.w = fmaf(ce[i], kk.w, e.w);
        }
      }
      *x0 = a;
      *x1 = e;
    }
    // ---- n <- decay n + sum_l w_l k_l: thread = feature, the last warps first (the first ones may have one more unit of C)
    for (int d = REC_THREADS - 1 - tid; d < DHQK; d += REC_THREADS) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int l = 0; l < REC_L; l += 4) {
        const float4 w = *reinterpret_cast<const float4*>(s_w + l);
        x.x = fmaf(w.x, tk[l * DP + d], x.x);
        x.y = fmaf(w.y, tk[(l + 1) * DP + d], x.y);
        x.z = fmaf(w.z, tk[(l + 2) * DP + d], x.z);
        x.w = fmaf(w.w, tk[(l + 3) * DP + d], x.w);
      }
      s_n[d] = fmaf(decay, s_n[d], sum4(x));
    }
    if (ly.nbuf == 1 && chunk + 1 < nchunks) {
      __syncthreads();   // the only buffer is free
      load_chunk(chunk + 1, 0);
    }
  }
  __syncthreads();

  // final state
  for (int u = tid; u < REC_COLS * DHQK; u += REC_THREADS) {
    const int d = u / REC_COLS, c = u % REC_COLS;
    if (col0 + c < DHV) p.c_out[(sidx * DHQK + d) * DHV + col0 + c] = s_c[c * DP + d];
  }
  if (blockIdx.x == 0) {
    for (int d = tid; d < DHQK; d += REC_THREADS) p.n_out[sidx * DHQK + d] = s_n[d];
    if (tid == 0) p.m_out[sidx] = (float)m_prev;
  }
}

int validate_seq_common(const xl_mlstm_seq_params* p) {
  if (!p || !p->q || !p->k || !p->v || !p->h || !p->igate || !p->fgate || !p->c_out || !p->n_out || !p->m_out)
    return XL_ERR_NULL_POINTER;
  const bool any0 = p->c0 || p->n0 || p->m0, all0 = p->c0 && p->n0 && p->m0;
  if (any0 && !all0) return XL_ERR_NULL_POINTER;
  if (all0 && (p->n0 == p->n_out || p->m0 == p->m_out)) return XL_ERR_ALIASING;
  if (p->B <= 0 || p->NH <= 0 || p->S <= 0 || p->DHQK <= 0 || p->DHV <= 0) return XL_ERR_BAD_SHAPE;
  if (p->cu_seqlens && p->num_docs <= 0) return XL_ERR_BAD_SHAPE;
  if (p->NH > 65535) return XL_ERR_BAD_SHAPE;
  const int nd = p->cu_seqlens ? p->num_docs : p->B;
  if (nd > 65535) return XL_ERR_TOO_LARGE;
  if (p->dtype != XL_F32 && p->dtype != XL_BF16) return XL_ERR_BAD_DTYPE;
  return XL_OK;
}

template <typename T>
static int launch_recurrent(const xl_mlstm_seq_params* p, size_t smem, cudaStream_t st) {
  auto kern = p->DHQK == 64    ? mlstm_recurrent_kernel<T, 64>
              : p->DHQK == 128 ? mlstm_recurrent_kernel<T, 128>
              : p->DHQK == 256 ? mlstm_recurrent_kernel<T, 256>
                               : mlstm_recurrent_kernel<T, 0>;
  XL_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int nd = p->cu_seqlens ? p->num_docs : p->B;
  // 16-byte copies of q and k rows (fp32): every row starts on a 16-byte boundary and is a whole number of pieces
  const bool vec = aligned16(p->q) && aligned16(p->k) && p->DHQK % 4 == 0 &&
                   !((p->q_sb | p->q_sh | p->q_st | p->k_sb | p->k_sh | p->k_st) & 3);
  kern<<<dim3((p->DHV + REC_COLS - 1) / REC_COLS, p->NH, nd), REC_THREADS, smem, st>>>(*p, vec ? 1 : 0);
  return check_launch("xl_mlstm_recurrent");
}

}  // namespace xl

extern "C" int xl_mlstm_recurrent(const xl_mlstm_seq_params* p, void* cuda_stream) {
  using namespace xl;
  int rc = validate_seq_common(p);
  if (rc != XL_OK) return rc;
  if (p->DHQK > 512) return XL_ERR_BAD_SHAPE;
  const size_t smem = RecLayout(p->DHQK).total * sizeof(float);
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  return p->dtype == XL_F32 ? launch_recurrent<float>(p, smem, st) : launch_recurrent<__nv_bfloat16>(p, smem, st);
}
