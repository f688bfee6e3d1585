// Operators next to the mLSTM cell in the reference's layer, each fused into one pass over its data:
//   xl_add_rmsnorm    residual add + RMSNorm                      (xlstm/xlstm_large/model.py:499-510, components.py:70-97)
//   xl_soft_cap       cap * tanh(x / cap) of gate pre-activations and logits  (components.py:5-22)
//   xl_headnorm_gate  per-head LayerNorm of the cell output read through its (B,NH,S,DH) strides, weight, output gate
//                     (xlstm/xlstm_large/model.py:435-449, components.py:171-242)
//   xl_causal_conv1d  depthwise causal convolution over time + SiLU in front of the sLSTM cell, with document
//                     boundaries (xlstm/components/conv.py:110-129, xlstm/blocks/slstm/layer.py:133-142)
//   xl_swiglu         silu(gate) * up of the feed-forward block (xlstm/xlstm_large/model.py:268-277)
// Both are bound by HBM traffic: every element is read once with 16-byte loads, kept in registers across the
// reduction, and written once.  Rounding points are those of the reference's eager operator sequence (fp32
// reductions; the normalised value rounded to the model dtype, then the weight product rounded, then the gate).
#include "common.cuh"

namespace xl {

constexpr int ADJ_MAXC = 4;  // most 16-byte vectors per thread (kernels are instantiated for 1, 2 and 4)

template <typename T> struct Vec16;
template <> struct Vec16<float> {
  static constexpr int N = 4;
  float v[4];
};
template <> struct Vec16<__nv_bfloat16> {
  static constexpr int N = 8;
  __nv_bfloat16 v[8];
};

template <typename T>
__device__ __forceinline__ Vec16<T> load16(const T* p) {
  Vec16<T> r;
  *reinterpret_cast<uint4*>(r.v) = *reinterpret_cast<const uint4*>(p);
  return r;
}
template <typename T>
__device__ __forceinline__ void store16(T* p, const Vec16<T>& r) {
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(r.v);
}

// The gate is rounded to T right away: for bf16 the hardware exponential and reciprocal (a few fp32 ulp) are far
// inside the rounding step and keep the kernel on the memory roofline (with expf and an IEEE division the kernel
// was bound by instruction issue: 0.49 ms against 0.25 ms of traffic at the 7B shapes); fp32 keeps the exact forms.
// out = round(round(sigmoid(o)) * round(round((h - mean) * r) * w)), the eager reference's rounding sequence.
__device__ __forceinline__ Vec16<float> normalise_weight_gate(const Vec16<float>& h, const Vec16<float>& o,
                                                              const Vec16<float>& w, float mean, float r) {
  Vec16<float> y;
#pragma unroll
  for (int i = 0; i < 4; ++i) y.v[i] = sigmoid_for<float>(o.v[i]) * (((h.v[i] - mean) * r) * w.v[i]);
  return y;
}
// bf16: two elements per instruction where the hardware has it -- one packed conversion per rounding point and
// packed bf16 multiplies (the product of two bf16 values rounded once, which is what "multiply in fp32, round to
// bf16" gives).  Element by element, with a conversion per rounding, the kernel was bound by instruction issue.
__device__ __forceinline__ Vec16<__nv_bfloat16> normalise_weight_gate(const Vec16<__nv_bfloat16>& h, const Vec16<__nv_bfloat16>& o,
                                                                      const Vec16<__nv_bfloat16>& w, float mean, float r) {
  Vec16<__nv_bfloat16> y;
  const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(h.v);
  const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(o.v);
  const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(w.v);
  __nv_bfloat162* y2 = reinterpret_cast<__nv_bfloat162*>(y.v);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 hf = __bfloat1622float2(h2[i]), of = __bfloat1622float2(o2[i]);
    const __nv_bfloat162 nw = __hmul2(__floats2bfloat162_rn((hf.x - mean) * r, (hf.y - mean) * r), w2[i]);
    const __nv_bfloat162 g = __floats2bfloat162_rn(sigmoid_for<__nv_bfloat16>(of.x), sigmoid_for<__nv_bfloat16>(of.y));
    y2[i] = __hmul2(g, nw);
  }
  return y;
}

// Without a gate (o == NULL): out = round((h - mean) * r * w), one rounding, as a group norm computes it
// (F.group_norm in MultiHeadLayerNorm.forward, xlstm/components/ln.py:52-68).
template <typename T>
__device__ __forceinline__ Vec16<T> normalise_weight(const Vec16<T>& h, const Vec16<T>& w, float mean, float r) {
  Vec16<T> y;
#pragma unroll
  for (int i = 0; i < Vec16<T>::N; ++i) y.v[i] = from_float<T>(((to_float(h.v[i]) - mean) * r) * to_float(w.v[i]));
  return y;
}

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// ------------------------------------------------------------------------------------------------------------
// residual add + RMSNorm: one CTA of 256 threads per row
// ------------------------------------------------------------------------------------------------------------
constexpr int RMS_THREADS = 256;

template <typename T, int NC>
__global__ void __launch_bounds__(RMS_THREADS) add_rmsnorm_kernel(const xl_add_rmsnorm_params p) {
  constexpr int V = Vec16<T>::N;
  __shared__ float s_part[RMS_THREADS / 32];
  const long long row = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  grid_dependency_wait();
  grid_dependents_launch();
  const T* x = static_cast<const T*>(p.x) + row * p.x_sr;
  const T* y = p.y ? static_cast<const T*>(p.y) + row * p.y_sr : nullptr;
  const T* w = static_cast<const T*>(p.weight);
  T* xo = p.x_out ? static_cast<T*>(p.x_out) + row * p.xo_sr : nullptr;
  T* nd = static_cast<T*>(p.normed) + row * p.n_sr;

  // every load of the row is issued before the first use (x, y and the weights: up to 12 vectors in flight per thread)
  Vec16<T> xv[NC], yv[NC], wv[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int e = (c * RMS_THREADS + tid) * V;
    if (e < p.D) {
      xv[c] = load16(x + e);
      if (y) yv[c] = load16(y + e);
    }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int e = (c * RMS_THREADS + tid) * V;
    if (e < p.D) wv[c] = load16(w + e);
  }
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int e = (c * RMS_THREADS + tid) * V;
    if (e < p.D) {
      if (y) {
#pragma unroll
        for (int i = 0; i < V; ++i) xv[c].v[i] = from_float<T>(to_float(xv[c].v[i]) + to_float(yv[c].v[i]));
        store16(xo + e, xv[c]);
      }
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const float f = to_float(xv[c].v[i]);
        ss = fmaf(f, f, ss);
      }
    }
  }
  ss = warp_sum(ss);
  if (lane == 0) s_part[warp] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < RMS_THREADS / 32; ++i) tot += s_part[i];
  const float r = rsqrtf(tot / (float)p.D + p.eps);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int e = (c * RMS_THREADS + tid) * V;
    if (e < p.D) {
      Vec16<T> o;
#pragma unroll
      for (int i = 0; i < V; ++i)
        o.v[i] = from_float<T>(to_float(from_float<T>(to_float(xv[c].v[i]) * r)) * to_float(wv[c].v[i]));
      store16(nd + e, o);
    }
  }
}

// ------------------------------------------------------------------------------------------------------------
// per-head LayerNorm + weight + output gate: one warp per (batch, R consecutive tokens, head)
// ------------------------------------------------------------------------------------------------------------
constexpr int HNG_WARPS = 8;
// Vectors of h a warp has in flight where there are enough rows to fill the machine all the same.  With one token per warp
// a block lived for one load latency and the launch rate of blocks bound it: 16 x 2048 tokens, 4 heads of 256 (134 MB):
// 40 us, 36 with four tokens.
constexpr int HNG_IN_FLIGHT = 4;
constexpr long long HNG_FULL = 148 * 64 * 8;   // rows (token, head) from which on

template <typename T, int NC, int R>
__global__ void __launch_bounds__(HNG_WARPS * 32) headnorm_gate_kernel(const xl_headnorm_gate_params p) {
  constexpr int V = Vec16<T>::N;
  const int lane = threadIdx.x & 31;
  // 32-bit index arithmetic on purpose (grid.y = batch row): with 64-bit divisions for (batch, token, head) the index
  // computation alone was more than half of the warp's instructions
  const unsigned unit = blockIdx.x * HNG_WARPS + (threadIdx.x >> 5);   // (group of R tokens, head) within the batch row
  if (unit >= ((unsigned)p.S + R - 1) / R * (unsigned)p.NH) return;
  const unsigned sg = unit / (unsigned)p.NH, head = unit - sg * (unsigned)p.NH, s0 = sg * R;
  const long long b = blockIdx.y;
  const T* h = static_cast<const T*>(p.h) + b * p.h_sb + head * p.h_sh + s0 * p.h_st;
  const T* o = static_cast<const T*>(p.o) + b * p.o_sb + s0 * p.o_st + (long long)head * p.DH;
  const T* w = static_cast<const T*>(p.weight) + (long long)head * p.DH;
  T* out = static_cast<T*>(p.out) + ((b * p.S + s0) * p.NH + head) * p.DH;

  // every load of the rows is issued before the first use
  Vec16<T> hv[R][NC], ov[R][NC], wv[NC];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int e = (c * 32 + lane) * V;
      if (e < p.DH && (R == 1 || s0 + r < (unsigned)p.S)) {
        hv[r][c] = load16(h + r * p.h_st + e);
        if (p.o) ov[r][c] = load16(o + r * p.o_st + e);
      }
    }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int e = (c * 32 + lane) * V;
    if (e < p.DH) wv[c] = load16(w + e);
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (R > 1 && s0 + r >= (unsigned)p.S) break;
    float sum = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int e = (c * 32 + lane) * V;
      if (e < p.DH) {
#pragma unroll
        for (int i = 0; i < V; ++i) sum += to_float(hv[r][c].v[i]);
      }
    }
    const float mean = warp_sum(sum) / (float)p.DH;
    float sq = 0.f;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int e = (c * 32 + lane) * V;
      if (e < p.DH) {
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const float d = to_float(hv[r][c].v[i]) - mean;
          sq = fmaf(d, d, sq);
        }
      }
    }
    const float rstd = rsqrtf(warp_sum(sq) / (float)p.DH + p.eps);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int e = (c * 32 + lane) * V;
      if (e < p.DH)
        store16(out + (long long)r * p.NH * p.DH + e, p.o ? normalise_weight_gate(hv[r][c], ov[r][c], wv[c], mean, rstd)
                                                          : normalise_weight<T>(hv[r][c], wv[c], mean, rstd));
    }
  }
}

// ------------------------------------------------------------------------------------------------------------
// soft cap: cap * tanh(x / cap), each operator's result rounded to T
// ------------------------------------------------------------------------------------------------------------
template <typename T, typename O, bool ROUND_EACH>
__global__ void __launch_bounds__(256) soft_cap_kernel(const T* __restrict__ x, O* __restrict__ out, long long n, float cap,
                                                       long long cols, long long x_row_stride, const T* __restrict__ bias) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  grid_dependency_wait();
  grid_dependents_launch();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    // (rows of `cols` elements `x_row_stride` apart: a column slice of a wider projection output; a bias per column is
    // added first, rounded to T as the reference's Linear rounds its output)
    float v;
    if (cols > 0) {
      const long long r = i / cols, c = i - r * cols;
      v = to_float(x[r * x_row_stride + c]);
      if (bias) v = to_float(from_float<T>(v + to_float(bias[c])));
    } else {
      v = to_float(x[i]);
    }
    if (ROUND_EACH) {
      const T q = from_float<T>(v / cap);
      const T t = from_float<T>(tanhf(to_float(q)));
      out[i] = from_float<O>(to_float(from_float<T>(cap * to_float(t))));
    } else {
      out[i] = from_float<O>(cap * tanhf(v / cap));
    }
  }
}

// ---------------------------------------------------------------------------------------------
// SwiGLU: out[r, j] = round(round(silu(gz[r, j])) * gz[r, F + j]) -- the eager sequence of the reference's feed-forward
// (act_fn(proj_up_gate(x)) * proj_up(x), xlstm/xlstm_large/model.py:268-277) on the output of the fused up-projection.
// One pass: reads 2F, writes F per row.
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) swiglu_kernel(const T* __restrict__ gz, T* __restrict__ out, long long rows, int F,
                                                     long long gz_row_stride) {
  constexpr int V = Vec16<T>::N;
  const long long nvec = rows * (long long)(F / V), stride = (long long)gridDim.x * blockDim.x;
  grid_dependency_wait();
  grid_dependents_launch();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nvec; i += stride) {
    const long long r = i / (F / V);
    const int c = (int)(i - r * (F / V)) * V;
    const Vec16<T> g = load16(gz + r * gz_row_stride + c), z = load16(gz + r * gz_row_stride + F + c);
    Vec16<T> o;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float gv = to_float(g.v[k]);
      const float sl = to_float(from_float<T>(gv * sigmoid_for<T>(gv)));
      o.v[k] = from_float<T>(sl * to_float(z.v[k]));
    }
    store16(out + r * (long long)F + c, o);
  }
}

// ---------------------------------------------------------------------------------------------
// Depthwise causal convolution over time, optional SiLU, document boundaries.
//   y[b,t,f] = bias[f] + sum_{lag=0}^{K-1} w[f][K-1-lag] x[b,t-lag,f]      (taps that reach in front of the first token of
//   the document -- or of the row -- read zero), out = silu(round(y)).
// A thread owns one 16-byte vector of features and walks CONV_TILE consecutive tokens with the last K-1 inputs in
// registers, so x is read once (plus a K-1 token halo per tile) and out written once: HBM-bound.  The loads of CONV_GROUP
// tokens are issued together -- one token at a time a thread waited out a load's latency per token -- and the taps are
// compiled for the kernel size, without a test per tap unless a document starts near.
// 16 x 2048 tokens x 1024 features, K = 4 (134 MB): 43 us, 148 before.
// ---------------------------------------------------------------------------------------------
constexpr int CONV_THREADS = 128, CONV_TILE = 32, CONV_GROUP = 8, CONV_MAXK = 8;

template <typename T, int K>
__global__ void __launch_bounds__(CONV_THREADS) causal_conv1d_kernel(const xl_conv1d_params p) {
  constexpr int V = Vec16<T>::N, W = K > 1 ? K - 1 : 1;
  const unsigned fblocks = (unsigned)(p.F / V + CONV_THREADS - 1) / CONV_THREADS;   // (one axis for both: either may be long)
  const unsigned tile = blockIdx.x / fblocks;
  const int f0 = ((blockIdx.x - tile * fblocks) * CONV_THREADS + threadIdx.x) * V;
  if (f0 >= p.F) return;
  const int b = blockIdx.y;
  const int t0 = tile * CONV_TILE, t1 = min(p.S, t0 + CONV_TILE);
  const T* x = static_cast<const T*>(p.x) + (long long)b * p.x_sb + f0;
  T* out = static_cast<T*>(p.out) + (long long)b * p.o_sb + f0;
  // win[l-1] = x[t-l]; wl[l] multiplies x[t-l] (tap K-1-l of the convolution's weight)
  Vec16<T> win[W];
#pragma unroll
  for (int l = 1; l < K; ++l) {
#pragma unroll
    for (int i = 0; i < V; ++i) win[l - 1].v[i] = from_float<T>(0.f);
    if (t0 - l >= 0) win[l - 1] = load16(x + (long long)(t0 - l) * p.x_st);
  }
  float wl[K][V], bias[V];
  const T *wp = static_cast<const T*>(p.weight) + (long long)f0 * K, *bp = static_cast<const T*>(p.bias) + f0;
  if ((reinterpret_cast<uintptr_t>(wp) | (p.bias ? reinterpret_cast<uintptr_t>(bp) : 0)) % 16 == 0) {   // V rows of K taps: K whole vectors
    Vec16<T> raw[K];
#pragma unroll
    for (int j = 0; j < K; ++j) raw[j] = load16(wp + j * V);
#pragma unroll
    for (int i = 0; i < V; ++i)
#pragma unroll
      for (int l = 0; l < K; ++l) wl[l][i] = to_float(raw[(i * K + K - 1 - l) / V].v[(i * K + K - 1 - l) % V]);
    Vec16<T> rb;
    if (p.bias) rb = load16(bp);
#pragma unroll
    for (int i = 0; i < V; ++i) bias[i] = p.bias ? to_float(rb.v[i]) : 0.f;
  } else {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      bias[i] = p.bias ? to_float(bp[i]) : 0.f;
#pragma unroll
      for (int l = 0; l < K; ++l) wl[l][i] = to_float(wp[i * K + (K - 1 - l)]);
    }
  }
  // tokens since the first token of the document that holds (b, t0); the next boundary on the flattened axis
  long long since = t0, next_b = 0x7fffffffffffffffLL;
  int idx = 0;
  const long long flat0 = (long long)b * p.S + t0;
  if (p.cu_seqlens) {
    int lo = 0, hi = p.num_docs;   // last offset <= flat0
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if ((long long)p.cu_seqlens[mid] <= flat0) lo = mid; else hi = mid - 1;
    }
    idx = lo;
    since = flat0 - (long long)p.cu_seqlens[idx];
    if (since > t0) since = t0;   // a row start is a start whatever the offsets say
    next_b = idx + 1 <= p.num_docs ? (long long)p.cu_seqlens[idx + 1] : next_b;
  }
  // one token; `reach`: tokens of its document in front of it (K and more: every tap is inside)
  auto token = [&](const Vec16<T>& cur, int t, long long reach) {
    Vec16<T> o;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      float acc = fmaf(wl[0][i], to_float(cur.v[i]), bias[i]);
#pragma unroll
      for (int l = 1; l < K; ++l)
        if (l <= reach) acc = fmaf(wl[l][i], to_float(win[l - 1].v[i]), acc);
      float y = to_float(from_float<T>(acc));            // the convolution's output is rounded to T ...
      if (p.act) y = y * sigmoid_for<T>(y);               // ... before the activation
      o.v[i] = from_float<T>(y);
    }
#pragma unroll
    for (int l = K - 1; l >= 2; --l) win[l - 1] = win[l - 2];
    if constexpr (K > 1) win[0] = cur;
    store16(out + (long long)t * p.o_st, o);
  };
  for (int tg = t0; tg < t1; tg += CONV_GROUP) {
    const long long flat = (long long)b * p.S + tg;
    Vec16<T> cur[CONV_GROUP];
#pragma unroll
    for (int j = 0; j < CONV_GROUP; ++j) cur[j] = load16(x + (long long)min(tg + j, t1 - 1) * p.x_st);
    if (tg + CONV_GROUP <= t1 && since >= K - 1 && flat + CONV_GROUP <= next_b) {   // inside one document, whole group
#pragma unroll
      for (int j = 0; j < CONV_GROUP; ++j) token(cur[j], tg + j, K);
      since += CONV_GROUP;
    } else {
#pragma unroll
      for (int j = 0; j < CONV_GROUP; ++j) {
        if (tg + j >= t1) break;
        while (flat + j >= next_b) {   // a document starts here (empty documents are stepped over)
          since = flat + j - next_b;
          ++idx;
          next_b = idx + 1 <= p.num_docs ? (long long)p.cu_seqlens[idx + 1] : 0x7fffffffffffffffLL;
        }
        token(cur[j], tg + j, since);
        ++since;
      }
    }
  }
}

}  // namespace xl

extern "C" int xl_add_rmsnorm(const xl_add_rmsnorm_params* p, void* cuda_stream) {
  using namespace xl;
  if (!p || !p->x || !p->weight || !p->normed) return XL_ERR_NULL_POINTER;
  if (p->y && !p->x_out) return XL_ERR_NULL_POINTER;
  if (p->dtype != XL_F32 && p->dtype != XL_BF16) return XL_ERR_BAD_DTYPE;
  const int V = p->dtype == XL_F32 ? 4 : 8;
  if (p->rows < 0 || p->D <= 0 || p->D % V != 0) return XL_ERR_BAD_SHAPE;
  if (p->D > RMS_THREADS * ADJ_MAXC * V) return XL_ERR_TOO_LARGE;
  if (p->rows > 0x7fffffffLL) return XL_ERR_TOO_LARGE;
  if (p->x_sr % V || p->n_sr % V || (p->y && (p->y_sr % V || p->xo_sr % V))) return XL_ERR_BAD_STRIDE;
  if (!aligned16(p->x) || !aligned16(p->weight) || !aligned16(p->normed) || (p->y && (!aligned16(p->y) || !aligned16(p->x_out))))
    return XL_ERR_BAD_ALIGNMENT;
  if (p->normed == p->x || (p->y && p->normed == p->x_out)) return XL_ERR_ALIASING;
  if (p->rows == 0) return XL_OK;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  const int nc = (p->D + RMS_THREADS * V - 1) / (RMS_THREADS * V);
  const dim3 grid((unsigned)p->rows);
#define XL_RMS_LAUNCH(T)                                                              \
  do {                                                                                \
    if (nc <= 1) (void)launch_dependent(add_rmsnorm_kernel<T, 1>, grid, dim3(RMS_THREADS), 0, st, *p);          \
    else if (nc <= 2) (void)launch_dependent(add_rmsnorm_kernel<T, 2>, grid, dim3(RMS_THREADS), 0, st, *p);     \
    else (void)launch_dependent(add_rmsnorm_kernel<T, 4>, grid, dim3(RMS_THREADS), 0, st, *p);                  \
  } while (0)
  if (p->dtype == XL_F32) XL_RMS_LAUNCH(float);
  else XL_RMS_LAUNCH(__nv_bfloat16);
#undef XL_RMS_LAUNCH
  return check_launch("xl_add_rmsnorm");
}

extern "C" int xl_headnorm_gate(const xl_headnorm_gate_params* p, void* cuda_stream) {
  using namespace xl;
  if (!p || !p->h || !p->weight || !p->out) return XL_ERR_NULL_POINTER;
  if (p->dtype != XL_F32 && p->dtype != XL_BF16) return XL_ERR_BAD_DTYPE;
  const int V = p->dtype == XL_F32 ? 4 : 8;
  if (p->B <= 0 || p->NH <= 0 || p->S <= 0 || p->DH <= 0 || p->DH % V != 0) return XL_ERR_BAD_SHAPE;
  if (p->DH > 32 * ADJ_MAXC * V) return XL_ERR_TOO_LARGE;
  if (p->h_sb % V || p->h_sh % V || p->h_st % V || (p->o && (p->o_sb % V || p->o_st % V))) return XL_ERR_BAD_STRIDE;
  if (!aligned16(p->h) || (p->o && !aligned16(p->o)) || !aligned16(p->weight) || !aligned16(p->out)) return XL_ERR_BAD_ALIGNMENT;
  if (p->out == p->h || p->out == p->o) return XL_ERR_ALIASING;
  const long long per_row = (long long)p->S * p->NH;
  if (per_row > 0x7fffffffLL || p->B > 65535) return XL_ERR_TOO_LARGE;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  const int nc = (p->DH + 32 * V - 1) / (32 * V);
  const bool many = per_row * p->B >= HNG_FULL;
#define XL_HNG_ROWS(T, NC, R)                                                                                                              \
  headnorm_gate_kernel<T, NC, (R)><<<dim3((unsigned)(((p->S + (R) - 1) / (R) * (long long)p->NH + HNG_WARPS - 1) / HNG_WARPS), (unsigned)p->B), \
                                     HNG_WARPS * 32, 0, st>>>(*p)
#define XL_HNG_LAUNCH(T, NC)                                      \
  do {                                                            \
    if (many) XL_HNG_ROWS(T, NC, HNG_IN_FLIGHT / NC);             \
    else XL_HNG_ROWS(T, NC, 1);                                   \
  } while (0)
#define XL_HNG_TYPE(T)                        \
  do {                                        \
    if (nc <= 1) XL_HNG_LAUNCH(T, 1);         \
    else if (nc <= 2) XL_HNG_LAUNCH(T, 2);    \
    else XL_HNG_ROWS(T, 4, 1);                \
  } while (0)
  if (p->dtype == XL_F32) XL_HNG_TYPE(float);
  else XL_HNG_TYPE(__nv_bfloat16);
#undef XL_HNG_TYPE
#undef XL_HNG_LAUNCH
#undef XL_HNG_ROWS
  return check_launch("xl_headnorm_gate");
}

extern "C" int xl_soft_cap(const xl_soft_cap_params* p, void* cuda_stream) {
  using namespace xl;
  if (!p || !p->x || !p->out) return XL_ERR_NULL_POINTER;
  if (p->dtype != XL_F32 && p->dtype != XL_BF16) return XL_ERR_BAD_DTYPE;
  if (p->n < 0 || !(p->cap > 0.f) || p->out_f32 < 0 || p->out_f32 > 2) return XL_ERR_BAD_SHAPE;
  if (p->cols < 0 || (p->cols > 0 && (p->n % p->cols != 0 || p->x_row_stride < p->cols))) return XL_ERR_BAD_SHAPE;
  if (p->bias && p->cols <= 0) return XL_ERR_BAD_SHAPE;
  if (p->n == 0) return XL_OK;
  if (p->out == p->x && ((p->dtype == XL_BF16 && p->out_f32) || (p->cols > 0 && p->x_row_stride != p->cols))) return XL_ERR_ALIASING;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  const long long want = (p->n + 255) / 256;
  const unsigned grid = (unsigned)(want < 148 * 16 ? want : 148 * 16);
  const long long cols = p->cols, rs = p->x_row_stride;
  if (p->dtype == XL_F32)
    (void)launch_dependent(soft_cap_kernel<float, float, false>, dim3(grid), dim3(256), 0, st, static_cast<const float*>(p->x), static_cast<float*>(p->out), p->n, p->cap, cols, rs, static_cast<const float*>(p->bias));
  else if (p->out_f32 == 2)
    (void)launch_dependent(soft_cap_kernel<__nv_bfloat16, float, false>, dim3(grid), dim3(256), 0, st, static_cast<const __nv_bfloat16*>(p->x), static_cast<float*>(p->out), p->n, p->cap, cols, rs, static_cast<const __nv_bfloat16*>(p->bias));
  else if (p->out_f32)
    (void)launch_dependent(soft_cap_kernel<__nv_bfloat16, float, true>, dim3(grid), dim3(256), 0, st, static_cast<const __nv_bfloat16*>(p->x), static_cast<float*>(p->out), p->n, p->cap, cols, rs, static_cast<const __nv_bfloat16*>(p->bias));
  else
    (void)launch_dependent(soft_cap_kernel<__nv_bfloat16, __nv_bfloat16, true>, dim3(grid), dim3(256), 0, st, static_cast<const __nv_bfloat16*>(p->x), static_cast<__nv_bfloat16*>(p->out), p->n, p->cap, cols, rs, static_cast<const __nv_bfloat16*>(p->bias));
  return check_launch("xl_soft_cap");
}

extern "C" int xl_swiglu(const xl_swiglu_params* p, void* cuda_stream) {
  using namespace xl;
  if (!p || !p->gz || !p->out) return XL_ERR_NULL_POINTER;
  if (p->dtype != XL_F32 && p->dtype != XL_BF16) return XL_ERR_BAD_DTYPE;
  const int V = p->dtype == XL_F32 ? 4 : 8;
  if (p->rows < 0 || p->F <= 0 || p->F % V != 0 || p->gz_row_stride < 2LL * p->F || p->gz_row_stride % V != 0) return XL_ERR_BAD_SHAPE;
  if (!aligned16(p->gz) || !aligned16(p->out)) return XL_ERR_BAD_ALIGNMENT;
  if (p->out == p->gz) return XL_ERR_ALIASING;
  if (p->rows == 0) return XL_OK;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  const long long want = (p->rows * (long long)(p->F / V) + 255) / 256;
  const unsigned grid = (unsigned)(want < 148 * 16 ? want : 148 * 16);
  if (p->dtype == XL_F32) (void)launch_dependent(swiglu_kernel<float>, dim3(grid), dim3(256), 0, st, static_cast<const float*>(p->gz), static_cast<float*>(p->out), p->rows, p->F, p->gz_row_stride);
  else (void)launch_dependent(swiglu_kernel<__nv_bfloat16>, dim3(grid), dim3(256), 0, st, static_cast<const __nv_bfloat16*>(p->gz), static_cast<__nv_bfloat16*>(p->out), p->rows, p->F, p->gz_row_stride);
  return check_launch("xl_swiglu");
}

extern "C" int xl_causal_conv1d(const xl_conv1d_params* p, void* cuda_stream) {
  using namespace xl;
  if (!p || !p->x || !p->weight || !p->out) return XL_ERR_NULL_POINTER;
  if (p->dtype != XL_F32 && p->dtype != XL_BF16) return XL_ERR_BAD_DTYPE;
  const int V = p->dtype == XL_F32 ? 4 : 8;
  if (p->B <= 0 || p->S <= 0 || p->F <= 0 || p->F % V != 0 || p->K < 1) return XL_ERR_BAD_SHAPE;
  if (p->K > CONV_MAXK || p->B > 65535) return XL_ERR_TOO_LARGE;
  if (p->cu_seqlens && p->num_docs <= 0) return XL_ERR_BAD_SHAPE;
  if (p->x_sb % V || p->x_st % V || p->o_sb % V || p->o_st % V || p->x_st < p->F || p->o_st < p->F) return XL_ERR_BAD_STRIDE;
  if (!aligned16(p->x) || !aligned16(p->out)) return XL_ERR_BAD_ALIGNMENT;
  if (p->out == p->x) return XL_ERR_ALIASING;   // a tile's halo is read by the neighbouring thread block
  if (p->S > 65535 * 64) return XL_ERR_TOO_LARGE;
  const int64_t blocks = (int64_t)((p->S + CONV_TILE - 1) / CONV_TILE) * ((p->F / V + CONV_THREADS - 1) / CONV_THREADS);
  if (blocks > 0x7fffffff) return XL_ERR_TOO_LARGE;
  const dim3 grid((unsigned)blocks, (unsigned)p->B);
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
#define XL_CONV_LAUNCH(KK)                                                                             \
  case KK:                                                                                             \
    if (p->dtype == XL_F32) causal_conv1d_kernel<float, KK><<<grid, CONV_THREADS, 0, st>>>(*p);        \
    else causal_conv1d_kernel<__nv_bfloat16, KK><<<grid, CONV_THREADS, 0, st>>>(*p);                   \
    break
  switch (p->K) {
    XL_CONV_LAUNCH(1); XL_CONV_LAUNCH(2); XL_CONV_LAUNCH(3); XL_CONV_LAUNCH(4);
    XL_CONV_LAUNCH(5); XL_CONV_LAUNCH(6); XL_CONV_LAUNCH(7); XL_CONV_LAUNCH(8);
  }
#undef XL_CONV_LAUNCH
  return check_launch("xl_causal_conv1d");
}
