// Native host path of the tensor-level entry points (xlstm_b200/ops.py): unpacks the tensors, checks them, allocates the
// outputs through PyTorch's caching allocator, fills the parameter block of include/xlstm_b200.h and calls the C entry on
// the current stream.
//
// What bounds a small call is the host: the kernels of a decode step or of a short prompt take 3 - 10 us, while the same
// work in Python (ctypes field by field, a device guard and a stream object per call) took 16 - 25 us.  Therefore plain
// METH_FASTCALL functions with positional arguments and no argument parser in between, and the allocator called directly.
// The interpreter lock is given up between the unpacking of the arguments and the wrapping of the results: an allocation or a
// launch on a full queue may block.
// No arithmetic happens here and there is no fallback: what the kernels do not cover raises.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <mutex>

#include "../../include/xlstm_b200.h"

namespace {

using at::Tensor;

constexpr int MAX_DEVICES = 64;

// Gives up the interpreter lock until lock() or the end of the scope (an exception on its way out, too).
class Unlocked {
 public:
  Unlocked() : state_(PyEval_SaveThread()) {}
  Unlocked(const Unlocked&) = delete;
  Unlocked& operator=(const Unlocked&) = delete;
  ~Unlocked() { lock(); }
  void lock() {
    if (state_) PyEval_RestoreThread(state_);
    state_ = nullptr;
  }

 private:
  PyThreadState* state_;
};

// ---------------------------------------------------------------------------------------------- arguments
const Tensor& tensor_arg(PyObject* o, const char* name) {
  TORCH_CHECK_VALUE(THPVariable_Check(o), name, " must be a tensor");
  return THPVariable_Unpack(o);
}
const Tensor* optional_arg(PyObject* o, const char* name) { return o == Py_None ? nullptr : &tensor_arg(o, name); }

double double_arg(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
int64_t int_arg(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
void want_args(Py_ssize_t have, Py_ssize_t want) {
  TORCH_CHECK_TYPE(have == want, "expected ", want, " arguments, got ", have);
}
void require_cuda(const Tensor& t) {
  TORCH_CHECK_VALUE(t.is_cuda(), "xlstm_b200 kernels need CUDA tensors (there is no CPU path)");
}
void require_cuda(const Tensor* t) {
  if (t) require_cuda(*t);
}

bool known_dtype(const Tensor& t) { return t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16; }
int32_t dtype_code(const Tensor& t) { return t.scalar_type() == at::kFloat ? XL_F32 : XL_BF16; }

// ---------------------------------------------------------------------------------------------- tensors
// The conversions below return the tensor itself in the usual case, so a call on ready inputs copies nothing.
Tensor last_contig(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }
Tensor as_float(const Tensor& t) { return t.scalar_type() == at::kFloat ? t : t.to(at::kFloat); }
Tensor float_contig(const Tensor& t) { return as_float(t).contiguous(); }

// `t` without the dimensions of size 1 between its first `lead` and its last
Tensor drop_units(const Tensor& t, int64_t lead) {
  Tensor r = t;
  while (r.dim() > lead + 1 && r.size(lead) == 1) r = r.squeeze(lead);
  return r;
}

Tensor empty_on(at::IntArrayRef sizes, at::ScalarType dtype, const Tensor& like) {
  return Tensor(at::detail::empty_cuda(sizes, dtype, like.device(), std::nullopt));
}

// The status word of a device: one int32 that kernels set when a bounded wait expires.  Lives until the process exits.
// Called without the interpreter lock (the allocation under the mutex may need it).
Tensor& status_tensor(int64_t index) {
  static std::mutex mutex;
  static std::atomic<Tensor*> words[MAX_DEVICES];
  TORCH_CHECK_VALUE(index >= 0 && index < MAX_DEVICES, "device index out of range");
  Tensor* word = words[index].load(std::memory_order_acquire);
  if (!word) {
    const std::lock_guard<std::mutex> hold(mutex);
    word = words[index].load(std::memory_order_relaxed);
    if (!word) {
      word = new Tensor(at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, (int8_t)index)));
      words[index].store(word, std::memory_order_release);
    }
  }
  return *word;
}
int32_t* status_ptr(const Tensor& like) { return static_cast<int32_t*>(status_tensor(like.device().index()).data_ptr()); }

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

PyObject* check_fn = nullptr;   // xlstm_b200._lib.check, which raises the package's error for a status code
void check(int rc, const char* where) {
  if (rc == XL_OK) return;
  if (!check_fn) {
    PyObject* mod = PyImport_ImportModule("xlstm_b200._lib");
    if (mod) check_fn = PyObject_GetAttrString(mod, "check");
    Py_XDECREF(mod);
    if (!check_fn) throw python_error();
  }
  PyObject* r = PyObject_CallFunction(check_fn, "is", rc, where);
  Py_XDECREF(r);
  throw python_error();
}

PyObject* pack(std::initializer_list<Tensor> ts) {
  PyObject* out = PyTuple_New((Py_ssize_t)ts.size());
  if (!out) throw python_error();
  Py_ssize_t k = 0;
  for (const Tensor& t : ts) PyTuple_SET_ITEM(out, k++, THPVariable_Wrap(t));
  return out;
}
PyObject* pack_pair(PyObject* a, PyObject* b) {
  PyObject* out = PyTuple_New(2);
  if (!out) throw python_error();
  PyTuple_SET_ITEM(out, 0, a);
  PyTuple_SET_ITEM(out, 1, b);
  return out;
}

// ---------------------------------------------------------------------------------------------- mLSTM over a sequence
// (q, k, v, i, f, c0, n0, m0, cu_seqlens on the device or None, documents, eps, kernel) -> (h, (c, n, m));
// kernel: 0 = chosen by shape and dtype, 1 = chunkwise, 2 = recurrent, 3 = chunkwise with documents whole
PyObject* mlstm_sequence(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 12);
  const Tensor &q0 = tensor_arg(a[0], "q"), &k0 = tensor_arg(a[1], "k"), &v_arg = tensor_arg(a[2], "v");
  const Tensor &i0 = tensor_arg(a[3], "i"), &f0 = tensor_arg(a[4], "f");
  const Tensor *c_in = optional_arg(a[5], "c_initial"), *n_in = optional_arg(a[6], "n_initial"), *m_in = optional_arg(a[7], "m_initial");
  const Tensor* cu = optional_arg(a[8], "cu_seqlens");
  const int64_t docs = int_arg(a[9]), choice = int_arg(a[11]);
  const double eps = double_arg(a[10]);
  Unlocked unlocked;
  for (const Tensor* t : {&q0, &k0, &v_arg, &i0, &f0, c_in, n_in, m_in, cu}) require_cuda(t);
  const Tensor v0 = drop_units(v_arg, 3);   // (B,NH,S,1,DHV) is taken, too
  TORCH_CHECK_VALUE(known_dtype(q0) && k0.scalar_type() == q0.scalar_type() && v0.scalar_type() == q0.scalar_type(),
                    "q,k,v must share a dtype (float32 or bfloat16), got ", q0.scalar_type(), ",", k0.scalar_type(), ",", v0.scalar_type());
  TORCH_CHECK_VALUE(q0.dim() == 4 && v0.dim() == 4, "q, k, v must be (B,NH,S,D)");
  const int64_t B = q0.size(0), NH = q0.size(1), S = q0.size(2), DQ = q0.size(3), DV = v0.size(3);
  TORCH_CHECK_VALUE(k0.sizes() == q0.sizes() && v0.sizes().slice(0, 3) == q0.sizes().slice(0, 3) && i0.sizes() == q0.sizes().slice(0, 3) &&
                        f0.sizes() == q0.sizes().slice(0, 3),
                    "inconsistent shapes for q,k,v,i,f");
  const c10::cuda::CUDAGuard guard(q0.device());
  const Tensor q = last_contig(q0), k = last_contig(k0), v = last_contig(v0);
  Tensor i = as_float(i0), f = as_float(f0);
  if (i.strides() != f.strides()) { i = i.contiguous(); f = f.contiguous(); }
  int64_t kernel = choice;
  if (kernel == 0) {
    bool chunk = q.scalar_type() == at::kBFloat16 && (DQ == 64 || DQ == 128 || DQ == 256) && DV % 128 == 0;
    for (const Tensor* t : {&q, &k, &v})
      chunk = chunk && t->stride(0) % 8 == 0 && t->stride(1) % 8 == 0 && t->stride(2) % 8 == 0 && reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 == 0;
    kernel = chunk ? 1 : 2;
  }
  const int64_t nd = cu ? docs : B;
  Tensor c0, n0, m0;
  if (c_in) {
    TORCH_CHECK_VALUE(n_in && m_in, "c_initial, n_initial and m_initial must be given together");
    c0 = float_contig(*c_in); n0 = float_contig(*n_in); m0 = float_contig(*m_in);
    TORCH_CHECK_VALUE(c0.sizes() == at::IntArrayRef({nd, NH, DQ, DV}) && n0.sizes() == at::IntArrayRef({nd, NH, DQ}) && m0.numel() == nd * NH,
                      "initial state shapes must be (N,NH,DHQK,DHV), (N,NH,DHQK), (N,NH[,1])");
  }
  const Tensor h = empty_on({B, NH, S, DV}, q.scalar_type(), q), c = empty_on({nd, NH, DQ, DV}, at::kFloat, q);
  const Tensor n = empty_on({nd, NH, DQ}, at::kFloat, q), m = empty_on({nd, NH, 1}, at::kFloat, q);
  xl_mlstm_seq_params p = {};
  p.q = q.data_ptr(); p.k = k.data_ptr(); p.v = v.data_ptr(); p.h = h.data_ptr();
  p.igate = i.const_data_ptr<float>(); p.fgate = f.const_data_ptr<float>();
  if (c_in) { p.c0 = c0.const_data_ptr<float>(); p.n0 = n0.const_data_ptr<float>(); p.m0 = m0.const_data_ptr<float>(); }
  p.c_out = c.data_ptr<float>(); p.n_out = n.data_ptr<float>(); p.m_out = m.data_ptr<float>();
  p.cu_seqlens = cu ? cu->const_data_ptr<int32_t>() : nullptr;
  p.status = status_ptr(q);
  p.B = B; p.NH = NH; p.S = S; p.DHQK = DQ; p.DHV = DV; p.num_docs = nd;
  p.q_sb = q.stride(0); p.q_sh = q.stride(1); p.q_st = q.stride(2);
  p.k_sb = k.stride(0); p.k_sh = k.stride(1); p.k_st = k.stride(2);
  p.v_sb = v.stride(0); p.v_sh = v.stride(1); p.v_st = v.stride(2);
  p.h_sb = h.stride(0); p.h_sh = h.stride(1); p.h_st = h.stride(2);
  p.g_sb = i.stride(0); p.g_sh = i.stride(1); p.g_st = i.stride(2);
  p.eps = (float)eps; p.dtype = dtype_code(q);
  int rc;
  if (kernel != 2) {
    // (stream-ordered: free for the allocator at return.  Where there is no room for it the documents stay whole, as for callers
    // of the C entry without scratch.)
    int64_t bytes = kernel == 3 ? 0 : xl_mlstm_chunkwise_scratch_bytes(&p);
    Tensor scratch;
    if (bytes) {
      try {
        scratch = empty_on({bytes}, at::kByte, q);
      } catch (const c10::OutOfMemoryError&) {
        bytes = 0;
      }
    }
    rc = xl_mlstm_chunkwise_parts(&p, bytes ? scratch.data_ptr() : nullptr, bytes, stream_of(q));
  } else {
    rc = xl_mlstm_recurrent(&p, stream_of(q));
  }
  unlocked.lock();
  check(rc, kernel != 2 ? "xl_mlstm_chunkwise" : "xl_mlstm_recurrent");
  return pack_pair(THPVariable_Wrap(h), pack({c, n, m}));
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------- mLSTM decode step
// What the plain step and the fused decode cell share: inputs, state pool, slots.  The members keep converted tensors
// alive until the launch.
struct StepArgs {
  Tensor q, k, v, m_in, slot, c, n, m;
  int64_t B, NH, DQ, DV;

  void fill(xl_mlstm_step_params& p, const Tensor& q0, const Tensor& k_arg, const Tensor& v_arg, const Tensor* c0, const Tensor* n0, const Tensor* m0,
            const Tensor* slot0, double eps, bool inplace) {
    const Tensor k0 = drop_units(k_arg, 2), v0 = drop_units(v_arg, 2);   // (B,NH,1,D) is taken, too
    TORCH_CHECK_VALUE(q0.dim() == 3 && v0.dim() == 3 && k0.sizes() == q0.sizes() && v0.size(0) == q0.size(0) && v0.size(1) == q0.size(1),
                      "step inputs: q, k (B,NH,DHQK) and v (B,NH,DHV)");
    TORCH_CHECK_VALUE(known_dtype(q0) && k0.scalar_type() == q0.scalar_type() && v0.scalar_type() == q0.scalar_type(),
                      "q,k,v must share a dtype (float32 or bfloat16)");
    B = q0.size(0); NH = q0.size(1); DQ = q0.size(2); DV = v0.size(2);
    q = last_contig(q0); k = last_contig(k0); v = last_contig(v0);
    int64_t N = B;
    if (slot0) {
      TORCH_CHECK_VALUE(c0, "`slot` addresses rows of a state pool: pass c, n, m");
      TORCH_CHECK_VALUE(slot0->dim() == 1 && slot0->numel() == B && (slot0->scalar_type() == at::kInt || slot0->scalar_type() == at::kLong),
                        "slot must be a (", B, ",) int32 (or int64) vector");
      TORCH_CHECK_VALUE(slot0->device() == q.device(), "slot lives on another device than the inputs");
      slot = slot0->to(at::kInt).contiguous();
    }
    if (c0) {
      TORCH_CHECK_VALUE(n0 && m0, "c, n and m must be given together");
      TORCH_CHECK_VALUE(c0->scalar_type() == at::kFloat && c0->is_contiguous() && n0->is_contiguous(), "state pool must be contiguous fp32");
      N = c0->size(0);
      m_in = m0->reshape({N, NH, 1}).contiguous();
      TORCH_CHECK_VALUE(slot0 || N == B, "without `slot` the state pool must have one row per stream");
      c = inplace ? *c0 : (slot0 ? c0->clone() : empty_on({N, NH, DQ, DV}, at::kFloat, q));   // (rows no slot names keep their contents)
      p.c_in = c0->const_data_ptr<float>(); p.n_in = n0->const_data_ptr<float>(); p.m_in = m_in.const_data_ptr<float>();
    } else {
      c = empty_on({N, NH, DQ, DV}, at::kFloat, q);
    }
    n = c0 && slot0 ? n0->clone() : empty_on({N, NH, DQ}, at::kFloat, q);
    m = c0 && slot0 ? m_in.clone() : empty_on({N, NH, 1}, at::kFloat, q);
    p.q = q.data_ptr(); p.k = k.data_ptr(); p.v = v.data_ptr();
    p.c_out = c.data_ptr<float>(); p.n_out = n.data_ptr<float>(); p.m_out = m.data_ptr<float>();
    p.slot = slot0 ? slot.const_data_ptr<int32_t>() : nullptr;
    p.status = status_ptr(q);
    p.B = B; p.NH = NH; p.DHQK = DQ; p.DHV = DV; p.n_slots = N;
    p.q_sb = q.stride(0); p.q_sh = q.stride(1);
    p.k_sb = k.stride(0); p.k_sh = k.stride(1);
    p.v_sb = v.stride(0); p.v_sh = v.stride(1);
    p.eps = (float)eps; p.dtype = dtype_code(q);
  }
  // the in-place C goes back as the very object the caller passed
  PyObject* result(PyObject* out, PyObject* c_obj, bool inplace) const {
    PyObject* st = PyTuple_New(3);
    if (!st) throw python_error();
    PyTuple_SET_ITEM(st, 0, c_obj != Py_None && inplace ? Py_NewRef(c_obj) : THPVariable_Wrap(c));
    PyTuple_SET_ITEM(st, 1, THPVariable_Wrap(n));
    PyTuple_SET_ITEM(st, 2, THPVariable_Wrap(m));
    return pack_pair(out, st);
  }
};

// (q, k, v, i, f, c, n, m, slot on the device or None, eps, inplace) -> (h, (c, n, m))
PyObject* mlstm_step(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 11);
  const Tensor &q = tensor_arg(a[0], "q"), &k = tensor_arg(a[1], "k"), &v = tensor_arg(a[2], "v");
  const Tensor &i0 = tensor_arg(a[3], "i"), &f0 = tensor_arg(a[4], "f");
  const Tensor *c = optional_arg(a[5], "c"), *n = optional_arg(a[6], "n"), *m = optional_arg(a[7], "m"), *slot = optional_arg(a[8], "slot");
  const double eps = double_arg(a[9]);
  const bool inplace = a[10] == Py_True;
  Unlocked unlocked;
  for (const Tensor* t : {&q, &k, &v, &i0, &f0, c, n, m}) require_cuda(t);
  const c10::cuda::CUDAGuard guard(q.device());
  StepArgs s;
  xl_mlstm_step_params p = {};
  s.fill(p, q, k, v, c, n, m, slot, eps, inplace);
  auto gate = [&](const Tensor& t) {   // (B,NH) or (B,NH,1), or whatever reshapes to (B,NH)
    const Tensor g = as_float(t);
    const bool direct = (g.dim() == 2 || (g.dim() == 3 && g.size(2) == 1)) && g.size(0) == s.B && g.size(1) == s.NH;
    return direct ? g : g.reshape({s.B, s.NH});
  };
  Tensor i = gate(i0), f = gate(f0);
  if (i.stride(0) != f.stride(0) || i.stride(1) != f.stride(1)) { i = i.contiguous(); f = f.contiguous(); }
  const Tensor h = empty_on({s.B, s.NH, s.DV}, q.scalar_type(), q);
  p.h = h.data_ptr();
  p.igate = i.const_data_ptr<float>(); p.fgate = f.const_data_ptr<float>();
  p.h_sb = h.stride(0); p.h_sh = h.stride(1);
  p.g_sb = i.stride(0); p.g_sh = i.stride(1);
  const int rc = xl_mlstm_step(&p, stream_of(q));
  unlocked.lock();
  check(rc, "xl_mlstm_step");
  return s.result(THPVariable_Wrap(h), a[5], inplace);
  END_HANDLE_TH_ERRORS
}

// (q, k, v, gates_raw, gate_bias or None, gate_cap, ogate, norm_weight, c, n, m, slot or None, eps, norm_eps) -> (hg, (c, n, m))
PyObject* mlstm_decode_cell(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 14);
  const Tensor &q = tensor_arg(a[0], "q"), &k = tensor_arg(a[1], "k"), &v = tensor_arg(a[2], "v"), &gates0 = tensor_arg(a[3], "gates_raw");
  const Tensor* bias0 = optional_arg(a[4], "gate_bias");
  const Tensor &o0 = tensor_arg(a[6], "ogate"), &w0 = tensor_arg(a[7], "norm_weight");
  const Tensor *c = optional_arg(a[8], "c"), *n = optional_arg(a[9], "n"), *m = optional_arg(a[10], "m"), *slot = optional_arg(a[11], "slot");
  const double cap = double_arg(a[5]), eps = double_arg(a[12]), norm_eps = double_arg(a[13]);
  Unlocked unlocked;
  for (const Tensor* t : {&q, &k, &v, &gates0, bias0, &o0, &w0, c, n, m}) require_cuda(t);
  const c10::cuda::CUDAGuard guard(q.device());
  TORCH_CHECK_VALUE(v.size(-1) <= 1024, "mlstm_decode_cell: head value width above 1024");
  StepArgs s;
  xl_mlstm_decode_cell_params p = {};
  s.fill(p.step, q, k, v, c, n, m, slot, eps, true);
  const int64_t H = s.NH * s.DV;
  // (B, width) rows with a contiguous last dimension: column slices of a wider projection output as they are
  auto rows = [&](const Tensor& t, int64_t width) {
    const Tensor r = last_contig(t);
    return r.dim() == 2 && r.size(0) == s.B && r.size(1) == width ? r : r.reshape({s.B, width});
  };
  const Tensor gates = rows(gates0, 2 * s.NH), o = rows(o0, H), w = w0.contiguous(), bias = bias0 ? bias0->contiguous() : Tensor();
  const auto dt = q.scalar_type();
  TORCH_CHECK_VALUE(gates.scalar_type() == dt && o.scalar_type() == dt && w.scalar_type() == dt && (!bias0 || bias.scalar_type() == dt),
                    "mlstm_decode_cell: gates, output gate, bias and norm weight in the dtype of q");
  TORCH_CHECK_VALUE(w.numel() == H && (!bias0 || bias.numel() == 2 * s.NH), "mlstm_decode_cell: norm weight (NH*DHV), gate bias (2*NH)");
  const Tensor hg = empty_on({s.B, H}, dt, q);
  p.gates_raw = gates.data_ptr(); p.gate_bias = bias0 ? bias.data_ptr() : nullptr;
  p.ogate = o.data_ptr(); p.norm_weight = w.data_ptr(); p.hg = hg.data_ptr();
  p.gr_sb = gates.stride(0); p.o_sb = o.stride(0); p.hg_sb = hg.stride(0);
  p.gate_cap = (float)cap; p.norm_eps = (float)norm_eps;
  const int rc = xl_mlstm_decode_cell(&p, stream_of(q));
  unlocked.lock();
  check(rc, "xl_mlstm_decode_cell");
  return s.result(THPVariable_Wrap(hg), a[8], true);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------- sLSTM
// (wx, R, bias, state0 or None, cu_seqlens on the device or None, documents, train_cache) -> (h, state[, cache])
PyObject* slstm_forward(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 7);
  const Tensor &wx0 = tensor_arg(a[0], "wx"), &R0 = tensor_arg(a[1], "R"), &bias0 = tensor_arg(a[2], "bias");
  const Tensor *st0 = optional_arg(a[3], "state0"), *cu = optional_arg(a[4], "cu_seqlens");
  const int64_t docs = int_arg(a[5]);
  const bool train = a[6] == Py_True;
  Unlocked unlocked;
  for (const Tensor* t : {&wx0, &R0, &bias0, st0, cu}) require_cuda(t);
  TORCH_CHECK_VALUE(wx0.scalar_type() == at::kBFloat16, "the sLSTM kernel computes on bf16 inputs (fp32 state); cast wx and R to bfloat16");
  TORCH_CHECK_VALUE(wx0.dim() == 3 && R0.dim() == 4, "inconsistent sLSTM shapes");
  const int64_t B = wx0.size(0), S = wx0.size(1), NH = R0.size(0), DH = R0.size(1), H = NH * DH;
  TORCH_CHECK_VALUE(wx0.size(2) == 4 * H && R0.sizes() == at::IntArrayRef({NH, DH, 4, DH}) && bias0.numel() == NH * 4 * DH, "inconsistent sLSTM shapes");
  const c10::cuda::CUDAGuard guard(wx0.device());
  const Tensor wx = wx0.contiguous(), R = R0.to(at::kBFloat16).contiguous(), bias = float_contig(bias0);
  const Tensor out = empty_on({B, NH, S, DH}, at::kBFloat16, wx), st = empty_on({4, B, H}, at::kFloat, wx);
  Tensor s0, cache;
  xl_slstm_params p = {};
  p.wx = wx.data_ptr(); p.R = R.data_ptr(); p.bias = bias.const_data_ptr<float>();
  if (st0) {
    s0 = float_contig(*st0);
    TORCH_CHECK_VALUE(s0.sizes() == at::IntArrayRef({4, B, H}), "state0 must be (4,B,H)");
    p.state0 = s0.const_data_ptr<float>();
  }
  p.h_out = out.data_ptr(); p.state_out = st.data_ptr<float>();
  p.cu_seqlens = cu ? cu->const_data_ptr<int32_t>() : nullptr;
  p.status = status_ptr(wx);
  p.B = B; p.S = S; p.NH = NH; p.DH = DH; p.num_docs = cu ? docs : 0; p.dtype = XL_BF16;
  if (train) {
    const int64_t bytes = xl_slstm_cache_bytes(B, S, NH, DH);
    TORCH_CHECK_VALUE(bytes > 0, "the sLSTM training path needs a head size of 64, 128 or 256");
    cache = empty_on({bytes}, at::kByte, wx);
    p.train_cache = cache.data_ptr();
  }
  const int rc = xl_slstm_forward(&p, stream_of(wx));
  unlocked.lock();
  check(rc, "xl_slstm_forward");
  return train ? pack({out, st, cache}) : pack({out, st});
  END_HANDLE_TH_ERRORS
}

// (cache, R, dh, dstate_out or None, state0 or None) -> (dwx, dstate0)
PyObject* slstm_backward(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 5);
  const Tensor &cache = tensor_arg(a[0], "cache"), &R0 = tensor_arg(a[1], "R"), &dh0 = tensor_arg(a[2], "dh");
  const Tensor *ds = optional_arg(a[3], "dstate_out"), *st0 = optional_arg(a[4], "state0");
  Unlocked unlocked;
  for (const Tensor* t : {&cache, &R0, &dh0, ds, st0}) require_cuda(t);
  TORCH_CHECK_VALUE(dh0.dim() == 4, "dh must be (B,NH,S,DH)");
  const int64_t B = dh0.size(0), NH = dh0.size(1), S = dh0.size(2), DH = dh0.size(3), H = NH * DH;
  TORCH_CHECK_VALUE(R0.sizes() == at::IntArrayRef({NH, DH, 4, DH}), "inconsistent sLSTM shapes");
  TORCH_CHECK_VALUE(cache.scalar_type() == at::kByte && cache.numel() == xl_slstm_cache_bytes(B, S, NH, DH),
                    "cache does not belong to a forward call of these sizes");
  const c10::cuda::CUDAGuard guard(dh0.device());
  const Tensor R = R0.to(at::kBFloat16).contiguous(), dh = dh0.to(at::kBFloat16).contiguous();
  const Tensor dwx = empty_on({B, S, 4 * H}, at::kBFloat16, dh), ds0 = empty_on({4, B, H}, at::kFloat, dh);
  xl_slstm_bwd_params p = {};
  p.cache = cache.data_ptr(); p.R = R.data_ptr(); p.dh = dh.data_ptr(); p.dwx = dwx.data_ptr(); p.dstate0 = ds0.data_ptr<float>();
  Tensor dso, s0;
  if (ds) {
    dso = float_contig(*ds);
    TORCH_CHECK_VALUE(dso.sizes() == at::IntArrayRef({4, B, H}), "dstate_out must be (4,B,H)");
    p.dstate_out = dso.const_data_ptr<float>();
  }
  if (st0) {
    s0 = float_contig(*st0);
    TORCH_CHECK_VALUE(s0.sizes() == at::IntArrayRef({4, B, H}), "state0 must be (4,B,H)");
    p.state0 = s0.const_data_ptr<float>();
  }
  p.status = status_ptr(dh);
  p.B = B; p.S = S; p.NH = NH; p.DH = DH; p.dtype = XL_BF16;
  const int rc = xl_slstm_backward(&p, stream_of(dh));
  unlocked.lock();
  check(rc, "xl_slstm_backward");
  return pack({dwx, ds0});
  END_HANDLE_TH_ERRORS
}

// (dwx (B,S,4,NH,DH), h (B,NH,S,DH), h0 (B,NH,DH) or None) -> (dR, dbias); all bf16 and as the kernel takes them (see ops.py)
PyObject* slstm_weight_grads(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 3);
  const Tensor &dwx = tensor_arg(a[0], "dwx"), &h = tensor_arg(a[1], "h");
  const Tensor* h0 = optional_arg(a[2], "h0");
  Unlocked unlocked;
  for (const Tensor* t : {&dwx, &h, h0}) {
    require_cuda(t);
    TORCH_CHECK_VALUE(!t || (t->scalar_type() == at::kBFloat16 && t->is_contiguous() && t->device() == dwx.device()),
                      "slstm_weight_grads: contiguous bf16 tensors on one device");
  }
  TORCH_CHECK_VALUE(h.dim() == 4, "h must be (B,NH,S,DH)");
  const int64_t B = h.size(0), NH = h.size(1), S = h.size(2), DH = h.size(3);
  TORCH_CHECK_VALUE(dwx.sizes() == at::IntArrayRef({B, S, 4, NH, DH}) && (!h0 || h0->sizes() == at::IntArrayRef({B, NH, DH})), "inconsistent sLSTM shapes");
  const c10::cuda::CUDAGuard guard(h.device());
  const Tensor dR = empty_on({NH, DH, 4, DH}, at::kFloat, h), db = empty_on({NH, 4, DH}, at::kFloat, h);
  const int64_t bytes = xl_slstm_weight_grads_scratch_bytes(B, S, NH, DH);
  const Tensor scratch = bytes ? empty_on({bytes}, at::kByte, h) : Tensor();   // (stream-ordered: free for the allocator at return)
  xl_slstm_wgrad_params p = {};
  p.dwx = dwx.data_ptr(); p.h = h.data_ptr(); p.h0 = h0 ? h0->data_ptr() : nullptr;
  p.dR = dR.data_ptr<float>(); p.dbias = db.data_ptr<float>();
  p.scratch = bytes ? scratch.data_ptr() : nullptr; p.scratch_bytes = bytes;
  p.status = status_ptr(h);
  p.B = B; p.S = S; p.NH = NH; p.DH = DH; p.dtype = XL_BF16;
  const int rc = xl_slstm_weight_grads(&p, stream_of(h));
  unlocked.lock();
  check(rc, "xl_slstm_weight_grads");
  return pack({dR, db});
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------- operators next to the cells
// (rows, D) view of (..., D) with contiguous rows
Tensor as_rows(const Tensor& t, int64_t D) {
  const Tensor r = t.dim() == 2 ? t : t.reshape({-1, D});
  return r.stride(-1) == 1 ? r : r.contiguous();
}

// (x, weight, y or None, eps, inplace) -> (x_new, normed)
PyObject* add_rmsnorm(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 5);
  const Tensor &x = tensor_arg(a[0], "x"), &w0 = tensor_arg(a[1], "weight");
  const Tensor* y = optional_arg(a[2], "y");
  const double eps = double_arg(a[3]);
  const bool inplace = a[4] == Py_True;
  Unlocked unlocked;
  for (const Tensor* t : {&x, &w0, y}) require_cuda(t);
  TORCH_CHECK_VALUE(known_dtype(x) && w0.scalar_type() == x.scalar_type() && (!y || (y->scalar_type() == x.scalar_type() && y->sizes() == x.sizes())),
                    "add_rmsnorm: x, y and weight must share one dtype (float32 or bfloat16) and x, y one shape");
  const int64_t D = x.size(-1);
  TORCH_CHECK_VALUE(w0.dim() == 1 && w0.size(0) == D, "add_rmsnorm: weight must have shape (D,)");
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor x2 = as_rows(x, D), w = w0.contiguous(), y2 = y ? as_rows(*y, D) : Tensor();
  const int64_t rows = x2.size(0);
  const bool over_x = y && inplace && x2.data_ptr() == x.data_ptr();
  const Tensor xo = !y || over_x ? x2 : empty_on(x.sizes(), x.scalar_type(), x);
  const Tensor normed = empty_on(x.sizes(), x.scalar_type(), x);
  xl_add_rmsnorm_params p = {};
  p.x = x2.data_ptr(); p.weight = w.data_ptr(); p.normed = normed.data_ptr();
  p.rows = rows; p.D = (int32_t)D; p.x_sr = x2.stride(0); p.n_sr = D;
  if (y) {
    p.y = y2.data_ptr(); p.x_out = xo.data_ptr();
    p.y_sr = y2.stride(0); p.xo_sr = over_x ? x2.stride(0) : D;
  }
  p.eps = (float)eps; p.dtype = dtype_code(x);
  const int rc = xl_add_rmsnorm(&p, stream_of(x));
  unlocked.lock();
  check(rc, "xl_add_rmsnorm");
  return pack_pair(!y || over_x ? Py_NewRef(a[0]) : THPVariable_Wrap(xo), THPVariable_Wrap(normed));
  END_HANDLE_TH_ERRORS
}

// (x (..., K), w (N, K), w_ahead) -> (..., N), bf16, at most 16 rows of x; w_ahead: the caller knows that the launch in front does not write w
PyObject* rows_linear(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 3);
  const Tensor &x = tensor_arg(a[0], "x"), &w0 = tensor_arg(a[1], "w");
  const bool w_ahead = a[2] == Py_True;
  Unlocked unlocked;
  for (const Tensor* t : {&x, &w0}) require_cuda(t);
  TORCH_CHECK_VALUE(x.scalar_type() == at::kBFloat16 && w0.scalar_type() == at::kBFloat16 && w0.dim() == 2 && x.dim() >= 1 && x.size(-1) == w0.size(1),
                    "rows_linear: bfloat16 x (..., K) and w (N, K)");
  const int64_t K = x.size(-1), N = w0.size(0);
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor x2 = as_rows(x, K), w = last_contig(w0);
  c10::SmallVector<int64_t, 5> sizes(x.sizes().begin(), x.sizes().end());
  sizes.back() = N;
  const Tensor y = empty_on(sizes, at::kBFloat16, x);
  xl_rows_linear_params p = {};
  p.x = x2.data_ptr(); p.w = w.data_ptr(); p.y = y.data_ptr(); p.status = status_ptr(x);
  p.x_sr = x2.size(0) > 1 ? x2.stride(0) : K; p.w_sr = N > 1 ? w.stride(0) : K;
  p.rows = (int32_t)x2.size(0); p.N = (int32_t)N; p.K = (int32_t)K; p.dtype = XL_BF16;
  const bool ahead = w_ahead && w.is_same(w0);   // (a copy of w made here is the launch in front)
  const int rc = ahead ? xl_rows_linear_ahead(&p, stream_of(x)) : xl_rows_linear(&p, stream_of(x));
  unlocked.lock();
  check(rc, "xl_rows_linear");
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

// (h, o_preact or None, weight, eps) -> (B, S, NH*DH)
PyObject* headnorm_gate(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 4);
  const Tensor &h0 = tensor_arg(a[0], "h"), &w0 = tensor_arg(a[2], "weight");
  const Tensor* o0 = optional_arg(a[1], "o_preact");
  const double eps = double_arg(a[3]);
  Unlocked unlocked;
  for (const Tensor* t : {&h0, o0, &w0}) require_cuda(t);
  TORCH_CHECK_VALUE(h0.dim() == 4 && known_dtype(h0) && (!o0 || o0->scalar_type() == h0.scalar_type()) && w0.scalar_type() == h0.scalar_type(),
                    "headnorm_gate: h must be (B,NH,S,DH); h, o_preact and weight must share float32 or bfloat16");
  const int64_t B = h0.size(0), NH = h0.size(1), S = h0.size(2), DH = h0.size(3);
  TORCH_CHECK_VALUE((!o0 || o0->sizes() == at::IntArrayRef({B, S, NH * DH})) && w0.sizes() == at::IntArrayRef({NH * DH}),
                    "headnorm_gate: o_preact must be (B,S,NH*DH) and weight (NH*DH,)");
  const c10::cuda::CUDAGuard guard(h0.device());
  const Tensor h = last_contig(h0), w = w0.contiguous(), o = o0 ? last_contig(*o0) : Tensor();
  const Tensor out = empty_on({B, S, NH * DH}, h.scalar_type(), h);
  xl_headnorm_gate_params p = {};
  p.h = h.data_ptr(); p.weight = w.data_ptr(); p.out = out.data_ptr();
  p.B = B; p.NH = NH; p.S = S; p.DH = DH;
  p.h_sb = h.stride(0); p.h_sh = h.stride(1); p.h_st = h.stride(2);
  if (o0) { p.o = o.data_ptr(); p.o_sb = o.stride(0); p.o_st = o.stride(1); }
  p.eps = (float)eps; p.dtype = dtype_code(h);
  const int rc = xl_headnorm_gate(&p, stream_of(h));
  unlocked.lock();
  check(rc, "xl_headnorm_gate");
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// (x, cap, out mode of the C entry: 0 x's dtype, 1 fp32, 2 fp32 without roundings in between, bias or None)
PyObject* soft_cap(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 4);
  const Tensor& x = tensor_arg(a[0], "x");
  const Tensor* bias0 = optional_arg(a[3], "bias");
  const double cap = double_arg(a[1]);
  const int64_t mode = int_arg(a[2]);
  Unlocked unlocked;
  for (const Tensor* t : {&x, bias0}) require_cuda(t);
  TORCH_CHECK_VALUE(known_dtype(x), "soft_cap: float32 or bfloat16 only");
  const int64_t cols = x.size(-1);
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor x2 = as_rows(x, cols), bias = bias0 ? bias0->contiguous() : Tensor();
  const Tensor out = empty_on(x.sizes(), mode ? at::kFloat : x.scalar_type(), x);
  xl_soft_cap_params p = {};
  p.x = x2.data_ptr(); p.out = out.data_ptr(); p.n = x.numel(); p.cap = (float)cap;
  p.dtype = dtype_code(x); p.out_f32 = (int32_t)mode;
  if (x2.size(0) > 0 && (x2.stride(0) != cols || bias0)) {
    p.cols = cols;
    p.x_row_stride = x2.stride(0);
    if (bias0) {
      TORCH_CHECK_VALUE(bias.dim() == 1 && bias.size(0) == cols && bias.scalar_type() == x.scalar_type(),
                        "soft_cap: bias must have the size of the last dimension and x's dtype");
      p.bias = bias.data_ptr();
    }
  }
  const int rc = xl_soft_cap(&p, stream_of(x));
  unlocked.lock();
  check(rc, "xl_soft_cap");
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

PyObject* swiglu(PyObject*, PyObject* gz_obj) {
  HANDLE_TH_ERRORS
  const Tensor& gz = tensor_arg(gz_obj, "gz");
  Unlocked unlocked;
  require_cuda(gz);
  TORCH_CHECK_VALUE(known_dtype(gz) && gz.size(-1) % 2 == 0, "swiglu: float32 or bfloat16, even last dimension");
  const int64_t F = gz.size(-1) / 2;
  const c10::cuda::CUDAGuard guard(gz.device());
  const Tensor g2 = as_rows(gz, 2 * F);
  c10::SmallVector<int64_t, 5> sizes(gz.sizes().begin(), gz.sizes().end());
  sizes.back() = F;
  const Tensor out = empty_on(sizes, gz.scalar_type(), gz);
  xl_swiglu_params p = {};
  p.gz = g2.data_ptr(); p.out = out.data_ptr(); p.rows = g2.size(0); p.F = (int32_t)F; p.gz_row_stride = g2.stride(0); p.dtype = dtype_code(gz);
  const int rc = xl_swiglu(&p, stream_of(gz));
  unlocked.lock();
  check(rc, "xl_swiglu");
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// (x, weight (F,K) or (F,1,K), bias or None, cu_seqlens on the device or None, documents, silu) -> (B, S, F)
PyObject* causal_conv1d(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 6);
  const Tensor &x0 = tensor_arg(a[0], "x"), &w0 = tensor_arg(a[1], "weight");
  const Tensor *bias0 = optional_arg(a[2], "bias"), *cu = optional_arg(a[3], "cu_seqlens");
  const int64_t docs = int_arg(a[4]);
  const bool silu = a[5] == Py_True;
  Unlocked unlocked;
  for (const Tensor* t : {&x0, &w0, bias0, cu}) require_cuda(t);
  TORCH_CHECK_VALUE(x0.dim() == 3 && known_dtype(x0), "causal_conv1d: x must be (B,S,F) in float32 or bfloat16");
  const int64_t B = x0.size(0), S = x0.size(1), F = x0.size(2), K = w0.size(-1);
  TORCH_CHECK_VALUE((w0.dim() == 2 || w0.dim() == 3) && w0.size(0) == F && w0.scalar_type() == x0.scalar_type() &&
                        (!bias0 || (bias0->sizes() == at::IntArrayRef({F}) && bias0->scalar_type() == x0.scalar_type())),
                    "causal_conv1d: weight must be (F,K) and bias (F,), both in x's dtype");
  const c10::cuda::CUDAGuard guard(x0.device());
  const Tensor x = last_contig(x0), w = (w0.dim() == 3 ? w0.select(1, 0) : w0).contiguous(), bias = bias0 ? bias0->contiguous() : Tensor();
  const Tensor out = empty_on({B, S, F}, x.scalar_type(), x);
  xl_conv1d_params p = {};
  p.x = x.data_ptr(); p.weight = w.data_ptr(); p.bias = bias0 ? bias.data_ptr() : nullptr; p.out = out.data_ptr();
  p.cu_seqlens = cu ? cu->const_data_ptr<int32_t>() : nullptr;
  p.B = B; p.S = S; p.F = F; p.K = K; p.num_docs = cu ? docs : 0; p.act = silu;
  p.x_sb = x.stride(0); p.x_st = x.stride(1);
  p.o_sb = out.stride(0); p.o_st = out.stride(1);
  p.dtype = dtype_code(x);
  const int rc = xl_causal_conv1d(&p, stream_of(x));
  unlocked.lock();
  check(rc, "xl_causal_conv1d");
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// (inputs: list of one or two, weights: list of one to four, in_sel: list) -> (..., slots * NH*DH)
PyObject* headwise_proj(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 3);
  TORCH_CHECK_VALUE(PyList_Check(a[0]) && PyList_Check(a[1]) && PyList_Check(a[2]), "headwise_proj: lists wanted");
  const int64_t nx = PyList_GET_SIZE(a[0]), n = PyList_GET_SIZE(a[1]);
  TORCH_CHECK_VALUE(n >= 1 && n <= 4 && nx >= 1 && nx <= 2 && PyList_GET_SIZE(a[2]) == n,
                    "headwise_proj: one to four weights, one or two inputs, in_sel entries index the inputs");
  xl_headwise_params p = {};
  Tensor xs[2], ws[4];
  for (int64_t j = 0; j < nx; ++j) { xs[j] = tensor_arg(PyList_GET_ITEM(a[0], j), "input"); require_cuda(xs[j]); }
  for (int64_t j = 0; j < n; ++j) {
    ws[j] = tensor_arg(PyList_GET_ITEM(a[1], j), "weight");
    require_cuda(ws[j]);
    const int64_t sel = int_arg(PyList_GET_ITEM(a[2], j));
    TORCH_CHECK_VALUE(sel >= 0 && sel < nx, "headwise_proj: one to four weights, one or two inputs, in_sel entries index the inputs");
    p.in_sel[j] = (int32_t)sel;
  }
  Unlocked unlocked;
  TORCH_CHECK_VALUE(ws[0].dim() == 3, "headwise_proj: weights must be bfloat16 (NH, DH, DH)");
  const int64_t NH = ws[0].size(0), DH = ws[0].size(1), D = NH * DH;
  TORCH_CHECK_VALUE(ws[0].size(2) == DH && (DH == 64 || DH == 128 || DH == 256), "headwise_proj: square per-head blocks of 64, 128 or 256 features only");
  c10::SmallVector<int64_t, 5> sizes(xs[0].sizes().begin(), xs[0].sizes().end());
  const c10::cuda::CUDAGuard guard(xs[0].device());
  for (int64_t j = 0; j < nx; ++j) {
    TORCH_CHECK_VALUE(xs[j].scalar_type() == at::kBFloat16 && xs[j].size(-1) == D && xs[j].sizes() == at::IntArrayRef(sizes),
                      "headwise_proj: inputs must be bfloat16 (..., NH*DH) of one shape");
    xs[j] = as_rows(xs[j], D);
    if (xs[j].stride(0) % 8) xs[j] = xs[j].contiguous();
    p.x[j] = xs[j].data_ptr();
    p.x_row_stride[j] = xs[j].stride(0);
  }
  for (int64_t j = 0; j < n; ++j) {
    TORCH_CHECK_VALUE(ws[j].scalar_type() == at::kBFloat16 && ws[j].sizes() == at::IntArrayRef({NH, DH, DH}),
                      "headwise_proj: weights must be bfloat16 (NH, DH, DH)");
    ws[j] = ws[j].contiguous();
    p.w[j] = ws[j].data_ptr();
  }
  sizes.back() = n * D;
  const Tensor out = empty_on(sizes, at::kBFloat16, xs[0]);
  p.out = out.data_ptr(); p.out_row_stride = n * D;
  p.status = status_ptr(out);
  p.rows = xs[0].size(0); p.NH = NH; p.DH = DH; p.n_slots = (int32_t)n; p.dtype = XL_BF16;
  const int rc = xl_headwise_proj(&p, stream_of(out));
  unlocked.lock();
  check(rc, "xl_headwise_proj");
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// Scratch of the greedy head, once per device (grown when more rows come) and shared by all calls on the device.  Called
// without the interpreter lock.
Tensor greedy_scratch(int64_t index, int64_t need, const Tensor& like) {
  static std::mutex mutex;
  static Tensor* scratch[MAX_DEVICES];
  TORCH_CHECK_VALUE(index < MAX_DEVICES, "device index out of range");
  const std::lock_guard<std::mutex> hold(mutex);
  if (!scratch[index] || scratch[index]->numel() < need) {
    const int64_t bytes = std::max(need, xl_softcap_argmax_scratch_bytes(256));
    Tensor* fresh = new Tensor(at::zeros({bytes}, at::TensorOptions().dtype(at::kByte).device(like.device())));
    delete scratch[index];
    scratch[index] = fresh;
  }
  return *scratch[index];
}

// (logits, cap) -> int64 tokens of shape logits.shape[:-1]
PyObject* softcap_argmax(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 2);
  const Tensor& logits = tensor_arg(a[0], "logits");
  const double cap = double_arg(a[1]);
  Unlocked unlocked;
  require_cuda(logits);
  TORCH_CHECK_VALUE(known_dtype(logits), "softcap_argmax: float32 or bfloat16 only");
  const int64_t V = logits.size(-1);
  const c10::cuda::CUDAGuard guard(logits.device());
  const Tensor x = as_rows(logits, V);
  const int64_t rows = x.size(0), need = xl_softcap_argmax_scratch_bytes((int32_t)rows), index = x.device().index();
  const Tensor sc = greedy_scratch(index, need, x);
  const Tensor out = empty_on(logits.sizes().slice(0, logits.dim() - 1), at::kLong, x);
  xl_greedy_params p = {};
  p.logits = x.data_ptr(); p.tokens = out.data_ptr<int64_t>(); p.scratch = sc.data_ptr(); p.scratch_bytes = sc.numel();
  p.rows = (int32_t)rows; p.V = (int32_t)V; p.row_stride = x.stride(0); p.cap = (float)cap; p.dtype = dtype_code(x);
  const int rc = xl_softcap_argmax(&p, stream_of(x));
  unlocked.lock();
  check(rc, "xl_softcap_argmax");
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------- host-side vectors
// A Python sequence of integers, or a tensor on the host that is one.
std::vector<int64_t> host_integers(PyObject* o) {
  std::vector<int64_t> out;
  PyObject* list = nullptr;   // (other tensors go the way their `tolist` goes: numbers truncate, a scalar or a matrix is no sequence of numbers)
  if (THPVariable_Check(o)) {
    const Tensor& t0 = THPVariable_Unpack(o);
    if (t0.dim() == 1 && (t0.scalar_type() == at::kInt || t0.scalar_type() == at::kLong)) {
      const Tensor t = t0.to(at::kLong).contiguous();
      out.assign(t.const_data_ptr<int64_t>(), t.const_data_ptr<int64_t>() + t.numel());
      return out;
    }
    list = PyObject_CallMethod(o, "tolist", nullptr);
    if (!list) throw python_error();
    o = list;
  }
  PyObject* seq = PySequence_Fast(o, "a sequence of integers is wanted");
  Py_XDECREF(list);
  if (!seq) throw python_error();
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
  out.reserve((size_t)n);
  for (Py_ssize_t j = 0; j < n; ++j) {
    PyObject* index = PyNumber_Long(PySequence_Fast_GET_ITEM(seq, j));
    const long long v = index ? PyLong_AsLongLong(index) : -1;
    Py_XDECREF(index);
    if (v == -1 && PyErr_Occurred()) { Py_DECREF(seq); throw python_error(); }
    out.push_back(v);
  }
  Py_DECREF(seq);
  return out;
}

// int32 vector on `device` (index; below 0: the host).  The copy leaves from pinned memory and is not waited for: from
// pageable memory every packed call synchronised the stream.  Not under capture, where that synchronisation was an error.
Tensor int32_vector(const std::vector<int64_t>& vals, int64_t device) {
  if (device >= 0) {
    // (a captured copy would read the host buffer at every replay, long after it has gone to somebody else)
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
    TORCH_CHECK(c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None,
                "offsets and slots from the host cannot enter a CUDA graph: pass an int32 tensor on the device");
  }
  Tensor host = at::empty({(int64_t)vals.size()}, at::TensorOptions().dtype(at::kInt).pinned_memory(device >= 0));
  int32_t* dst = host.data_ptr<int32_t>();
  for (size_t j = 0; j < vals.size(); ++j) {
    TORCH_CHECK(vals[j] >= INT32_MIN && vals[j] <= INT32_MAX, vals[j], " does not fit into 32 bits");
    dst[j] = (int32_t)vals[j];
  }
  return device < 0 ? host : host.to(at::Device(at::kCUDA, (int8_t)device), at::kInt, /*non_blocking=*/true);
}

// (offsets on the host, B, S, device index or -1) -> (int32 offsets on the device, documents), checked
PyObject* document_offsets(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 4);
  const std::vector<int64_t> cu = host_integers(a[0]);
  const int64_t B = int_arg(a[1]), S = int_arg(a[2]), n = (int64_t)cu.size();
  const int64_t device = int_arg(a[3]);
  Unlocked unlocked;
  TORCH_CHECK_VALUE(n >= 2 && cu.front() == 0 && cu.back() == B * S, "cu_seqlens must start at 0 and end at B*S=", B * S);
  for (int64_t j = 0; j + 1 < n; ++j) {
    TORCH_CHECK_VALUE(cu[j + 1] >= cu[j], "cu_seqlens must be non-decreasing");
    TORCH_CHECK_VALUE(cu[j + 1] == cu[j] || cu[j] / S == (cu[j + 1] - 1) / S, "document [", cu[j], ",", cu[j + 1], ") straddles two rows of length ", S);
  }
  const Tensor offsets = int32_vector(cu, device);
  unlocked.lock();
  return pack_pair(THPVariable_Wrap(offsets), PyLong_FromLongLong(n - 1));
  END_HANDLE_TH_ERRORS
}

// (slots on the host, B, pool rows, device index or -1) -> int32 slots on the device, checked
PyObject* slot_vector(PyObject*, PyObject* const* a, Py_ssize_t na) {
  HANDLE_TH_ERRORS
  want_args(na, 4);
  const std::vector<int64_t> slots = host_integers(a[0]);
  const int64_t B = int_arg(a[1]), n = int_arg(a[2]), device = int_arg(a[3]);
  Unlocked unlocked;
  TORCH_CHECK_VALUE((int64_t)slots.size() == B, "slot must have one entry per stream (", B, "), got ", slots.size());
  std::vector<bool> taken((size_t)std::max<int64_t>(n, 0), false);
  for (const int64_t s : slots) TORCH_CHECK_VALUE(s < n, "slot entries must be below the pool size ", n);
  for (const int64_t s : slots) {
    if (s < 0) continue;
    TORCH_CHECK_VALUE(!taken[(size_t)s], "two active streams name the same pool row");
    taken[(size_t)s] = true;
  }
  const Tensor rows = int32_vector(slots, device);
  unlocked.lock();
  return THPVariable_Wrap(rows);
  END_HANDLE_TH_ERRORS
}

PyObject* status_word(PyObject*, PyObject* index) {
  HANDLE_TH_ERRORS
  const int64_t device = int_arg(index);
  Unlocked unlocked;
  const Tensor& word = status_tensor(device);
  unlocked.lock();
  return THPVariable_Wrap(word);
  END_HANDLE_TH_ERRORS
}

#define XL_FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    XL_FAST(mlstm_sequence), XL_FAST(mlstm_step), XL_FAST(mlstm_decode_cell), XL_FAST(slstm_forward), XL_FAST(slstm_backward), XL_FAST(slstm_weight_grads), XL_FAST(rows_linear),
    XL_FAST(add_rmsnorm), XL_FAST(headnorm_gate), XL_FAST(soft_cap), XL_FAST(causal_conv1d), XL_FAST(headwise_proj), XL_FAST(softcap_argmax),
    XL_FAST(document_offsets), XL_FAST(slot_vector),
    {"swiglu", swiglu, METH_O, nullptr}, {"status_word", status_word, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", "Native host path of xlstm_b200.ops.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "built_for", XL_BUILT_FOR) < 0) Py_CLEAR(m);   // the PyTorch it is compiled against
  return m;
}
