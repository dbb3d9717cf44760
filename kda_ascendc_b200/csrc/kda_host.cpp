// Host path of the public Python functions: argument checks, output allocation and the C-ABI call of one
// forward in a single native call.
//
// What it replaces per call is the interpreter: some forty tensor-attribute reads and comparisons, ctypes
// argument packing and two context managers, 35-50 us on a B200 host against 6 us of device time for a
// decode step.  The rules and messages of the argument checks stay in api.py: the functions here accept a call only
// when every check would pass, and return None otherwise, so that the Python path decides what is wrong
// (or serves the rarer options: debug outputs, stage timing).
//
// CPython's vectorcall protocol and the tensor type's own accessors are used directly; nothing here keeps
// state between calls.
#include <Python.h>

#include <cstdlib>
#include <cstring>
#include <exception>
#include <vector>

#include <ATen/ATen.h>
#include <ATen/core/grad_mode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/kda_b200.h"

namespace {

constexpr int64_t kD = 128;
constexpr int64_t kBT = 16;

// A null result of an argument accessor means "take the Python path".
struct Miss {};

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) throw Miss();
  return THPVariable_Unpack(o);
}
bool truth(PyObject* o) {
  if (o == Py_True) return true;
  if (o == Py_False || o == Py_None) return false;
  throw Miss();
}
double number(PyObject* o) {
  if (PyFloat_CheckExact(o)) return PyFloat_AS_DOUBLE(o);
  if (PyLong_CheckExact(o)) {
    const double x = PyLong_AsDouble(o);
    if (x != -1.0 || PyErr_Occurred() == nullptr) return x;   // else beyond a double: the handler of Miss clears the error
  }
  throw Miss();
}
void need(bool ok) {
  if (!ok) throw Miss();
}

struct Inputs {
  const at::Tensor *q, *k, *v, *g, *beta;
  int64_t B, T, Hq, H;
  c10::Device dev = c10::Device(c10::kCPU);
};

// The shared validator's rules on q, k, v, g and beta (api.py:_validate_kda_inputs).
Inputs take_inputs(PyObject* const* a, bool contiguous) {
  Inputs in;
  in.q = &tensor(a[0]); in.k = &tensor(a[1]); in.v = &tensor(a[2]); in.g = &tensor(a[3]); in.beta = &tensor(a[4]);
  need(in.q->dim() == 4 && in.k->dim() == 4 && in.v->dim() == 4 && in.g->dim() == 4 && in.beta->dim() == 3);
  const auto qs = in.q->sizes(), ks = in.k->sizes(), vs = in.v->sizes(), gs = in.g->sizes(), bs = in.beta->sizes();
  in.B = qs[0]; in.T = qs[1]; in.Hq = qs[2]; in.H = vs[2];
  need(in.B > 0 && in.T > 0 && in.Hq > 0 && in.H > 0 && qs[3] == kD && vs[3] == kD && in.H % in.Hq == 0);
  need(in.B < 0x7fffffff && in.T < 0x7fffffff && in.H < 0x7fffffff);
  need(ks == qs && vs[0] == in.B && vs[1] == in.T && gs[0] == in.B && gs[1] == in.T && gs[2] == in.H && gs[3] == kD &&
       bs[0] == in.B && bs[1] == in.T && bs[2] == in.H);
  need(in.q->scalar_type() == at::kBFloat16 && in.k->scalar_type() == at::kBFloat16 && in.v->scalar_type() == at::kBFloat16 &&
       (in.g->scalar_type() == at::kBFloat16 || in.g->scalar_type() == at::kFloat) && in.beta->scalar_type() == at::kFloat);
  in.dev = in.q->device();
  need(in.dev.is_cuda() && in.k->device() == in.dev && in.v->device() == in.dev && in.g->device() == in.dev &&
       in.beta->device() == in.dev);
  if (contiguous)
    need(in.q->is_contiguous() && in.k->is_contiguous() && in.v->is_contiguous() && in.g->is_contiguous() && in.beta->is_contiguous());
  else
    need(in.q->stride(3) == 1 && in.k->stride(3) == 1 && in.v->stride(3) == 1 && in.g->stride(3) == 1);
  return in;
}

// An optional fp32 contiguous tensor of the given shape on the inputs' device; null for None.
const at::Tensor* side_tensor(PyObject* o, const Inputs& in, at::IntArrayRef shape) {
  if (o == Py_None) return nullptr;
  const at::Tensor& t = tensor(o);
  need(t.scalar_type() == at::kFloat && t.device() == in.dev && t.sizes() == shape && t.is_contiguous());
  return &t;
}

void set_strides(int64_t (&dst)[3], const at::Tensor& t) {
  dst[0] = t.stride(0); dst[1] = t.stride(1); dst[2] = t.stride(2);
}

KdaFwdArgs base_args(const Inputs& in, double scale, double lower_bound, uint32_t flags) {
  KdaFwdArgs a;
  memset(&a, 0, sizeof(a));
  a.q = in.q->data_ptr(); a.k = in.k->data_ptr(); a.v = in.v->data_ptr(); a.g = in.g->data_ptr();
  a.beta = static_cast<const float*>(in.beta->data_ptr());
  a.B = static_cast<int32_t>(in.B); a.T = static_cast<int32_t>(in.T); a.H = static_cast<int32_t>(in.H);
  a.Hq = in.Hq == in.H ? 0 : static_cast<int32_t>(in.Hq);
  a.g_dtype = in.g->scalar_type() == at::kBFloat16 ? KDA_G_BF16 : KDA_G_FP32;
  set_strides(a.q_stride, *in.q); set_strides(a.k_stride, *in.k); set_strides(a.v_stride, *in.v);
  set_strides(a.g_stride, *in.g); set_strides(a.beta_stride, *in.beta);
  a.scale = static_cast<float>(scale);
  a.lower_bound = static_cast<float>(lower_bound);
  a.flags = flags;
  return a;
}

// The adapter's extra rules: no autograd through these calls, and dt_bias may come as [H, 128].
void need_no_grad(const Inputs& in) {
  if (!c10::GradMode::is_enabled()) return;
  need(!in.q->requires_grad() && !in.k->requires_grad() && !in.v->requires_grad() && !in.g->requires_grad() && !in.beta->requires_grad());
}
const at::Tensor* bias_tensor(PyObject* o, const Inputs& in, bool fla) {
  if (fla && o != Py_None && tensor(o).dim() == 2) return side_tensor(o, in, {in.H, kD});
  return side_tensor(o, in, {in.H * kD});
}

// The C calls run without the interpreter lock (a launch can wait for room in the stream's queue).  The
// destructor takes the lock back, also when `f` throws.
class ReleasedLock {
 public:
  ReleasedLock() : state_(PyEval_SaveThread()) {}
  ~ReleasedLock() { PyEval_RestoreThread(state_); }
  ReleasedLock(const ReleasedLock&) = delete;
  ReleasedLock& operator=(const ReleasedLock&) = delete;

 private:
  PyThreadState* state_;
};
template <class F>
int unlocked(F f) {
  const ReleasedLock released;
  return f();
}

// cu_seqlens as 32-bit host values: a list or tuple of integers, or a 1-D integer tensor on any device (one
// device-to-host read if it lives on a GPU).
std::vector<int32_t> host_offsets(PyObject* o) {
  std::vector<int32_t> cu;
  if (PyList_CheckExact(o) || PyTuple_CheckExact(o)) {
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
    cu.resize(static_cast<size_t>(n));
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* x = PySequence_Fast_GET_ITEM(o, i);
      need(PyLong_CheckExact(x));
      const long v = PyLong_AsLong(x);
      need(v >= 0 && v <= 0x7fffffff);
      cu[static_cast<size_t>(i)] = static_cast<int32_t>(v);
    }
    return cu;
  }
  at::Tensor t = tensor(o);
  need(t.dim() == 1 && (t.scalar_type() == at::kInt || t.scalar_type() == at::kLong));
  if (t.is_cuda()) unlocked([&] { t = t.cpu(); return 0; });
  need(t.is_cpu());
  cu.resize(static_cast<size_t>(t.numel()));
  const int64_t st = t.numel() > 0 ? t.stride(0) : 1;
  for (size_t i = 0; i < cu.size(); ++i) {
    const int64_t v = t.scalar_type() == at::kInt ? static_cast<const int32_t*>(t.data_ptr())[static_cast<int64_t>(i) * st]
                                                  : static_cast<const int64_t*>(t.data_ptr())[static_cast<int64_t>(i) * st];
    need(v >= 0 && v <= 0x7fffffff);
    cu[i] = static_cast<int32_t>(v);
  }
  return cu;
}

float* fptr(const at::Tensor* t) { return t == nullptr ? nullptr : static_cast<float*>(t->data_ptr()); }

// A failed C call: the message goes out as the exception api.py:_check raises for it.
PyObject* raise_for(int rc) {
  PyErr_SetString(rc == KDA_ERR_INVALID_ARG ? PyExc_ValueError : PyExc_RuntimeError, kda_last_error());
  return nullptr;
}

// The C++ exception being handled, as the Python exception that PyTorch's own bindings raise for it (out of memory
// keeps its type; an error raised in Python under an ATen call is that error).
PyObject* raise_current() {
  torch::translate_exception_to_python(std::current_exception());
  return nullptr;
}

PyObject* result(at::Tensor o, PyObject* ht) {   // steals ht
  PyObject* out = PyTuple_New(2);
  PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(std::move(o)));
  PyTuple_SET_ITEM(out, 1, ht);
  return out;
}

// chunk(q, k, v, g, beta, scale, initial_state, output_final_state, l2norm, gate, beta_sigmoid, safe_gate, lower_bound,
//       A_log, dt_bias, state_v_first, cu_seqlens, fla) -> (o, ht) | None
// `fla`: the call comes through the flash-linear-attention adapter and has to pass its rules as well.
PyObject* chunk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 18) Py_RETURN_NONE;
  try {
    const char* prof = getenv("KDA_PROFILE");
    need(prof == nullptr || strcmp(prof, "1") != 0);
    const Inputs in = take_inputs(a, true);
    const bool v_first = truth(a[15]), gate = truth(a[9]);
    const double scale = a[5] == Py_None ? 0.08838834764831845 : number(a[5]);   // 128^-0.5
    double lb = -5.0;
    if (a[12] != Py_None) lb = number(a[12]);
    if (gate) need(truth(a[11]) && a[12] != Py_None && lb > -11.0 && lb < 0.0 && a[13] != Py_None);
    const bool fla = truth(a[17]);
    if (fla) need_no_grad(in);
    std::vector<int32_t> cu;
    int64_t n_states = in.B, n_chunks = 0;
    if (a[16] != Py_None) {
      need(in.B == 1);
      cu = host_offsets(a[16]);
      need(cu.size() >= 2 && cu.back() == in.T);
      n_states = static_cast<int64_t>(cu.size()) - 1;
      n_chunks = kda_varlen_fill_tables(cu.data(), static_cast<int32_t>(n_states), static_cast<int32_t>(in.H), nullptr, nullptr);
      need(n_chunks > 0);
    }
    const at::Tensor* h0 = side_tensor(a[6], in, {n_states, in.H, kD, kD});
    const at::Tensor* a_log = side_tensor(a[13], in, {in.H});
    const at::Tensor* bias = bias_tensor(a[14], in, fla);
    const uint32_t flags = (gate ? KDA_FLAG_GATE_IN_KERNEL : 0u) | (truth(a[8]) ? KDA_FLAG_QK_L2NORM : 0u) |
                           (truth(a[10]) ? KDA_FLAG_BETA_SIGMOID : 0u) | (v_first ? 0u : KDA_FLAG_STATE_K_FIRST);
    const bool want_ht = truth(a[7]);
    KdaFwdArgs args = base_args(in, scale, lb, flags);
    args.A_log = fptr(a_log); args.dt_bias = fptr(bias); args.h0 = fptr(h0);

    const c10::cuda::CUDAGuard guard(in.dev);
    const auto opt = in.q->options();
    at::Tensor o = at::empty({in.B, in.T, in.H, kD}, opt.dtype(at::kBFloat16));
    at::Tensor ht;
    if (want_ht) ht = at::empty({n_states, in.H, kD, kD}, opt.dtype(at::kFloat));
    const int64_t ws_tokens = n_chunks > 0 ? kBT * n_chunks : in.T;
    const at::Tensor ws = at::empty({static_cast<int64_t>(kda_fwd_workspace_bytes(args.B, static_cast<int32_t>(ws_tokens), args.H))},
                                    opt.dtype(at::kByte));
    at::Tensor tab;   // [n_chunks + n_seqs][4]: the chunk table, then the sequence table
    if (n_chunks > 0) {
      at::Tensor host = at::empty({n_chunks + n_states, 4}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
      int32_t* p = static_cast<int32_t*>(host.data_ptr());
      kda_varlen_fill_tables(cu.data(), static_cast<int32_t>(n_states), args.H, p, p + 4 * n_chunks);
      tab = host.to(opt.dtype(at::kInt), /*non_blocking=*/true);
      args.n_seqs = static_cast<int32_t>(n_states);
      args.n_chunks = static_cast<int32_t>(n_chunks);
      args.chunk_table = static_cast<const int32_t*>(tab.data_ptr());
      args.seq_table = args.chunk_table + 4 * n_chunks;
    }
    args.o = o.data_ptr();
    set_strides(args.o_stride, o);
    args.ht = want_ht ? static_cast<float*>(ht.data_ptr()) : nullptr;
    args.workspace = ws.data_ptr();
    void* stream = c10::cuda::getCurrentCUDAStream(in.dev.index()).stream();
    const int rc = unlocked([&] { return kda_fwd(&args, stream); });
    if (rc != KDA_OK) return raise_for(rc);
    PyObject* pht = Py_None;
    if (want_ht) pht = THPVariable_Wrap(std::move(ht)); else Py_INCREF(pht);
    return result(std::move(o), pht);
  } catch (const Miss&) {
    PyErr_Clear();
    Py_RETURN_NONE;
  } catch (...) {
    return raise_current();
  }
}

// recurrent(q, k, v, g, beta, scale, initial_state, output_final_state, lower_bound, A_log, dt_bias, inplace_state,
//           state_v_first, max_tokens, fla) -> (o, ht) | None
PyObject* recurrent(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 15) Py_RETURN_NONE;
  try {
    const Inputs in = take_inputs(a, false);
    const bool fla = truth(a[14]);
    if (fla) need_no_grad(in);
    const bool inplace = truth(a[11]), v_first = truth(a[12]);
    const double scale = a[5] == Py_None ? 0.08838834764831845 : number(a[5]);
    need(a[8] != Py_None && a[9] != Py_None);
    const double lb = number(a[8]);
    need(lb > -11.0 && lb < 0.0);
    const at::Tensor* h0 = side_tensor(a[6], in, {in.B, in.H, kD, kD});
    const at::Tensor* a_log = side_tensor(a[9], in, {in.H});
    const at::Tensor* bias = bias_tensor(a[10], in, fla);
    need(!inplace || h0 != nullptr);
    const bool want_ht = truth(a[7]);
    KdaFwdArgs args = base_args(in, scale, lb,
                                KDA_FLAG_GATE_IN_KERNEL | KDA_FLAG_QK_L2NORM | KDA_FLAG_BETA_SIGMOID | (v_first ? 0u : KDA_FLAG_STATE_K_FIRST));
    args.A_log = fptr(a_log); args.dt_bias = fptr(bias); args.h0 = fptr(h0);

    const c10::cuda::CUDAGuard guard(in.dev);
    const auto opt = in.q->options();
    at::Tensor o = at::empty({in.B, in.T, in.H, kD}, opt.dtype(at::kBFloat16));
    at::Tensor ht, ws;
    PyObject* pht = Py_None;
    if (inplace) {
      args.ht = fptr(h0);
      pht = a[6];
    } else if (want_ht) {
      ht = at::empty({in.B, in.H, kD, kD}, opt.dtype(at::kFloat));
      args.ht = static_cast<float*>(ht.data_ptr());
    }
    args.o = o.data_ptr();
    set_strides(args.o_stride, o);
    void* stream = c10::cuda::getCurrentCUDAStream(in.dev.index()).stream();
    int rc;
    if (in.T > static_cast<int64_t>(number(a[13]))) {
      ws = at::empty({static_cast<int64_t>(kda_fwd_workspace_bytes(args.B, args.T, args.H))}, opt.dtype(at::kByte));
      args.workspace = ws.data_ptr();
      rc = unlocked([&] { return kda_fwd(&args, stream); });
    } else {
      rc = unlocked([&] { return kda_recurrent_fwd(&args, stream); });
    }
    if (rc != KDA_OK) return raise_for(rc);
    if (!inplace && want_ht) pht = THPVariable_Wrap(std::move(ht)); else Py_INCREF(pht);
    return result(std::move(o), pht);
  } catch (const Miss&) {
    PyErr_Clear();
    Py_RETURN_NONE;
  } catch (...) {
    return raise_current();
  }
}

// run_plan(argument block address, device index, stream or None, recurrent) -> None: one C call of a plan with
// its device current (the library sizes grids and caches kernel attributes for the current device).
PyObject* run_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 4) {
    PyErr_SetString(PyExc_TypeError, "run_plan takes 4 arguments");
    return nullptr;
  }
  const KdaFwdArgs* args = static_cast<const KdaFwdArgs*>(PyLong_AsVoidPtr(a[0]));
  const long dev = PyLong_AsLong(a[1]);
  if (PyErr_Occurred()) return nullptr;
  try {
    void* stream;
    if (a[2] == Py_None) {
      stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(dev)).stream();
    } else {
      stream = PyLong_AsVoidPtr(a[2]);
      if (PyErr_Occurred()) return nullptr;
    }
    const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(dev));
    const bool rec = a[3] == Py_True;
    const int rc = unlocked([&] { return rec ? kda_recurrent_fwd(args, stream) : kda_fwd(args, stream); });
    if (rc != KDA_OK) return raise_for(rc);
  } catch (...) {
    return raise_current();
  }
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"chunk", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(chunk)), METH_FASTCALL, nullptr},
    {"recurrent", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(recurrent)), METH_FASTCALL, nullptr},
    {"run_plan", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(run_plan)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_kda_host", "Native host path of the KDA functions.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__kda_host() { return PyModule_Create(&kModule); }
