// Host side of the Python operators (`ttt_tk_b200.ops`): argument validation, the C ABI's argument structs and the
// launch, in native code.  For short sequences a call is bound by its host time, and checking 15 to 42 tensors one
// attribute at a time from Python took most of it.  Measured: the forward's enqueue 50 -> 4.2 us; forwards of one
// mini-batch in a row 57 -> 8.9 us each (the kernel's own time), of four TTT-Linear mini-batches 44 -> 10.6.
//
// Plain CPython functions (METH_FASTCALL, positional arguments in the operators' order); every failed check raises
// RuntimeError like the reference's TORCH_CHECKs (kernels/ttt/ttt.cu:621-630, kernels/ttt_backward/ttt.cu:1507-1760).
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/python_variable.h>

#include <initializer_list>
#include <stdexcept>
#include <string>

#include "../../include/ttt_mlp_b200.h"

namespace {

constexpr int64_t CS = 64, F = 64, HID = 256;
constexpr at::ScalarType kBf = at::kBFloat16, kF32 = at::kFloat;

[[noreturn]] void fail(const std::string& msg) { throw std::runtime_error(msg); }

std::string shape_text(at::IntArrayRef s) {
  std::string o = "(";
  for (size_t i = 0; i < s.size(); ++i) o += (i ? ", " : "") + std::to_string(s[i]);
  return o + (s.size() == 1 ? ",)" : ")");
}

const char* dtype_text(at::ScalarType t) {
  return t == kBf ? "torch.bfloat16" : t == kF32 ? "torch.float32" : t == at::kByte ? "torch.uint8" : at::toString(t);
}

struct Call {
  int64_t B = 0, H = 0, NC = 0, cgs = 0, n = 0;
  c10::Device dev{c10::kCPU};

  // XQ, checkpoint_group_size and the first checkpoint tensor give the call's dimensions
  Call(PyObject* xq, PyObject* cgs_obj, PyObject* w1_checkpoints) {
    if (!THPVariable_Check(xq) || THPVariable_Unpack(xq).dim() != 5) fail("XQ must be 5-D [B, H, NC, 64, 64]");
    const at::Tensor& t = THPVariable_Unpack(xq);
    B = t.size(0); H = t.size(1); NC = t.size(2);
    if (t.size(4) != F) fail("head dimension must be 64");
    if (t.size(3) != CS) fail("mini-batch size must be 64");
    if (NC < 1) fail("need at least one mini-batch");
    PyObject* l = PyNumber_Long(cgs_obj);
    if (!l) throw std::logic_error("");        // the Python error is set
    cgs = PyLong_AsLongLong(l);
    Py_DECREF(l);
    if (cgs == -1 && PyErr_Occurred()) throw std::logic_error("");
    if (cgs < 1) fail("checkpoint_group_size must be >= 1");
    if (cgs > INT32_MAX) fail("checkpoint_group_size is too large");
    n = (NC + cgs - 1) / cgs;
    if (!THPVariable_Check(w1_checkpoints) || THPVariable_Unpack(w1_checkpoints).dim() != 5 ||
        THPVariable_Unpack(w1_checkpoints).size(2) != n)
      fail("checkpoint tensors must hold ceil(NC / checkpoint_group_size) = " + std::to_string(n) + " states");
    dev = t.device();
  }

  const at::Tensor& tensor(PyObject* o, const char* name, at::ScalarType dt) const {
    if (!THPVariable_Check(o)) fail(std::string(name) + " must be a tensor");
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor");
    if (t.device() != dev) fail(std::string(name) + " must be on " + dev.str());
    if (t.scalar_type() != dt)
      fail(std::string(name) + " must have dtype " + dtype_text(dt) + ", got " + dtype_text(t.scalar_type()));
    if (!t.is_contiguous()) fail(std::string(name) + " must be contiguous");
    return t;
  }
  void* ptr(PyObject* o, const char* name, at::ScalarType dt, std::initializer_list<int64_t> shape) const {
    const at::Tensor& t = tensor(o, name, dt);
    const at::IntArrayRef want(shape.begin(), shape.size());
    if (t.sizes() != want)
      fail(std::string(name) + " must have shape " + shape_text(want) + ", got " + shape_text(t.sizes()));
    return t.data_ptr();
  }
  float* f32(PyObject* o, const char* name, std::initializer_list<int64_t> shape) const {
    return static_cast<float*>(ptr(o, name, kF32, shape));
  }
  void* tok(PyObject* o, const char* name) const { return ptr(o, name, kBf, {B, H, NC, CS, F}); }
  void* eta(PyObject* o, const char* name) const {
    if (!THPVariable_Check(o)) fail(std::string(name) + " must be a tensor");
    const at::IntArrayRef s = THPVariable_Unpack(o).sizes();
    const bool r = s.size() == 4 || (s.size() == 5 && s[4] == 1);
    if (!r || s[0] != B || s[1] != H || s[2] != NC || s[3] != CS)
      fail(std::string(name) + " must have shape [B, H, NC, 64] or [B, H, NC, 64, 1], got " + shape_text(s));
    return tensor(o, name, kBf).data_ptr();
  }
  // items of a `final_state` sequence of `count` tensors, or nullptr for None
  static PyObject* items(PyObject* o, Py_ssize_t count, const char* what) {
    if (o == Py_None) return nullptr;
    PyObject* f = PySequence_Fast(o, "final_state must be a sequence");
    if (!f) throw std::logic_error("");
    if (PySequence_Fast_GET_SIZE(f) != count) {
      Py_DECREF(f);
      fail(std::string("final_state must be ") + what);
    }
    return f;
  }
  template <class Args>
  void dims(Args& a, PyObject* flags) const {
    a.B = static_cast<int32_t>(B);
    a.H = static_cast<int32_t>(H);
    a.NC = static_cast<int32_t>(NC);
    a.checkpoint_group_size = static_cast<int32_t>(cgs);
    a.num_checkpoints = static_cast<int32_t>(n);
    a.flags = static_cast<uint32_t>(PyLong_AsUnsignedLong(flags));
  }
};

struct Ref {        // a new reference, given back at the end of its scope
  PyObject* o;
  explicit Ref(PyObject* p) : o(p) {}
  ~Ref() { Py_XDECREF(o); }
};

template <class Args, class Fn>
PyObject* launch(const Call& c, Args& a, Fn fn, const char* what) {
  const c10::cuda::CUDAGuard guard(c.dev);
  void* stream = at::cuda::getCurrentCUDAStream(c.dev.index()).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS      // a call with the synchronise flag blocks
  rc = fn(&a, stream);
  Py_END_ALLOW_THREADS
  if (rc != 0)
    fail(std::string(what) + " failed (code " + std::to_string(rc) + "): " + ttt_b200_last_error());
  Py_RETURN_NONE;
}

template <class Fn>
PyObject* guarded(Fn fn) {
  try {
    return fn();
  } catch (const std::logic_error&) {      // a Python error is set already
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "internal error");
  return nullptr;
}

PyObject* wrong_count(const char* what) {
  PyErr_Format(PyExc_TypeError, "%s: wrong number of arguments", what);
  return nullptr;
}

// forward(XQ, XK, XV, last_eta, norm_weight, norm_bias, W1, b1, W2, b2, 4 checkpoint tensors, Out, cgs, final, flags)
PyObject* forward(PyObject*, PyObject* const* v, Py_ssize_t nargs) {
  if (nargs != 18) return wrong_count("forward");
  return guarded([&]() -> PyObject* {
    const Call c(v[0], v[15], v[10]);
    const int64_t B = c.B, H = c.H, n = c.n;
    ttt_b200_fwd_args a = {};
    a.XQ = c.tok(v[0], "XQ");
    a.XK = c.tok(v[1], "XK");
    a.XV = c.tok(v[2], "XV");
    a.last_eta = c.eta(v[3], "last_eta");
    a.ttt_norm_weight = c.f32(v[4], "ttt_norm_weight", {1, H, 1, F});
    a.ttt_norm_bias = c.f32(v[5], "ttt_norm_bias", {1, H, 1, F});
    a.W1 = c.f32(v[6], "W1", {B, H, F, HID});
    a.b1 = c.f32(v[7], "b1", {B, H, 1, HID});
    a.W2 = c.f32(v[8], "W2", {B, H, HID, F});
    a.b2 = c.f32(v[9], "b2", {B, H, 1, F});
    a.W1_checkpoints = c.f32(v[10], "W1_checkpoints", {B, H, n, F, HID});
    a.b1_checkpoints = c.f32(v[11], "b1_checkpoints", {B, H, n, 1, HID});
    a.W2_checkpoints = c.f32(v[12], "W2_checkpoints", {B, H, n, HID, F});
    a.b2_checkpoints = c.f32(v[13], "b2_checkpoints", {B, H, n, 1, F});
    a.Out = c.tok(v[14], "Out");
    const Ref fin(Call::items(v[16], 4, "(W1, b1, W2, b2)"));
    if (fin.o) {
      PyObject** f = PySequence_Fast_ITEMS(fin.o);
      a.W1_final = c.f32(f[0], "W1_final", {B, H, F, HID});
      a.b1_final = c.f32(f[1], "b1_final", {B, H, 1, HID});
      a.W2_final = c.f32(f[2], "W2_final", {B, H, HID, F});
      a.b2_final = c.f32(f[3], "b2_final", {B, H, 1, F});
    }
    c.dims(a, v[17]);
    return launch(c, a, ttt_b200_forward, "ttt_forward");
  });
}

// linear_forward(XQ, XK, XV, last_eta, norm_weight, norm_bias, W1, b1, 2 checkpoint tensors, Out, cgs, final, flags)
PyObject* linear_forward(PyObject*, PyObject* const* v, Py_ssize_t nargs) {
  if (nargs != 14) return wrong_count("linear_forward");
  return guarded([&]() -> PyObject* {
    const Call c(v[0], v[11], v[8]);
    const int64_t B = c.B, H = c.H, n = c.n;
    ttt_b200_linear_fwd_args a = {};
    a.XQ = c.tok(v[0], "XQ");
    a.XK = c.tok(v[1], "XK");
    a.XV = c.tok(v[2], "XV");
    a.last_eta = c.eta(v[3], "last_eta");
    a.ttt_norm_weight = c.f32(v[4], "ttt_norm_weight", {1, H, 1, F});
    a.ttt_norm_bias = c.f32(v[5], "ttt_norm_bias", {1, H, 1, F});
    a.W1 = c.f32(v[6], "W1", {B, H, F, F});
    a.b1 = c.f32(v[7], "b1", {B, H, 1, F});
    a.W1_checkpoints = c.f32(v[8], "W1_checkpoints", {B, H, n, F, F});
    a.b1_checkpoints = c.f32(v[9], "b1_checkpoints", {B, H, n, 1, F});
    a.Out = c.tok(v[10], "Out");
    const Ref fin(Call::items(v[12], 2, "(W1, b1)"));
    if (fin.o) {
      PyObject** f = PySequence_Fast_ITEMS(fin.o);
      a.W1_final = c.f32(f[0], "W1_final", {B, H, F, F});
      a.b1_final = c.f32(f[1], "b1_final", {B, H, 1, F});
    }
    c.dims(a, v[13]);
    return launch(c, a, ttt_b200_linear_forward, "ttt_linear_forward");
  });
}

// linear_backward(XQ, XK, XV, last_eta, norm_weight, norm_bias, 2 checkpoint tensors, dL/dW1_last, dL/db1_last, dL/dXQW,
//                 d_norm_weight, d_norm_bias, dL/dW1_init, dL/db1_init, d_eta, dXQ, dXK, dXV, cgs, scratch, flags)
PyObject* linear_backward(PyObject*, PyObject* const* v, Py_ssize_t nargs) {
  if (nargs != 22) return wrong_count("linear_backward");
  return guarded([&]() -> PyObject* {
    const Call c(v[0], v[19], v[6]);
    const int64_t B = c.B, H = c.H, n = c.n;
    ttt_b200_linear_bwd_args a = {};
    a.XQ = c.tok(v[0], "XQ");
    a.XK = c.tok(v[1], "XK");
    a.XV = c.tok(v[2], "XV");
    a.grad_L_XQW_mini_batch = c.tok(v[10], "grad_L_XQW_mini_batch");
    a.grad_L_XQ = c.tok(v[16], "grad_L_XQ");
    a.grad_L_XK = c.tok(v[17], "grad_L_XK");
    a.grad_L_XV = c.tok(v[18], "grad_L_XV");
    a.last_eta = c.eta(v[3], "last_eta");
    a.grad_L_last_eta = c.eta(v[15], "grad_L_last_eta");
    a.ttt_norm_weight = c.f32(v[4], "ttt_norm_weight", {1, H, 1, F});
    a.ttt_norm_bias = c.f32(v[5], "ttt_norm_bias", {1, H, 1, F});
    a.W1_checkpoints = c.f32(v[6], "W1_checkpoints", {B, H, n, F, F});
    a.b1_checkpoints = c.f32(v[7], "b1_checkpoints", {B, H, n, 1, F});
    a.grad_L_W1_last = c.f32(v[8], "grad_L_W1_last", {B, H, F, F});
    a.grad_L_b1_last = c.f32(v[9], "grad_L_b1_last", {B, H, 1, F});
    a.grad_L_ttt_norm_weight = c.f32(v[11], "grad_L_ttt_norm_weight", {B, H, 1, F});
    a.grad_L_ttt_norm_bias = c.f32(v[12], "grad_L_ttt_norm_bias", {B, H, 1, F});
    a.grad_L_W1_init = c.f32(v[13], "grad_L_W1_init", {B, H, F, F});
    a.grad_L_b1_init = c.f32(v[14], "grad_L_b1_init", {B, H, 1, F});
    const uint64_t need = ttt_b200_linear_backward_scratch_bytes(static_cast<int>(B), static_cast<int>(H),
                                                                 static_cast<int>(c.cgs));
    at::Tensor own;
    if (v[20] == Py_None) {
      own = at::empty({static_cast<int64_t>(need)}, at::TensorOptions().dtype(at::kByte).device(c.dev));
    } else {
      bool ok = THPVariable_Check(v[20]);
      if (ok) {
        own = THPVariable_Unpack(v[20]);
        ok = own.is_cuda() && own.device() == c.dev && own.is_contiguous() && own.scalar_type() == at::kByte &&
             static_cast<uint64_t>(own.numel()) >= need;
      }
      if (!ok)
        fail("scratch must be a contiguous uint8 CUDA tensor of at least " + std::to_string(need) + " bytes");
    }
    a.scratch = own.data_ptr();
    a.scratch_bytes = static_cast<uint64_t>(own.numel());
    c.dims(a, v[21]);
    return launch(c, a, ttt_b200_linear_backward, "ttt_linear_backward");
  });
}

// backward(the 42 tensors of ttt_backward in its order, cgs, flags)
PyObject* backward(PyObject*, PyObject* const* v, Py_ssize_t nargs) {
  if (nargs != 44) return wrong_count("backward");
  return guarded([&]() -> PyObject* {
    const Call c(v[0], v[42], v[6]);
    const int64_t B = c.B, H = c.H, n = c.n, g = c.cgs;
    ttt_b200_bwd_args a = {};
    a.XQ = c.tok(v[0], "XQ");
    a.XK = c.tok(v[1], "XK");
    a.XV = c.tok(v[2], "XV");
    a.last_eta = c.eta(v[3], "last_eta");
    a.ttt_norm_weight = c.f32(v[4], "ttt_norm_weight", {1, H, 1, F});
    a.ttt_norm_bias = c.f32(v[5], "ttt_norm_bias", {1, H, 1, F});
    a.W1_checkpoints = c.f32(v[6], "W1_checkpoints", {B, H, n, F, HID});
    a.b1_checkpoints = c.f32(v[7], "b1_checkpoints", {B, H, n, 1, HID});
    a.W2_checkpoints = c.f32(v[8], "W2_checkpoints", {B, H, n, HID, F});
    a.b2_checkpoints = c.f32(v[9], "b2_checkpoints", {B, H, n, 1, F});
    a.Out = c.tok(v[10], "Out");
    a.W1_init_group = c.f32(v[11], "W1_init_group", {B, H, g, F, HID});
    a.b1_init_group = c.f32(v[12], "b1_init_group", {B, H, g, 1, HID});
    a.W2_init_group = c.f32(v[13], "W2_init_group", {B, H, g, HID, F});
    a.b2_init_group = c.f32(v[14], "b2_init_group", {B, H, g, 1, F});
    a.x_hat_ln_group = c.ptr(v[15], "x_hat_ln_group", kBf, {B, H, g, CS, F});
    a.std_ln_group = c.f32(v[16], "std_ln_group", {B, H, g, CS, 1});
    a.X2_group = c.ptr(v[17], "X2_group", kBf, {B, H, g, CS, HID});
    a.Z1_group = c.ptr(v[18], "Z1_group", kBf, {B, H, g, CS, HID});
    a.Z1_bar_group = c.ptr(v[19], "Z1_bar_group", kBf, {B, H, g, CS, HID});
    a.X2_bar_group = c.ptr(v[20], "X2_bar_group", kBf, {B, H, g, CS, HID});
    a.grad_l_wrt_Z2_group = c.ptr(v[21], "grad_l_wrt_Z2_group", kBf, {B, H, g, CS, F});
    a.grad_l_wrt_Z1_group = c.ptr(v[22], "grad_l_wrt_Z1_group", kBf, {B, H, g, CS, HID});
    a.x_hat_fused_group = c.ptr(v[23], "x_hat_fused_group", kBf, {B, H, g, CS, F});
    a.grad_x_hat_fused_group = c.ptr(v[24], "grad_x_hat_fused_group", kBf, {B, H, g, CS, F});
    a.grad_output_fused_group = c.ptr(v[25], "grad_output_fused_group", kBf, {B, H, g, CS, F});
    a.std_fused_group = c.f32(v[26], "std_fused_group", {B, H, g, CS, 1});
    a.grad_L_W1_last = c.f32(v[27], "grad_L_W1_last", {B, H, F, HID});
    a.grad_L_b1_last = c.f32(v[28], "grad_L_b1_last", {B, H, 1, HID});
    a.grad_L_W2_last = c.f32(v[29], "grad_L_W2_last", {B, H, HID, F});
    a.grad_L_b2_last = c.f32(v[30], "grad_L_b2_last", {B, H, 1, F});
    a.grad_L_XQW_mini_batch = c.tok(v[31], "grad_L_XQW_mini_batch");
    a.grad_L_ttt_norm_weight = c.f32(v[32], "grad_L_ttt_norm_weight", {B, H, 1, F});
    a.grad_L_ttt_norm_bias = c.f32(v[33], "grad_L_ttt_norm_bias", {B, H, 1, F});
    a.grad_L_W1_init = c.f32(v[34], "grad_L_W1_init", {B, H, F, HID});
    a.grad_L_b1_init = c.f32(v[35], "grad_L_b1_init", {B, H, 1, HID});
    a.grad_L_W2_init = c.f32(v[36], "grad_L_W2_init", {B, H, HID, F});
    a.grad_L_b2_init = c.f32(v[37], "grad_L_b2_init", {B, H, 1, F});
    a.grad_L_last_eta = c.eta(v[38], "grad_L_last_eta");
    a.grad_L_XQ = c.tok(v[39], "grad_L_XQ");
    a.grad_L_XK = c.tok(v[40], "grad_L_XK");
    a.grad_L_XV = c.tok(v[41], "grad_L_XV");
    c.dims(a, v[43]);
    return launch(c, a, ttt_b200_backward, "ttt_backward");
  });
}

PyMethodDef kMethods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(forward)), METH_FASTCALL, nullptr},
    {"backward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(backward)), METH_FASTCALL, nullptr},
    {"linear_forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear_forward)), METH_FASTCALL, nullptr},
    {"linear_backward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear_backward)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_ttt_host", "Validation and launch of the TTT operators.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ttt_host() { return PyModule_Create(&kModule); }
