// The host side of a call from Python: checks, outputs, workspace and the library's entry point in one native call.
//
// What bounds a call of a short sequence is the time to enqueue it: a forward of 8 heads of 64 rows took 32.5 us, its kernels 15.5.  The
// interpreter's checks of the tensors' attributes, its three allocations and the conversion of 26 arguments by ctypes took 15 of them.
// With this code 17.4 us; a training step of 2 heads of 64 rows fp32 158 -> 110 us, of which 79 are autograd's own, of the dot-product-sum
// of 16 heads of 1024 rows 172 -> 125.  These functions take the calls that need no help: five or eight contiguous, 16-byte aligned CUDA tensors of one
// shape, type and device, which is the current one.  For any other call they return None and change nothing: the Python code then
// copies, converts, switches devices or raises, as its own checks say.
//
// An extension module rather than a dispatcher operator: the autograd functions, their hooks and saved tensors stay where they are.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <climits>
#include <map>

#include "tritt.h"

namespace {

enum { kTdpFwd = TRITT_OP_TDP_FWD, kTdpBwd = TRITT_OP_TDP_BWD, kDpsFwd = TRITT_OP_DPS_FWD, kDpsBwd = TRITT_OP_DPS_BWD };
constexpr int kDevices = 64;
constexpr int kNotPlain = INT_MIN;   // no code of the library's

// Everything below is read and written with the interpreter's lock held.
struct Entries {   // (the addresses come from Python, which has loaded the library)
  decltype(&tritt_tdp_fwd) tdp_fwd;
  decltype(&tritt_tdp_bwd) tdp_bwd;
  decltype(&tritt_dps_fwd) dps_fwd;
  decltype(&tritt_dps_bwd) dps_bwd;
  decltype(&tritt_dps_bwd_saved) dps_bwd_saved;
  decltype(&tritt_workspace_bytes_flags) workspace_bytes;
  decltype(&tritt_tdp_fwd_workspace) tdp_fwd_workspace;
} lib{};
volatile int* status_words[kDevices] = {};
std::map<std::array<int, 12>, size_t> workspace_sizes;

// The call's tensors have one shape [B, N, T, D], type and device.
struct Shape {
  int B, N, T, D, dtype, device;
  at::ScalarType type;
};

bool usable(const at::Tensor& t) {
  return t.defined() && !t.unsafeGetTensorImpl()->is_python_dispatch() && t.layout() == at::kStrided && t.is_cuda() && t.has_storage() &&
         t.is_contiguous() && !t.is_neg() && t.numel() > 0;
}
bool aligned(const void* p) { return p != nullptr && (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

bool read_shape(const at::Tensor& q, Shape& s) {
  if (!usable(q) || q.dim() != 4) return false;
  s.type = q.scalar_type();
  s.dtype = s.type == at::kFloat ? TRITT_F32 : s.type == at::kHalf ? TRITT_F16 : s.type == at::kBFloat16 ? TRITT_BF16 : -1;
  for (int i = 0; i < 4; ++i)
    if (q.size(i) > INT_MAX) return false;
  s.B = (int)q.size(0);
  s.N = (int)q.size(1);
  s.T = (int)q.size(2);
  s.D = (int)q.size(3);
  s.device = q.device().index();
  return s.dtype >= 0 && (s.D & (s.D - 1)) == 0 && s.device >= 0 && s.device < kDevices && s.device == c10::cuda::current_device();
}

// (not a subclass: what is allocated like one of those is of its type)
bool is_tensor(PyObject* o) { return (PyObject*)Py_TYPE(o) == THPVariableClass; }

// Address of a tensor of the call's shape; null: not one.
void* operand(PyObject* o, const Shape& s) {
  if (!is_tensor(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!usable(t) || t.dim() != 4 || t.size(0) != s.B || t.size(1) != s.N || t.size(2) != s.T || t.size(3) != s.D ||
      t.scalar_type() != s.type || t.device().index() != s.device)
    return nullptr;
  void* p = t.data_ptr();
  return aligned(p) ? p : nullptr;
}

bool read_int(PyObject* o, int none, int& v) {
  if (o == Py_None) {
    v = none;
    return none >= 0;
  }
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  const long x = PyLong_AsLongAndOverflow(o, &overflow);
  if (overflow || x > INT_MAX || x < INT_MIN) return false;
  v = (int)x;
  return true;
}
bool read_float(PyObject* o, float& v) {
  if (!PyFloat_CheckExact(o)) return false;
  v = (float)PyFloat_AS_DOUBLE(o);
  return true;
}

// The scalars of a call, from argument i on: scale, causal, flags, windows (four, or the one of the dot-product-sum).
struct Scalars {
  float scale;
  int causal, flags, w[4];
  int* status;
};
bool read_scalars(PyObject* const* a, int op, const Shape& s, Scalars& c) {
  if (!read_float(a[0], c.scale) || !PyBool_Check(a[1]) || !read_int(a[2], -1, c.flags)) return false;
  c.causal = a[1] == Py_True;
  const int windows = op < kDpsFwd ? 4 : 1;
  for (int i = 0; i < windows; ++i)
    if (!read_int(a[3 + i], op < kDpsFwd ? s.T : -1, c.w[i])) return false;
  // (a kernel of an earlier call gave up, or the word is not there yet: Python reports, or makes it)
  c.status = const_cast<int*>(status_words[s.device]);
  return lib.tdp_fwd != nullptr && c.status != nullptr && *status_words[s.device] == 0;
}

size_t workspace_size(int op, const Shape& s, const Scalars& c) {
  std::array<int, 12> key = {op, s.B, s.N, s.T, s.D, s.dtype, op < kDpsFwd ? c.flags : 0, 0, 0, 0, 0, 0};
  if (op == kTdpFwd) {   // (what the forward makes use of depends on the mask)
    key[7] = c.causal;
    for (int i = 0; i < 4; ++i) key[8 + i] = c.w[i];
  }
  const auto it = workspace_sizes.find(key);
  if (it != workspace_sizes.end()) return it->second;
  if (workspace_sizes.size() >= 1024) workspace_sizes.clear();
  const size_t n = op == kTdpFwd ? lib.tdp_fwd_workspace(s.B, s.N, s.T, s.D, s.dtype, c.causal, c.w[0], c.w[1], c.w[2], c.w[3], 1, c.flags)
                                 : lib.workspace_bytes(op, s.B, s.N, s.T, s.D, s.dtype, key[6]);
  return workspace_sizes[key] = n < 256 ? 256 : n;
}

// The interpreter's lock is not held while device memory is allocated (which may wait for the device) and kernels are launched.
struct Unlocked {
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

// An output's address; null: something stands in for plain tensors (a mode), Python's own calls shall meet it
void* fresh(const at::Tensor& t) {
  if (!usable(t)) return nullptr;
  void* p = t.data_ptr();
  return aligned(p) ? p : nullptr;
}

PyObject* wrap_all(at::Tensor* t, int n) {
  PyObject* r = PyTuple_New(n);
  if (!r) return nullptr;
  for (int i = 0; i < n; ++i) {
    PyObject* o = THPVariable_Wrap(t[i]);
    if (!o) {
      Py_DECREF(r);
      return nullptr;
    }
    PyTuple_SET_ITEM(r, i, o);
  }
  return r;
}

// forward(op, q, k1, k2, v1, v2, scale, causal, flags, windows...) -> (o, log-sum-exp, workspace), the library's error code, or None
PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int op;
  if (n < 10 || !read_int(a[0], -1, op) || n != (op < kDpsFwd ? 13 : 10) || !is_tensor(a[1])) Py_RETURN_NONE;
  Shape s;
  Scalars c;
  const at::Tensor& q = THPVariable_Unpack(a[1]);
  if (!read_shape(q, s) || !read_scalars(a + 6, op, s, c)) Py_RETURN_NONE;
  void* in[5];
  for (int i = 0; i < 5; ++i)
    if (!(in[i] = operand(a[1 + i], s))) Py_RETURN_NONE;
  const size_t bytes = workspace_size(op, s, c);
  at::Tensor out[3];
  int rc;
  {
    Unlocked unlocked;
    out[0] = at::empty_like(q);
    out[1] = at::empty({s.B, s.N, s.T}, q.options().dtype(at::kFloat));
    out[2] = at::empty({(int64_t)bytes}, q.options().dtype(at::kByte));
    void *const o = fresh(out[0]), *const l = fresh(out[1]), *const w = fresh(out[2]);
    void* const stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)s.device).stream();
    if (!o || !l || !w)
      rc = kNotPlain;
    else if (op == kTdpFwd)
      rc = lib.tdp_fwd(in[0], in[1], in[2], in[3], in[4], o, (float*)l, s.B, s.N, s.T, s.D, s.dtype, c.scale, c.causal, c.w[0], c.w[1],
                       c.w[2], c.w[3], 1, 0, w, bytes, c.status, c.flags, stream);
    else
      rc = lib.dps_fwd(in[0], in[1], in[2], in[3], in[4], o, (float*)l, s.B, s.N, s.T, s.D, s.dtype, c.scale, c.causal, c.w[0], w, bytes,
                       c.status, c.flags, stream);
  }
  if (rc == kNotPlain) Py_RETURN_NONE;
  if (rc != 0) return PyLong_FromLong(rc);
  return wrap_all(out, op == kTdpFwd ? 2 : 3);
  END_HANDLE_TH_ERRORS
}

// backward(op, q, k1, k2, v1, v2, o, do, log-sum-exp, scale, causal, flags, windows..., the forward's workspace or None)
// -> the five gradients, the library's error code, or None
PyObject* backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int op;
  if (n < 14 || !read_int(a[0], -1, op) || n != (op < kDpsFwd ? 17 : 14) || !is_tensor(a[1]) || !is_tensor(a[8]))
    Py_RETURN_NONE;
  Shape s;
  Scalars c;
  const at::Tensor& q = THPVariable_Unpack(a[1]);
  if (!read_shape(q, s) || !read_scalars(a + 9, op, s, c)) Py_RETURN_NONE;
  void* in[7];
  for (int i = 0; i < 7; ++i)
    if (!(in[i] = operand(a[1 + i], s))) Py_RETURN_NONE;
  const at::Tensor& lse = THPVariable_Unpack(a[8]);
  if (!usable(lse) || lse.dim() != 3 || lse.size(0) != s.B || lse.size(1) != s.N || lse.size(2) != s.T || lse.scalar_type() != at::kFloat ||
      lse.device().index() != s.device || !aligned(lse.data_ptr()))
    Py_RETURN_NONE;
  const void* saved = nullptr;
  size_t saved_bytes = 0;
  if (a[n - 1] != Py_None) {
    if (op != kDpsBwd || !is_tensor(a[n - 1])) Py_RETURN_NONE;
    const at::Tensor& w = THPVariable_Unpack(a[n - 1]);
    if (!usable(w) || w.scalar_type() != at::kByte || w.device().index() != s.device) Py_RETURN_NONE;
    saved = w.data_ptr();
    saved_bytes = (size_t)w.numel();
  }
  const float* const l = (const float*)lse.data_ptr();
  const size_t bytes = workspace_size(op, s, c);
  at::Tensor out[6];
  int rc = 0;
  {
    Unlocked unlocked;
    void* p[6];
    for (int i = 0; i < 6; ++i) {
      out[i] = i < 5 ? at::empty_like(q) : at::empty({(int64_t)bytes}, q.options().dtype(at::kByte));
      if (!(p[i] = fresh(out[i]))) rc = kNotPlain;
    }
    void* const stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)s.device).stream();
    if (rc == kNotPlain)
      ;
    else if (op == kTdpBwd)
      rc = lib.tdp_bwd(in[0], in[1], in[2], in[3], in[4], in[5], in[6], l, p[0], p[1], p[2], p[3], p[4], s.B, s.N, s.T, s.D, s.dtype,
                       c.scale, c.causal, c.w[0], c.w[1], c.w[2], c.w[3], 1, 0, p[5], bytes, c.status, c.flags, stream);
    else if (!saved)
      rc = lib.dps_bwd(in[0], in[1], in[2], in[3], in[4], in[5], in[6], l, p[0], p[1], p[2], p[3], p[4], s.B, s.N, s.T, s.D, s.dtype,
                       c.scale, c.causal, c.w[0], p[5], bytes, c.status, c.flags, stream);
    else
      rc = lib.dps_bwd_saved(in[0], in[1], in[2], in[3], in[4], in[5], in[6], l, p[0], p[1], p[2], p[3], p[4], s.B, s.N, s.T, s.D, s.dtype,
                             c.scale, c.causal, c.w[0], p[5], bytes, saved, saved_bytes, c.status, c.flags, stream);
  }
  if (rc == kNotPlain) Py_RETURN_NONE;
  if (rc != 0) return PyLong_FromLong(rc);
  return wrap_all(out, 5);
  END_HANDLE_TH_ERRORS
}

// init(addresses of tritt_tdp_fwd, tritt_tdp_bwd, tritt_dps_fwd, tritt_dps_bwd, tritt_dps_bwd_saved, tritt_workspace_bytes_flags,
// tritt_tdp_fwd_workspace)
PyObject* init(PyObject*, PyObject* args) {
  unsigned long long f[7];
  if (!PyArg_ParseTuple(args, "KKKKKKK", f, f + 1, f + 2, f + 3, f + 4, f + 5, f + 6)) return nullptr;
  lib = {(decltype(lib.tdp_fwd))f[0],       (decltype(lib.tdp_bwd))f[1],         (decltype(lib.dps_fwd))f[2],          (decltype(lib.dps_bwd))f[3],
         (decltype(lib.dps_bwd_saved))f[4], (decltype(lib.workspace_bytes))f[5], (decltype(lib.tdp_fwd_workspace))f[6]};
  Py_RETURN_NONE;
}

// set_status(device, address of its status word)
PyObject* set_status(PyObject*, PyObject* args) {
  int device;
  unsigned long long address;
  if (!PyArg_ParseTuple(args, "iK", &device, &address)) return nullptr;
  if (device >= 0 && device < kDevices) status_words[device] = (volatile int*)address;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"init", init, METH_VARARGS, nullptr},
                         {"set_status", set_status, METH_VARARGS, nullptr},
                         {"forward", (PyCFunction)(void (*)(void))forward, METH_FASTCALL, nullptr},
                         {"backward", (PyCFunction)(void (*)(void))backward, METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  PyObject* m = PyModule_Create(&module);
  // (the version whose headers this was compiled with: objects' layouts are its own)
  if (m && PyModule_AddStringConstant(m, "torch_version", TRITT_TORCH_VERSION) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
