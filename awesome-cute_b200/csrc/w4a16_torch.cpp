// The call path from Python tensors to the C ABI (include/w4a16.h), compiled: what marlin.py's mul(), Layer.forward()
// and quantize_pack_device() do per call.
//
// A decode GEMM takes a few microseconds on the device, and a Python-level call (tensor attributes, the current-stream
// query, fifteen ctypes conversions) takes longer than that: 8.5 us for mul(), 18.6 us for Layer.forward() with its
// views and module look-ups, so small layers ran at the host's pace.  Here the tensors are read through torch's C++
// interface.  These functions only serve the calls that are right: whatever they cannot serve (arguments of another
// type, wrong shapes, CPU tensors) they leave to the Python code, which raises the reference's errors
// (gemm/marlin_gemm/marlin_gemm.cpp:19-56); an error code of the library goes back to it as a number.  The arithmetic and every
// check of the library itself stay behind the C ABI, whose entry points arrive as addresses (bind()), so that this file does
// not link against the library.
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <exception>

#include "../../include/w4a16.h"

namespace {

decltype(&w4a16_marlin_gemm) g_gemm = nullptr;
decltype(&w4a16_quantize_pack_device) g_pack = nullptr;

// Without the interpreter lock, which comes back also when an exception passes.
struct Unlocked {
  PyThreadState *state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

PyObject *bind(PyObject *, PyObject *const *args, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "bind(gemm, quantize_pack_device)");
    return nullptr;
  }
  g_gemm = reinterpret_cast<decltype(g_gemm)>(PyLong_AsVoidPtr(args[0]));
  g_pack = reinterpret_cast<decltype(g_pack)>(PyLong_AsVoidPtr(args[1]));
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

// `serve` with torch's exceptions turned into "not served" (the Python code then meets the same condition itself)
template <class F>
PyObject *guarded(F serve) {
  try {
    return serve();
  } catch (const std::exception &) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
}

// The reference's argument checks, short of the messages; true when the call may go to the library.
bool gemm_args(int64_t k, int64_t n, const at::Tensor &A, const at::Tensor &s, const at::Tensor &ws, int max_par, int &groupsize) {
  if (s.dim() < 1 || !A.is_cuda()) return false;
  const int64_t groups = s.size(0);
  if (groups < 1) return false;
  groupsize = groups == 1 ? -1 : (int)(k / groups);
  return (groups == 1 || groupsize * groups == k) && ws.numel() >= n / 128 * max_par && !((n | k) >> 31);
}

int call_gemm(const at::Tensor &A, const at::Tensor &B, const at::Tensor &C, const at::Tensor &s, const at::Tensor &ws, int64_t m,
              int64_t n, int64_t k, int groupsize, int thread_k, int thread_n, int sms, int max_par) {
  const c10::cuda::OptionalCUDAGuard guard(A.device());
  const int dev = A.get_device();
  void *stream = c10::cuda::getCurrentCUDAStream(dev).stream();
  const void *a = A.data_ptr(), *b = B.data_ptr(), *sp = s.data_ptr();
  void *c = C.data_ptr(), *w = ws.data_ptr();
  const Unlocked unlocked;   // (a full launch queue makes the launch wait for the GPU)
  return g_gemm(a, b, c, sp, (int)m, (int)n, (int)k, w, groupsize, dev, stream, thread_k, thread_n, sms, max_par);
}

// mul(A, B, C, s, workspace, thread_k, thread_n, sms, max_par) -> the library's code, or None when not served
PyObject *mul(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  if (nargs != 9) Py_RETURN_NONE;
  for (int i = 0; i < 5; ++i)
    if (!THPVariable_Check(args[i])) Py_RETURN_NONE;
  int v[4];
  for (int i = 0; i < 4; ++i) {
    if (!PyLong_Check(args[5 + i])) Py_RETURN_NONE;
    int over = 0;
    const long x = PyLong_AsLongAndOverflow(args[5 + i], &over);
    if (over || x != (int)x) Py_RETURN_NONE;
    v[i] = (int)x;
  }
  return guarded([&]() -> PyObject * {
    const at::Tensor &A = THPVariable_Unpack(args[0]), &B = THPVariable_Unpack(args[1]), &C = THPVariable_Unpack(args[2]),
                     &s = THPVariable_Unpack(args[3]), &ws = THPVariable_Unpack(args[4]);
    int groupsize;
    if (A.dim() < 2 || C.dim() < 2 || A.size(0) >> 31 || !gemm_args(A.size(1), C.size(1), A, s, ws, v[3], groupsize)) Py_RETURN_NONE;
    return PyLong_FromLong(call_gemm(A, B, C, s, ws, A.size(0), C.size(1), A.size(1), groupsize, v[0], v[1], v[2], v[3]));
  });
}

// forward(A, B, s, workspace) -> C [..., n], the library's code if that is an error, or None when not served.  A contiguous, as
// its view (-1, k) is what is read.
PyObject *forward(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  if (nargs != 4) Py_RETURN_NONE;
  for (int i = 0; i < 4; ++i)
    if (!THPVariable_Check(args[i])) Py_RETURN_NONE;
  return guarded([&]() -> PyObject * {
    const at::Tensor &A = THPVariable_Unpack(args[0]), &B = THPVariable_Unpack(args[1]), &s = THPVariable_Unpack(args[2]),
                     &ws = THPVariable_Unpack(args[3]);
    int groupsize;
    if (A.dim() < 1 || s.dim() < 2 || A.numel() == 0 || !A.is_contiguous()) Py_RETURN_NONE;
    const int64_t k = A.size(-1), n = s.size(1);
    if ((A.numel() / k) >> 31 || !gemm_args(k, n, A, s, ws, 16, groupsize)) Py_RETURN_NONE;
    c10::SmallVector<int64_t, 4> shape(A.sizes().begin(), A.sizes().end());
    shape.back() = n;
    at::Tensor C = at::empty(shape, A.options().requires_grad(false));
    if (const int rc = call_gemm(A, B, C, s, ws, A.numel() / k, n, k, groupsize, -1, -1, -1, 16)) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(C));
  });
}

// quantize_pack(weight_nk, scales, groupsize) -> (B, s_packed), the library's code if that is an error, or None when not served
PyObject *quantize_pack(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  if (nargs != 3 || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1]) || !PyLong_Check(args[2])) Py_RETURN_NONE;
  int over = 0;
  const long gs = PyLong_AsLongAndOverflow(args[2], &over);
  if (over || (gs != -1 && gs != 128)) Py_RETURN_NONE;
  return guarded([&]() -> PyObject * {
    const at::Tensor &w = THPVariable_Unpack(args[0]), &s = THPVariable_Unpack(args[1]);
    if (!w.is_cuda() || !s.is_cuda() || w.scalar_type() != at::kHalf || s.scalar_type() != at::kHalf || w.dim() != 2 ||
        !w.is_contiguous() || !s.is_contiguous())
      Py_RETURN_NONE;
    const int64_t n = w.size(0), k = w.size(1);
    if ((n | k) >> 31) Py_RETURN_NONE;
    const c10::cuda::OptionalCUDAGuard guard(w.device());
    at::Tensor B = at::empty({k / 16, 2 * n}, w.options().dtype(at::kInt).requires_grad(false));
    at::Tensor sp = at::empty({gs == -1 ? 1 : k / gs, n}, w.options().requires_grad(false));
    void *stream = c10::cuda::getCurrentCUDAStream(w.get_device()).stream();
    int rc;
    {
      const Unlocked unlocked;
      rc = g_pack(w.data_ptr(), s.data_ptr(), (int)k, (int)n, (int)gs, B.data_ptr(), sp.data_ptr(), stream);
    }
    if (rc) return PyLong_FromLong(rc);
    PyObject *b = THPVariable_Wrap(std::move(B));
    if (!b) return nullptr;
    PyObject *p = THPVariable_Wrap(std::move(sp));
    if (!p) {
      Py_DECREF(b);
      return nullptr;
    }
    PyObject *t = PyTuple_Pack(2, b, p);
    Py_DECREF(b);
    Py_DECREF(p);
    return t;
  });
}

#define FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f))
PyMethodDef methods[] = {{"bind", FAST(bind), METH_FASTCALL, nullptr},
                         {"mul", FAST(mul), METH_FASTCALL, nullptr},
                         {"forward", FAST(forward), METH_FASTCALL, nullptr},
                         {"quantize_pack", FAST(quantize_pack), METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_calls(void) { return PyModule_Create(&module); }
