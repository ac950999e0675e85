// The call path of the small ops (router, routing sort, top-k reduce) from Python: checks, output tensors and the
// C-ABI call in one native function.
//
// These ops take 3 to 10 us on the device and a call through Python and ctypes 9 to 18 us of host time, which therefore
// was what a caller waited for.  A function here serves the plain call - ordinary contiguous CUDA tensors on the current
// device, arguments of the plain Python types, no dispatch or function mode - and returns None for any other, which the
// Python form then handles or refuses as it always has.  A failing C call returns its status.
// Time of a call in a loop of calls: topk_softmax (one row) 11.3 -> 5.9 us, moe_align_block_size (131072 slots) 17.9 -> 10.4,
// moe_sum_reduce (one token) 8.9 -> 3.9.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/xkb200.h"

namespace {

decltype(&xkb_topk_softmax) g_topk_softmax;
decltype(&xkb_moe_align_block_size) g_align;
decltype(&xkb_moe_align_workspace_bytes) g_align_bytes;
decltype(&xkb_moe_sum_reduce) g_sum_reduce;

bool modes_active() {
  return at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set();
}

// The tensor behind `obj` if it is a plain one, else nullptr.
const at::Tensor* plain(PyObject* obj) {
  if (!THPVariable_CheckExact(obj)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(obj);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage() || !t.is_contiguous() || t.is_neg() ||
      t.is_conj() || t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                                              c10::DispatchKey::FuncTorchGradWrapper,
                                                              c10::DispatchKey::Functionalize})) ||
      t.get_device() != c10::cuda::current_device())
    return nullptr;
  return &t;
}

int code_of(at::ScalarType t) {   // -1: not a type of the library
  return t == at::kBFloat16 ? XKB_BF16 : t == at::kFloat ? XKB_F32 : t == at::kHalf ? XKB_F16 : -1;
}

bool plain_int(PyObject* obj, int64_t* value) {
  if (!PyLong_CheckExact(obj)) return false;
  int overflow = 0;
  *value = PyLong_AsLongLongAndOverflow(obj, &overflow);
  return overflow == 0;
}

void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// a tuple of new references (nullptr: an error is set)
template <typename... Objects>
PyObject* tuple_of(Objects... objects) {
  PyObject* const all[] = {objects...};
  PyObject* t = PyTuple_New(sizeof...(objects));
  bool ok = t != nullptr;
  for (size_t i = 0; i < sizeof...(objects); ++i) {
    ok = ok && all[i] != nullptr;
    if (t != nullptr) PyTuple_SET_ITEM(t, (Py_ssize_t)i, all[i]);
    else Py_XDECREF(all[i]);
  }
  if (!ok) { Py_XDECREF(t); return nullptr; }
  return t;
}

// topk_softmax(gating [M, E], topk, renormalize) -> (weights, ids)
PyObject* topk_softmax(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t topk;
  if (n != 3 || modes_active() || !plain_int(args[1], &topk) || !PyBool_Check(args[2])) Py_RETURN_NONE;
  const at::Tensor* g = plain(args[0]);
  if (g == nullptr || g->dim() != 2 || code_of(g->scalar_type()) < 0) Py_RETURN_NONE;
  const int64_t M = g->size(0), E = g->size(1);
  if (topk < 1 || topk > E || E > 0x7fffffff) Py_RETURN_NONE;
  at::Tensor w = at::empty({M, topk}, g->options().dtype(at::kFloat));
  at::Tensor ids = at::empty({M, topk}, g->options().dtype(at::kInt));
  const int code = code_of(g->scalar_type()), renorm = args[2] == Py_True;
  void* const stream = stream_of(*g);
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = g_topk_softmax(g->const_data_ptr(), code, static_cast<float*>(w.mutable_data_ptr()),
                          static_cast<int32_t*>(ids.mutable_data_ptr()), M, (int)E, (int)topk, renorm, stream);
  Py_END_ALLOW_THREADS
  if (status != 0) return PyLong_FromLong(status);
  return tuple_of(THPVariable_Wrap(std::move(w)), THPVariable_Wrap(std::move(ids)));
  END_HANDLE_TH_ERRORS
}

// moe_align_block_size(topk_ids, block_size, num_experts) -> (sorted_ids, expert_ids, num_post), untruncated
PyObject* moe_align_block_size(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  int64_t block, E;
  if (n != 3 || modes_active() || !plain_int(args[1], &block) || !plain_int(args[2], &E)) Py_RETURN_NONE;
  const at::Tensor* ids = plain(args[0]);
  if (ids == nullptr || ids->scalar_type() != at::kInt) Py_RETURN_NONE;
  const int64_t numel = ids->numel();
  if (block < 1 || block > (1 << 20) || E < 0 || E > 1024 || numel >= (1ll << 30)) Py_RETURN_NONE;
  const int64_t max_pad = numel + (E + 1) * (block - 1), max_blocks = (max_pad + block - 1) / block;
  if (max_blocks == 0) Py_RETURN_NONE;
  const at::TensorOptions opt = ids->options();
  at::Tensor sorted = at::empty({max_pad}, opt), experts = at::empty({max_blocks}, opt), post = at::empty({1}, opt), ws;
  void* ws_ptr = nullptr;
  int64_t ws_bytes = 0;
  if (numel > 8192) {   // up to there the sort takes no scratch memory
    ws_bytes = (g_align_bytes(numel, (int)E) + 3) / 4 * 4;
    ws = at::empty({ws_bytes / 4}, opt);
    ws_ptr = ws.mutable_data_ptr();
  }
  void* const stream = stream_of(*ids);
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = g_align(static_cast<const int32_t*>(ids->const_data_ptr()), numel, (int)E, (int)block, nullptr, 0,
                   static_cast<int32_t*>(sorted.mutable_data_ptr()), static_cast<int32_t*>(experts.mutable_data_ptr()),
                   static_cast<int32_t*>(post.mutable_data_ptr()), nullptr, ws_ptr, ws_bytes, stream);
  Py_END_ALLOW_THREADS
  if (status != 0) return PyLong_FromLong(status);
  return tuple_of(THPVariable_Wrap(std::move(sorted)), THPVariable_Wrap(std::move(experts)),
                  THPVariable_Wrap(std::move(post)));
  END_HANDLE_TH_ERRORS
}

// moe_sum_reduce(y [M, top_k, H], w [M, top_k] or None, routed_scaling_factor) -> [M, H]
PyObject* moe_sum_reduce(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 3 || modes_active() || !PyFloat_CheckExact(args[2])) Py_RETURN_NONE;
  const at::Tensor* y = plain(args[0]);
  if (y == nullptr || y->dim() != 3 || (y->scalar_type() != at::kBFloat16 && y->scalar_type() != at::kFloat)) Py_RETURN_NONE;
  const int64_t M = y->size(0), top_k = y->size(1), H = y->size(2);
  if (top_k > 0x7fffffff) Py_RETURN_NONE;
  const at::Tensor* w = nullptr;
  if (args[1] != Py_None) {
    w = plain(args[1]);
    if (w == nullptr || w->dim() != 2 || w->size(0) != M || w->size(1) != top_k || w->get_device() != y->get_device() ||
        (w->scalar_type() != at::kBFloat16 && w->scalar_type() != at::kFloat))
      Py_RETURN_NONE;
  }
  at::Tensor out = at::empty({M, H}, y->options());
  const int y_code = code_of(y->scalar_type()), w_code = w == nullptr ? XKB_F32 : code_of(w->scalar_type());
  const float factor = (float)PyFloat_AS_DOUBLE(args[2]);
  void* const stream = stream_of(*y);
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = g_sum_reduce(y->const_data_ptr(), y_code, w == nullptr ? nullptr : w->const_data_ptr(), w_code,
                        out.mutable_data_ptr(), y_code, M, (int)top_k, H, factor, stream);
  Py_END_ALLOW_THREADS
  if (status != 0) return PyLong_FromLong(status);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// bind(topk_softmax, align, align_workspace_bytes, sum_reduce): the library's functions, as addresses
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 4) { PyErr_SetString(PyExc_TypeError, "bind: four addresses expected"); return nullptr; }
  void* p[4];
  for (int i = 0; i < 4; ++i) {
    p[i] = PyLong_AsVoidPtr(args[i]);
    if (p[i] == nullptr) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind: null address");
      return nullptr;
    }
  }
  g_topk_softmax = reinterpret_cast<decltype(g_topk_softmax)>(p[0]);
  g_align = reinterpret_cast<decltype(g_align)>(p[1]);
  g_align_bytes = reinterpret_cast<decltype(g_align_bytes)>(p[2]);
  g_sum_reduce = reinterpret_cast<decltype(g_sum_reduce)>(p[3]);
  Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyMethodDef method(const char* name) {
  return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(F)), METH_FASTCALL, nullptr};
}
PyMethodDef g_methods[] = {method<topk_softmax>("topk_softmax"), method<moe_align_block_size>("moe_align_block_size"),
                           method<moe_sum_reduce>("moe_sum_reduce"), method<bind>("bind"), {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_torch_calls", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_calls() { return PyModule_Create(&g_module); }
