// _dxb_call: whole eager calls, from tensors to a launched kernel: the registered GEMM kernels, and the
// two ends of a weight's life (packing and unpacking).
//
// A GEMM of this package lasts 5 to 15 us, and a call made of Python statements (attribute
// reads, data_ptr(), dictionary look-ups, torch.empty) costs about as much host time as that, so
// chains of small calls were bound by the host: 13.4 us per call against 5.5 us of GPU time at one
// token.  call() does the same steps natively.  It serves the plain case only -- tensors of the right
// types, contiguous, on the current device, weight already repacked, workspace already there -- and
// returns None for everything else, errors included, which ops.py then handles as before.
//
//   bind(gemm_ex, scratch_bytes, capture_id, quantize, quantize_scratch_bytes, dequantize_ex, relaid)
//                                              addresses in the loaded library, the cache of repacked weights
//   set_workspace(device, stream, ptr, bytes, scratch, scratch_bytes)
//                                              what ops.py holds for that stream (0 bytes: nothing)
//   call(bits, x, qweight, scales, zeros, bias, group_size, max_ctas, layout, epilogue, pinned) -> Tensor | None
//   quantize(weight, bits, group_size, symmetric) -> (qweight, scales, zeros | None) | None
//   dequantize(qweight, scales, zeros, group_size, bits, layout) -> Tensor | None
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <unordered_map>

#include "../../include/dexter_b200.h"

namespace {

using GemmEx = decltype(&dxb_wq_gemm_ex);
using GemmScratch = decltype(&dxb_scratch_bytes);
using CaptureId = decltype(&dxb_capture_id);
using Quantize = decltype(&dxb_quantize);
using ScratchBytes = decltype(&dxb_quantize_scratch_bytes);
using Dequantize = decltype(&dxb_dequantize_ex);

GemmEx g_gemm = nullptr;
GemmScratch g_gemm_scratch = nullptr;
CaptureId g_capture_id = nullptr;
Quantize g_quantize = nullptr;
ScratchBytes g_scratch_bytes = nullptr;
Dequantize g_dequantize = nullptr;
// id(qweight) -> (weak reference, version, repacked copy or None, address, streams that may read it, ...), owned by ops.py
PyObject* g_relaid = nullptr;

struct Mix {
  size_t operator()(const std::pair<uint64_t, uint64_t>& k) const {
    return static_cast<size_t>((k.first ^ (k.second * 0x9E3779B97F4A7C15ull)) * 0xFF51AFD7ED558CCDull);
  }
};
// All state below is only touched with the interpreter lock held.
struct Workspace {
  void* ptr;  // for calls that leave counters and partial sums alone
  size_t bytes;
  void* scratch;  // for the others, outside captures
  size_t scratch_bytes;
};
std::unordered_map<std::pair<uint64_t, uint64_t>, Workspace, Mix> g_workspaces;  // (device, stream)
std::unordered_map<std::pair<uint64_t, uint64_t>, size_t, Mix> g_need;           // (shape words) -> dxb_scratch_bytes

template <class F>
F at_address(unsigned long long v) { return reinterpret_cast<F>(static_cast<uintptr_t>(v)); }

PyObject* bind(PyObject*, PyObject* args) {
  unsigned long long gemm = 0, gemm_scratch = 0, capture_id = 0, quantize = 0, scratch = 0, dequantize = 0;
  PyObject* relaid = nullptr;
  if (!PyArg_ParseTuple(args, "KKKKKKO!", &gemm, &gemm_scratch, &capture_id, &quantize, &scratch, &dequantize, &PyDict_Type,
                        &relaid))
    return nullptr;
  g_gemm = at_address<GemmEx>(gemm);
  g_gemm_scratch = at_address<GemmScratch>(gemm_scratch);
  g_capture_id = at_address<CaptureId>(capture_id);
  g_quantize = at_address<Quantize>(quantize);
  g_scratch_bytes = at_address<ScratchBytes>(scratch);
  g_dequantize = at_address<Dequantize>(dequantize);
  Py_INCREF(relaid);
  Py_XSETREF(g_relaid, relaid);
  Py_RETURN_NONE;
}

PyObject* set_workspace(PyObject*, PyObject* args) {
  int device = 0;
  unsigned long long stream = 0, ptr = 0, bytes = 0, scratch = 0, scratch_bytes = 0;
  if (!PyArg_ParseTuple(args, "iKKKKK", &device, &stream, &ptr, &bytes, &scratch, &scratch_bytes)) return nullptr;
  g_workspaces[{static_cast<uint64_t>(device), stream}] = {at_address<void*>(ptr), static_cast<size_t>(bytes),
                                                           at_address<void*>(scratch), static_cast<size_t>(scratch_bytes)};
  Py_RETURN_NONE;
}

// A plain torch.Tensor or Parameter (no subclass that might want to see the call itself).
const at::Tensor* plain_tensor(PyObject* o) {
  return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr;
}

// Looks an int4 weight up in the cache of repacked copies: false when ops.py has not seen it yet, it has changed
// since, or this stream has not waited for the copy; else `copy` is its repacked copy, or nullptr where its
// shape takes none.
bool repacked(PyObject* obj, const at::Tensor& q, cudaStream_t stream, const at::Tensor** copy) {
  *copy = nullptr;
  PyObject* key = PyLong_FromVoidPtr(obj);
  if (!key) { PyErr_Clear(); return false; }
  PyObject* hit = PyDict_GetItemWithError(g_relaid, key);  // borrowed
  Py_DECREF(key);
  if (!hit || !PyTuple_CheckExact(hit) || PyTuple_GET_SIZE(hit) < 5) { PyErr_Clear(); return false; }
  if (PyWeakref_GetObject(PyTuple_GET_ITEM(hit, 0)) != obj) return false;
  if (q.is_inference() || PyLong_AsUnsignedLong(PyTuple_GET_ITEM(hit, 1)) != q._version() ||
      PyLong_AsVoidPtr(PyTuple_GET_ITEM(hit, 3)) != q.const_data_ptr()) {
    PyErr_Clear();
    return false;
  }
  PyObject* item = PyTuple_GET_ITEM(hit, 2);
  if (item == Py_None) return true;
  PyObject* raw = PyLong_FromVoidPtr(stream);
  if (!raw) { PyErr_Clear(); return false; }
  const int known = PySet_Contains(PyTuple_GET_ITEM(hit, 4), raw);
  Py_DECREF(raw);
  if (known != 1) { PyErr_Clear(); return false; }
  if (!THPVariable_CheckExact(item)) return false;
  *copy = &THPVariable_Unpack(item);
  return true;
}

PyObject* call(PyObject* const* a, Py_ssize_t n_args) {
  if (n_args != 11) {
    PyErr_SetString(PyExc_TypeError, "_dxb_call.call takes exactly 11 arguments");
    return nullptr;
  }
  if (!g_gemm) Py_RETURN_NONE;
  const long bits = PyLong_AsLong(a[0]), group = PyLong_AsLong(a[6]), max_ctas = PyLong_AsLong(a[7]);
  const long layout = PyLong_AsLong(a[8]), epilogue = PyLong_AsLong(a[9]);
  if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
  // A caller that came through the registry honours its DEXTER_KERNEL pin, which is parsed there.
  if (a[10] == Py_True && std::getenv("DEXTER_KERNEL") != nullptr) Py_RETURN_NONE;
  const at::Tensor *x = plain_tensor(a[1]), *q = plain_tensor(a[2]), *s = plain_tensor(a[3]);
  const at::Tensor *z = a[4] == Py_None ? nullptr : plain_tensor(a[4]);
  const at::Tensor *b = a[5] == Py_None ? nullptr : plain_tensor(a[5]);
  if (!x || !q || !s || (a[4] != Py_None && !z) || (a[5] != Py_None && !b)) Py_RETURN_NONE;
  if (!x->is_cuda() || x->scalar_type() != at::kBFloat16 || s->scalar_type() != at::kBFloat16 ||
      q->scalar_type() != at::kByte || q->dim() != 2 || s->dim() != 2 || (z && z->scalar_type() != at::kBFloat16) ||
      (b && b->scalar_type() != at::kBFloat16))
    Py_RETURN_NONE;
  const auto dev = x->device();
  if (dev.index() != c10::cuda::current_device() || q->device() != dev || s->device() != dev ||
      (z && z->device() != dev) || (b && b->device() != dev))
    Py_RETURN_NONE;
  if (!q->is_contiguous() || !s->is_contiguous() || (z && !z->is_contiguous()) || (b && !b->is_contiguous()))
    Py_RETURN_NONE;
  const int64_t n = q->size(1), k = bits == 4 ? 2 * q->size(0) : q->size(0);
  const int64_t cells = group > 0 ? k / group * n : 0;
  if (s->numel() < cells || (z && z->numel() < cells) || (b && b->numel() < n)) Py_RETURN_NONE;
  const int64_t dims = x->dim();
  if (dims < 1 || x->size(dims - 1) != k || k <= 0) Py_RETURN_NONE;
  int64_t m, ldx;
  if (dims == 2) {
    m = x->size(0);
    ldx = x->stride(0);
    if (x->stride(1) != 1 || ldx % 8) Py_RETURN_NONE;
  } else {
    if (!x->is_contiguous() || k % 8) Py_RETURN_NONE;
    m = x->numel() / k;
    ldx = k;
  }
  const void* xp = x->const_data_ptr();
  if (m <= 0 || reinterpret_cast<uintptr_t>(xp) % 16 || m > INT32_MAX || n > INT32_MAX || k > INT32_MAX) Py_RETURN_NONE;

  dxb_gemm_opts opts = {};
  opts.weight_layout = static_cast<int>(layout);
  opts.epilogue = static_cast<int>(epilogue);
  opts.max_ctas = static_cast<int>(max_ctas);
  const auto stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  if (layout == DXB_LAYOUT_DEXTER && bits == 4) {
    const at::Tensor* copy;
    if (!repacked(a[2], *q, stream, &copy)) Py_RETURN_NONE;
    if (copy) {
      q = copy;
      opts.weight_layout = DXB_LAYOUT_B200;
    }
  }

  const auto ws = g_workspaces.find({static_cast<uint64_t>(dev.index()), reinterpret_cast<uint64_t>(stream)});
  if (ws == g_workspaces.end()) Py_RETURN_NONE;
  const std::pair<uint64_t, uint64_t> shape{(static_cast<uint64_t>(m) << 32) | static_cast<uint64_t>(n),
                                            (static_cast<uint64_t>(k) << 32) | (static_cast<uint64_t>(max_ctas & 0xFFFFFF) << 8) |
                                                static_cast<uint64_t>(bits)};
  auto need = g_need.find(shape);
  if (need == g_need.end()) {
    if (g_need.size() > 4096) g_need.clear();
    need = g_need.emplace(shape, g_gemm_scratch(static_cast<int>(m), static_cast<int>(n), static_cast<int>(k),
                                                static_cast<int>(bits), static_cast<int>(max_ctas))).first;
  }
  void* space = ws->second.ptr;
  size_t space_bytes = ws->second.bytes;
  if (need->second > 0) {  // a captured call gets scratch of its graph's own, from ops.py
    if (ws->second.scratch_bytes < need->second || g_capture_id(stream) != 0) Py_RETURN_NONE;
    space = ws->second.scratch;
    space_bytes = ws->second.scratch_bytes;
  }

  at::Tensor out;
  if (dims == 2) {
    out = at::empty({m, n}, x->options());
  } else {
    auto sizes = x->sizes().vec();
    sizes.back() = n;
    out = at::empty(sizes, x->options());
  }
  const int rc = g_gemm(static_cast<int>(bits), xp, ldx, q->const_data_ptr(), s->const_data_ptr(),
                        z ? z->const_data_ptr() : nullptr, b ? b->const_data_ptr() : nullptr, out.mutable_data_ptr(), n,
                        static_cast<int>(m), static_cast<int>(n), static_cast<int>(k), static_cast<int>(group),
                        space, space_bytes, &opts, stream);
  if (rc != DXB_OK) Py_RETURN_NONE;  // the general path reports it
  return THPVariable_Wrap(std::move(out));
}

PyObject* quantize(PyObject* const* a, Py_ssize_t n_args) {
  if (n_args != 4) {
    PyErr_SetString(PyExc_TypeError, "_dxb_call.quantize takes exactly 4 arguments");
    return nullptr;
  }
  const at::Tensor* w = plain_tensor(a[0]);
  const long bits = PyLong_AsLong(a[1]), group = PyLong_AsLong(a[2]);
  if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
  const bool symmetric = a[3] == Py_True;
  if (!g_quantize || !w || (bits != 4 && bits != 8) || !w->is_cuda() || w->scalar_type() != at::kBFloat16 || w->dim() != 2 ||
      !w->is_contiguous() || w->device().index() != c10::cuda::current_device())
    Py_RETURN_NONE;
  const int64_t n = w->size(0), k = w->size(1);
  if (n <= 0 || k <= 0 || group <= 0 || k % group || n > INT32_MAX || k > INT32_MAX) Py_RETURN_NONE;
  const auto bytes = w->options().dtype(at::kByte);
  at::Tensor q = at::empty({bits == 4 ? k / 2 : k, n}, bytes), s = at::empty({k / group, n}, w->options()), z, scratch;
  if (!symmetric) z = at::empty({k / group, n}, w->options());
  const size_t need = g_scratch_bytes(static_cast<int>(n), static_cast<int>(k), static_cast<int>(group), static_cast<int>(bits));
  if (need) scratch = at::empty({static_cast<int64_t>(need)}, bytes);
  const auto stream = c10::cuda::getCurrentCUDAStream(w->device().index()).stream();
  const int rc = g_quantize(w->const_data_ptr(), q.mutable_data_ptr(), s.mutable_data_ptr(),
                            symmetric ? nullptr : z.mutable_data_ptr(), need ? scratch.mutable_data_ptr() : nullptr,
                            static_cast<int>(n), static_cast<int>(k), static_cast<int>(group), static_cast<int>(bits),
                            symmetric ? 1 : 0, stream);
  if (rc != DXB_OK) Py_RETURN_NONE;  // shapes the kernel does not take
  PyObject* zeros = Py_NewRef(Py_None);
  if (!symmetric) Py_SETREF(zeros, THPVariable_Wrap(std::move(z)));
  return Py_BuildValue("(NNN)", THPVariable_Wrap(std::move(q)), THPVariable_Wrap(std::move(s)), zeros);
}

PyObject* dequantize(PyObject* const* a, Py_ssize_t n_args) {
  if (n_args != 6) {
    PyErr_SetString(PyExc_TypeError, "_dxb_call.dequantize takes exactly 6 arguments");
    return nullptr;
  }
  const at::Tensor *q = plain_tensor(a[0]), *s = plain_tensor(a[1]);
  const at::Tensor* z = a[2] == Py_None ? nullptr : plain_tensor(a[2]);
  const long group = PyLong_AsLong(a[3]), bits = PyLong_AsLong(a[4]), layout = PyLong_AsLong(a[5]);
  if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
  if (!g_dequantize || !q || !s || (a[2] != Py_None && !z) || !q->is_cuda() || q->scalar_type() != at::kByte || q->dim() != 2 ||
      !q->is_contiguous() || s->scalar_type() != at::kBFloat16 || !s->is_contiguous() ||
      (z && (z->scalar_type() != at::kBFloat16 || !z->is_contiguous())))
    Py_RETURN_NONE;
  const auto dev = q->device();
  if (dev.index() != c10::cuda::current_device() || s->device() != dev || (z && z->device() != dev)) Py_RETURN_NONE;
  const int64_t n = q->size(1), k = q->size(0) * (bits == 4 ? 2 : 1);
  if (n <= 0 || k <= 0 || n > INT32_MAX || k > INT32_MAX || group > INT32_MAX) Py_RETURN_NONE;
  const int64_t cells = group > 0 ? k / group * n : 0;
  if (s->numel() < cells || (z && z->numel() < cells)) Py_RETURN_NONE;
  at::Tensor out = at::empty({k, n}, s->options());
  const auto stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const int rc = g_dequantize(q->const_data_ptr(), s->const_data_ptr(), z ? z->const_data_ptr() : nullptr,
                              out.mutable_data_ptr(), static_cast<int>(n), static_cast<int>(k), static_cast<int>(group),
                              static_cast<int>(bits), static_cast<int>(layout), stream);
  if (rc != DXB_OK) Py_RETURN_NONE;  // the general path reports it
  return THPVariable_Wrap(std::move(out));
}

// Any C++ exception sends the call down the general path, which raises what there is to raise: tensors
// without storage or strides (vmap, sparse) throw from the plainest accessors, allocations when memory is short.
template <PyObject* (*F)(PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  try {
    return F(a, n_args);
  } catch (...) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
}
template <PyObject* (*F)(PyObject* const*, Py_ssize_t)>
PyCFunction fastcall() {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<F>));
}
PyMethodDef methods[] = {
    {"bind", bind, METH_VARARGS, "bind(addresses in the library..., relaid)"},
    {"set_workspace", set_workspace, METH_VARARGS, "set_workspace(device, stream, ptr, bytes)"},
    {"call", fastcall<call>(), METH_FASTCALL, "one eager GEMM, or None where the general path has to take it"},
    {"quantize", fastcall<quantize>(), METH_FASTCALL, "a weight packed, or None where the general path has to do it"},
    {"dequantize", fastcall<dequantize>(), METH_FASTCALL, "the dense weight, or None where the general path has to make it"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_dxb_call", "native eager call", -1, methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dxb_call() { return PyModule_Create(&module_def); }
