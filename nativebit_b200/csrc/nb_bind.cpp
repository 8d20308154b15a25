// The host side of PackedLinear's call as one native function (a CPython module over torch's C++ tensors and the C ABI).  One
// activation row through 2560 x 2560 is 4.9 us on the device and was 16.2 us of host code: 2.4 of them the launch, the rest views,
// attribute and device look-ups, and fifteen arguments converted one by one.
//
// `linear` takes the calls it knows to be plain, and answers None to everything else (another device than the current one,
// tensor subclasses, no rows, gaps between rows, a workspace that is missing or too small, any status but success): the
// general path then does what it always did, its errors included.
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/nativebit_b200.h"

namespace {

constexpr int64_t kBlock = 128, kGemvRows = 16, kFusedRows = 1024;

int tag(at::ScalarType t) {
  return t == at::kFloat ? (int)NB_F32 : t == at::kHalf ? (int)NB_F16 : t == at::kBFloat16 ? (int)NB_BF16 : -1;
}

// workspaces[(device, stream)], held for the call (another thread may replace the entry meanwhile), or an undefined tensor.
at::Tensor workspace(PyObject* workspaces, int device, void* stream) {
  PyObject* key = Py_BuildValue("(iK)", device, (unsigned long long)(uintptr_t)stream);
  if (!key) return {};
  PyObject* ws = PyDict_GetItemWithError(workspaces, key);        // borrowed
  Py_DECREF(key);
  return ws && THPVariable_Check(ws) ? THPVariable_Unpack(ws) : at::Tensor();
}

// Whether a copy made of the tensors and versions in `of`, (packed, codebook, version, version), is one of these tensors as they are now.
bool copy_of(PyObject* of, PyObject* packed, PyObject* codebook) {
  if (!packed || !codebook || !PyTuple_CheckExact(of) || PyTuple_GET_SIZE(of) != 4 ||
      PyTuple_GET_ITEM(of, 0) != packed || PyTuple_GET_ITEM(of, 1) != codebook)
    return false;
  for (int i = 0; i < 2; ++i) {
    const at::Tensor& t = THPVariable_Unpack(PyTuple_GET_ITEM(of, i));
    if (PyLong_AsLongLong(PyTuple_GET_ITEM(of, 2 + i)) != (t.is_inference() ? -1 : t._version())) return false;
  }
  return true;
}

// The weights of the last launch over the packed bytes, [packed, codebook, version, version] or [] (or just whether to order it): whether
// these are others.
bool unseen(PyObject* seen, PyObject* packed, PyObject* codebook) {
  if (!PyList_CheckExact(seen)) return PyObject_IsTrue(seen) == 1;
  if (PyList_GET_SIZE(seen) != 4 || PyList_GET_ITEM(seen, 0) != packed || PyList_GET_ITEM(seen, 1) != codebook) return true;
  for (int i = 0; i < 2; ++i) {
    const at::Tensor& t = THPVariable_Unpack(i ? codebook : packed);
    if (PyLong_AsLongLong(PyList_GET_ITEM(seen, 2 + i)) != (t.is_inference() ? -1 : t._version())) return true;
  }
  return false;
}
void note_seen(PyObject* seen, PyObject* packed, PyObject* codebook) {
  if (!PyList_CheckExact(seen)) return;
  const at::Tensor &p = THPVariable_Unpack(packed), &c = THPVariable_Unpack(codebook);
  PyObject* now = Py_BuildValue("[OOLL]", packed, codebook, (long long)(p.is_inference() ? -1 : p._version()),
                                (long long)(c.is_inference() ? -1 : c._version()));
  if (now) PyList_SetSlice(seen, 0, PyList_GET_SIZE(seen), now);
  Py_XDECREF(now);
}

// all_current([(a module's buffers, what its copy was made of), ..]) -> whether every copy is of the module's present weights
PyObject* all_current(PyObject*, PyObject* list) {
  HANDLE_TH_ERRORS
  if (!PyList_Check(list)) {
    PyErr_SetString(PyExc_TypeError, "all_current takes a list");
    return nullptr;
  }
  static PyObject *const packed = PyUnicode_InternFromString("packed_indices"), *const codebook = PyUnicode_InternFromString("codebook");
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) {
    PyObject* item = PyList_GET_ITEM(list, i);
    if (!PyTuple_CheckExact(item) || PyTuple_GET_SIZE(item) != 2 || !PyDict_Check(PyTuple_GET_ITEM(item, 0))) Py_RETURN_FALSE;
    PyObject* buffers = PyTuple_GET_ITEM(item, 0);
    if (!copy_of(PyTuple_GET_ITEM(item, 1), PyDict_GetItemWithError(buffers, packed), PyDict_GetItemWithError(buffers, codebook))) {
      if (PyErr_Occurred()) return nullptr;
      Py_RETURN_FALSE;
    }
  }
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// linear(x, packed, codebook, w_stream or None, what it was made of, n, k, bits, seen (`unseen`), gemv workspaces, prefill
// workspaces) -> y or None
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  if (count != 11) {
    PyErr_SetString(PyExc_TypeError, "linear takes eleven arguments");
    return nullptr;
  }
  if (!THPVariable_CheckExact(a[0]) || !THPVariable_CheckExact(a[1]) || !THPVariable_CheckExact(a[2]) || !PyDict_Check(a[9]) || !PyDict_Check(a[10]))
    Py_RETURN_NONE;
  const at::Tensor &x = THPVariable_Unpack(a[0]), &packed = THPVariable_Unpack(a[1]), &codebook = THPVariable_Unpack(a[2]);
  const int64_t n = PyLong_AsLongLong(a[5]), k = PyLong_AsLongLong(a[6]);
  const int bits = (int)PyLong_AsLong(a[7]);
  if (PyErr_Occurred()) return nullptr;
  const int xt = tag(x.scalar_type()), ct = tag(codebook.scalar_type());
  if (xt < 0 || (ct != NB_F16 && ct != NB_F32) || !x.is_cuda() || x.layout() != at::kStrided || x.dim() < 1 || x.size(-1) != k || !x.is_contiguous() ||
      n < 1 || k < 1 || n > INT32_MAX || k > INT32_MAX)
    Py_RETURN_NONE;
  const at::Device device = x.device();
  const int64_t m = x.numel() / k;
  if (m < 1 || m > kFusedRows || packed.device() != device || codebook.device() != device || device.index() != c10::cuda::current_device()) Py_RETURN_NONE;
  void* const stream = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  at::DimVector shape(x.sizes());
  shape.back() = n;
  int rc = NB_ERR_ARG;
  const bool ordered = m <= kGemvRows && unseen(a[8], a[1], a[2]);
  const bool few = nb_chain_takes_packed((int)m, (int)n, (int)k, bits, xt) != 0;     // over the packed bytes; more rows of a small matrix over its copy
  if (few || (m > kGemvRows && THPVariable_CheckExact(a[3]) && nb_chain_takes((int)m, (int)n, (int)k, bits, xt))) {
    const at::Tensor &w = THPVariable_Unpack(a[few ? 1 : 3]), ws = workspace(a[10], device.index(), stream);
    if (!ws.defined()) Py_RETURN_NONE;
    if (few ? packed.scalar_type() != at::kByte || !packed.is_contiguous() || !codebook.is_contiguous() ||
                  packed.numel() < n * (k / 8) * bits || codebook.numel() != (n * (k / kBlock)) << bits
            : w.device() != device || !copy_of(a[4], a[1], a[2]))
      Py_RETURN_NONE;
    at::Tensor y = at::empty(shape, x.options().requires_grad(false).memory_format(c10::MemoryFormat::Contiguous));
    nb_chain_args args = {};
    args.w = static_cast<const uint8_t*>(w.const_data_ptr());
    if (few) {
      args.codebook = codebook.const_data_ptr();
      args.codebook_dtype = ct;
      args.ordered = ordered;
    }
    args.x = x.const_data_ptr();
    args.y = y.mutable_data_ptr();
    args.status = static_cast<int*>(ws.mutable_data_ptr());         // the workspace's head
    args.M = (int)m; args.N = (int)n; args.K = (int)k; args.bits = bits;
    args.x_dtype = args.y_dtype = xt;
    Py_BEGIN_ALLOW_THREADS
    rc = nb_chain_linear(&args, stream);
    Py_END_ALLOW_THREADS
    if (rc == NB_OK) {
      if (few && ordered) note_seen(a[8], a[1], a[2]);
      return THPVariable_Wrap(std::move(y));
    }
  } else if (m <= kGemvRows) {
    const at::Tensor ws = workspace(a[9], device.index(), stream);
    if (!ws.defined()) Py_RETURN_NONE;
    at::Tensor y = at::empty(shape, x.options().requires_grad(false).memory_format(c10::MemoryFormat::Contiguous));
    const void *xp = x.const_data_ptr(), *cp = codebook.const_data_ptr();
    const uint8_t* pp = static_cast<const uint8_t*>(packed.const_data_ptr());
    void *yp = y.mutable_data_ptr(), *wp = ws.mutable_data_ptr();
    const size_t wn = ws.nbytes();
    Py_BEGIN_ALLOW_THREADS
    rc = (ordered ? nb_gemv_ordered : nb_gemv)(xp, xt, (int)m, pp, cp, ct, bits, kBlock, (int)n, (int)k, yp, xt, wp, wn, stream);
    Py_END_ALLOW_THREADS
    if (rc == NB_OK) {
      if (ordered) note_seen(a[8], a[1], a[2]);
      return THPVariable_Wrap(std::move(y));
    }
  } else if (xt != NB_F16 && m * (xt == NB_F32 ? 2 : 1) <= kFusedRows && THPVariable_CheckExact(a[3])) {       // (that kernel writes bf16 or fp32)
    const at::Tensor &w = THPVariable_Unpack(a[3]), ws = workspace(a[10], device.index(), stream);
    if (!ws.defined() || w.device() != device || !copy_of(a[4], a[1], a[2])) Py_RETURN_NONE;
    at::Tensor y = at::empty(shape, x.options().requires_grad(false).memory_format(c10::MemoryFormat::Contiguous));
    const void* xp = x.const_data_ptr();
    const uint8_t* pw = static_cast<const uint8_t*>(w.const_data_ptr());
    void *yp = y.mutable_data_ptr(), *wp = ws.mutable_data_ptr();
    const size_t wn = ws.nbytes();
    Py_BEGIN_ALLOW_THREADS
    rc = nb_gemm_prefill_fused(xp, xt, (int)m, pw, bits, (int)n, (int)k, yp, xt, wp, wn, stream);
    Py_END_ALLOW_THREADS
    if (rc == NB_OK) return THPVariable_Wrap(std::move(y));
  }
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {{"linear", (PyCFunction)(void (*)(void))linear, METH_FASTCALL, nullptr}, {"all_current", all_current, METH_O, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_bind", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__bind(void) { return PyModule_Create(&module); }
