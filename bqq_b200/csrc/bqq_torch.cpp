// Native side of the Python module's calls (bqq_modules.py): checks the tensors of a layer and of one call, allocates
// the output and calls the C ABI, without the interpreter in between.
//
// Bound: a decode forward of a small layer is 5 us of GPU work; the same steps in Python (attribute look-ups through
// nn.Module.__getattr__, tensor property calls, a device context, ctypes argument conversion) took 30 us of host time.
// Measured, one forward among others of 2048 x 2048 with 2 bit layers at batch 1: 33.0 -> 6.6 us (3.5 us of it are the
// caller's no_grad and nn.Module.__call__).
//
// Every function returns None when anything is not the plain case (packed state missing or stale, another current
// device, an unusual tensor, scratch too small, autograd wanted): the caller then takes its Python route, which
// rebuilds the state or raises the right error.  Nothing is remembered from one call for the next except the layer's
// plane pointers (as long as the buffers they were packed from are unchanged) and the addresses of the scratch buffers
// that bqq_modules._workspace owns and never frees.  The interpreter lock is held throughout.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <vector>

#include "bqq_b200.h"

namespace {

PyObject *s_fast, *s_params, *s_buffers, *s_a, *s_b, *s_c, *s_d, *s_bias;

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return BQQ_F32;
    case at::kBFloat16: return BQQ_BF16;
    case at::kHalf: return BQQ_F16;
    default: return -1;
  }
}
const at::ScalarType kTypes[3] = {at::kFloat, at::kBFloat16, at::kHalf};

// ---- scratch buffers, as registered by bqq_modules._workspace --------------------------------------
enum Kind { kDecode = 0, kPrefill = 1 };
struct Scratch {
  int device, kind;
  cudaStream_t stream;
  void* ptr;
  size_t bytes;
};
std::vector<Scratch> g_scratch;

Scratch* find_scratch(int device, cudaStream_t stream, int kind) {
  for (Scratch& s : g_scratch)
    if (s.stream == stream && s.kind == kind && s.device == device) return &s;
  return nullptr;
}

PyObject* set_scratch(PyObject*, PyObject* args) {
  int device, kind;
  unsigned long long stream, ptr, bytes;
  if (!PyArg_ParseTuple(args, "iKiKK", &device, &stream, &kind, &ptr, &bytes)) return nullptr;
  Scratch* s = find_scratch(device, (cudaStream_t)stream, kind);
  if (!s) {
    g_scratch.push_back({device, kind, (cudaStream_t)stream, nullptr, 0});
    s = &g_scratch.back();
  }
  s->ptr = (void*)ptr;
  s->bytes = (size_t)bytes;
  Py_RETURN_NONE;
}

// ---- the packed state of one layer -------------------------------------------------------------------
struct Source {                    // a buffer the planes were packed from
  PyObject* name;
  const void* data;
  uint32_t version;
  int64_t numel;
  at::ScalarType type;
};
struct LayerObject {
  PyObject_HEAD
  BqqLayer layer;                  // coefficient and bias pointers are filled in on every call
  Source src[2];
  int device;
  int64_t in_f, out_f;
};

const at::Tensor* plain_tensor(PyObject* o) {
  if (!o || !THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided) return nullptr;
  return &t;
}

bool fill_source(Source* s, PyObject* name, PyObject* tensor) {
  const at::Tensor* t = plain_tensor(tensor);
  if (!t || t->is_inference()) return false;          // no version counter
  Py_INCREF(name);
  *s = {name, t->data_ptr(), t->_version(), t->numel(), t->scalar_type()};
  return true;
}
bool source_unchanged(const Source& s, PyObject* buffers) {
  const at::Tensor* t = plain_tensor(PyDict_GetItemWithError(buffers, s.name));
  return t && !t->is_inference() && t->data_ptr() == s.data && t->_version() == s.version && t->numel() == s.numel && t->scalar_type() == s.type;
}

void layer_dealloc(PyObject* o) {
  LayerObject* l = (LayerObject*)o;
  for (Source& s : l->src) Py_XDECREF(s.name);
  Py_TYPE(o)->tp_free(o);
}
PyTypeObject LayerType = {PyVarObject_HEAD_INIT(nullptr, 0)};

// Layer(dims, zplanes, yplanes, name0, tensor0, name1, tensor1) or None
PyObject* make_layer(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  int d[6];
  PyObject *zp, *yp, *n0, *t0, *n1, *t1;
  if (!PyArg_ParseTuple(args, "(iiiiii)OOUOUO", d, d + 1, d + 2, d + 3, d + 4, d + 5, &zp, &yp, &n0, &t0, &n1, &t1))
    return nullptr;
  const at::Tensor *z = plain_tensor(zp), *y = plain_tensor(yp);
  if (!z || !y) Py_RETURN_NONE;
  LayerObject* l = (LayerObject*)LayerType.tp_alloc(&LayerType, 0);
  if (!l) return nullptr;
  if (!fill_source(&l->src[0], n0, t0) || !fill_source(&l->src[1], n1, t1)) {
    Py_DECREF(l);
    Py_RETURN_NONE;
  }
  l->layer.dims = {d[0], d[1], d[2], d[3], d[4], d[5]};
  l->layer.zplanes = (const uint32_t*)z->data_ptr();
  l->layer.yplanes = (const uint32_t*)y->data_ptr();
  l->device = z->device().index();
  l->in_f = (int64_t)d[2] * d[4];
  l->out_f = (int64_t)d[1] * d[3];
  return (PyObject*)l;
  END_HANDLE_TH_ERRORS
}

// ---- one call ------------------------------------------------------------------------------------------
bool grad_wanted(const at::Tensor& t) { return t.requires_grad(); }

// A coefficient (or the bias): plain, contiguous, on the layer's device.
const at::Tensor* coefficient(PyObject* params, PyObject* name, int device) {
  const at::Tensor* t = plain_tensor(PyDict_GetItemWithError(params, name));
  return t && t->is_contiguous() && t->device().index() == device ? t : nullptr;
}

// Fills `layer` from the module's dictionary; nullptr when the Python route has to be taken.
LayerObject* open_layer(PyObject* dict, BqqLayer* layer, bool grad) {
  PyObject* o = PyDict_GetItemWithError(dict, s_fast);
  if (!o || Py_TYPE(o) != &LayerType) return nullptr;
  LayerObject* l = (LayerObject*)o;
  if (at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set()) return nullptr;
  PyObject* params = PyDict_GetItemWithError(dict, s_params);
  PyObject* buffers = PyDict_GetItemWithError(dict, s_buffers);
  if (!params || !buffers || !PyDict_Check(params) || !PyDict_Check(buffers)) return nullptr;
  if (!source_unchanged(l->src[0], buffers) || !source_unchanged(l->src[1], buffers)) return nullptr;
  if (c10::cuda::current_device() != l->device) return nullptr;
  *layer = l->layer;
  const at::Tensor* t[4];
  PyObject* names[4] = {s_a, s_b, s_c, s_d};
  for (int k = 0; k < 4; ++k) {
    t[k] = coefficient(params, names[k], l->device);
    if (!t[k] || t[k]->scalar_type() != t[0]->scalar_type() || (grad && grad_wanted(*t[k]))) return nullptr;
  }
  layer->coef_dtype = dtype_code(t[0]->scalar_type());
  if (layer->coef_dtype < 0) return nullptr;
  layer->a = t[0]->data_ptr();
  layer->b = t[1]->data_ptr();
  layer->c = t[2]->data_ptr();
  layer->d = t[3]->data_ptr();
  PyObject* bias = PyDict_GetItemWithError(params, s_bias);
  if (!bias) bias = PyDict_GetItemWithError(dict, s_bias);
  if (!bias && PyDict_GetItemWithError(buffers, s_bias)) return nullptr;
  layer->bias = nullptr;
  layer->bias_dtype = 0;
  if (bias && bias != Py_None) {
    const at::Tensor* b = coefficient(params, s_bias, l->device);
    if (!b || dtype_code(b->scalar_type()) < 0 || (grad && grad_wanted(*b))) return nullptr;
    layer->bias = b->data_ptr();
    layer->bias_dtype = dtype_code(b->scalar_type());
  }
  return l;
}

// Rows of X [..., width] as (pointer, rows, pitch); false when X has to be copied or is of another kind.
bool rows_of(const at::Tensor& x, int64_t width, int64_t* rows, int64_t* ld) {
  const int64_t nd = x.dim();
  if (nd < 1 || x.size(nd - 1) != width || x.is_conj() || x.is_neg()) return false;
  if (nd == 2 && x.stride(1) == 1) {
    *rows = x.size(0);
    *ld = *rows == 1 ? width : x.stride(0);
  } else if (x.is_contiguous()) {
    *rows = x.numel() / (width ? width : 1);
    *ld = width;
  } else {
    return false;
  }
  return *rows > 0 && *rows < (1ll << 31) && *ld >= width;
}

at::Tensor new_output(const at::Tensor& x, int64_t out_f) {
  at::DimVector sizes(x.sizes());
  sizes.back() = out_f;
  return at::Tensor(at::detail::empty_cuda(sizes, x.scalar_type(), x.device(), std::nullopt));
}

PyObject* raise_code(const char* what, int rc) {
  PyErr_Format(PyExc_RuntimeError, "%s failed: %s (code %d)", what, bqq_strerror(rc), rc);
  return nullptr;
}

// forward(module.__dict__, X) -> Y or None
PyObject* forward(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2) { PyErr_SetString(PyExc_TypeError, "forward(dict, X)"); return nullptr; }
  const at::Tensor* x = plain_tensor(args[1]);
  if (!x) Py_RETURN_NONE;
  const bool grad = c10::GradMode::is_enabled();
  BqqLayer layer;
  LayerObject* l = open_layer(args[0], &layer, grad);
  const int code = dtype_code(x->scalar_type());
  int64_t m, ldx;
  if (!l || code < 0 || x->device().index() != l->device || (grad && grad_wanted(*x)) || !rows_of(*x, l->in_f, &m, &ldx))
    Py_RETURN_NONE;
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(l->device).stream();
  const Scratch* ws = find_scratch(l->device, stream, m <= BQQ_DECODE_MAX_M ? kDecode : kPrefill);
  if (!ws || ws->bytes < bqq_forward_workspace_bytes(&layer.dims, (int)m)) Py_RETURN_NONE;
  at::Tensor y = new_output(*x, l->out_f);
  const int rc = bqq_forward(&layer, x->data_ptr(), code, (int)m, ldx, y.data_ptr(), code, l->out_f, ws->ptr, ws->bytes,
                             stream);
  if (rc) return raise_code(m <= BQQ_DECODE_MAX_M ? "bqq_forward_decode" : "bqq_forward_prefill", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// forward_fused(module.__dict__, X, rms_weight or None, eps, swiglu, residual or None) -> Y or None (up to 16 rows)
PyObject* forward_fused(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6) { PyErr_SetString(PyExc_TypeError, "forward_fused(dict, X, rms_weight, eps, swiglu, residual)"); return nullptr; }
  const at::Tensor* x = plain_tensor(args[1]);
  if (!x) Py_RETURN_NONE;
  const bool grad = c10::GradMode::is_enabled(), norm = args[2] != Py_None, res = args[5] != Py_None;
  const int swiglu = PyObject_IsTrue(args[4]);
  const double eps = PyFloat_AsDouble(args[3]);
  if (swiglu < 0 || PyErr_Occurred()) return nullptr;
  BqqLayer layer;
  LayerObject* l = open_layer(args[0], &layer, grad);
  const int code = dtype_code(x->scalar_type());
  int64_t m, ldx;
  if (!l || code < 0 || (norm && swiglu) || x->device().index() != l->device || (grad && grad_wanted(*x)) ||
      !rows_of(*x, swiglu ? 2 * l->in_f : l->in_f, &m, &ldx) || m > BQQ_DECODE_MAX_M)
    Py_RETURN_NONE;
  BqqFusion f = {};
  if (norm) {
    const at::Tensor* w = plain_tensor(args[2]);
    if (!w || dtype_code(w->scalar_type()) < 0 || !w->is_contiguous() || w->numel() != l->in_f ||
        w->device().index() != l->device)
      Py_RETURN_NONE;
    f.prologue = BQQ_PRO_RMSNORM;
    f.norm_weight = w->data_ptr();
    f.norm_dtype = dtype_code(w->scalar_type());
    f.eps = (float)eps;
  } else if (swiglu) {
    f.prologue = BQQ_PRO_SWIGLU;
  }
  if (res) {
    const at::Tensor* r = plain_tensor(args[5]);
    int64_t rm, ldr;
    if (!r || dtype_code(r->scalar_type()) < 0 || r->device().index() != l->device || !rows_of(*r, l->out_f, &rm, &ldr) ||
        rm != m)
      Py_RETURN_NONE;
    f.residual = r->data_ptr();
    f.ld_residual = ldr;
    f.residual_dtype = dtype_code(r->scalar_type());
  }
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(l->device).stream();
  const Scratch* ws = find_scratch(l->device, stream, kDecode);
  if (!ws || ws->bytes < bqq_decode_workspace_bytes(&layer.dims, (int)m)) Py_RETURN_NONE;
  at::Tensor y = new_output(*x, l->out_f);
  const int rc = bqq_forward_decode_fused(&layer, x->data_ptr(), code, (int)m, ldx, y.data_ptr(), code, l->out_f, &f,
                                          ws->ptr, ws->bytes, stream);
  if (rc) return raise_code("bqq_forward_decode_fused", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// weight(module.__dict__, dtype code) -> W [out, in] or None
PyObject* weight(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2) { PyErr_SetString(PyExc_TypeError, "weight(dict, code)"); return nullptr; }
  const long code = PyLong_AsLong(args[1]);
  if (code == -1 && PyErr_Occurred()) return nullptr;
  BqqLayer layer;
  LayerObject* l = open_layer(args[0], &layer, false);
  if (!l || code < 0 || code > 2) Py_RETURN_NONE;
  at::Tensor w(at::detail::empty_cuda({l->out_f, l->in_f}, kTypes[code], at::Device(at::kCUDA, (int8_t)l->device), std::nullopt));
  const int rc = bqq_reconstruct_weight(&layer, w.data_ptr(), (int)code, 1.f,
                                        c10::cuda::getCurrentCUDAStream(l->device).stream());
  if (rc) return raise_code("bqq_reconstruct_weight", rc);
  return THPVariable_Wrap(std::move(w));
  END_HANDLE_TH_ERRORS
}

// ---- host-buffer forward bound to its arguments -----------------------------------------------------------
struct HostCallObject {
  PyObject_HEAD
  vectorcallfunc call;
  BqqLayer layer;
  const void* x;
  void* y;
  int x_dtype, m, y_dtype, device;
  long long ldx, ldy;
  void* ws;
  size_t ws_bytes;
  cudaStream_t stream;
  PyObject *result, *keep;         // the output tensor; whatever owns the bound memory
};
PyTypeObject HostCallType = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* host_call(PyObject* self, PyObject* const*, size_t nargs, PyObject* kw) {
  HANDLE_TH_ERRORS
  HostCallObject* h = (HostCallObject*)self;
  if (PyVectorcall_NARGS(nargs) || (kw && PyTuple_GET_SIZE(kw))) {
    PyErr_SetString(PyExc_TypeError, "run() takes no arguments");
    return nullptr;
  }
  const int current = c10::cuda::current_device();
  if (current != h->device) c10::cuda::set_device(h->device);
  const int rc = bqq_forward_host(&h->layer, h->x, h->x_dtype, h->m, h->ldx, h->y, h->y_dtype, h->ldy, h->ws, h->ws_bytes,
                                  h->stream);
  if (current != h->device) c10::cuda::set_device(current);
  if (rc) return raise_code("bqq_forward_host", rc);
  Py_INCREF(h->result);
  return h->result;
  END_HANDLE_TH_ERRORS
}
int host_traverse(PyObject* o, visitproc visit, void* arg) {
  Py_VISIT(((HostCallObject*)o)->result);
  Py_VISIT(((HostCallObject*)o)->keep);
  return 0;
}
int host_clear(PyObject* o) {
  Py_CLEAR(((HostCallObject*)o)->result);
  Py_CLEAR(((HostCallObject*)o)->keep);
  return 0;
}
void host_dealloc(PyObject* o) {
  PyObject_GC_UnTrack(o);
  host_clear(o);
  Py_TYPE(o)->tp_free(o);
}

// host_call(layer address, x, x_dtype, m, ldx, y, y_dtype, ldy, ws, ws_bytes, stream, device, result, keep)
PyObject* make_host_call(PyObject*, PyObject* args) {
  unsigned long long layer, x, y, ws, ws_bytes, stream;
  int xd, m, yd, device;
  long long ldx, ldy;
  PyObject *result, *keep;
  if (!PyArg_ParseTuple(args, "KKiiLKiLKKKiOO", &layer, &x, &xd, &m, &ldx, &y, &yd, &ldy, &ws, &ws_bytes, &stream, &device,
                        &result, &keep))
    return nullptr;
  HostCallObject* h = (HostCallObject*)HostCallType.tp_alloc(&HostCallType, 0);
  if (!h) return nullptr;
  h->call = host_call;
  h->layer = *(const BqqLayer*)layer;
  h->x = (const void*)x; h->x_dtype = xd; h->m = m; h->ldx = ldx;
  h->y = (void*)y; h->y_dtype = yd; h->ldy = ldy;
  h->ws = (void*)ws; h->ws_bytes = (size_t)ws_bytes;
  h->stream = (cudaStream_t)stream; h->device = device;
  Py_INCREF(result); h->result = result;
  Py_INCREF(keep); h->keep = keep;
  return (PyObject*)h;
}

PyMethodDef kMethods[] = {
    {"set_scratch", set_scratch, METH_VARARGS, "set_scratch(device, stream, kind, address, bytes)"},
    {"make_layer", make_layer, METH_VARARGS, "make_layer(dims, zplanes, yplanes, name0, tensor0, name1, tensor1)"},
    {"forward", (PyCFunction)(void (*)(void))forward, METH_FASTCALL, "forward(dict, X)"},
    {"forward_fused", (PyCFunction)(void (*)(void))forward_fused, METH_FASTCALL,
     "forward_fused(dict, X, rms_weight, eps, swiglu, residual)"},
    {"weight", (PyCFunction)(void (*)(void))weight, METH_FASTCALL, "weight(dict, code)"},
    {"make_host_call", make_host_call, METH_VARARGS, "make_host_call(layer, x, ..., result, keep)"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_bqq_torch", "Native calls of bqq_modules", -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__bqq_torch(void) {
  LayerType.tp_name = "bqq_b200._bqq_torch.Layer";
  LayerType.tp_basicsize = sizeof(LayerObject);
  LayerType.tp_flags = Py_TPFLAGS_DEFAULT;
  LayerType.tp_dealloc = layer_dealloc;
  HostCallType.tp_name = "bqq_b200._bqq_torch.HostCall";
  HostCallType.tp_basicsize = sizeof(HostCallObject);
  HostCallType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC | Py_TPFLAGS_HAVE_VECTORCALL;
  HostCallType.tp_vectorcall_offset = offsetof(HostCallObject, call);
  HostCallType.tp_call = PyVectorcall_Call;
  HostCallType.tp_traverse = host_traverse;
  HostCallType.tp_clear = host_clear;
  HostCallType.tp_dealloc = host_dealloc;
  if (PyType_Ready(&LayerType) < 0 || PyType_Ready(&HostCallType) < 0) return nullptr;
  s_fast = PyUnicode_InternFromString("_bqq_fast");
  s_params = PyUnicode_InternFromString("_parameters");
  s_buffers = PyUnicode_InternFromString("_buffers");
  s_a = PyUnicode_InternFromString("a");
  s_b = PyUnicode_InternFromString("b");
  s_c = PyUnicode_InternFromString("c");
  s_d = PyUnicode_InternFromString("d");
  s_bias = PyUnicode_InternFromString("bias");
  return PyModule_Create(&kModule);
}
