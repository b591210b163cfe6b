// Host side of the calls that small batches make most: checks, allocations and the C-ABI call in one step.
//
// With the checks in Python and ctypes in between, a layer of 32 tokens spent 28 us on the host for 13 us of launches, a gate 7 for 3,
// a linear of one row 11 for 3; the device takes less than that.  The functions here take the usual form of a call (plain CUDA
// tensors of the current device, contiguous, of the types and shapes that need no conversion) and answer None for every other one: the caller
// then goes on as before, with the same checks, conversions and errors.  They call the same entry points of the C ABI with the same
// arguments, and keep nothing from one call to the next.
//
// The module is bound to the C ABI by the addresses that bind() is given, those of the library that the package has loaded.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TracerMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <exception>

#include "../../include/lightop_b200.h"

namespace {

struct Abi {
  decltype(&lo_topk_softmax) topk_softmax = nullptr;
  decltype(&lo_fused_moe_workspace_bytes) moe_workspace = nullptr;
  decltype(&lo_fused_moe_channel_workspace_bytes) channel_workspace = nullptr;
  decltype(&lo_fused_moe_block_int8) moe = nullptr;
  decltype(&lo_fused_moe_channel_int8) channel = nullptr;
  decltype(&lo_block_int8_linear_dynamic_scratch_bytes) linear_scratch = nullptr;
  decltype(&lo_block_int8_linear_dynamic) linear = nullptr;
} abi;
PyObject *check_status = nullptr;      // _lib.check(status, name): raises for a status other than 0

// A tensor as its data pointer says: torch.Tensor or Parameter itself, and none of the dispatch keys by which a wrapper (vmap,
// functionalisation, a subclass, lazy conjugation) stands in for other data.
bool plain(PyObject *o) {
  if (!THPVariable_CheckExact(o)) return false;
  static const uint64_t usual = (c10::DispatchKeySet(c10::DispatchKey::CUDA) | c10::DispatchKeySet(c10::DispatchKey::AutogradCUDA) |
                                 c10::DispatchKeySet(c10::DispatchKey::ADInplaceOrView) | c10::DispatchKeySet(c10::DispatchKey::AutocastCUDA)).raw_repr();
  return (THPVariable_Unpack(o).key_set().raw_repr() & ~usual) == 0;
}
// The device that is current, or -1 where a mode is active that is to see the allocations and conversions of the general path.
int current_device() {
  if (at::impl::torch_function_mode_enabled() || c10::impl::dispatch_mode_enabled() || at::tracer::impl::is_dispatch_enabled()) return -1;
  return (int)c10::cuda::current_device();
}
// The argument as a contiguous tensor on `device` (has_storage: not one without memory), null otherwise.
const at::Tensor *tensor(PyObject *o, int device) {
  if (!plain(o)) return nullptr;
  const at::Tensor &t = THPVariable_Unpack(o);
  return t.is_cuda() && t.get_device() == device && t.has_storage() && t.is_contiguous() ? &t : nullptr;
}
const at::Tensor *typed(PyObject *o, int device, at::ScalarType type) {
  const at::Tensor *t = tensor(o, device);
  return t != nullptr && t->scalar_type() == type ? t : nullptr;
}
bool shaped(const at::Tensor &t, std::initializer_list<int64_t> sizes) { return t.sizes() == at::IntArrayRef(sizes); }
int code_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return LO_F32;
    case at::kHalf: return LO_F16;
    case at::kBFloat16: return LO_BF16;
    case at::kInt: return LO_I32;
    case at::kLong: return LO_I64;
    default: return -1;
  }
}
bool integer(PyObject *o, int64_t *v) {
  if (!PyLong_CheckExact(o)) return false;
  int over = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &over);
  return over == 0;
}
// [128, 128] as a list or tuple of two ints
bool blocks_of_128(PyObject *o) {
  if (!(PyList_CheckExact(o) || PyTuple_CheckExact(o)) || PySequence_Fast_GET_SIZE(o) != 2) return false;
  int64_t a = 0, b = 0;
  return integer(PySequence_Fast_GET_ITEM(o, 0), &a) && integer(PySequence_Fast_GET_ITEM(o, 1), &b) && a == 128 && b == 128;
}
// Scratch of the stream's pool for the kernels of one call: given back on return, reused in the order of the stream.
c10::DataPtr scratch(size_t bytes) { return c10::cuda::CUDACachingAllocator::get()->allocate(bytes); }
// null with an exception set where the status is not 0
bool succeeded(int status, const char *what) {
  if (status == 0) return true;
  PyObject *r = PyObject_CallFunction(check_status, "is", status, what);
  Py_XDECREF(r);
  if (r != nullptr) PyErr_Format(PyExc_RuntimeError, "%s: status %d", what, status);
  return false;
}
PyObject *none() { Py_RETURN_NONE; }

// topk_softmax(weights, ids, gating, renormalize): True, or None
PyObject *topk_softmax(PyObject *, PyObject *const *a, Py_ssize_t n) {
  if (n != 4) return none();
  try {
    const int dev = current_device();
    if (dev < 0) return none();
    const at::Tensor *w = typed(a[0], dev, at::kFloat), *ids = tensor(a[1], dev), *g = tensor(a[2], dev);
    if (!w || !ids || !g || g->dim() != 2 || w->dim() != 2 || !PyBool_Check(a[3])) return none();
    const at::ScalarType it = ids->scalar_type(), gt = g->scalar_type();
    const int64_t M = g->size(0), E = g->size(1), k = w->size(1);
    if ((it != at::kInt && it != at::kLong) || (gt != at::kFloat && gt != at::kHalf && gt != at::kBFloat16) || !shaped(*w, {M, k}) || !shaped(*ids, {M, k})) return none();
    void *stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = abi.topk_softmax(g->data_ptr(), code_of(gt), M, (int)E, (int)k, a[3] == Py_True, static_cast<float *>(w->data_ptr()), ids->data_ptr(), code_of(it), nullptr,
                          stream);
    Py_END_ALLOW_THREADS
    if (!succeeded(st, "topk_softmax")) return nullptr;
    Py_RETURN_TRUE;
  } catch (const std::exception &) {
    return none();      // (an allocation that failed: the general path meets it again and raises)
  }
}

// fused_experts(x, w1, w2, weights, ids, cache13, w1_scale, w2_scale, expert_map, shared_output, block_shape, per_channel, experts, weight_on_input, factor,
//               inplace, status word): the layer's output, or None
PyObject *fused_experts(PyObject *, PyObject *const *a, Py_ssize_t n) {
  if (n != 17) return none();
  try {
    const int dev = current_device();
    if (dev < 0) return none();
    const bool channel = a[10] == Py_None;
    if (channel ? a[11] != Py_True : (a[11] != Py_False || !blocks_of_128(a[10]))) return none();
    const at::Tensor *x = typed(a[0], dev, at::kBFloat16), *w1 = typed(a[1], dev, at::kChar), *w2 = typed(a[2], dev, at::kChar);
    const at::Tensor *w = typed(a[3], dev, at::kFloat), *ids = tensor(a[4], dev);
    const at::Tensor *s1 = typed(a[6], dev, at::kFloat), *s2 = typed(a[7], dev, at::kFloat), *status = typed(a[16], dev, at::kInt);
    if (!x || !w1 || !w2 || !w || !ids || !s1 || !s2 || !status || x->dim() != 2 || w1->dim() != 3 || ids->dim() != 2) return none();
    const at::Tensor *cache = nullptr, *map = nullptr, *shared = nullptr;
    if (a[5] != Py_None && !(cache = typed(a[5], dev, at::kBFloat16))) return none();
    if (a[8] != Py_None && (!(map = typed(a[8], dev, at::kInt)) || map->dim() != 1)) return none();
    if (a[9] != Py_None && !(shared = typed(a[9], dev, at::kBFloat16))) return none();
    const at::ScalarType it = ids->scalar_type();
    const int64_t M = x->size(0), H = x->size(1), E = w1->size(0), N = w1->size(1), I = N / 2, k = ids->size(1);
    int64_t experts = 0;
    if ((it != at::kInt && it != at::kLong) || M < 1 || k < 1 || !shaped(*ids, {M, k}) || !shaped(*w, {M, k}) || w1->size(2) != H || N % 256 != 0 || H % 128 != 0 ||
        !shaped(*w2, {E, H, I}) || (shared && !shaped(*shared, {M, H})) || !integer(a[12], &experts))
      return none();
    if (channel ? (s1->numel() != E * N || s2->numel() != E * H) : (!shaped(*s1, {E, N / 128, H / 128}) || !shaped(*s2, {E, H / 128, I / 128}))) return none();
    if (experts == -1) experts = E;
    if (experts < -0x7fffffffLL || experts > 0x7fffffffLL || E > 0x7fffffffLL || k > 0x7fffffffLL) return none();
    // tokens in one piece: LMSLIM_FUSED_MOE_CHUNK_SIZE as the general path reads it
    int64_t most = 16384;
    if (const char *env = std::getenv("LMSLIM_FUSED_MOE_CHUNK_SIZE")) {
      char *end = nullptr;
      most = std::strtoll(env, &end, 10);
      if (end == env || *end != 0) return none();
    }
    if (M > most || !PyBool_Check(a[13]) || !PyBool_Check(a[15]) || (a[13] == Py_True && k != 1)) return none();
    double factor = 1.0;
    if (PyFloat_CheckExact(a[14])) factor = PyFloat_AS_DOUBLE(a[14]);
    else if (a[14] != Py_None) return none();
    if (cache && cache->numel() < M * k * H) return none();

    at::Tensor out = a[15] == Py_True ? *x : at::empty({M, H}, x->options());
    c10::DataPtr own_cache;
    void *c3 = cache ? cache->data_ptr() : nullptr;
    if (!cache) {
      own_cache = scratch((size_t)(M * k * H) * 2);
      c3 = own_cache.get();
    }
    const size_t bytes = channel ? abi.channel_workspace(M, (int)E, (int)experts, (int)k, H, I) : abi.moe_workspace(M, (int)E, (int)experts, (int)k, H, I);
    const c10::DataPtr ws = scratch(bytes);
    void *stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    const int8_t *p1 = static_cast<const int8_t *>(w1->data_ptr()), *p2 = static_cast<const int8_t *>(w2->data_ptr());
    const float *ps1 = static_cast<const float *>(s1->data_ptr()), *ps2 = static_cast<const float *>(s2->data_ptr()), *pw = static_cast<const float *>(w->data_ptr());
    const int32_t *pmap = map ? static_cast<const int32_t *>(map->data_ptr()) : nullptr;
    const void *px = x->data_ptr(), *pids = ids->data_ptr(), *psh = shared ? shared->data_ptr() : nullptr;
    void *po = out.data_ptr();
    int32_t *pst = static_cast<int32_t *>(status->data_ptr());
    const int on_input = a[13] == Py_True;
    int st;
    Py_BEGIN_ALLOW_THREADS
    if (channel)
      st = abi.channel(px, LO_BF16, p1, p2, ps1, ps2, pw, pids, code_of(it), pmap, (int)experts, M, (int)E, (int)k, H, I, c3, psh, po, on_input, (float)factor, ws.get(), bytes,
                       pst, stream);
    else
      st = abi.moe(px, p1, p2, ps1, ps2, pw, pids, code_of(it), pmap, (int)experts, M, (int)E, (int)k, H, I, c3, psh, po, on_input, (float)factor, ws.get(), bytes, pst,
                   stream);
    Py_END_ALLOW_THREADS
    if (!succeeded(st, "fused_experts_impl_int8")) return nullptr;
    if (a[15] == Py_True) {
      Py_INCREF(a[0]);
      return a[0];
    }
    return THPVariable_Wrap(std::move(out));
  } catch (const std::exception &) {
    return none();
  }
}

// linear(x, w, block_size, w_scale, status word): bf16 result for bf16 x, or None
PyObject *linear(PyObject *, PyObject *const *a, Py_ssize_t n) {
  if (n != 5) return none();
  try {
    const int dev = current_device();
    if (dev < 0 || !blocks_of_128(a[2])) return none();
    const at::Tensor *x = typed(a[0], dev, at::kBFloat16), *w = typed(a[1], dev, at::kChar), *s = typed(a[3], dev, at::kFloat), *status = typed(a[4], dev, at::kInt);
    if (!x || !w || !s || !status || w->dim() != 2 || x->dim() < 1) return none();
    const int64_t N = w->size(0), K = w->size(1);
    if (N < 1 || K < 1 || K % 128 != 0 || x->size(-1) != K || x->numel() == 0 || !shaped(*s, {(N + 127) / 128, K / 128})) return none();
    const int64_t M = x->numel() / K;
    at::DimVector sizes(x->sizes().begin(), x->sizes().end());
    sizes.back() = N;
    at::Tensor out = at::empty(sizes, x->options());
    const size_t bytes = abi.linear_scratch(M, N, K, LO_BF16);
    c10::DataPtr ws;
    if (bytes) ws = scratch(bytes);
    void *stream = c10::cuda::getCurrentCUDAStream(dev).stream();
    int st;
    Py_BEGIN_ALLOW_THREADS
    st = abi.linear(x->data_ptr(), LO_BF16, static_cast<const int8_t *>(w->data_ptr()), static_cast<const float *>(s->data_ptr()), M, N, K, out.data_ptr(), ws.get(), bytes,
                    static_cast<int32_t *>(status->data_ptr()), stream);
    Py_END_ALLOW_THREADS
    if (!succeeded(st, "apply_w8a8_block_int8_linear")) return nullptr;
    return THPVariable_Wrap(std::move(out));
  } catch (const std::exception &) {
    return none();
  }
}

// bind({name of the C ABI: address}, check)
PyObject *bind(PyObject *, PyObject *args) {
  PyObject *names = nullptr, *check = nullptr;
  if (!PyArg_ParseTuple(args, "O!O", &PyDict_Type, &names, &check)) return nullptr;
  bool ok = true;
  auto take = [&](const char *name, auto &fn) {
    PyObject *v = ok ? PyDict_GetItemString(names, name) : nullptr;
    void *p = v ? PyLong_AsVoidPtr(v) : nullptr;
    if (!p) ok = false;
    else fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(p);
  };
  take("lo_topk_softmax", abi.topk_softmax);
  take("lo_fused_moe_workspace_bytes", abi.moe_workspace);
  take("lo_fused_moe_channel_workspace_bytes", abi.channel_workspace);
  take("lo_fused_moe_block_int8", abi.moe);
  take("lo_fused_moe_channel_int8", abi.channel);
  take("lo_block_int8_linear_dynamic_scratch_bytes", abi.linear_scratch);
  take("lo_block_int8_linear_dynamic", abi.linear);
  if (!ok) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_KeyError, "bind: a function of the C ABI is missing");
    return nullptr;
  }
  Py_INCREF(check);
  Py_XSETREF(check_status, check);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, "Addresses of the C ABI and the function that raises for a status."},
                         {"topk_softmax", (PyCFunction)(void (*)(void))topk_softmax, METH_FASTCALL, "topk_softmax of plain tensors; None: not taken."},
                         {"fused_experts", (PyCFunction)(void (*)(void))fused_experts, METH_FASTCALL, "Fused layer of plain tensors; None: not taken."},
                         {"linear", (PyCFunction)(void (*)(void))linear, METH_FASTCALL, "Dense linear of plain tensors; None: not taken."},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Host side of the calls that small batches make most.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" PyMODINIT_FUNC PyInit__host(void) {
  PyObject *m = PyModule_Create(&module);
  // the torch and the Python that this was compiled against: the build looks for the text in the file, the package compares it with what it runs on
  if (m != nullptr && PyModule_AddStringConstant(m, "built_for", LIGHTOP_BUILT_FOR) != 0) Py_CLEAR(m);
  return m;
}
