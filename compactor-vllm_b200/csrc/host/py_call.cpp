// Python calls of the C ABI that take tensors.  A short call (a decode step over few keys, a short prompt) is one kernel of 10 us, and
// what such a call costs on the host is what it costs: ctypes takes 4 to 5 us for 20 to 30 arguments and 0.3 us for every
// tensor's address, and a dozen properties of the tensors 0.2 us each.  Two layers:
//   * bind(name, address, otherwise): the function of include/cvllm.h at `address` as a callable that takes None, int, float and CUDA
//     tensors; with anything else among the arguments (a number of numpy's, a ctypes array) the call goes to `otherwise` (the ctypes
//     function), tensors as their addresses.
//   * decode_attention / prefill_attention: the whole of the two entry points for the plain form of their arguments (ordinary
//     CUDA tensors of the documented types, shapes and strides).  They return None where anything is out of the ordinary, or
//     where the library refuses; the caller then goes the long way, which converts, or says what is wrong.
// Nothing is kept between calls.  Measured, us: eight prompts of 17 to 256 tokens back to back 18.4 -> 12.3 (the kernel's time), one call
// and a wait for it 44.9 -> 27.8; decoding 8 x 384 rows with a wait 36.4 -> 27.9; a biased attention step with a wait 111 -> 98.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>
#include <cstring>
#include <tuple>
#include <type_traits>
#include <utility>

#include "cvllm.h"

namespace {

// An argument of type T from a Python object: 1 converted, 0 of a kind that is not ours, -1 an error is set.
template <class T>
int convert(PyObject* o, T& out) {
  if constexpr (std::is_pointer_v<T>) {
    if (o == Py_None) {
      out = nullptr;
      return 1;
    }
    if (THPVariable_CheckExact(o)) {
      const at::Tensor& t = THPVariable_Unpack(o);
      if (!t.is_cuda()) {
        PyErr_SetString(PyExc_AssertionError, "cvllm kernels need CUDA tensors (no CPU fallback exists)");
        return -1;
      }
      out = reinterpret_cast<T>(t.data_ptr());
      return 1;
    }
    if (THPVariable_Check(o)) {   // a subclass says for itself where it lies
      PyObject* cuda = PyObject_GetAttrString(o, "is_cuda");
      if (!cuda) return -1;
      const bool yes = PyObject_IsTrue(cuda) == 1;
      Py_DECREF(cuda);
      if (!yes) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_AssertionError, "cvllm kernels need CUDA tensors (no CPU fallback exists)");
        return -1;
      }
      PyObject* at = PyObject_CallMethod(o, "data_ptr", nullptr);
      if (!at) return -1;
      out = reinterpret_cast<T>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(at)));
      Py_DECREF(at);
      return PyErr_Occurred() ? -1 : 1;
    }
    if (!PyLong_Check(o)) return 0;
    out = reinterpret_cast<T>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLongMask(o)));
    return PyErr_Occurred() ? -1 : 1;
  } else if constexpr (std::is_floating_point_v<T>) {
    if (!PyFloat_Check(o) && !PyLong_Check(o)) return 0;
    out = static_cast<T>(PyFloat_AsDouble(o));
    return PyErr_Occurred() ? -1 : 1;
  } else {
    if (!PyLong_Check(o)) return 0;
    out = static_cast<T>(PyLong_AsUnsignedLongLongMask(o));   // as ctypes: the low bits
    return PyErr_Occurred() ? -1 : 1;
  }
}

// A bound function's state: (capsule with the address, the ctypes function).
template <class F>
struct Bound;
template <class... A>
struct Bound<int(A...)> {
  template <size_t... I>
  static int call(void* address, PyObject* const* args, int& result, std::index_sequence<I...>) {
    std::tuple<A...> a;
    int state = 1;
    ((state = state == 1 ? convert(args[I], std::get<I>(a)) : state), ...);
    if (state != 1) return state;
    Py_BEGIN_ALLOW_THREADS
    result = reinterpret_cast<int (*)(A...)>(address)(std::get<I>(a)...);
    Py_END_ALLOW_THREADS
    return 1;
  }
  // a tensor where the ABI takes a pointer -> its address, anything else as it came: 1 and a new reference, or -1
  template <class T>
  static int address(PyObject* o, PyObject*& out) {
    if constexpr (std::is_pointer_v<T>) {
      if (THPVariable_Check(o)) {
        T at;
        if (convert(o, at) != 1) return -1;
        out = PyLong_FromVoidPtr(const_cast<void*>(static_cast<const void*>(at)));
        return out ? 1 : -1;
      }
    }
    out = Py_NewRef(o);
    return 1;
  }
  template <size_t... I>
  static PyObject* long_way(PyObject* otherwise, PyObject* const* args, Py_ssize_t n, std::index_sequence<I...>) {
    PyObject* list = PyTuple_New(n);
    if (!list) return nullptr;
    int state = 1;
    auto put = [&](Py_ssize_t i, auto convert_one) {
      PyObject* item = nullptr;
      if (state == 1 && i < n && (state = convert_one(args[i], item)) == 1) PyTuple_SET_ITEM(list, i, item);
    };
    (put(I, address<A>), ...);
    for (Py_ssize_t i = sizeof...(A); i < n; ++i) put(i, address<int>);
    PyObject* result = state == 1 ? PyObject_CallObject(otherwise, list) : nullptr;
    Py_DECREF(list);
    return result;
  }
  static PyObject* run(PyObject* self, PyObject* const* args, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    int result = 0, state = 0;
    if (n == static_cast<Py_ssize_t>(sizeof...(A)))
      state = call(PyCapsule_GetPointer(PyTuple_GET_ITEM(self, 0), nullptr), args, result, std::index_sequence_for<A...>{});
    if (state < 0) return nullptr;
    if (state == 0) return long_way(PyTuple_GET_ITEM(self, 1), args, n, std::index_sequence_for<A...>{});
    return PyLong_FromLong(result);
    END_HANDLE_TH_ERRORS
  }
};

#define CVLLM_BOUND(X)                                                                                                         \
  X(cvllm_decode_attention) X(cvllm_decode_step) X(cvllm_decode_store_kv) X(cvllm_prefill_store_all)                          \
  X(cvllm_prefill_attention_bounded) X(cvllm_rope_qknorm_store) X(cvllm_row_norm_rope_store)                                  \
  X(cvllm_bias_attn_varlen_dist) X(cvllm_bias_attn_decode_stream) X(cvllm_bias_attn_decode_dist)                              \
  X(cvllm_leverage_scores) X(cvllm_leverage_scores_from_sketch) X(cvllm_chunk_attn_scores) X(cvllm_snapkv_scores)             \
  X(cvllm_snapkv_scores_bounded) X(cvllm_select_store_topk_bounded) X(cvllm_causal_conv) X(cvllm_causal_conv_mode)            \
  X(cvllm_conv_state_update) X(cvllm_delta_rule) X(cvllm_delta_rule_chunks) X(cvllm_rmsnorm) X(cvllm_residual_norm)           \
  X(cvllm_gated_act)

PyMethodDef kBound[] = {
#define X(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&Bound<decltype(name)>::run)), METH_FASTCALL, nullptr},
    CVLLM_BOUND(X)
#undef X
    {nullptr, nullptr, 0, nullptr}};

PyObject* bind(PyObject*, PyObject* args) {
  const char* name = nullptr;
  unsigned long long address = 0;
  PyObject* otherwise = nullptr;
  if (!PyArg_ParseTuple(args, "sKO", &name, &address, &otherwise)) return nullptr;
  for (PyMethodDef* d = kBound; d->ml_name; ++d)
    if (std::strcmp(d->ml_name, name) == 0) {
      PyObject* capsule = PyCapsule_New(reinterpret_cast<void*>(address), nullptr, nullptr);
      if (!capsule) return nullptr;
      PyObject* state = PyTuple_Pack(2, capsule, otherwise);
      Py_DECREF(capsule);
      if (!state) return nullptr;
      PyObject* fn = PyCFunction_NewEx(d, state, nullptr);
      Py_DECREF(state);
      return fn;
    }
  Py_RETURN_NONE;
}

// an ordinary CUDA tensor: no subclass, conjugate or negative view, and memory of its own (a tensor that vmap or a transform of
// torch.func stands in for has none); the caller checks shapes and strides
const at::Tensor* plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && t.has_storage() && !t.is_conj() && !t.is_neg() ? &t : nullptr;
}
bool index_on(const at::Tensor& t, const at::Device& dev) {
  return t.scalar_type() == at::kInt && t.device() == dev && t.is_contiguous();
}
int dtype_of(const at::Tensor& t) {
  return t.scalar_type() == at::kBFloat16 ? CVLLM_BF16 : t.scalar_type() == at::kHalf ? CVLLM_F16 : -1;
}
bool int_of(PyObject* o, int64_t& v) {
  if (!PyLong_CheckExact(o)) return false;
  v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) {
    PyErr_Clear();
    return false;
  }
  return true;
}
bool scale_of(PyObject* o, int64_t D, float& scale) {
  if (o == Py_None) scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(D)));
  else if (PyFloat_CheckExact(o)) scale = static_cast<float>(PyFloat_AS_DOUBLE(o));
  else return false;
  return true;
}
bool fits_int(int64_t v) { return v >= 0 && v <= 0x7fffffff; }
bool power_of_two(int64_t v) { return v > 0 && (v & (v - 1)) == 0; }

// decode_attention(address, workspaces, q, k, v, seq_lens_bh, page_table, batch_mapping, HKV, PAGE_SIZE, sm_scale) -> out or None.
// workspaces: (device, stream, ("decode_attn", B, HQ, HKV)) -> byte tensor
PyObject* decode_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 11) Py_RETURN_NONE;
  const at::Tensor *q = plain(a[2]), *k = plain(a[3]), *v = plain(a[4]), *lens = plain(a[5]), *pt = plain(a[6]), *bm = plain(a[7]);
  int64_t HKV, PS;
  float scale;
  if (!q || !k || !v || !lens || !pt || !bm || !int_of(a[8], HKV) || !int_of(a[9], PS)) Py_RETURN_NONE;
  if (q->dim() != 3 || k->dim() != 2 || v->dim() != 2 || pt->dim() != 3 || lens->dim() != 2) Py_RETURN_NONE;
  const int64_t B = q->size(0), HQ = q->size(1), D = q->size(2), NLP = pt->size(2);
  const at::Device dev = q->device();
  const int dtype = dtype_of(*q);
  if (dtype < 0 || !scale_of(a[10], D, scale) || B < 1 || B > 32767 || HKV < 1 || HQ % HKV || HQ > 65536 || PS < 1 || PS % 32 || PS > 65536 ||
      !power_of_two(D) || D > 4096 || !fits_int(NLP))
    Py_RETURN_NONE;
  if (k->scalar_type() != q->scalar_type() || v->scalar_type() != q->scalar_type() || k->device() != dev || v->device() != dev ||
      !q->is_contiguous() || !k->is_contiguous() || !v->is_contiguous() || !index_on(*lens, dev) || !index_on(*pt, dev) ||
      !index_on(*bm, dev) || pt->size(1) != HKV)
    Py_RETURN_NONE;
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  PyObject* key = Py_BuildValue("(iK(sLLL))", static_cast<int>(dev.index()), reinterpret_cast<unsigned long long>(stream), "decode_attn",
                                static_cast<long long>(B), static_cast<long long>(HQ), static_cast<long long>(HKV));
  if (!key) return nullptr;
  PyObject* ws = PyDict_GetItemWithError(a[1], key);
  Py_DECREF(key);
  if (!ws) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  const at::Tensor* work = plain(ws);
  if (!work) Py_RETURN_NONE;
  const at::Tensor space = *work;     // held for the call: another thread may replace the entry
  const auto call = reinterpret_cast<decltype(&cvllm_decode_attention)>(PyCapsule_GetPointer(a[0], nullptr));
  if (!call) return nullptr;
  at::Tensor out = at::empty({B, HQ, D}, q->options());
  // all that may throw or set an error comes before the lock is released
  const void *q_at = q->data_ptr(), *k_at = k->data_ptr(), *v_at = v->data_ptr();
  void *out_at = out.data_ptr(), *space_at = space.data_ptr();
  const int32_t *lens_at = lens->data_ptr<int32_t>(), *pt_at = pt->data_ptr<int32_t>(), *bm_at = bm->data_ptr<int32_t>();
  const size_t space_bytes = static_cast<size_t>(space.numel());
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = call(q_at, out_at, k_at, v_at, lens_at, pt_at, bm_at, space_at, space_bytes, static_cast<int>(B), static_cast<int>(HQ),
            static_cast<int>(HKV), static_cast<int>(D), static_cast<int>(PS), static_cast<int>(NLP), scale, dtype, 0, stream);
  Py_END_ALLOW_THREADS
  if (rc != CVLLM_OK) Py_RETURN_NONE;
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// prefill_attention(address, q, k, v, k_cache, v_cache, seq_lens_bh, page_table, batch_mapping, cu_seqlens_q, max_seqlen_q,
// max_seqlen_k_cache, HKV, PAGE_SIZE, sm_scale) -> out or None
PyObject* prefill_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 15) Py_RETURN_NONE;
  const at::Tensor *q = plain(a[1]), *k = plain(a[2]), *v = plain(a[3]), *kc = plain(a[4]), *vc = plain(a[5]), *lens = plain(a[6]),
                   *pt = plain(a[7]), *bm = plain(a[8]), *cu = plain(a[9]);
  int64_t max_q, max_past, HKV, PS;
  float scale;
  if (!q || !k || !v || !kc || !vc || !lens || !pt || !bm || !cu || !int_of(a[10], max_q) || !int_of(a[11], max_past) ||
      !int_of(a[12], HKV) || !int_of(a[13], PS))
    Py_RETURN_NONE;
  if (q->dim() != 3 || k->dim() != 3 || v->dim() != 3 || kc->dim() != 2 || vc->dim() != 2 || pt->dim() != 3) Py_RETURN_NONE;
  const int64_t T = q->size(0), HQ = q->size(1), D = q->size(2), B = cu->numel() - 1, rows = kc->size(0), NLP = pt->size(2);
  const at::Device dev = q->device();
  const int dtype = dtype_of(*q);
  if (dtype < 0 || !scale_of(a[14], D, scale) || T < 1 || !fits_int(T) || B < 1 || !fits_int(B) || HKV < 1 || HQ % HKV || HQ > 65536 ||
      PS < 1 || PS > 65536 || rows % PS || !power_of_two(D) || D > 4096 || !fits_int(NLP) || !fits_int(max_q))
    Py_RETURN_NONE;
  for (const at::Tensor* t : {k, v}) {
    if (t->scalar_type() != q->scalar_type() || t->device() != dev || t->size(0) != T || t->size(1) != HKV || t->size(2) != D ||
        t->stride(2) != 1 || t->stride(1) != D)
      Py_RETURN_NONE;
  }
  for (const at::Tensor* t : {kc, vc}) {
    if (t->scalar_type() != q->scalar_type() || t->device() != dev || t->size(0) != rows || t->size(1) != D || !t->is_contiguous())
      Py_RETURN_NONE;
  }
  if (q->stride(2) != 1 || q->stride(1) != D || !index_on(*lens, dev) || !index_on(*pt, dev) || !index_on(*bm, dev) || !index_on(*cu, dev))
    Py_RETURN_NONE;
  if (max_past > 0x7fffffff) max_past = 0x7fffffff;
  if (max_past < -1) Py_RETURN_NONE;
  const auto call = reinterpret_cast<decltype(&cvllm_prefill_attention_bounded)>(PyCapsule_GetPointer(a[0], nullptr));
  if (!call) return nullptr;
  at::Tensor out = at::empty({T, HQ, D}, q->options());
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  // all that may throw or set an error comes before the lock is released
  const void *q_at = q->data_ptr(), *k_at = k->data_ptr(), *v_at = v->data_ptr(), *kc_at = kc->data_ptr(), *vc_at = vc->data_ptr();
  void* out_at = out.data_ptr();
  const int32_t *lens_at = lens->data_ptr<int32_t>(), *pt_at = pt->data_ptr<int32_t>(), *bm_at = bm->data_ptr<int32_t>(),
                *cu_at = cu->data_ptr<int32_t>();
  const int64_t q_stride = q->stride(0), k_stride = k->stride(0), v_stride = v->stride(0), out_stride = out.stride(0);
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = call(q_at, k_at, v_at, out_at, kc_at, vc_at, lens_at, pt_at, bm_at, cu_at, static_cast<int>(B), static_cast<int>(T),
            static_cast<int>(HQ), static_cast<int>(HKV), static_cast<int>(D), static_cast<int>(PS), static_cast<int>(NLP), rows, q_stride,
            k_stride, v_stride, out_stride, static_cast<int>(max_q), static_cast<int>(max_past), scale, dtype, stream);
  Py_END_ALLOW_THREADS
  if (rc != CVLLM_OK) Py_RETURN_NONE;
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

PyObject* address_of(PyObject*, PyObject* arg) {
  const unsigned long long address = PyLong_AsUnsignedLongLong(arg);
  if (PyErr_Occurred()) return nullptr;
  return PyCapsule_New(reinterpret_cast<void*>(address), nullptr, nullptr);
}

PyMethodDef kMethods[] = {
    {"bind", bind, METH_VARARGS, "bind(name, address, otherwise): a function of the C ABI that takes tensors, or None"},
    {"address", address_of, METH_O, "address(int): an address as decode_attention and prefill_attention take it"},
    {"decode_attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(decode_attention)), METH_FASTCALL, nullptr},
    {"prefill_attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(prefill_attention)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_cvllm_call", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__cvllm_call(void) { return PyModule_Create(&kModule); }
