// torch_ops.cpp — the operators of ops.py that a program calls once per layer and token, from Python to the C ABI without Python in between.
//
// What the path costs: checks, an empty result, the stream and a ctypes call with a dozen converted arguments took 4.7 of the 8.8 µs of a
// small Linear.  Host µs a call, from Python / from here: a Linear of one row 8.8 / 4.9, an attention row over 20 keys 8.2 / 4.3, a fused GEMV
// 8.6 / 5.1, a norm or a sum 6.2 / 3.9; what is left is the result's allocation and the launch.
//
// A function takes what its ops.py namesake was given.  It answers None for everything but the plain case — a tensor that is no ordinary strided
// CUDA tensor of the type the operator takes, or not contiguous; a shape that ops.py refuses; an active torch-function mode — and
// ops.py then goes its own way, which copies, converts or raises; a status other than 0 comes back as a number.  Everything else is the same
// call of the C ABI: the result comes from torch's caching allocator (captured graphs, dispatch modes and the deterministic fill see
// it), the launch goes to the current stream of the current device, and the GIL is free meanwhile.
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/TensorSubclassLikeUtils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <dlfcn.h>

#include "b200_decode.h"

namespace {

// The C ABI of the library that _lib.py has loaded, whatever its file is called: this module is linked to none.
#define B200_FUNCTIONS(F) \
  F(gemv_bf16) F(gemm_bf16) F(rmsnorm_bf16) F(silu_mul_bf16) F(add_bf16) F(attn_bf16) F(gemv_fused_bf16) F(attn_decode_workspace_bytes) F(attn_decode_bf16)
struct {
#define B200_FIELD(f) decltype(&b200_##f) f;
  B200_FUNCTIONS(B200_FIELD)
} abi;

PyObject* bind(PyObject*, PyObject* handle) {   // what dlopen gave; before any other function here
  void* const lib = PyLong_AsVoidPtr(handle);
  if (lib == nullptr) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "no library");
#define B200_BIND(f)                                                             \
  abi.f = reinterpret_cast<decltype(abi.f)>(dlsym(lib, "b200_" #f));             \
  if (abi.f == nullptr) return PyErr_Format(PyExc_AttributeError, "the library does not export b200_" #f);
  B200_FUNCTIONS(B200_BIND)
  Py_RETURN_NONE;
}

// an ordinary contiguous CUDA tensor of this type, or null
const at::Tensor* plain(PyObject* o, at::ScalarType type = at::kBFloat16) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || t.layout() != at::kStrided || !t.is_cuda() || t.scalar_type() != type || !t.unsafeGetTensorImpl()->has_storage() ||
      at::isTensorSubclassLike(t) || t.key_set().has(c10::DispatchKey::Functionalize) || t._is_zerotensor() || !t.is_contiguous() || t.is_neg() ||
      t.is_conj())
    return nullptr;
  return &t;
}
// the same, or None
bool plain_or_none(PyObject* o, const at::Tensor*& t, at::ScalarType type = at::kBFloat16) {
  t = nullptr;
  return o == Py_None || (t = plain(o, type)) != nullptr;
}
bool modes() { return at::impl::torch_function_mode_enabled(); }
void* ptr(const at::Tensor* t) { return t == nullptr ? nullptr : t->data_ptr(); }

// A result of shape `sizes` on x's device, handed to `call` with the current stream: the tensor, or the status that is not 0.
template <typename F>
PyObject* run(const at::Tensor& x, at::IntArrayRef sizes, F call) {
  at::Tensor y;
  int rc;
  {
    pybind11::gil_scoped_release free;
    y = at::empty(sizes, at::TensorOptions().dtype(at::kBFloat16).device(x.device()));
    rc = call(y.data_ptr(), (void*)c10::cuda::getCurrentCUDAStream().stream());
  }
  return rc == 0 ? THPVariable_Wrap(y) : PyLong_FromLong(rc);
}

// x's sizes with another last one
c10::SmallVector<int64_t, 6> with_last(const at::Tensor& x, int64_t n) {
  c10::SmallVector<int64_t, 6> s(x.sizes().begin(), x.sizes().end());
  s.back() = n;
  return s;
}

PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n_args) {   // x, weight, bias or None
  HANDLE_TH_ERRORS
  const at::Tensor *x, *w, *b;
  if (n_args != 3 || modes() || !(x = plain(a[0])) || !(w = plain(a[1])) || !plain_or_none(a[2], b) || w->dim() != 2 || x->dim() < 1) Py_RETURN_NONE;
  const int64_t n = w->size(0), k = w->size(1);
  if (k < 1 || x->size(-1) != k || x->numel() < 1) Py_RETURN_NONE;
  const int64_t m = x->numel() / k;
  return run(*x, with_last(*x, n), [&](void* y, void* st) { return abi.gemv_bf16(y, x->data_ptr(), w->data_ptr(), ptr(b), m, n, k, st); });
  END_HANDLE_TH_ERRORS
}

PyObject* gemm(PyObject*, PyObject* const* a, Py_ssize_t n_args) {   // a, weight
  HANDLE_TH_ERRORS
  const at::Tensor *x, *w;
  if (n_args != 2 || modes() || !(x = plain(a[0])) || !(w = plain(a[1])) || w->dim() != 2 || x->dim() < 1) Py_RETURN_NONE;
  const int64_t n = w->size(0), k = w->size(1);
  if (k < 1 || x->size(-1) != k || x->numel() < 1) Py_RETURN_NONE;
  const int64_t m = x->numel() / k;
  return run(*x, with_last(*x, n), [&](void* y, void* st) { return abi.gemm_bf16(y, x->data_ptr(), w->data_ptr(), m, n, k, st); });
  END_HANDLE_TH_ERRORS
}

PyObject* rms_norm(PyObject*, PyObject* const* a, Py_ssize_t n_args) {   // x, weight or None, eps
  HANDLE_TH_ERRORS
  const at::Tensor *x, *w;
  if (n_args != 3 || modes() || !(x = plain(a[0])) || !plain_or_none(a[1], w) || !PyFloat_Check(a[2]) || x->dim() < 1 || x->numel() < 1) Py_RETURN_NONE;
  const int64_t dim = x->size(-1);
  const float eps = (float)PyFloat_AS_DOUBLE(a[2]);
  return run(*x, x->sizes(), [&](void* y, void* st) { return abi.rmsnorm_bf16(y, x->data_ptr(), ptr(w), x->numel() / dim, dim, eps, st); });
  END_HANDLE_TH_ERRORS
}

PyObject* silu_mul(PyObject*, PyObject* const* a, Py_ssize_t n_args) {   // x
  HANDLE_TH_ERRORS
  const at::Tensor* x;
  if (n_args != 1 || modes() || !(x = plain(a[0])) || x->dim() < 1 || x->numel() < 1 || x->size(-1) % 2 != 0) Py_RETURN_NONE;
  const int64_t n = x->size(-1) / 2;
  return run(*x, with_last(*x, n), [&](void* y, void* st) { return abi.silu_mul_bf16(y, x->data_ptr(), x->numel() / (2 * n), n, st); });
  END_HANDLE_TH_ERRORS
}

PyObject* add(PyObject*, PyObject* const* a, Py_ssize_t n_args) {   // a, b of one shape
  HANDLE_TH_ERRORS
  const at::Tensor *x, *z;
  if (n_args != 2 || modes() || !(x = plain(a[0])) || !(z = plain(a[1])) || x->sizes() != z->sizes()) Py_RETURN_NONE;
  return run(*x, x->sizes(), [&](void* y, void* st) { return abi.add_bf16(y, x->data_ptr(), z->data_ptr(), x->numel(), st); });
  END_HANDLE_TH_ERRORS
}

PyObject* flash_attention(PyObject*, PyObject* const* a, Py_ssize_t n_args) {   // q, k, v, causal
  HANDLE_TH_ERRORS
  const at::Tensor *q, *k, *v;
  if (n_args != 4 || modes() || !(q = plain(a[0])) || !(k = plain(a[1])) || !(v = plain(a[2])) || !PyBool_Check(a[3]) || q->dim() != 4 || k->dim() < 3)
    Py_RETURN_NONE;
  const int64_t B = q->size(0), Sq = q->size(1), Hq = q->size(2), D = q->size(3), Skv = k->size(1), Hkv = k->size(2);
  const int causal = a[3] == Py_True;
  return run(*q, q->sizes(), [&](void* y, void* st) {
    return abi.attn_bf16(y, q->data_ptr(), k->data_ptr(), v->data_ptr(), B, Sq, Skv, Hq, Hkv, D, causal, st);
  });
  END_HANDLE_TH_ERRORS
}

PyObject* gemv_fused(PyObject*, PyObject* const* a, Py_ssize_t n_args) {   // x, weight, norm or None, eps, bias or None, residual or None, silu
  HANDLE_TH_ERRORS
  const at::Tensor *x, *w, *norm, *b, *r;
  if (n_args != 7 || modes() || !(x = plain(a[0])) || !(w = plain(a[1])) || !plain_or_none(a[2], norm) || !PyFloat_Check(a[3]) ||
      !plain_or_none(a[4], b) || !plain_or_none(a[5], r) || !PyBool_Check(a[6]) || w->dim() != 2)
    Py_RETURN_NONE;
  const int silu = a[6] == Py_True, nseg = silu ? 2 : 1;
  const int64_t n = w->size(0) / nseg, k = w->size(1);
  const float eps = (float)PyFloat_AS_DOUBLE(a[3]);
  return run(*x, {n}, [&](void* y, void* st) {
    return abi.gemv_fused_bf16(y, x->data_ptr(), w->data_ptr(), n, k, nseg, ptr(norm), eps, ptr(b), ptr(r), silu, st);
  });
  END_HANDLE_TH_ERRORS
}

// qkv, kcache, vcache, q_heads, kv_heads, head_dim, pos or None, fixed_len, rope table or None, q_norm or None, k_norm or None, eps
PyObject* attn_decode(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  const at::Tensor *qkv, *kc, *vc, *pos, *rope, *qn, *kn;
  if (n_args != 12 || modes() || !(qkv = plain(a[0])) || !(kc = plain(a[1])) || !(vc = plain(a[2])) || !PyLong_Check(a[3]) || !PyLong_Check(a[4]) ||
      !PyLong_Check(a[5]) || !plain_or_none(a[6], pos, at::kInt) || !PyLong_Check(a[7]) || !plain_or_none(a[8], rope, at::kFloat) ||
      !plain_or_none(a[9], qn) || !plain_or_none(a[10], kn) || !PyFloat_Check(a[11]) || kc->dim() < 1)
    Py_RETURN_NONE;
  const int64_t Hq = PyLong_AsLongLong(a[3]), Hkv = PyLong_AsLongLong(a[4]), hd = PyLong_AsLongLong(a[5]), len = PyLong_AsLongLong(a[7]);
  if (PyErr_Occurred()) {   // a number that no int64 holds
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const int64_t ctx = kc->size(0);
  if (Hq < 1 || Hq > (1 << 20) || hd < 1 || hd > 1024) Py_RETURN_NONE;
  if (abi.attn_decode_workspace_bytes(Hq, Hkv, hd, ctx) < 0) Py_RETURN_NONE;
  const float eps = (float)PyFloat_AS_DOUBLE(a[11]);
  return run(*qkv, {Hq * hd}, [&](void* y, void* st) {
    // no workspace is taken: any address will do
    return abi.attn_decode_bf16(y, qkv->data_ptr(), ptr(qn), ptr(kn), eps, (const float*)ptr(rope), (const int32_t*)ptr(pos), len, kc->data_ptr(),
                                vc->data_ptr(), Hq, Hkv, hd, ctx, y, st);
  });
  END_HANDLE_TH_ERRORS
}

#define B200_OP(f) {#f, (PyCFunction)(void (*)(void))f, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {{"_bind", bind, METH_O, nullptr}, B200_OP(linear),     B200_OP(gemm),        B200_OP(rms_norm),
                         B200_OP(silu_mul),                B200_OP(add),        B200_OP(flash_attention),
                         B200_OP(gemv_fused),              B200_OP(attn_decode), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "b200ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_b200ops() { return PyModule_Create(&module); }
