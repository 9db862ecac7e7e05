// The step from torch tensors to the C ABI, in native code: checks dtypes and layouts, allocates the outputs, takes
// the current stream and calls the library.  A layer of a short prompt or of a few decode rows lasts 50-100 us on the
// GPU; the same step written in Python (per-argument attribute calls, ctypes conversion, a Stream object) cost 10-20 us
// per call and four calls a layer, so the GPU waited for the host.  One call here is 2-4 us, launch included.
//
// Exceptions keep the Python wrappers' types: TypeError for a wrong dtype or device, ValueError for a shape that does
// not fit, AssertionError for a violated layout contract; library errors go through _abi.check.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <algorithm>

#include <ATen/Functions.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/b200tp.h"

namespace {

PyObject* g_check = nullptr;  // _abi.check(rc, what): raises

struct Raised {};  // a Python exception is set

[[noreturn]] void raise(PyObject* type, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  PyErr_FormatV(type, fmt, ap);
  va_end(ap);
  throw Raised{};
}
void expect(bool ok, const char* what) {
  if (!ok) raise(PyExc_AssertionError, "%s", what);
}
void check(int rc, const char* what) {
  if (rc == B2_OK) return;
  PyObject* r = PyObject_CallFunction(g_check, "is", rc, what);
  Py_XDECREF(r);
  throw Raised{};
}

// One call of the library.  The GIL is released around it: a launch waits when the stream's queue is full, and other Python
// threads have to go on meanwhile.  (Arguments are converted by the caller, with the GIL held; the library's error text is per thread.)
struct Unlocked {
  PyThreadState* const state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};
template <class... P, class... A>
void launch(const char* what, int (*f)(P...), A... args) {
  const int rc = [&] {
    const Unlocked unlocked;
    return f(args...);
  }();
  check(rc, what);
}

// ---- arguments -----------------------------------------------------------------
const at::Tensor& tensor(PyObject* o, const char* what) {
  if (!THPVariable_Check(o)) raise(PyExc_TypeError, "%s: expected a tensor, got %s", what, Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
at::Tensor optional_tensor(PyObject* o, const char* what) { return o == Py_None ? at::Tensor() : tensor(o, what); }
int64_t integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw Raised{};
  return v;
}
float number(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw Raised{};
  return static_cast<float>(v);
}
b2_ctx* context(PyObject* o) {
  if (o == Py_None) return nullptr;
  void* p = PyLong_AsVoidPtr(o);
  if (p == nullptr && PyErr_Occurred()) throw Raised{};
  return static_cast<b2_ctx*>(p);
}
void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
template <class T>
const T* cptr(const at::Tensor& t) { return static_cast<const T*>(ptr(t)); }
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// a CUDA bf16 tensor whose last dimension is contiguous
at::Tensor bf16_rows(const at::Tensor& t, const char* what) {
  if (t.scalar_type() != at::kBFloat16 || !t.is_cuda())
    raise(PyExc_TypeError, "%s: expected a CUDA bf16 tensor, got %s on %s", what, c10::toString(t.scalar_type()), t.device().str().c_str());
  return t.dim() > 0 && t.stride(-1) != 1 ? t.contiguous() : t;
}
// the same as rows a TMA map can describe: 2-D, 16-byte aligned base and row stride
struct Rows {
  at::Tensor t;
  int64_t rows, cols, ld;
};
Rows matrix(const at::Tensor& x, const char* what) {
  at::Tensor t = bf16_rows(x, what);
  if (t.dim() != 2) t = t.reshape({-1, t.size(-1)});
  if ((t.size(0) > 1 && t.stride(0) % 8 != 0) || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0) t = t.clone(at::MemoryFormat::Contiguous);
  return {t, t.size(0), t.size(1), t.size(0) > 1 ? t.stride(0) : t.size(1)};
}
at::Tensor empty_rows(int64_t rows, int64_t cols, const at::Tensor& like) {
  return at::detail::empty_cuda({rows, cols}, at::kBFloat16, like.device(), std::nullopt);
}
// out [rows, N] in the leading shape of x
at::Tensor leading(const at::Tensor& out, const at::Tensor& x, int64_t n) {
  if (x.dim() == 2) return out;
  std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end() - 1);
  shape.push_back(n);
  return out.view(shape);
}
// [tokens, heads, head_dim] whose heads lie one after the other in each token's row, in 16-byte vectors
bool heads_in_rows(const at::Tensor& t) {
  return t.stride(2) == 1 && (t.size(1) == 1 || t.stride(1) == t.size(2)) && t.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}
PyObject* wrap(const at::Tensor& t) { return THPVariable_Wrap(t); }
PyObject* wrap(const at::Tensor& a, const at::Tensor& b) {
  PyObject* p = PyTuple_New(2);
  if (p == nullptr) throw Raised{};
  PyTuple_SET_ITEM(p, 0, wrap(a));
  PyTuple_SET_ITEM(p, 1, wrap(b));
  return p;
}

using Args = PyObject* const*;

// gemm(ctx, x, w, bias)
PyObject* gemm(Args a) {
  const at::Tensor& x = tensor(a[1], "gemm input");
  const Rows in = matrix(x, "gemm input");
  const at::Tensor w = bf16_rows(tensor(a[2], "gemm weight"), "gemm weight");
  if (w.dim() != 2 || w.size(1) != in.cols) raise(PyExc_ValueError, "gemm: input has %lld features, weight has %lld", (long long)in.cols, (long long)w.size(-1));
  const at::Tensor bias = optional_tensor(a[3], "gemm bias");
  const int64_t n = w.size(0);
  const at::Tensor out = empty_rows(in.rows, n, x);
  if (in.rows)
    launch("b2_gemm", b2_gemm, context(a[0]), in.t.data_ptr(), in.ld, w.data_ptr(), w.stride(0), ptr(bias), out.data_ptr(), n, in.rows, n, in.cols, stream());
  return wrap(leading(out, x, n));
}

// gemm_silu_mul(ctx, x, w_pairs)
PyObject* gemm_silu_mul(Args a) {
  const at::Tensor& x = tensor(a[1], "gemm_silu_mul input");
  const Rows in = matrix(x, "gemm_silu_mul input");
  const at::Tensor& w = tensor(a[2], "gemm_silu_mul weight");
  if (w.dim() != 2 || w.size(1) != in.cols || w.size(0) % 2) raise(PyExc_ValueError, "gemm_silu_mul: input has %lld features, paired weight has %lld rows of %lld", (long long)in.cols, (long long)w.size(0), (long long)w.size(-1));
  const int64_t n = w.size(0) / 2;
  const at::Tensor out = empty_rows(in.rows, n, x);
  if (in.rows)
    launch("b2_gemm_silu_mul", b2_gemm_silu_mul, context(a[0]), in.t.data_ptr(), in.ld, w.data_ptr(), w.stride(0), out.data_ptr(), n, in.rows, n, in.cols, stream());
  return wrap(leading(out, x, n));
}

struct Cache {
  void *k = nullptr, *v = nullptr;
  const int32_t* slots = nullptr;
};
Cache cache_of(const at::Tensor& k, const at::Tensor& v, const at::Tensor& slots, int64_t row) {
  Cache c;
  if (!k.defined() || k.numel() == 0) return c;
  expect(k.stride(1) == row && slots.defined() && slots.scalar_type() == at::kInt, "k_cache rows must be contiguous and slot_mapping int32");
  c.k = k.data_ptr();
  c.v = v.data_ptr();
  c.slots = slots.const_data_ptr<int32_t>();
  return c;
}

// qkv_fused(ctx, x, w, bias, nq, nkv, head_dim, q_norm_w, k_norm_w, eps, positions, cos_sin, k_cache, v_cache, slot_mapping)
PyObject* qkv_fused(Args a) {
  const at::Tensor& x = tensor(a[1], "qkv input");
  const Rows in = matrix(x, "qkv input");
  const at::Tensor& w = tensor(a[2], "qkv weight");
  const at::Tensor bias = optional_tensor(a[3], "qkv bias");
  const int64_t nq = integer(a[4]), nkv = integer(a[5]), hd = integer(a[6]), n = w.size(0);
  expect(n == (nq + 2 * nkv) * hd && w.size(1) == in.cols, "qkv_fused: weight shape");
  const at::Tensor qw = optional_tensor(a[7], "q_norm_w"), kw = optional_tensor(a[8], "k_norm_w");
  const at::Tensor& pos = tensor(a[10], "positions");
  const at::Tensor& cs = tensor(a[11], "cos_sin");
  expect(pos.scalar_type() == at::kLong && cs.scalar_type() == at::kFloat && cs.is_contiguous(), "positions must be int64, cos_sin contiguous fp32");
  const at::Tensor kc = optional_tensor(a[12], "k_cache"), vc = optional_tensor(a[13], "v_cache"), sm = optional_tensor(a[14], "slot_mapping");
  const Cache c = cache_of(kc, vc, sm, nkv * hd);
  const at::Tensor out = empty_rows(in.rows, n, x);
  if (in.rows)
    launch("b2_qkv_fused", b2_qkv_fused, context(a[0]), in.t.data_ptr(), in.ld, w.data_ptr(), w.stride(0), ptr(bias), out.data_ptr(), n, in.rows, nq, nkv, hd, in.cols,
           ptr(qw), ptr(kw), number(a[9]), pos.const_data_ptr<int64_t>(), cs.const_data_ptr<float>(), c.k, c.v, c.slots, stream());
  return wrap(out);
}

// rowpar_fused(ctx, x, w, bias, residual, norm_w, eps): None when the two-shot form serves this size
PyObject* rowpar_fused(Args a) {
  b2_ctx* ctx = context(a[0]);
  const at::Tensor& x = tensor(a[1], "row-parallel input");
  const Rows in = matrix(x, "row-parallel input");
  const at::Tensor& w = tensor(a[2], "row-parallel weight");
  const at::Tensor bias = optional_tensor(a[3], "bias"), norm_w = optional_tensor(a[5], "norm weight");
  const int64_t n = w.size(0);
  at::Tensor residual, res_out;
  if (norm_w.defined()) {
    residual = bf16_rows(tensor(a[4], "residual"), "residual").contiguous();
    res_out = at::detail::empty_cuda(residual.sizes(), at::kBFloat16, residual.device(), std::nullopt);
  }
  if (in.rows) {
    const int form = b2_rowpar_form(ctx, in.rows, n);
    if (form < 0) check(-form, "b2_rowpar_form");
    if (form == B2_FORM_TWOSHOT) Py_RETURN_NONE;
  }
  const at::Tensor out = empty_rows(in.rows, n, x);
  if (in.rows)
    launch("b2_rowpar_fused", b2_rowpar_fused, ctx, in.t.data_ptr(), in.ld, w.data_ptr(), w.stride(0), ptr(bias), in.rows, n, in.cols, ptr(residual), ptr(norm_w),
           number(a[6]), out.data_ptr(), ptr(res_out), stream());
  return norm_w.defined() ? wrap(out, res_out) : wrap(leading(out, x, n));
}

// rmsnorm(x, w, eps)
PyObject* rmsnorm(Args a) {
  at::Tensor x = bf16_rows(tensor(a[0], "rmsnorm input"), "rmsnorm input");
  const at::Tensor& w = tensor(a[1], "rmsnorm weight");
  const int64_t dim = x.dim() > 0 ? x.size(-1) : 0;
  if (x.dim() == 3 && dim <= 256 && heads_in_rows(x)) {  // heads of q or k, read from the rows of the projection
    const at::Tensor out = at::detail::empty_cuda(x.sizes(), at::kBFloat16, x.device(), std::nullopt);
    launch("b2_rmsnorm", b2_head_rmsnorm, x.data_ptr(), x.stride(0), x.size(1), w.data_ptr(), number(a[2]), x.size(0), dim, out.data_ptr(), x.size(1) * dim, stream());
    return wrap(out);
  }
  const Rows in = matrix(x, "rmsnorm input");
  const at::Tensor out = empty_rows(in.rows, in.cols, x);
  launch("b2_rmsnorm", b2_rmsnorm, in.t.data_ptr(), in.ld, w.data_ptr(), number(a[2]), in.rows, in.cols, out.data_ptr(), in.cols, stream());
  return wrap(x.dim() == 2 ? out : out.view(x.sizes()));
}

// add_rmsnorm(x, residual, w, eps)
PyObject* add_rmsnorm(Args a) {
  const at::Tensor x = bf16_rows(tensor(a[0], "add_rmsnorm input"), "add_rmsnorm input").contiguous();
  const at::Tensor r = bf16_rows(tensor(a[1], "residual"), "residual").contiguous();
  const int64_t dim = x.size(-1), rows = x.numel() / dim;
  const at::Tensor out = at::detail::empty_cuda(x.sizes(), at::kBFloat16, x.device(), std::nullopt);
  const at::Tensor res_out = at::detail::empty_cuda(x.sizes(), at::kBFloat16, x.device(), std::nullopt);
  launch("b2_add_rmsnorm", b2_add_rmsnorm, x.data_ptr(), r.data_ptr(), tensor(a[2], "add_rmsnorm weight").data_ptr(), number(a[3]), rows, dim, out.data_ptr(), res_out.data_ptr(), stream());
  return wrap(out, res_out);
}

// silu_and_mul(x)
PyObject* silu_and_mul(Args a) {
  const at::Tensor& x = tensor(a[0], "silu_and_mul input");
  const Rows in = matrix(x, "silu_and_mul input");
  const int64_t n = in.cols / 2;
  const at::Tensor out = empty_rows(in.rows, n, x);
  launch("b2_silu_and_mul", b2_silu_and_mul, in.t.data_ptr(), in.ld, in.rows, n, out.data_ptr(), stream());
  return wrap(leading(out, x, n));
}

// store_kvcache(key, value, k_cache, v_cache, slot_mapping)
PyObject* store_kvcache(Args a) {
  const at::Tensor &k = tensor(a[0], "key"), &v = tensor(a[1], "value"), &kc = tensor(a[2], "k_cache"), &vc = tensor(a[3], "v_cache"), &sm = tensor(a[4], "slot_mapping");
  const int64_t n = k.size(0), hd = k.size(2), d = k.size(1) * hd;
  // the reference's own preconditions (nanovllm/layers/attention.py:36-39)
  expect(k.stride(-1) == 1 && v.stride(-1) == 1, "key and value must be contiguous in the last dimension");
  expect(k.stride(1) == hd && v.stride(1) == hd, "heads must be contiguous");
  expect(kc.stride(1) == d && vc.stride(1) == d, "cache rows must be contiguous");
  expect(sm.numel() == n, "one slot per token");
  expect(k.element_size() == 2 && kc.element_size() == 2 && sm.scalar_type() == at::kInt, "16-bit elements, int32 slots");
  launch("b2_store_kvcache", b2_store_kvcache, k.data_ptr(), k.stride(0), v.data_ptr(), v.stride(0), kc.data_ptr(), vc.data_ptr(), sm.const_data_ptr<int32_t>(), n, d, stream());
  Py_RETURN_NONE;
}

// qk_norm_rope_store(qkv, nq, nkv, head_dim, q_norm_w, k_norm_w, eps, positions, cos_sin, k_cache, v_cache, slot_mapping)
PyObject* qk_norm_rope_store(Args a) {
  const at::Tensor& qkv = tensor(a[0], "qkv");
  expect(qkv.dim() == 2 && qkv.stride(1) == 1 && qkv.scalar_type() == at::kBFloat16, "qkv must be a bf16 matrix with contiguous rows");
  const int64_t nq = integer(a[1]), nkv = integer(a[2]), hd = integer(a[3]);
  const at::Tensor qw = optional_tensor(a[4], "q_norm_w"), kw = optional_tensor(a[5], "k_norm_w");
  const at::Tensor &pos = tensor(a[7], "positions"), &cs = tensor(a[8], "cos_sin");
  expect(pos.scalar_type() == at::kLong && cs.scalar_type() == at::kFloat && cs.is_contiguous(), "positions must be int64, cos_sin contiguous fp32");
  const at::Tensor kc = optional_tensor(a[9], "k_cache"), vc = optional_tensor(a[10], "v_cache"), sm = optional_tensor(a[11], "slot_mapping");
  const Cache c = cache_of(kc, vc, sm, nkv * hd);
  launch("b2_qk_norm_rope_store", b2_qk_norm_rope_store, qkv.data_ptr(), qkv.stride(0), qkv.size(0), nq, nkv, hd, ptr(qw), ptr(kw), number(a[6]), pos.const_data_ptr<int64_t>(),
         cs.const_data_ptr<float>(), c.k, c.v, c.slots, stream());
  Py_RETURN_NONE;
}

// rope(positions, q, k, cos_sin, head_dim): rotated copies; q, k [tokens, heads, head_dim], or flattened over the heads
PyObject* rope(Args a) {
  at::Tensor pos = tensor(a[0], "positions");
  const at::Tensor& cs = tensor(a[3], "cos_sin");
  const int64_t hd = integer(a[4]), t = pos.numel();
  expect(cs.scalar_type() == at::kFloat && cs.is_contiguous(), "cos_sin must be contiguous fp32");
  if (pos.scalar_type() != at::kLong) pos = pos.to(at::kLong);
  pos = pos.contiguous();
  at::Tensor in[2];
  int64_t heads[2], ld[2];
  for (int i = 0; i < 2; ++i) {
    at::Tensor x = tensor(a[1 + i], i == 0 ? "query" : "key");
    if (x.scalar_type() != at::kBFloat16) x = x.to(at::kBFloat16);
    if (x.dim() != 3 || x.size(0) != t || x.size(2) != hd) x = x.reshape({t, t > 0 ? x.numel() / (t * hd) : 1, hd});
    if (!x.is_cuda()) raise(PyExc_TypeError, "rotary embedding: expected CUDA tensors");
    if (!heads_in_rows(x)) x = x.clone(at::MemoryFormat::Contiguous);
    heads[i] = x.size(1);
    ld[i] = t > 1 ? x.stride(0) : heads[i] * hd;
    in[i] = x;
  }
  const at::Tensor qo = at::detail::empty_cuda(tensor(a[1], "query").sizes(), at::kBFloat16, in[0].device(), std::nullopt);
  const at::Tensor ko = at::detail::empty_cuda(tensor(a[2], "key").sizes(), at::kBFloat16, in[1].device(), std::nullopt);
  launch("b2_rope", b2_rope, in[0].data_ptr(), ld[0], in[1].data_ptr(), ld[1], t, heads[0], heads[1], hd, pos.const_data_ptr<int64_t>(), cs.const_data_ptr<float>(),
         qo.data_ptr(), ko.data_ptr(), stream());
  return wrap(qo, ko);
}

// embed(ctx, ids, w, vocab_start, vocab_end)
PyObject* embed(Args a) {
  at::Tensor ids = tensor(a[1], "token ids");
  const at::Tensor& w = tensor(a[2], "embedding weight");
  expect(ids.scalar_type() == at::kLong && ids.is_cuda(), "token ids must be CUDA int64");
  ids = ids.contiguous();
  const int64_t m = ids.numel(), h = w.size(1);
  const at::Tensor out = at::detail::empty_cuda({m, h}, w.scalar_type(), w.device(), std::nullopt);
  launch("b2_embed", b2_embed, context(a[0]), ids.const_data_ptr<int64_t>(), w.data_ptr(), integer(a[3]), integer(a[4]), m, h, out.data_ptr(), stream());
  if (ids.dim() == 1) return wrap(out);
  std::vector<int64_t> shape(ids.sizes().begin(), ids.sizes().end());
  shape.push_back(h);
  return wrap(out.view(shape));
}

// ---- attention -----------------------------------------------------------------
// The kernels read lengths, tables, keys and values through raw pointers.  What makes a call not theirs (head layout, strides,
// alignment) is left to the caller's general path; what is wrong with it is an error here, before anything is launched.
void same_device(const at::Tensor& t, const at::Tensor& q, const char* what) {
  if (t.device() != q.device()) raise(PyExc_TypeError, "%s is on %s, the query on %s", what, t.device().str().c_str(), q.device().str().c_str());
}
void on_current_gpu(const at::Tensor& q, const char* what) {
  if (!q.is_cuda() || q.device().index() != c10::cuda::current_device()) raise(PyExc_TypeError, "%s: expected a tensor on the current GPU, got %s", what, q.device().str().c_str());
}
void int32_vector(const at::Tensor& t, int64_t n, const char* what) {
  if (t.dim() != 1 || t.size(0) != n) raise(PyExc_ValueError, "%s: expected %lld elements, got %lld in %lld dimensions", what, (long long)n, (long long)t.numel(), (long long)t.dim());
  expect(t.scalar_type() == at::kInt && t.is_contiguous(), "lengths must be contiguous int32");
}
void block_table_rows(const at::Tensor& t, int64_t n) {
  if (t.size(0) != n) raise(PyExc_ValueError, "block_tables: %lld rows for %lld sequences", (long long)t.size(0), (long long)n);
  expect(t.scalar_type() == at::kInt, "int32 block tables");
}
void values_like_keys(const at::Tensor& k, const at::Tensor& v, int64_t hd) {
  if (k.size(-1) != hd) raise(PyExc_ValueError, "keys have head dimension %lld, the query %lld", (long long)k.size(-1), (long long)hd);
  if (v.sizes() != k.sizes()) raise(PyExc_ValueError, "keys and values differ in shape");
  if (k.scalar_type() != at::kBFloat16 || v.scalar_type() != at::kBFloat16)
    raise(PyExc_TypeError, "expected bf16 keys and values, got %s and %s", c10::toString(k.scalar_type()), c10::toString(v.scalar_type()));
}
bool on_16_bytes(const at::Tensor& t) { return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0; }
// rows of `heads` heads side by side that the kernels' vector loads and tensor maps can address
bool row_layout(const at::Tensor& t, int64_t heads, int64_t hd) {
  return t.stride(-1) == 1 && t.stride(-2) == hd && on_16_bytes(t) && (t.size(0) <= 1 || (t.stride(0) % 8 == 0 && t.stride(0) >= heads * hd));
}
bool table_layout(const at::Tensor& t) { return t.dim() == 2 && t.size(1) > 0 && t.stride(1) == 1 && (t.size(0) <= 1 || t.stride(0) >= t.size(1)); }

// paged_attention(ctx, q, k_cache, v_cache, context_lens, block_tables, scale): None when the kernel does not serve the call
PyObject* paged_attention(Args a) {
  const at::Tensor &q = tensor(a[1], "q"), &kc = tensor(a[2], "k_cache"), &vc = tensor(a[3], "v_cache"), &lens = tensor(a[4], "context_lens"),
                   &tables = tensor(a[5], "block_tables");
  if (q.dim() != 3 || kc.dim() != 4) Py_RETURN_NONE;
  const int64_t n = q.size(0), nq = q.size(1), hd = q.size(2), nkv = kc.size(2), bs = kc.size(1);
  if (!b2_paged_attention_supported(n, nq, nkv, hd, bs) || q.scalar_type() != at::kBFloat16 || !row_layout(q, nq, hd) || kc.size(0) == 0 ||
      !kc.is_contiguous() || !vc.is_contiguous() || !on_16_bytes(kc) || !on_16_bytes(vc) || !table_layout(tables))
    Py_RETURN_NONE;
  values_like_keys(kc, vc, hd);
  int32_vector(lens, n, "context_lens");
  block_table_rows(tables, n);
  on_current_gpu(q, "q");
  same_device(kc, q, "k_cache");
  same_device(vc, q, "v_cache");
  same_device(lens, q, "context_lens");
  same_device(tables, q, "block_tables");
  const at::Tensor out = at::detail::empty_cuda({n, nq, hd}, at::kBFloat16, q.device(), std::nullopt);
  launch("b2_paged_attention_decode", b2_paged_attention_decode, context(a[0]), q.data_ptr(), n > 1 ? q.stride(0) : nq * hd, kc.data_ptr(), vc.data_ptr(), kc.size(0), bs,
         tables.const_data_ptr<int32_t>(), n > 1 ? tables.stride(0) : tables.size(1), tables.size(1), lens.const_data_ptr<int32_t>(), n, nq, nkv, hd, number(a[6]),
         out.data_ptr(), stream());
  return wrap(out);
}

// prefill_attention(ctx, q, k, v, cu_q, cu_k, max_q, block_tables, scale): None when the kernel does not serve the call.
// k, v: [rows, nkv, head_dim], or the caches when block_tables is given
PyObject* prefill_attention(Args a) {
  const at::Tensor &q = tensor(a[1], "q"), &k = tensor(a[2], "k"), &v = tensor(a[3], "v"), &cu_q = tensor(a[4], "cu_seqlens_q"), &cu_k = tensor(a[5], "cu_seqlens_k");
  const at::Tensor tables = optional_tensor(a[7], "block_tables");
  const bool paged = tables.defined();
  if (q.dim() != 3 || k.dim() != (paged ? 4 : 3)) Py_RETURN_NONE;
  const int64_t n = q.size(0), nq = q.size(1), hd = q.size(2), nkv = k.size(-2), bs = paged ? k.size(1) : 0, rows = paged ? k.size(0) * bs : k.size(0);
  if (!b2_prefill_attention_supported(nq, nkv, hd, bs) || q.scalar_type() != at::kBFloat16 || k.scalar_type() != at::kBFloat16 || !row_layout(q, nq, hd) || rows == 0 ||
      rows > (1 << 30) || cu_q.numel() > 65536 || v.strides() != k.strides() || !on_16_bytes(v))
    Py_RETURN_NONE;
  if (paged ? !k.is_contiguous() || !on_16_bytes(k) || !table_layout(tables) : !row_layout(k, nkv, hd)) Py_RETURN_NONE;
  // Wide groups, many sequences of a few tokens: a CTA's tile of 128 rows is mostly empty and takes 5 us however few there are, so that more than two
  // of them an SM cost more than the library's tiles of 64 rows.  Time there over time here, 300 to 2000 tiles of prompts without a cached part: of
  // 1 token 0.2-0.9, of 16 to 64 0.88-1.02, of 80 1.2-1.4, of 96 1.19-1.35, of lengths around 96 1.2-1.4: the line is where it pays in all of them.  Up
  // to two an SM (290 tiles) 16 to 64 tokens 1.0-1.08.  Over 768 cached tokens 1 token 0.2-0.6, 16 to 64 1.02-1.19: the line is the same for all.
  constexpr int64_t kRows = 96, kTwoAnSm = 2 * 148;
  if (nq > 2 * nkv && n < kRows * (cu_q.numel() - 1) && (cu_q.numel() - 1) * (nq / 2) > kTwoAnSm) Py_RETURN_NONE;
  if (c10::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad())) Py_RETURN_NONE;  // (forward only)
  const int64_t n_seqs = cu_q.numel() - 1, max_q = integer(a[6]);
  values_like_keys(k, v, hd);
  int32_vector(cu_q, std::max<int64_t>(1, n_seqs + 1), "cu_seqlens_q");
  int32_vector(cu_k, n_seqs + 1, "cu_seqlens_k");
  if (paged) block_table_rows(tables, n_seqs);
  if (n > 0 && (n_seqs < 1 || max_q < 1)) raise(PyExc_ValueError, "%lld query tokens in %lld sequences of at most %lld", (long long)n, (long long)n_seqs, (long long)max_q);
  on_current_gpu(q, "q");
  same_device(k, q, "k");
  same_device(v, q, "v");
  same_device(cu_q, q, "cu_seqlens_q");
  same_device(cu_k, q, "cu_seqlens_k");
  if (paged) same_device(tables, q, "block_tables");
  const at::Tensor out = at::detail::empty_cuda({n, nq, hd}, at::kBFloat16, q.device(), std::nullopt);
  if (n)
    launch("b2_prefill_attention", b2_prefill_attention, context(a[0]), q.data_ptr(), n > 1 ? q.stride(0) : nq * hd, k.data_ptr(), v.data_ptr(),
           paged || rows == 1 ? nkv * hd : k.stride(0), rows, paged ? tables.const_data_ptr<int32_t>() : nullptr,
           paged ? (n_seqs > 1 ? tables.stride(0) : tables.size(1)) : 0, paged ? tables.size(1) : 0, bs, cu_q.const_data_ptr<int32_t>(),
           cu_k.const_data_ptr<int32_t>(), n_seqs, max_q, n, nq, nkv, hd, number(a[8]), out.data_ptr(), stream());
  return wrap(out);
}

// ---- the decoder layers of a decode step -----------------------------------------------------
// a contiguous bf16 tensor on the query's device that the kernel's 16-byte accesses can address
bool plain(const at::Tensor& t, const at::Tensor& x, at::IntArrayRef shape) {
  return t.scalar_type() == at::kBFloat16 && t.device() == x.device() && t.sizes() == shape && t.is_contiguous() && on_16_bytes(t);
}

// decode_stack(ctx, x, positions, layers, final_norm, nq, nkv, head_dim, inter, eps, qk_eps, scale, cos_sin, context_lens,
//              slot_mapping, block_tables): None when the kernel does not serve the call.
// layers: per layer (qkv_w, o_w, gate_up_w in pairs, down_w, in_norm, post_norm, q_norm, k_norm, k_cache, v_cache)
PyObject* decode_stack(Args a) {
  b2_ctx* ctx = context(a[0]);
  const at::Tensor &x = tensor(a[1], "decode input"), &pos = tensor(a[2], "positions"), &final_norm = tensor(a[4], "final norm"), &cs = tensor(a[12], "cos_sin"),
                   &lens = tensor(a[13], "context_lens"), &slots = tensor(a[14], "slot_mapping"), &tables = tensor(a[15], "block_tables");
  if (!PyList_Check(a[3])) raise(PyExc_TypeError, "decode_stack: layers must be a list");
  const Py_ssize_t n_layers = PyList_GET_SIZE(a[3]);
  const int64_t nq = integer(a[5]), nkv = integer(a[6]), hd = integer(a[7]), inter = integer(a[8]);
  if (x.dim() != 2 || n_layers < 1) Py_RETURN_NONE;
  const int64_t n = x.size(0), h = x.size(1);
  std::vector<b2_stack_layer> layers(n_layers);
  int64_t blocks = 0, bs = 0;
  for (Py_ssize_t i = 0; i < n_layers; ++i) {
    PyObject* l = PyList_GET_ITEM(a[3], i);
    if (!PyTuple_Check(l) || PyTuple_GET_SIZE(l) != 10) raise(PyExc_TypeError, "decode_stack: a layer is a tuple of 10");
    at::Tensor w[10];
    for (int k = 0; k < 10; ++k) w[k] = optional_tensor(PyTuple_GET_ITEM(l, k), "decode_stack layer");
    if (!w[8].defined() || !w[9].defined() || w[8].dim() != 4) Py_RETURN_NONE;
    if (i == 0) {
      blocks = w[8].size(0);
      bs = w[8].size(1);
    }
    const int64_t q = nq * hd, rows = (nq + 2 * nkv) * hd;
    if (!plain(w[0], x, {rows, h}) || !plain(w[1], x, {h, q}) || !plain(w[2], x, {2 * inter, h}) || !plain(w[3], x, {h, inter}) || !plain(w[4], x, {h}) ||
        !plain(w[5], x, {h}) || w[6].defined() != w[7].defined() || (w[6].defined() && (!plain(w[6], x, {hd}) || !plain(w[7], x, {hd}))) ||
        !plain(w[8], x, {blocks, bs, nkv, hd}) || !plain(w[9], x, {blocks, bs, nkv, hd}))
      Py_RETURN_NONE;
    layers[i] = {ptr(w[0]), ptr(w[1]), ptr(w[2]), ptr(w[3]), ptr(w[4]), ptr(w[5]), ptr(w[6]), ptr(w[7]), ptr(w[8]), ptr(w[9])};
  }
  if (n == 0 || blocks == 0 || !plain(x, x, {n, h}) || !plain(final_norm, x, {h}) || !table_layout(tables) || tables.scalar_type() != at::kInt || !cs.is_contiguous() ||
      cs.scalar_type() != at::kFloat || cs.size(-1) != hd || !on_16_bytes(cs) || pos.scalar_type() != at::kLong || !pos.is_contiguous() || pos.numel() != n)
    Py_RETURN_NONE;
  const int64_t bytes = b2_decode_stack_workspace(ctx, n, n_layers, h, nq, nkv, hd, inter, bs);
  if (bytes == 0) Py_RETURN_NONE;
  on_current_gpu(x, "decode input");
  int32_vector(lens, n, "context_lens");
  if (slots.numel() < n) raise(PyExc_ValueError, "slot_mapping: %lld slots for %lld rows", (long long)slots.numel(), (long long)n);
  expect(slots.scalar_type() == at::kInt && slots.is_contiguous(), "slot_mapping must be contiguous int32");  // (its first n, as the layers)
  block_table_rows(tables, n);
  for (const at::Tensor* t : {&pos, &cs, &lens, &slots, &tables}) same_device(*t, x, "an operand of the decode step");
  const at::Tensor out = empty_rows(n, h, x), ws = at::detail::empty_cuda({bytes}, at::kByte, x.device(), std::nullopt);
  const float eps = number(a[9]), qk_eps = number(a[10]), scale = number(a[11]);
  void* const on_stream = stream();
  const int rc = [&] {
    const Unlocked unlocked;
    return b2_decode_stack(ctx, layers.data(), n_layers, final_norm.data_ptr(), h, nq, nkv, hd, inter, eps, qk_eps, scale, cs.const_data_ptr<float>(), x.data_ptr(), n,
                           pos.const_data_ptr<int64_t>(), lens.const_data_ptr<int32_t>(), slots.const_data_ptr<int32_t>(), tables.const_data_ptr<int32_t>(),
                           n > 1 ? tables.stride(0) : tables.size(1), tables.size(1), bs, blocks, out.data_ptr(), ws.data_ptr(), bytes, on_stream);
  }();
  if (rc == B2_ERR_UNSUPPORTED) Py_RETURN_NONE;  // (the CTAs cannot all be resident)
  check(rc, "b2_decode_stack");
  return wrap(out);
}

PyObject* init(Args a) {
  Py_INCREF(a[0]);
  Py_XDECREF(g_check);
  g_check = a[0];
  Py_RETURN_NONE;
}

template <PyObject* (*F)(Args), Py_ssize_t N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != N) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", N, n);
    return nullptr;
  }
  try {
    return F(args);
  } catch (const Raised&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

#define B2_ENTRY(name, n) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(&entry<name, n>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {B2_ENTRY(init, 1), B2_ENTRY(gemm, 4), B2_ENTRY(gemm_silu_mul, 3), B2_ENTRY(qkv_fused, 15), B2_ENTRY(rowpar_fused, 7),
                         B2_ENTRY(rmsnorm, 3), B2_ENTRY(add_rmsnorm, 4), B2_ENTRY(silu_and_mul, 1), B2_ENTRY(store_kvcache, 5),
                         B2_ENTRY(qk_norm_rope_store, 12), B2_ENTRY(rope, 5), B2_ENTRY(embed, 5), B2_ENTRY(paged_attention, 7), B2_ENTRY(prefill_attention, 9),
                         B2_ENTRY(decode_stack, 16), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_b2torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__b2torch(void) { return PyModule_Create(&module_def); }
