// Host path of the package as a CPython extension over ATen: cache state, append, attention and dequantisation calls.
//
// A step of an attention layer is three calls of the C ABI on small operands; written in Python (descriptors through ctypes, device
// context managers, tensor allocations) it cost about 72 us per step, several times the kernels of the early scales.  Here it is one
// call per step (about 9 us): the quantizers' state lives in a C++ object (the base class of VAR_Q.quant.VAR_Q), descriptors are
// filled in place and tensors come straight from the caching allocator.  Every function declines (returns None / False) what it does
// not handle -- unusual dtypes and layouts, the whole-cache modes after their first step, anything erroneous -- and the Python code
// next to it takes over, so that errors and rare modes have one implementation.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/autograd/python_variable.h>

#include "varq_b200.h"

namespace {

enum Method : int { M_TENSOR, M_SCALE_HEAD_DIM, M_HEAD_DIM, M_SCALE, M_TOKEN, M_TOKEN_HEAD, M_COUNT };
const char* const METHOD_NAMES[M_COUNT] = {"G_TENSOR", "G_SCALE_HEAD_DIM", "G_HEAD_DIM", "G_SCALE", "G_TOKEN", "G_TOKEN_HEAD"};
bool share_l(int m) { return m == M_TENSOR || m == M_SCALE || m == M_SCALE_HEAD_DIM || m == M_HEAD_DIM; }
bool share_h(int m) { return m == M_TENSOR || m == M_SCALE || m == M_TOKEN; }
bool per_dim(int m) { return m == M_SCALE_HEAD_DIM || m == M_HEAD_DIM; }
bool requant(int m) { return m == M_TENSOR || m == M_HEAD_DIM; }

enum { T_CODES, T_CODES_NEXT, T_SCALE, T_ZP, T_SCALE_NEXT, T_ZP_NEXT, T_ROT, T_RB, T_COUNT };
struct Cache {
    PyObject_HEAD
    // settings
    long long quant_bits, method, pack, symmetric, reduce_batch, group_size, max_tokens, debug, bhlc;
    double eps;
    // state
    at::Tensor t[T_COUNT];
    long long has_shape, B, H, D, words, nB, nH, nG, lcap, rcap, n_tokens, n_rows;
    long long pend_set, pend[3];  // tokens, rows, replaces_cache
    long long last_set, last[2];
    long long meta_set, meta_c, meta_bits;
};

PyTypeObject* cache_type = nullptr;
bool is_cache(PyObject* o) { return PyObject_TypeCheck(o, cache_type); }

// ---------------------------------------------------------------- small helpers
int dtype_code(at::ScalarType s) { return s == at::kFloat ? VARQ_F32 : s == at::kHalf ? VARQ_F16 : s == at::kBFloat16 ? VARQ_BF16 : -1; }
int store_bits(const Cache* c) { return c->pack ? (int)c->quant_bits : 8; }

PyObject* raise(int rc) {
    PyErr_Format(rc == VARQ_ERR_CUDA ? PyExc_RuntimeError : PyExc_ValueError, "[VAR-Q] %s", varq_last_error());
    return nullptr;
}

at::Tensor empty(at::IntArrayRef shape, at::ScalarType s, c10::DeviceIndex dev) {
    return at::detail::empty_cuda(shape, s, c10::Device(c10::kCUDA, dev), c10::nullopt);
}
// Scratch of one call, from the caching allocator on the current stream: it goes back when the call returns and is reused in the order of
// that stream, and what a captured call used belongs to the graph's pool for the graph's lifetime.  (A buffer kept between calls would have to
// outlive every graph that holds its address, and would be shared by a replay and by calls on the stream that it was captured on.)
at::Tensor scratch(size_t bytes, c10::DeviceIndex dev) { return bytes ? empty({(long long)bytes}, at::kByte, dev) : at::Tensor(); }
void* scratch_ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// (B, L, H, D) strides of a 4-D tensor in the cache's item layout; false if the call does not handle it
bool view4(const at::Tensor& x, bool bhlc, varq_tensor_t& d, long long& B, long long& L, long long& H, long long& D) {
    if (!x.is_cuda() || x.dim() != 4) return false;
    const int dt = dtype_code(x.scalar_type());
    if (dt < 0 || x.stride(3) != 1) return false;
    const int l = bhlc ? 2 : 1, h = bhlc ? 1 : 2;
    B = x.size(0); L = x.size(l); H = x.size(h); D = x.size(3);
    if (B <= 0 || L <= 0 || H <= 0 || D <= 0 || B > INT32_MAX || L > INT32_MAX || H > INT32_MAX || D > INT32_MAX) return false;
    d.ptr = x.data_ptr(); d.dtype = dt; d._pad = 0;
    d.stride_b = x.stride(0); d.stride_l = x.stride(l); d.stride_h = x.stride(h);
    return true;
}

long long group_of(const Cache* c, long long D) { return per_dim((int)c->method) ? 1 : c->group_size ? c->group_size : D; }

void param_desc(const Cache* c, int scale, int zp, long long row0, long long D, varq_qparams_t& p) {
    const at::Tensor &s = c->t[scale], &z = c->t[zp];
    const long long cap = s.size(2), nG = c->nG;
    p.scale = s.data_ptr<float>() + row0 * nG;
    p.zp = z.defined() ? z.data_ptr<float>() + row0 * nG : nullptr;
    p.row_of_token = nullptr;
    p.stride_b = c->nH * cap * nG; p.stride_r = nG; p.stride_h = cap * nG; p.stride_g = 1;
    p.share_b = c->reduce_batch != 0; p.share_l = share_l((int)c->method); p.share_h = share_h((int)c->method); p.group = (int)group_of(c, D);
    p.row_begin = nullptr; p.n_rows = 0; p._pad = 0;
}
void codes_desc(const Cache* c, int which, long long tok0, varq_tensor_t& d) {
    const long long cap = c->t[which].size(2), W = c->words;
    d.ptr = c->t[which].data_ptr<int32_t>() + tok0 * W; d.dtype = 0; d._pad = 0;
    d.stride_b = c->H * cap * W; d.stride_l = W; d.stride_h = cap * W;
}

// Room for n more tokens and `rows` more parameter rows; caches grow by doubling and start with a few hundred tokens (a schedule's first
// steps are tiny), unless a capacity hint was given.
void ensure(Cache* c, long long n, long long rows, long long B, long long H, long long D, c10::DeviceIndex dev) {
    const bool sl = share_l((int)c->method);
    if (!c->has_shape) {
        c->has_shape = 1; c->B = B; c->H = H; c->D = D;
        const long long vpw = 32 / store_bits(c);
        c->words = (D + vpw - 1) / vpw;
        c->nB = c->reduce_batch ? 1 : B; c->nH = share_h((int)c->method) ? 1 : H; c->nG = D / group_of(c, D);
        c->lcap = c->rcap = 0;
    }
    const long long need_l = c->n_tokens + n;
    if (!c->t[T_CODES].defined() || need_l > c->lcap) {
        long long cap = std::max({need_l, c->max_tokens, 2 * c->lcap});
        if (!c->max_tokens) cap = std::max(cap, 256ll);
        cap = (cap + 63) / 64 * 64;
        at::Tensor codes = empty({B, H, cap, c->words}, at::kInt, dev), rot;
        if (sl) rot = empty({cap}, at::kInt, dev);
        if (c->t[T_CODES].defined() && c->n_tokens) {
            codes.narrow(2, 0, c->n_tokens).copy_(c->t[T_CODES].narrow(2, 0, c->n_tokens));
            if (sl) rot.narrow(0, 0, c->n_tokens).copy_(c->t[T_ROT].narrow(0, 0, c->n_tokens));
        }
        c->t[T_CODES] = codes; c->t[T_ROT] = rot; c->lcap = cap;
        c->t[T_CODES_NEXT] = at::Tensor();
    }
    const long long need_r = c->n_rows + rows;
    if (!c->t[T_SCALE].defined() || need_r > c->rcap) {
        const long long cap = std::max({sl ? 64ll : c->lcap, need_r, 2 * c->rcap});
        at::Tensor s = empty({c->nB, c->nH, cap, c->nG}, at::kFloat, dev), z, rb;
        if (!c->symmetric) z = empty({c->nB, c->nH, cap, c->nG}, at::kFloat, dev);
        if (c->t[T_SCALE].defined() && c->n_rows) {
            s.narrow(2, 0, c->n_rows).copy_(c->t[T_SCALE].narrow(2, 0, c->n_rows));
            if (z.defined()) z.narrow(2, 0, c->n_rows).copy_(c->t[T_ZP].narrow(2, 0, c->n_rows));
        }
        if (sl) {
            rb = empty({cap + 1}, at::kInt, dev);
            if (c->t[T_RB].defined() && c->n_rows) rb.narrow(0, 0, c->n_rows + 1).copy_(c->t[T_RB].narrow(0, 0, c->n_rows + 1));
            c->t[T_RB] = rb;
        }
        c->t[T_SCALE] = s; c->t[T_ZP] = z; c->rcap = cap;
        c->t[T_SCALE_NEXT] = at::Tensor(); c->t[T_ZP_NEXT] = at::Tensor();
    }
}

// Whether the native path takes this step, and its shape
bool can_append(const Cache* c, const at::Tensor& x, varq_tensor_t& d, long long& B, long long& L, long long& H, long long& D) {
    if (!view4(x, c->bhlc, d, B, L, H, D)) return false;
    if (requant((int)c->method) && c->n_tokens) return false;
    if (c->pack && c->quant_bits != 2 && c->quant_bits != 4 && c->quant_bits != 8) return false;
    const long long group = group_of(c, D);
    if (group < 1 || D % group) return false;
    if (c->has_shape && (c->B != B || c->H != H || c->D != D)) return false;
    if (c->meta_set && c->pack && (c->meta_c != D || c->meta_bits != store_bits(c))) return false;
    if (c->t[T_CODES].defined() && c->t[T_CODES].device() != x.device()) return false;
    return true;
}
void fill_job(Cache* c, const varq_tensor_t& d, varq_append_job_t& j) {
    const bool sl = share_l((int)c->method);
    j.x = d; j.bits = (int)c->quant_bits; j.store_bits = store_bits(c); j.eps = (float)c->eps;
    j.token0 = (int)c->n_tokens; j.row0 = (int)c->n_rows; j._pad = 0;
    codes_desc(c, T_CODES, c->n_tokens, j.codes);
    param_desc(c, T_SCALE, T_ZP, c->n_rows, c->D, j.p);
    j.row_of_token = sl ? c->t[T_ROT].data_ptr<int32_t>() + c->n_tokens : nullptr;
    j.row_begin = sl ? c->t[T_RB].data_ptr<int32_t>() + c->n_rows : nullptr;
}
void set_pending(Cache* c, long long L) {
    c->pend_set = 1; c->pend[0] = L; c->pend[1] = share_l((int)c->method) ? 1 : L; c->pend[2] = 0;
    c->meta_set = 1; c->meta_c = c->D; c->meta_bits = store_bits(c);
}
void commit(Cache* c) {
    c->n_tokens += c->pend[0]; c->n_rows += c->pend[1];
    c->last_set = 1; c->last[0] = c->pend[0]; c->last[1] = c->pend[1];
    c->pend_set = 0;
}

// quantize (and commit) one or two tensors; 1 done, 0 declined, -1 error set
int append_n(Cache** c, const at::Tensor** x, int n, float norm_eps, bool commit_too) {
    varq_tensor_t d[2];
    long long B = 0, L = 0, H = 0, D = 0;
    for (int i = 0; i < n; ++i) {
        long long b, l, h, dd;
        if (!can_append(c[i], *x[i], d[i], b, l, h, dd)) return 0;
        if (i == 0) { B = b; L = l; H = h; D = dd; }
        else if (b != B || l != L || h != H || dd != D || x[i]->device() != x[0]->device()) return 0;
    }
    const c10::DeviceIndex dev = x[0]->device().index();
    const c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, dev));
    const auto st = c10::cuda::getCurrentCUDAStream(dev);
    varq_append_job_t jobs[2];
    for (int i = 0; i < n; ++i) {
        ensure(c[i], L, share_l((int)c[i]->method) ? 1 : L, B, H, D, dev);
        fill_job(c[i], d[i], jobs[i]);
    }
    size_t ws = varq_append_workspace_bytes(jobs, n, (int)B, (int)L, (int)H, (int)D, norm_eps);
    at::Tensor buf = scratch(ws, dev);
    int rc = varq_append(jobs, n, (int)B, (int)L, (int)H, (int)D, norm_eps, scratch_ptr(buf), ws, st.stream());
    if (rc == VARQ_ERR_UNSUPPORTED && norm_eps >= 0.f) return 0;
    if (rc == VARQ_ERR_WORKSPACE) {
        for (int i = 0; i < n; ++i) ws = std::max(ws, varq_quant_workspace_bytes((int)B, (int)L, (int)H, (int)D, jobs[i].x.dtype, jobs[i].store_bits, &jobs[i].p));
        buf = scratch(ws, dev);
        rc = varq_append(jobs, n, (int)B, (int)L, (int)H, (int)D, norm_eps, scratch_ptr(buf), ws, st.stream());
    }
    if (rc != VARQ_OK) { raise(rc); return -1; }
    for (int i = 0; i < n; ++i) { set_pending(c[i], L); if (commit_too) commit(c[i]); }
    return 1;
}

void cache_desc(const Cache* c, varq_tensor_t& codes, varq_qparams_t& p) {
    codes_desc(c, T_CODES, 0, codes);
    param_desc(c, T_SCALE, T_ZP, 0, c->D, p);
    if (c->t[T_ROT].defined()) {
        p.row_of_token = c->t[T_ROT].data_ptr<int32_t>();
        p.row_begin = c->t[T_RB].data_ptr<int32_t>();
        p.n_rows = (int)c->n_rows;
    }
}

// attention over the committed caches; new reference, nullptr with an error set, or Py_None (declined)
PyObject* attend_impl(const at::Tensor& q, Cache* k, Cache* v, double scale, PyObject* out_dtype, bool norm, const at::Tensor* mul, double eps) {
    varq_tensor_t qd, od, kc, vc;
    varq_qparams_t kp, vp;
    long long B, Lq, H, D;
    if (!k->n_tokens || k->n_tokens != v->n_tokens || !view4(q, k->bhlc, qd, B, Lq, H, D)) Py_RETURN_NONE;
    if (B != k->B || H != k->H || D != k->D || B != v->B || H != v->H || D != v->D) Py_RETURN_NONE;
    if (q.device() != k->t[T_CODES].device() || q.device() != v->t[T_CODES].device()) Py_RETURN_NONE;
    at::ScalarType os = norm ? at::kFloat : q.scalar_type();
    if (out_dtype != Py_None) {
        if (!THPDtype_Check(out_dtype)) Py_RETURN_NONE;
        os = reinterpret_cast<THPDtype*>(out_dtype)->scalar_type;
        if (dtype_code(os) < 0) Py_RETURN_NONE;
    }
    const c10::DeviceIndex dev = q.device().index();
    const c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, dev));
    const auto st = c10::cuda::getCurrentCUDAStream(dev);
    at::Tensor out = empty({B, Lq, H, D}, os, dev);
    od.ptr = out.data_ptr(); od.dtype = dtype_code(os); od._pad = 0;
    od.stride_b = Lq * H * D; od.stride_l = H * D; od.stride_h = D;
    cache_desc(k, kc, kp);
    cache_desc(v, vc, vp);
    const long long Lk = k->n_tokens;
    const size_t ws = varq_attn_workspace_bytes((int)B, (int)H, (int)Lq, (int)Lk, (int)D, store_bits(k), store_bits(v));
    const at::Tensor buf = scratch(ws, dev);
    void* const wp = scratch_ptr(buf);
    int rc;
    if (norm)
        rc = varq_attn_fwd_qnorm(&qd, &kc, &vc, &kp, &vp, (int)B, (int)H, (int)Lq, (int)Lk, (int)D, store_bits(k), store_bits(v), (float)scale,
                                 mul ? mul->data_ptr<float>() : nullptr, (float)eps, &od, wp, ws, st.stream());
    else
        rc = varq_attn_fwd(&qd, &kc, &vc, &kp, &vp, (int)B, (int)H, (int)Lq, (int)Lk, (int)D, store_bits(k), store_bits(v), (float)scale, &od, wp, ws, st.stream());
    if (rc != VARQ_OK) return raise(rc);
    return THPVariable_Wrap(out);
}

at::Tensor dequant_impl(Cache* c, int codes, int scale, int zp, long long tok0, long long n, long long row0, bool rot, int* rc) {
    varq_tensor_t cd, od;
    varq_qparams_t p;
    const c10::DeviceIndex dev = c->t[codes].device().index();
    const c10::cuda::OptionalCUDAGuard guard(c10::Device(c10::kCUDA, dev));
    at::Tensor out = c->bhlc ? empty({c->B, c->H, n, c->D}, at::kFloat, dev) : empty({c->B, n, c->H, c->D}, at::kFloat, dev);
    codes_desc(c, codes, tok0, cd);
    param_desc(c, scale, zp, row0, c->D, p);
    if (rot) p.row_of_token = c->t[T_ROT].data_ptr<int32_t>() + tok0;
    else if (p.share_l) p.stride_r = 0;       // one row describes every token of the range
    od.ptr = out.data_ptr(); od.dtype = VARQ_F32; od._pad = 0;
    od.stride_b = n * c->H * c->D;
    od.stride_l = c->bhlc ? c->D : c->H * c->D; od.stride_h = c->bhlc ? n * c->D : c->D;
    *rc = varq_unpack_dequant(&cd, (int)c->B, (int)n, (int)c->H, (int)c->D, store_bits(c), &p, &od, c10::cuda::getCurrentCUDAStream(dev).stream());
    return out;
}
PyObject* wrap_dequant(const at::Tensor& t, int rc) { return rc == VARQ_OK ? THPVariable_Wrap(t) : raise(rc); }

#define GUARD_BEGIN try {
#define GUARD_END } catch (const std::exception& e) { if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what()); return nullptr; }

bool want(Py_ssize_t n, Py_ssize_t expected) {
    if (n == expected) return true;
    PyErr_SetString(PyExc_TypeError, "wrong number of arguments");
    return false;
}
PyObject* bool_result(int r) { if (r < 0) return nullptr; return PyBool_FromLong(r); }

// append(cache, item, commit) -> bool
PyObject* py_append(PyObject*, PyObject* const* a, Py_ssize_t n) {
    GUARD_BEGIN
    if (!want(n, 3)) return nullptr;
    if (!is_cache(a[0]) || !THPVariable_Check(a[1])) Py_RETURN_FALSE;
    Cache* c = reinterpret_cast<Cache*>(a[0]);
    const at::Tensor& x = THPVariable_Unpack(a[1]);
    const at::Tensor* px = &x;
    return bool_result(append_n(&c, &px, 1, -1.f, a[2] == Py_True));
    GUARD_END
}
// attend(q, k_cache, v_cache, scale, out_dtype) -> Tensor or None
PyObject* py_attend(PyObject*, PyObject* const* a, Py_ssize_t n) {
    GUARD_BEGIN
    if (!want(n, 5)) return nullptr;
    if (!THPVariable_Check(a[0]) || !is_cache(a[1]) || !is_cache(a[2])) Py_RETURN_NONE;
    const double scale = PyFloat_AsDouble(a[3]);
    if (scale == -1.0 && PyErr_Occurred()) return nullptr;
    return attend_impl(THPVariable_Unpack(a[0]), reinterpret_cast<Cache*>(a[1]), reinterpret_cast<Cache*>(a[2]), scale, a[4], false, nullptr, 0.0);
    GUARD_END
}
// what both step functions ask of q, k, v and the caches before anything is changed
bool step_ok(PyObject* const* qkv, PyObject* kc, PyObject* vc, PyObject* out_dtype) {
    if (!THPVariable_Check(qkv[0]) || !THPVariable_Check(qkv[1]) || !THPVariable_Check(qkv[2]) || !is_cache(kc) || !is_cache(vc) || kc == vc) return false;
    const Cache *k = reinterpret_cast<Cache*>(kc), *v = reinterpret_cast<Cache*>(vc);
    const at::Tensor &q = THPVariable_Unpack(qkv[0]), &x = THPVariable_Unpack(qkv[1]);
    varq_tensor_t d;
    long long B, L, H, D;
    if (k->debug || v->debug || k->bhlc != v->bhlc || k->n_tokens != v->n_tokens || (out_dtype != Py_None && !THPDtype_Check(out_dtype))) return false;
    if (!view4(q, k->bhlc, d, B, L, H, D) || x.dim() != 4 || q.device() != x.device()) return false;
    return B == x.size(0) && H == x.size(k->bhlc ? 1 : 2) && D == x.size(3);
}
PyObject* finish_step(PyObject* out) {
    if (out == Py_None) { Py_DECREF(out); PyErr_SetString(PyExc_ValueError, "[VAR-Q]: q does not match the cache"); return nullptr; }
    return out;
}
// step(q, k, v, k_cache, v_cache, scale, out_dtype) -> Tensor or None (nothing done)
PyObject* py_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
    GUARD_BEGIN
    if (!want(n, 7)) return nullptr;
    if (!step_ok(a, a[3], a[4], a[6])) Py_RETURN_NONE;
    Cache* c[2] = {reinterpret_cast<Cache*>(a[3]), reinterpret_cast<Cache*>(a[4])};
    const at::Tensor* x[2] = {&THPVariable_Unpack(a[1]), &THPVariable_Unpack(a[2])};
    const double scale = PyFloat_AsDouble(a[5]);
    if (scale == -1.0 && PyErr_Occurred()) return nullptr;
    const int r = append_n(c, x, 2, -1.f, true);
    if (r < 0) return nullptr;
    if (r == 0) Py_RETURN_NONE;
    return finish_step(attend_impl(THPVariable_Unpack(a[0]), c[0], c[1], scale, a[6], false, nullptr, 0.0));
    GUARD_END
}
// step_normalised(q, k, v, scale_mul or None, k_cache, v_cache, scale, out_dtype, eps) -> Tensor or None (nothing done)
PyObject* py_step_normalised(PyObject*, PyObject* const* a, Py_ssize_t n) {
    GUARD_BEGIN
    if (!want(n, 9)) return nullptr;
    if (!step_ok(a, a[4], a[5], a[7])) Py_RETURN_NONE;
    Cache* c[2] = {reinterpret_cast<Cache*>(a[4]), reinterpret_cast<Cache*>(a[5])};
    const at::Tensor *x[2] = {&THPVariable_Unpack(a[1]), &THPVariable_Unpack(a[2])}, &q = THPVariable_Unpack(a[0]);
    at::Tensor mul;
    if (a[3] != Py_None) {
        if (!THPVariable_Check(a[3])) Py_RETURN_NONE;
        mul = THPVariable_Unpack(a[3]);
        if (mul.requires_grad()) mul = mul.detach();
        if (mul.numel() != q.size(c[0]->bhlc ? 1 : 2) || !mul.is_cuda() || mul.device() != q.device()) Py_RETURN_NONE;
        if (mul.scalar_type() != at::kFloat || !mul.is_contiguous()) mul = mul.to(at::kFloat).reshape({-1}).contiguous();
    }
    const double scale = PyFloat_AsDouble(a[6]), eps = PyFloat_AsDouble(a[8]);
    if (PyErr_Occurred()) return nullptr;
    const int r = append_n(c, x, 2, (float)eps, true);
    if (r < 0) return nullptr;
    if (r == 0) Py_RETURN_NONE;
    return finish_step(attend_impl(q, c[0], c[1], scale, a[7], true, mul.defined() ? &mul : nullptr, eps));
    GUARD_END
}
// use_var_q(cache, item) -> Tensor or None (nothing done)
PyObject* py_use(PyObject*, PyObject* const* a, Py_ssize_t n) {
    GUARD_BEGIN
    if (!want(n, 2)) return nullptr;
    if (!is_cache(a[0]) || !THPVariable_Check(a[1])) Py_RETURN_NONE;
    Cache* c = reinterpret_cast<Cache*>(a[0]);
    if (c->debug) Py_RETURN_NONE;
    const at::Tensor& x = THPVariable_Unpack(a[1]);
    const at::Tensor* px = &x;
    const int r = append_n(&c, &px, 1, -1.f, true);
    if (r < 0) return nullptr;
    if (r == 0) Py_RETURN_NONE;
    int rc = VARQ_OK;
    const at::Tensor out = dequant_impl(c, T_CODES, T_SCALE, T_ZP, 0, c->n_tokens, 0, c->t[T_ROT].defined(), &rc);
    return wrap_dequant(out, rc);
    GUARD_END
}
// dequant(cache, which) -> Tensor or None; which: 0 the whole committed cache, 1 the step quantized last
PyObject* py_dequant(PyObject*, PyObject* const* a, Py_ssize_t n) {
    GUARD_BEGIN
    if (!want(n, 2)) return nullptr;
    if (!is_cache(a[0])) Py_RETURN_NONE;
    Cache* c = reinterpret_cast<Cache*>(a[0]);
    const long which = PyLong_AsLong(a[1]);
    int rc = VARQ_OK;
    if (which == 0) {
        if (!c->n_tokens) Py_RETURN_NONE;
        const at::Tensor out = dequant_impl(c, T_CODES, T_SCALE, T_ZP, 0, c->n_tokens, 0, c->t[T_ROT].defined(), &rc);
        return wrap_dequant(out, rc);
    }
    if (c->pend_set) {
        const bool rep = c->pend[2] != 0;
        const at::Tensor out = dequant_impl(c, rep ? T_CODES_NEXT : T_CODES, rep ? T_SCALE_NEXT : T_SCALE, rep ? T_ZP_NEXT : T_ZP, rep ? 0 : c->n_tokens, c->pend[0],
                                            rep ? 0 : c->n_rows, false, &rc);
        return wrap_dequant(out, rc);
    }
    if (!c->n_tokens || !c->last_set) Py_RETURN_NONE;
    const at::Tensor out = dequant_impl(c, T_CODES, T_SCALE, T_ZP, c->n_tokens - c->last[0], c->last[0], c->n_rows - c->last[1], false, &rc);
    return wrap_dequant(out, rc);
    GUARD_END
}

// ---------------------------------------------------------------- attributes
enum Field : long { F_BITS, F_METHOD, F_PACK, F_SYM, F_REDUCE, F_GROUP, F_MAX, F_DEBUG, F_FMT, F_EPS, F_SHAPE, F_PEND, F_LAST, F_META,
                    F_WORDS, F_NB, F_NH, F_NG, F_LCAP, F_RCAP, F_NTOK, F_NROWS, F_T0 };
long long* int_field(Cache* c, long f) {
    switch (f) {
        case F_BITS: return &c->quant_bits; case F_PACK: return &c->pack; case F_SYM: return &c->symmetric; case F_REDUCE: return &c->reduce_batch;
        case F_DEBUG: return &c->debug; case F_WORDS: return &c->words; case F_NB: return &c->nB; case F_NH: return &c->nH; case F_NG: return &c->nG;
        case F_LCAP: return &c->lcap; case F_RCAP: return &c->rcap; case F_NTOK: return &c->n_tokens; case F_NROWS: return &c->n_rows;
        case F_GROUP: return &c->group_size; case F_MAX: return &c->max_tokens;
    }
    return nullptr;
}
PyObject* get_field(PyObject* self, void* closure) {
    GUARD_BEGIN
    Cache* c = reinterpret_cast<Cache*>(self);
    const long f = (long)(intptr_t)closure;
    if (f >= F_T0) { const at::Tensor& t = c->t[f - F_T0]; if (!t.defined()) Py_RETURN_NONE; return THPVariable_Wrap(t); }
    switch (f) {
        case F_METHOD: return PyUnicode_FromString(METHOD_NAMES[c->method]);
        case F_FMT: return PyUnicode_FromString(c->bhlc ? "BHLc" : "BLHc");
        case F_EPS: return PyFloat_FromDouble(c->eps);
        case F_PACK: case F_SYM: case F_REDUCE: case F_DEBUG: return PyBool_FromLong(*int_field(c, f) != 0);
        case F_GROUP: case F_MAX: if (!*int_field(c, f)) Py_RETURN_NONE; return PyLong_FromLongLong(*int_field(c, f));
        case F_SHAPE: if (!c->has_shape) Py_RETURN_NONE; return Py_BuildValue("(LLL)", c->B, c->H, c->D);
        case F_PEND: if (!c->pend_set) Py_RETURN_NONE; return Py_BuildValue("(LLO)", c->pend[0], c->pend[1], c->pend[2] ? Py_True : Py_False);
        case F_LAST: if (!c->last_set) Py_RETURN_NONE; return Py_BuildValue("(LL)", c->last[0], c->last[1]);
        case F_META: {
            if (!c->meta_set) Py_RETURN_NONE;
            const long long vpw = 32 / c->meta_bits;
            return Py_BuildValue("{s:L,s:L,s:L,s:L}", "orig_c", c->meta_c, "vals_per_word", vpw, "pad_len", (vpw - c->meta_c % vpw) % vpw, "bits", c->meta_bits);
        }
    }
    return PyLong_FromLongLong(*int_field(c, f));
    GUARD_END
}
int set_field(PyObject* self, PyObject* v, void* closure) {
    Cache* c = reinterpret_cast<Cache*>(self);
    const long f = (long)(intptr_t)closure;
    if (!v) { PyErr_SetString(PyExc_AttributeError, "cannot delete this attribute"); return -1; }
    if (f >= F_T0) {
        if (v == Py_None) { c->t[f - F_T0] = at::Tensor(); return 0; }
        if (!THPVariable_Check(v)) { PyErr_SetString(PyExc_TypeError, "a tensor or None is expected"); return -1; }
        c->t[f - F_T0] = THPVariable_Unpack(v);
        return 0;
    }
    switch (f) {
        case F_METHOD: {
            const char* s = PyUnicode_AsUTF8(v);
            if (!s) return -1;
            for (int m = 0; m < M_COUNT; ++m) if (!strcmp(s, METHOD_NAMES[m])) { c->method = m; return 0; }
            PyErr_Format(PyExc_ValueError, "Invalid quant_method: %s", s);
            return -1;
        }
        case F_FMT: { const char* s = PyUnicode_AsUTF8(v); if (!s) return -1; c->bhlc = !strcmp(s, "BHLc"); return 0; }
        case F_EPS: c->eps = PyFloat_AsDouble(v); return PyErr_Occurred() ? -1 : 0;
        case F_PACK: case F_SYM: case F_REDUCE: case F_DEBUG: { const int t = PyObject_IsTrue(v); if (t < 0) return -1; *int_field(c, f) = t; return 0; }
        case F_SHAPE: c->has_shape = v != Py_None; return c->has_shape && !PyArg_ParseTuple(v, "LLL", &c->B, &c->H, &c->D) ? -1 : 0;
        case F_PEND: c->pend_set = v != Py_None; return c->pend_set && !PyArg_ParseTuple(v, "LLL", &c->pend[0], &c->pend[1], &c->pend[2]) ? -1 : 0;
        case F_LAST: c->last_set = v != Py_None; return c->last_set && !PyArg_ParseTuple(v, "LL", &c->last[0], &c->last[1]) ? -1 : 0;
        case F_META: {
            c->meta_set = v != Py_None;
            if (!c->meta_set) return 0;
            PyObject *oc = PyMapping_GetItemString(v, "orig_c"), *ob = oc ? PyMapping_GetItemString(v, "bits") : nullptr;
            if (oc) { c->meta_c = PyLong_AsLongLong(oc); Py_DECREF(oc); }
            if (ob) { c->meta_bits = PyLong_AsLongLong(ob); Py_DECREF(ob); }
            return PyErr_Occurred() ? -1 : 0;
        }
    }
    if (v == Py_None && (f == F_GROUP || f == F_MAX)) { *int_field(c, f) = 0; return 0; }
    *int_field(c, f) = PyLong_AsLongLong(v);
    return PyErr_Occurred() ? -1 : 0;
}
#define FIELD(NAME, ID) {NAME, get_field, set_field, nullptr, reinterpret_cast<void*>((intptr_t)(ID))}
PyGetSetDef cache_getset[] = {
    FIELD("quant_bits", F_BITS), FIELD("quant_method", F_METHOD), FIELD("pack_to_int32", F_PACK), FIELD("symmetric", F_SYM), FIELD("reduce_batch", F_REDUCE),
    FIELD("group_size", F_GROUP), FIELD("_max_tokens", F_MAX), FIELD("debug", F_DEBUG), FIELD("_fmt", F_FMT), FIELD("eps", F_EPS), FIELD("_shape", F_SHAPE),
    FIELD("_pending", F_PEND), FIELD("_last", F_LAST), FIELD("_pack_meta", F_META), FIELD("_words", F_WORDS), FIELD("_nB", F_NB), FIELD("_nH", F_NH),
    FIELD("_nG", F_NG), FIELD("_lcap", F_LCAP), FIELD("_rcap", F_RCAP), FIELD("_n_tokens", F_NTOK), FIELD("_n_rows", F_NROWS),
    FIELD("_codes", F_T0 + T_CODES), FIELD("_codes_next", F_T0 + T_CODES_NEXT), FIELD("_scale_tbl", F_T0 + T_SCALE), FIELD("_zp_tbl", F_T0 + T_ZP),
    FIELD("_scale_next", F_T0 + T_SCALE_NEXT), FIELD("_zp_next", F_T0 + T_ZP_NEXT), FIELD("_row_of_token", F_T0 + T_ROT), FIELD("_row_begin", F_T0 + T_RB),
    {nullptr, nullptr, nullptr, nullptr, nullptr}};

PyObject* cache_new(PyTypeObject* type, PyObject*, PyObject*) {
    PyObject* self = type->tp_alloc(type, 0);       // zeroed
    if (!self) return nullptr;
    Cache* c = reinterpret_cast<Cache*>(self);
    for (auto& t : c->t) new (&t) at::Tensor();
    c->quant_bits = 8; c->method = M_SCALE_HEAD_DIM; c->pack = c->symmetric = c->reduce_batch = 1; c->eps = 1e-12;
    return self;
}
void cache_dealloc(PyObject* self) {
    Cache* c = reinterpret_cast<Cache*>(self);
    for (auto& t : c->t) t.~Tensor();
    PyTypeObject* type = Py_TYPE(self);
    type->tp_free(self);
    Py_DECREF(type);
}
int cache_init(PyObject*, PyObject*, PyObject*) { return 0; }
PyType_Slot cache_slots[] = {{Py_tp_new, (void*)cache_new}, {Py_tp_dealloc, (void*)cache_dealloc}, {Py_tp_init, (void*)cache_init}, {Py_tp_getset, cache_getset},
                             {Py_tp_doc, (void*)"State of one quantized cache: settings, packed codes, parameter tables."}, {0, nullptr}};
PyType_Spec cache_spec = {"VAR_Q._host.Cache", sizeof(Cache), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE, cache_slots};

#define FAST(NAME, FN, DOC) {NAME, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(FN)), METH_FASTCALL, DOC}
PyMethodDef methods[] = {
    FAST("append", py_append, "append(cache, item, commit) -> bool"),
    FAST("attend", py_attend, "attend(q, k_cache, v_cache, scale, out_dtype) -> Tensor or None"),
    FAST("step", py_step, "step(q, k, v, k_cache, v_cache, scale, out_dtype) -> Tensor or None"),
    FAST("step_normalised", py_step_normalised, "step_normalised(q, k, v, scale_mul, k_cache, v_cache, scale, out_dtype, eps) -> Tensor or None"),
    FAST("use_var_q", py_use, "use_var_q(cache, item) -> Tensor or None"),
    FAST("dequant", py_dequant, "dequant(cache, which) -> Tensor or None"),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Host path of the VAR_Q package.", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" PyMODINIT_FUNC PyInit__host(void) {
    PyObject* m = PyModule_Create(&module);
    if (!m) return nullptr;
    PyObject* t = PyType_FromSpec(&cache_spec);
    if (!t) { Py_DECREF(m); return nullptr; }
    cache_type = reinterpret_cast<PyTypeObject*>(t);
    Py_INCREF(t);
    if (PyModule_AddObject(m, "Cache", t) < 0) { Py_DECREF(t); Py_DECREF(m); return nullptr; }
    return m;
}
