// The tensor-level calls of ops_seq.py that small steps make most, from Python tensors to the library's entry points without ctypes: what bounds
// such a step is the host's work between two launches.  us a call: a product of 8 rows 10.6 -> 4.6 (its kernel 4.3); routed experts of one token, four
// calls, 61 -> 37; attention over a cache of 100 keys 25 -> 13.
//
// Every function gets what its wrapper got, in order, and answers with the wrapper's result; with None where the arguments are not the plain
// case (other types, tensor subclasses, modes that watch calls, memory without an address: the wrapper goes on and says what is wrong); or with the
// library's status as an int where that is not 0.  The entry points' addresses come from the library that Python loaded (bind), so there is one of it.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../../include/umbrella_b200_seq.h"

namespace {

struct Entries {
    decltype(&umbs_gemm) gemm;
    decltype(&umbs_gemm_sorted) gemm_sorted;
    decltype(&umbs_moe_route) moe_route;
    decltype(&umbs_add_norm) add_norm;
    decltype(&umbs_kv_pool) kv_pool;
    decltype(&umbs_cached_attention_ex) cached_attention;
    decltype(&umbs_ring_append) ring_append;
    decltype(&umbs_window_attention_gated) window_attention;
    decltype(&umbs_retention_ex) retention;
} g{};
constexpr int kEntries = sizeof(Entries) / sizeof(void*);

struct NotPlain {};                                         // the wrapper's own way

using Args = PyObject* const*;

const at::Tensor* tensor_or_null(PyObject* o) {
    if (o == Py_None) return nullptr;
    if (!THPVariable_CheckExact(o)) throw NotPlain();
    return &THPVariable_Unpack(o);
}
const at::Tensor& tensor(PyObject* o) {
    const at::Tensor* t = tensor_or_null(o);
    if (t == nullptr) throw NotPlain();
    return *t;
}
long integer(PyObject* o) {
    const long v = PyLong_Check(o) ? PyLong_AsLong(o) : -1;     // (True and False are ints)
    if (!PyLong_Check(o) || (v == -1 && PyErr_Occurred())) throw NotPlain();
    return v;
}
int small(PyObject* o) {
    const long v = integer(o);
    if (v != (int)v) throw NotPlain();
    return (int)v;
}
long integer_or(PyObject* o, long none) { return o == Py_None ? none : integer(o); }
float number(PyObject* o) {
    if (!PyFloat_Check(o) && !PyLong_Check(o)) throw NotPlain();
    const double v = PyFloat_AsDouble(o);
    if (v == -1. && PyErr_Occurred()) throw NotPlain();
    return (float)v;
}
bool truth(PyObject* o) {
    if (!PyBool_Check(o)) throw NotPlain();
    return o == Py_True;
}
template <typename T = void> T* at_(const at::Tensor& t) { return (T*)t.mutable_data_ptr(); }
template <typename T = void> T* at_(const at::Tensor* t) { return t != nullptr ? (T*)t->mutable_data_ptr() : nullptr; }
int mode_of(at::ScalarType t) {
    if (t == at::kBFloat16) return UMBS_BF16;
    if (t == at::kFloat) return UMBS_F32;
    throw NotPlain();
}
int mode(const at::Tensor& t) {
    if (!t.is_cuda()) throw NotPlain();
    return mode_of(t.scalar_type());
}
at::Tensor empty(at::IntArrayRef s, at::ScalarType t, const at::Tensor& like) { return at::empty(s, at::TensorOptions(t).device(like.device())); }
void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
template <typename F> int call(F f) {
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = f();
    Py_END_ALLOW_THREADS
    return rc;
}
PyObject* result(int rc, at::Tensor t) { return rc != 0 ? PyLong_FromLong(rc) : THPVariable_Wrap(std::move(t)); }

template <typename F> PyObject* guarded(Py_ssize_t n, Py_ssize_t want, F f) {
    if (n != want) {
        PyErr_SetString(PyExc_TypeError, "wrong number of arguments");
        return nullptr;
    }
    try {
        if (g.gemm != nullptr && !at::impl::torch_function_mode_enabled() && !c10::impl::TorchDispatchModeTLS::any_modes_set()) return f();
    } catch (...) {                                         // (only in front of the first launch: everything is read and made before it)
        PyErr_Clear();
    }
    Py_RETURN_NONE;
}

// a, w, out_f32, groups, a_goff, c_goff, n, k, grp_off, row_src, rows, dual, limit, max_rows
PyObject* gemm(PyObject*, Args p, Py_ssize_t n_args) {
    return guarded(n_args, 14, [&]() -> PyObject* {
        const at::Tensor &a = tensor(p[0]), &w = tensor(p[1]);
        const int md = mode(a), wd = (int)w.dim();
        if (a.dim() < 1 || wd < 2 || w.scalar_type() != a.scalar_type() || a.stride(-1) != 1 || !w.is_contiguous()) throw NotPlain();
        const bool f32 = truth(p[2]), dual = truth(p[11]);
        const int groups = small(p[3]), a_goff = small(p[4]), c_goff = small(p[5]);
        const int64_t w1 = w.size(wd - 1), w2 = w.size(wd - 2), K = integer_or(p[7], w1), N = integer_or(p[6], w2 / (dual ? 2 : 1));
        const at::Tensor *off = tensor_or_null(p[8]), *src = tensor_or_null(p[9]);
        const int64_t M = integer_or(p[10], a.size(0)), most = integer_or(p[13], M), cols = groups == 1 || off != nullptr ? N : (int64_t)groups * c_goff;
        if (K != (int)K || N != (int)N || M != (int)M || most != (int)most || M < 0 || cols < 0) throw NotPlain();
        const float limit = number(p[12]);
        const at::TensorOptions to = at::TensorOptions(f32 ? at::kFloat : a.scalar_type()).device(a.device());
        void *pa = at_(a), *pw = at_(w), *st = stream();
        int32_t *po = at_<int32_t>(off), *ps = at_<int32_t>(src);
        const int64_t lda = a.stride(0);
        if (off != nullptr && a_goff == 0 && c_goff == 0) {
            at::Tensor out = at::empty({M, cols}, to);
            void* pc = at_(out);
            return result(call([&] { return g.gemm_sorted(md, pa, lda, pw, w1, w2 * w1, pc, cols, f32, (int)most, (int)M, (int)N, (int)K, groups, po, ps, dual, limit, st); }), out);
        }
        // (zeros only where the product may leave gaps: see the wrapper)
        at::Tensor out = groups == 1 && off == nullptr && most >= M ? at::empty({M, cols}, to) : at::zeros({M, cols}, to);
        void* pc = at_(out);
        return result(call([&] { return g.gemm(md, pa, lda, a_goff, pw, w1, w2 * w1, pc, cols, c_goff, f32, (int)most, (int)N, (int)K, groups, po, ps, dual, limit, st); }), out);
    });
}

// h, w_router, top
PyObject* moe_route(PyObject*, Args p, Py_ssize_t n_args) {
    return guarded(n_args, 3, [&]() -> PyObject* {
        const at::Tensor &h = tensor(p[0]), &r = tensor(p[1]);
        const int md = mode(h), top = small(p[2]);
        if (h.dim() != 2 || r.dim() < 1 || top < 1) throw NotPlain();
        const int64_t n = h.size(0), width = h.size(1), E = r.size(0);
        if (n != (int)n || width != (int)width || E != (int)E || n * top != (int)(n * top)) throw NotPlain();
        at::Tensor sel_w = empty({n, top}, at::kFloat, h), off = empty({E + 1}, at::kInt, h), tok = empty({n * top}, at::kInt, h), pos = empty({n * top}, at::kInt, h),
                   scratch = empty({2 * E + n * top}, at::kInt, h);
        at::Tensor sel_e = scratch.narrow(0, 2 * E, n * top).view({n, top});
        void *ph = at_(h), *st = stream();
        float *pr = at_<float>(r), *pw = at_<float>(sel_w);
        int32_t *po = at_<int32_t>(off), *pt = at_<int32_t>(tok), *pp = at_<int32_t>(pos), *pc = at_<int32_t>(scratch);
        const int rc = call([&] { return g.moe_route(md, ph, (int)n, (int)width, pr, (int)E, top, pw, po, pt, pp, pc, st); });
        if (rc != 0) return PyLong_FromLong(rc);
        return Py_BuildValue("(NNNNN)", THPVariable_Wrap(sel_w), THPVariable_Wrap(off), THPVariable_Wrap(tok), THPVariable_Wrap(pos), THPVariable_Wrap(sel_e));
    });
}

// x, w, b, eps, kind, w_offset, dtype's number (UMBS_*), rows, delta, pair_out, sel_w, pair_pos, shared, shared_gate, scale, mult, want_copy
PyObject* add_norm(PyObject*, Args p, Py_ssize_t n_args) {
    return guarded(n_args, 17, [&]() -> PyObject* {
        const at::Tensor &x = tensor(p[0]), *w = tensor_or_null(p[1]), *b = tensor_or_null(p[2]), *rows = tensor_or_null(p[7]), *delta = tensor_or_null(p[8]),
                         *pair = tensor_or_null(p[9]), *sel = tensor_or_null(p[10]), *pos = tensor_or_null(p[11]), *shared = tensor_or_null(p[12]),
                         *gate = tensor_or_null(p[13]), *scale = tensor_or_null(p[14]);
        const int md = small(p[6]), kind = small(p[4]);
        if (!x.is_cuda() || x.dim() != 2 || (sel != nullptr && sel->dim() < 2)) throw NotPlain();
        const float eps = number(p[3]), w_offset = number(p[5]);
        const bool copied = truth(p[16]);
        const int64_t n = rows != nullptr ? rows->numel() : x.size(0), width = x.size(1);
        if (n != (int)n || width != (int)width) throw NotPlain();
        umbs_delta_t d{};
        const bool any = delta != nullptr || pair != nullptr || shared != nullptr;
        if (any) {
            d.delta = at_<float>(delta);
            d.pair_out = at_<float>(pair);
            d.sel_w = at_<float>(sel);
            d.pair_pos = at_<int32_t>(pos);
            d.top = sel != nullptr ? (int)sel->size(1) : 0;
            d.shared = at_<float>(shared);
            d.shared_gate = at_<float>(gate);
            d.scale = at_<float>(scale);
            d.mult = number(p[15]);
        }
        at::Tensor y = empty({n, width}, md == UMBS_BF16 ? at::kBFloat16 : at::kFloat, x), copy;
        if (copied) copy = empty({n, width}, at::kFloat, x);
        float *px = at_<float>(x), *pw = at_<float>(w), *pb = at_<float>(b), *pc = copied ? at_<float>(copy) : nullptr;
        int32_t* pr = at_<int32_t>(rows);
        void *py = at_(y), *st = stream();
        const int rc = call([&] { return g.add_norm(md, px, any ? &d : nullptr, pr, (int)n, kind, pw, pb, w_offset, (int)width, eps, py, pc, st); });
        if (rc != 0 || !copied) return result(rc, y);
        return Py_BuildValue("(NN)", THPVariable_Wrap(y), THPVariable_Wrap(copy));
    });
}

// q, kv, kv_cache, the batch's address, heads, kv_heads, dim, vdim, scale, mode, window, pool, pool_cache, head_bias, gate, gate_per_head, append, split, sink
PyObject* cached_attention(PyObject*, Args p, Py_ssize_t n_args) {
    return guarded(n_args, 19, [&]() -> PyObject* {
        const at::Tensor &q = tensor(p[0]), &kv = tensor(p[1]), &cache = tensor(p[2]), *pools = tensor_or_null(p[12]), *bias = tensor_or_null(p[13]),
                         *gate = tensor_or_null(p[14]), *sink = tensor_or_null(p[18]);
        const umbs_batch_t* b = (const umbs_batch_t*)integer(p[3]);
        const int md = mode(q), heads = small(p[4]), kvh = small(p[5]), dim = small(p[6]), vdim = small(p[7]), how = small(p[9]), window = small(p[10]), pool = small(p[11]);
        const float scale = number(p[8]);
        const bool per_head = truth(p[15]), append = truth(p[16]), split = truth(p[17]);
        if (b == nullptr || q.dim() < 1 || cache.dim() < 2 || (pools != nullptr && pools->dim() < 2) || (gate != nullptr && gate->dim() < 1) || (pool > 0 && pools == nullptr) ||
            heads < 0 || vdim < 0)
            throw NotPlain();
        const int row = kvh * (dim + vdim), kv_len = (int)cache.size(1), pool_len = pools != nullptr ? (int)pools->size(1) : 0;
        at::Tensor out = empty({q.size(0), (int64_t)heads * vdim}, q.scalar_type(), q), part;
        const int64_t parts = 2048 * ((int64_t)vdim + 2);
        if (split) part = empty({parts}, at::kFloat, q);
        umbs_attn_opts_t o{};
        o.sink = at_<float>(sink);
        void *pq = at_(q), *pkv = at_(kv), *pc = at_(cache), *pp = at_(pools), *po = at_(out), *st = stream();
        float *pb = at_<float>(bias), *pg = at_<float>(gate), *ps = split ? at_<float>(part) : nullptr;
        const int64_t ldg = gate != nullptr ? gate->stride(0) : 0;
        const int rc = call([&] {
            int e = pool > 0 ? g.kv_pool(md, pkv, pc, kv_len, pp, pool_len, b, row, pool, st) : 0;
            if (e == 0)
                e = g.cached_attention(md, how, pq, pkv, pc, kv_len, pp, pool_len, b, heads, kvh, dim, vdim, window, pool, scale, pb, pg, ldg, per_head, &o, ps,
                                       split ? parts * 4 : 0, po, st);
            return e == 0 && append ? g.ring_append(md, pkv, pc, kv_len, b, row, st) : e;
        });
        return result(rc, out);
    });
}

// q, k, k_shared, v, the batch's address, heads, scale, window, sink, use_sink, gate, gate_per_head
PyObject* window_attention(PyObject*, Args p, Py_ssize_t n_args) {
    return guarded(n_args, 12, [&]() -> PyObject* {
        const at::Tensor &q = tensor(p[0]), &k = tensor(p[1]), *ks = tensor_or_null(p[2]), &v = tensor(p[3]), *sink = tensor_or_null(p[8]), *gate = tensor_or_null(p[10]);
        const umbs_batch_t* b = (const umbs_batch_t*)integer(p[4]);
        const int md = mode(q), heads = small(p[5]), window = small(p[7]);
        const float scale = number(p[6]);
        const bool use_sink = truth(p[9]), per_head = truth(p[11]);
        if (b == nullptr || heads < 1 || q.dim() != 2 || k.dim() != 2 || v.dim() != 2 || (ks != nullptr && ks->dim() != 2) || (gate != nullptr && gate->dim() < 1)) throw NotPlain();
        const int sd = ks != nullptr ? (int)ks->size(1) : 0, dim = (int)(k.size(1) / heads), vdim = (int)(v.size(1) / heads);
        if (q.size(1) != (int64_t)heads * (dim + sd)) throw NotPlain();
        at::Tensor out = empty({q.size(0), (int64_t)heads * vdim}, q.scalar_type(), q);
        void *pq = at_(q), *pk = at_(k), *pks = at_(ks), *pv = at_(v), *po = at_(out), *st = stream();
        float *psk = at_<float>(sink), *pg = at_<float>(gate);
        return result(call([&] {
            return g.window_attention(md, pq, q.stride(0), pk, k.stride(0), pks, ks != nullptr ? ks->stride(0) : 0, sd, pv, v.stride(0), b, heads, dim, vdim, window, scale,
                                      use_sink ? UMBS_ATTN_SOFTMAX_SINK : UMBS_ATTN_SOFTMAX, psk, pg, gate != nullptr ? gate->stride(0) : 0, per_head, po,
                                      (int64_t)heads * vdim, st);
        }), out);
    });
}

// qkvg, the batch's address, heads, dim, vdim, rot_dims, inv_freq, decay, eps, state, dtype's number, segments, k_scale, norm_w, norm_parts, gate_act
PyObject* retention(PyObject*, Args p, Py_ssize_t n_args) {
    return guarded(n_args, 16, [&]() -> PyObject* {
        const at::Tensor &x = tensor(p[0]), *freq = tensor_or_null(p[6]), *decay = tensor_or_null(p[7]), *state = tensor_or_null(p[9]), *norm = tensor_or_null(p[13]);
        const umbs_batch_t* b = (const umbs_batch_t*)integer(p[1]);
        const int heads = small(p[2]), dim = small(p[3]), vdim = small(p[4]), rot = small(p[5]), md = small(p[10]);
        if (b == nullptr || !x.is_cuda() || x.dim() < 1 || heads < 1 || dim < 1 || vdim < 1 || rot < 0) throw NotPlain();
        const float eps = number(p[8]);
        umbs_retention_opts_t o{};
        o.k_scale = number(p[12]);
        o.norm_w = at_<float>(norm);
        o.norm_parts = small(p[14]);
        o.gate_act = small(p[15]);
        const int64_t T = x.size(0), hv = (int64_t)heads * vdim, segs = truth(p[11]) && T >= 128 ? 32 * hv * dim : 0;
        at::Tensor seg, o32 = empty({T, hv}, at::kFloat, x), out = empty({T, hv}, md == UMBS_BF16 ? at::kBFloat16 : at::kFloat, x),
                   table = empty({T, rot > 1 ? rot : 1}, at::kFloat, x);
        if (segs > 0) seg = empty({segs}, at::kFloat, x);
        float *px = at_<float>(x), *pf = at_<float>(freq), *pd = at_<float>(decay), *ps = at_<float>(state), *p32 = at_<float>(o32), *pt = at_<float>(table),
              *pg = segs > 0 ? at_<float>(seg) : nullptr;
        void *po = at_(out), *st = stream();
        const int64_t ld = x.stride(0);
        return result(call([&] { return g.retention(md, px, ld, b, heads, dim, vdim, rot, pf, pd, eps, ps, p32, pt, pg, segs * 4, &o, po, st); }), out);
    });
}

// the entry points' addresses, in the order of Entries
PyObject* bind(PyObject*, Args p, Py_ssize_t n_args) {
    if (n_args != kEntries) {
        PyErr_SetString(PyExc_TypeError, "wrong number of entry points");
        return nullptr;
    }
    void* at[kEntries];
    for (int i = 0; i < kEntries; ++i) {
        at[i] = PyLong_AsVoidPtr(p[i]);
        if (at[i] == nullptr) {
            if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "no address");
            return nullptr;
        }
    }
    memcpy(&g, at, sizeof g);
    Py_RETURN_NONE;
}

#define UMBS_CALL(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {UMBS_CALL(bind), UMBS_CALL(gemm), UMBS_CALL(moe_route), UMBS_CALL(add_norm), UMBS_CALL(cached_attention), UMBS_CALL(window_attention),
                         UMBS_CALL(retention), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_ = {PyModuleDef_HEAD_INIT, "_seq_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__seq_calls(void) { return PyModule_Create(&module_); }
