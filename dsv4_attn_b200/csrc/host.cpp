// The operator surface's fast path (CPython extension module `_host`): one call from api.py checks the tensors, allocates what
// the caller did not pass, fills the C ABI's parameter block and launches.
//
// The kernels of a decode step run for 5 to 60 us each; the same work written in Python (attribute look-ups, ctypes
// fields, torch.empty, the stream query) took 15 to 35 us a call on the build's hosts and was what a step of small
// kernels waited for.  Here a call takes 3 to 6 us.
//
// A function returns the call's result; an int, the library's error code, when a launch failed; or None when
// anything about the arguments is not the ordinary case.  api.py then goes through its own checks, which name what is
// wrong, so that messages and exception types are defined in one place.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/dsv4_attn.h"

namespace {

// Entry points of the library api.py has loaded (which an environment variable may choose), by address.
struct Library {
    decltype(&dsv4_csa_sparse_decode_fwd) csa;
    decltype(&dsv4_hca_dense_decode_fwd) hca;
    decltype(&dsv4_hca_packed_decode_fwd) packed;
    decltype(&hca_decode_fwd) planes;
    decltype(&dsv4_rope_norm_fwd) rope_norm;
    decltype(&dsv4_kv_quantize_insert) insert;
    decltype(&dsv4_csa_compress_reduce_fwd) csa_compress;
    decltype(&dsv4_hca_compress_fwd) hca_compress;
    decltype(&dsv4_indexer_topk_fwd) indexer;
    decltype(&dsv4_attn_combine) combine;
    decltype(&dsv4_attn_plan) plan;
    decltype(&dsv4_attn_plan_splits) plan_splits;
} lib;

constexpr int kLatent = 512, kQk = 576, kEntry = DSV4_ENTRY_BYTES, kPage = DSV4_PAGE_ENTRIES;

const at::Tensor* any_tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// A contiguous CUDA tensor of the given type and rank (rank < 0: any), or null.
const at::Tensor* tensor(PyObject* o, at::ScalarType type, int64_t rank) {
    const at::Tensor* t = any_tensor(o);
    if (t == nullptr || !t->is_cuda() || t->scalar_type() != type || !t->is_contiguous() || (rank >= 0 && t->dim() != rank)) return nullptr;
    return t;
}
// The same where the argument may be None: false when it is neither.
bool optional_tensor(PyObject* o, at::ScalarType type, int64_t rank, const at::Tensor** t) {
    *t = nullptr;
    if (o == Py_None) return true;
    *t = tensor(o, type, rank);
    return *t != nullptr;
}
bool has_shape(const at::Tensor* t, at::IntArrayRef s) { return t == nullptr || t->sizes() == s; }
template <typename T = void>
T* ptr(const at::Tensor* t) { return t == nullptr ? nullptr : static_cast<T*>(t->data_ptr()); }
bool integer(PyObject* o, int64_t* v) {
    if (!PyLong_Check(o)) return false;
    *v = PyLong_AsLongLong(o);
    if (*v == -1 && PyErr_Occurred()) { PyErr_Clear();  return false; }
    return true;
}
bool number(PyObject* o, float* v) {
    const double d = PyFloat_AsDouble(o);
    if (d == -1.0 && PyErr_Occurred()) { PyErr_Clear();  return false; }
    *v = float(d);
    return true;
}
bool fits32(int64_t v) { return v >= 0 && v <= 0x7FFFFFFF; }
void* stream_of(const at::Tensor* t) { return c10::cuda::getCurrentCUDAStream(t->device().index()).stream(); }
// Other Python threads run while the allocator or a launch makes this one wait (the launch queue may be full of work that one of them has to feed).
struct NoGil {
    PyThreadState* state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};
template <typename... P, typename... A>
int launch(int (*entry)(P...), A&&... args) {
    NoGil released;
    return entry(args...);
}
at::Tensor empty(at::IntArrayRef s, at::ScalarType type, const at::Tensor* like) {
    NoGil released;
    return at::Tensor(at::detail::empty_cuda(s, type, like->device(), std::nullopt));
}

// An output the caller passed (checked) or that is allocated here; result() hands it to Python.
struct Output {
    PyObject* given = nullptr;
    const at::Tensor* t = nullptr;
    at::Tensor own;
    bool take(PyObject* o, at::ScalarType type, at::IntArrayRef s, const at::Tensor* like) {
        if (o == Py_None) {
            own = empty(s, type, like);
            t = &own;
            return true;
        }
        given = o;
        t = tensor(o, type, int64_t(s.size()));
        return t != nullptr && t->sizes() == s;
    }
    PyObject* result() {
        if (given != nullptr) { Py_INCREF(given);  return given; }
        return THPVariable_Wrap(std::move(own));
    }
};
PyObject* pair(Output& a, Output& b) {
    PyObject* x = a.result();
    PyObject* y = b.result();
    PyObject* r = PyTuple_New(2);
    PyTuple_SET_ITEM(r, 0, x);
    PyTuple_SET_ITEM(r, 1, y);
    return r;
}
PyObject* none() { Py_RETURN_NONE; }
PyObject* code(int rc) { return PyLong_FromLong(rc); }

// What the two packed-record decode calls share.
struct Decode {
    const at::Tensor *q, *pool, *table, *sink, *status, *po = nullptr, *pl = nullptr;
    at::Tensor own_po, own_pl;
    Output out, lse;
    int64_t B, s_q, H, splits;
    void* sched = nullptr;

    // plan: None or the tuple (kind, B, s_q, H, topk, sched, partial_o, partial_lse) of a Plan
    bool fill(PyObject* q_, PyObject* pool_, PyObject* table_, PyObject* sink_, PyObject* splits_, PyObject* out_, PyObject* lse_, PyObject* workspace,
              PyObject* status_, PyObject* plan, int64_t kind, int64_t topk, int64_t max_len) {
        q = tensor(q_, at::kBFloat16, 4);
        pool = tensor(pool_, at::kByte, 3);
        table = tensor(table_, at::kInt, 2);
        if (q == nullptr || pool == nullptr || table == nullptr) return false;
        B = q->size(0);  s_q = q->size(1);  H = q->size(2);
        if (q->size(3) != kQk || pool->size(1) != kPage || pool->size(2) != kEntry || table->size(0) != B) return false;
        if (!fits32(B * s_q) || !fits32(H) || !fits32(table->size(1))) return false;
        if (!optional_tensor(sink_, at::kFloat, 1, &sink) || !has_shape(sink, {H})) return false;
        status = status_ == Py_None ? nullptr : any_tensor(status_);
        if (status_ != Py_None && status == nullptr) return false;
        if (plan != Py_None) {
            int64_t v[5];
            if (!PyTuple_Check(plan) || PyTuple_GET_SIZE(plan) != 8) return false;
            for (int i = 0; i < 5; ++i)
                if (!integer(PyTuple_GET_ITEM(plan, i), &v[i])) return false;
            if (v[0] != kind || v[1] != B || v[2] != s_q || v[3] != H || (kind == DSV4_PLAN_CSA && v[4] != topk)) return false;
            const at::Tensor* s = any_tensor(PyTuple_GET_ITEM(plan, 5));
            po = any_tensor(PyTuple_GET_ITEM(plan, 6));
            pl = any_tensor(PyTuple_GET_ITEM(plan, 7));
            if (s == nullptr || po == nullptr || pl == nullptr) return false;
            sched = s->data_ptr();
            splits = 1;
        } else if (splits_ == Py_None) {
            splits = lib.plan_splits(int(B * s_q), int(H), int(max_len), 0);
            if (splits < 1) return false;
        } else if (!integer(splits_, &splits) || splits < 1 || splits > DSV4_MAX_SPLITS) {
            return false;
        }
        if (!out.take(out_, at::kBFloat16, {B, s_q, H, kLatent}, q) || !lse.take(lse_, at::kFloat, {B, s_q, H}, q)) return false;
        if (plan == Py_None && splits > 1) {
            const int64_t rows = splits * B * s_q * H;
            if (workspace == Py_None) {
                own_po = empty({rows * kLatent}, at::kFloat, q);
                own_pl = empty({rows}, at::kFloat, q);
                po = &own_po;
                pl = &own_pl;
            } else {
                if (!PyTuple_Check(workspace) || PyTuple_GET_SIZE(workspace) != 2) return false;
                po = tensor(PyTuple_GET_ITEM(workspace, 0), at::kFloat, -1);
                pl = tensor(PyTuple_GET_ITEM(workspace, 1), at::kFloat, -1);
                if (po == nullptr || pl == nullptr || po->numel() < rows * kLatent || pl->numel() < rows) return false;
            }
        }
        return true;
    }
};

// (q, kv_pool, block_table, indices, sm_scale, kv_len, topk_len, attn_sink, num_splits, out, lse, workspace, status, plan)
PyObject* csa(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 14) return none();
    const at::Tensor *idx = tensor(a[3], at::kInt, 3), *kv_len, *topk_len;
    Dsv4CsaSparseDecodeParams p{};
    if (idx == nullptr || !number(a[4], &p.sm_scale) || !optional_tensor(a[5], at::kInt, 2, &kv_len) || !optional_tensor(a[6], at::kInt, 2, &topk_len)) return none();
    const int64_t topk = idx->size(2);
    Decode d;
    if (!fits32(topk) || !d.fill(a[0], a[1], a[2], a[7], a[8], a[9], a[10], a[11], a[12], a[13], DSV4_PLAN_CSA, topk, topk)) return none();
    if (idx->size(0) != d.B || idx->size(1) != d.s_q || !has_shape(kv_len, {d.B, d.s_q}) || !has_shape(topk_len, {d.B, d.s_q})) return none();
    p.B = int(d.B);  p.s_q = int(d.s_q);  p.H = int(d.H);  p.topk = int(topk);  p.max_pages = int(d.table->size(1));  p.num_splits = int(d.splits);
    p.num_pages = d.pool->size(0);
    p.q = ptr(d.q);  p.kv_pool = ptr(d.pool);  p.block_table = ptr<int32_t>(d.table);  p.indices = ptr<int32_t>(idx);
    p.kv_len = ptr<int32_t>(kv_len);  p.topk_len = ptr<int32_t>(topk_len);  p.attn_sink = ptr<float>(d.sink);
    p.out = ptr(d.out.t);  p.lse = ptr<float>(d.lse.t);  p.partial_o = ptr<float>(d.po);  p.partial_lse = ptr<float>(d.pl);
    p.status = ptr<int32_t>(d.status);  p.sched = d.sched;
    const int rc = launch(lib.csa, &p, stream_of(d.q));
    return rc != 0 ? code(rc) : pair(d.out, d.lse);
}

// (q, kv_pool, block_table, kv_len, win_pool, win_len, sm_scale, attn_sink, num_splits, out, lse, workspace, status, max_len, plan)
PyObject* hca(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 15) return none();
    const at::Tensor *kv_len = tensor(a[3], at::kInt, 2), *win = tensor(a[4], at::kByte, 3), *win_len = tensor(a[5], at::kInt, 2);
    const at::Tensor* table = tensor(a[2], at::kInt, 2);
    Dsv4HcaDenseDecodeParams p{};
    if (kv_len == nullptr || win == nullptr || win_len == nullptr || table == nullptr || win->size(2) != kEntry || !number(a[6], &p.sm_scale)) return none();
    int64_t max_len;
    if (a[13] == Py_None) max_len = table->size(1) * kPage + win->size(1);
    else if (!integer(a[13], &max_len)) return none();
    Decode d;
    if (!fits32(max_len) || !d.fill(a[0], a[1], a[2], a[7], a[8], a[9], a[10], a[11], a[12], a[14], DSV4_PLAN_HCA, 0, max_len)) return none();
    if (!has_shape(kv_len, {d.B, d.s_q}) || !has_shape(win_len, {d.B, d.s_q}) || win->size(0) != d.B || !fits32(win->size(1))) return none();
    p.B = int(d.B);  p.s_q = int(d.s_q);  p.H = int(d.H);  p.max_pages = int(d.table->size(1));  p.win_cap = int(win->size(1));  p.num_splits = int(d.splits);
    p.num_pages = d.pool->size(0);
    p.q = ptr(d.q);  p.kv_pool = ptr(d.pool);  p.block_table = ptr<int32_t>(d.table);  p.kv_len = ptr<int32_t>(kv_len);
    p.win_pool = ptr(win);  p.win_len = ptr<int32_t>(win_len);  p.attn_sink = ptr<float>(d.sink);
    p.out = ptr(d.out.t);  p.lse = ptr<float>(d.lse.t);  p.partial_o = ptr<float>(d.po);  p.partial_lse = ptr<float>(d.pl);
    p.status = ptr<int32_t>(d.status);  p.sched = d.sched;
    const int rc = launch(lib.hca, &p, stream_of(d.q));
    return rc != 0 ? code(rc) : pair(d.out, d.lse);
}

// (q, kv_pages, block_table, m_cur, swa_pages, swa_block_table, swa_len, sm_scale, page_size, attn_sink, num_splits, out, lse, workspace, status)
PyObject* packed(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 15) return none();
    const at::Tensor* q = tensor(a[0], at::kBFloat16, 3);
    const at::Tensor *m_cur = tensor(a[3], at::kInt, 1), *swa_len = tensor(a[6], at::kInt, 1), *sink;
    Dsv4HcaPackedDecodeParams p{};
    int64_t page, splits;
    if (q == nullptr || m_cur == nullptr || swa_len == nullptr || !number(a[7], &p.sm_scale) || !integer(a[8], &page)) return none();
    const int64_t B = q->size(0), H = q->size(1);
    if (q->size(2) != 512 || (page != 16 && page != 32 && page != 64) || !has_shape(m_cur, {B}) || !has_shape(swa_len, {B}) || !fits32(B) || !fits32(H)) return none();
    if (!optional_tensor(a[9], at::kFloat, 1, &sink) || !has_shape(sink, {H})) return none();
    const at::Tensor *pool[2] = {nullptr, nullptr}, *table[2] = {nullptr, nullptr};
    int64_t cap = 0;
    for (int i = 0; i < 2; ++i) {
        if (a[1 + 3 * i] == Py_None) continue;
        pool[i] = tensor(a[1 + 3 * i], at::kByte, 2);
        table[i] = tensor(a[2 + 3 * i], at::kInt, 2);
        if (pool[i] == nullptr || table[i] == nullptr || pool[i]->size(1) != page * 584 || table[i]->size(0) != B) return none();
        cap += table[i]->size(1) * page;
    }
    if ((pool[0] == nullptr && pool[1] == nullptr) || !fits32(cap)) return none();
    if (a[10] == Py_None) splits = lib.plan_splits(int(B), int(H), int(cap), 0);
    else if (!integer(a[10], &splits)) return none();
    if (splits < 1 || splits > DSV4_MAX_SPLITS) return none();
    const at::Tensor* status = a[14] == Py_None ? nullptr : any_tensor(a[14]);
    if ((a[14] != Py_None && status == nullptr) || a[13] != Py_None) return none();
    Output out, lse;
    if (a[11] != Py_None || a[12] != Py_None) return none();       // caller's outputs are not checked by the slow path either: leave them to it
    if (!out.take(a[11], at::kBFloat16, {B, H, 512}, q) || !lse.take(a[12], at::kFloat, {B, H}, q)) return none();
    at::Tensor po, pl;
    if (splits > 1) {
        po = empty({splits * B * H * 512}, at::kFloat, q);
        pl = empty({splits * B * H}, at::kFloat, q);
        p.partial_o = ptr<float>(&po);
        p.partial_lse = ptr<float>(&pl);
    }
    p.B = int(B);  p.H = int(H);  p.page_size = int(page);  p.num_splits = int(splits);
    p.max_pages = pool[0] ? int(table[0]->size(1)) : 0;  p.swa_max_pages = pool[1] ? int(table[1]->size(1)) : 0;
    p.num_pages = pool[0] ? pool[0]->size(0) : 0;  p.swa_num_pages = pool[1] ? pool[1]->size(0) : 0;
    p.q = ptr(q);  p.kv_pages = ptr(pool[0]);  p.block_table = ptr<int32_t>(table[0]);  p.m_cur = ptr<int32_t>(m_cur);
    p.swa_pages = ptr(pool[1]);  p.swa_block_table = ptr<int32_t>(table[1]);  p.swa_len = ptr<int32_t>(swa_len);
    p.attn_sink = ptr<float>(sink);  p.out = ptr(out.t);  p.lse = ptr<float>(lse.t);  p.status = ptr<int32_t>(status);
    const int rc = launch(lib.packed, &p, stream_of(q));
    return rc != 0 ? code(rc) : pair(out, lse);
}

// (Q, Kc, Kc_s, Kc_rope, Kswa, Kswa_s, Kswa_rope, sink_logits, sm_scale, M_cur, swa_len, O, partial_O, partial_lse)
PyObject* planes(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 14) return none();
    const at::Tensor* q = tensor(a[0], at::kBFloat16, 3);
    float sm_scale;
    int64_t M, W;
    if (q == nullptr || !number(a[8], &sm_scale) || !integer(a[9], &M) || !integer(a[10], &W) || !fits32(M) || !fits32(W) || !fits32(M + W)) return none();
    const at::Tensor* t[7];                                         // Kc .. Kswa_rope, sink: taken as they are, as by the slow path
    for (int i = 0; i < 7; ++i) {
        t[i] = a[1 + i] == Py_None ? nullptr : any_tensor(a[1 + i]);
        if (a[1 + i] != Py_None && t[i] == nullptr) return none();
    }
    if (t[0] == nullptr || t[3] == nullptr) return none();
    const int64_t B = q->size(0), H = q->size(1), dq = q->size(2), c = t[0]->size(-1), S = (M + W) / 128;
    if (!fits32(B) || !fits32(H) || !fits32(dq)) return none();
    const at::Tensor *po = a[12] == Py_None ? nullptr : any_tensor(a[12]), *pl = a[13] == Py_None ? nullptr : any_tensor(a[13]);
    if ((a[12] != Py_None && po == nullptr) || (a[13] != Py_None && pl == nullptr)) return none();
    at::Tensor own_o, own_po, own_pl;
    const at::Tensor* o = a[11] == Py_None ? nullptr : any_tensor(a[11]);
    if (a[11] != Py_None && o == nullptr) return none();
    if (o == nullptr) {
        own_o = empty({B, H, dq}, at::kBFloat16, q);
        o = &own_o;
    }
    if (po == nullptr && S > 1) {
        own_po = empty({S * B * H * dq}, at::kFloat, q);
        own_pl = empty({S * B * H}, at::kFloat, q);
        po = &own_po;
        pl = &own_pl;
    }
    const int rc = launch(lib.planes, ptr(q), ptr(t[0]), ptr(t[1]), ptr(t[2]), ptr(t[3]), ptr(t[4]), ptr(t[5]), ptr(t[6]), ptr(o), ptr(po), ptr(pl), sm_scale, int(B), int(H),
                              int(c), int(dq - c), int(M), int(W), stream_of(q));
    if (rc != 0) return code(rc);
    if (a[11] != Py_None) { Py_INCREF(a[11]);  return a[11]; }
    return THPVariable_Wrap(std::move(own_o));
}

// (x, positions, norm_weight, eps, n_rope, theta, inverse, out)
PyObject* rope_norm(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 8) return none();
    const at::Tensor *x = tensor(a[0], at::kBFloat16, 3), *pos = tensor(a[1], at::kInt, 1), *w;
    Dsv4RopeNormParams p{};
    int64_t n_rope;
    if (x == nullptr || pos == nullptr || !optional_tensor(a[2], at::kBFloat16, 1, &w) || !number(a[3], &p.eps) || !integer(a[4], &n_rope) || !number(a[5], &p.theta))
        return none();
    const int64_t rows = x->size(0), vecs = x->size(1), c = x->size(2);
    if (!has_shape(pos, {rows}) || !has_shape(w, {c}) || n_rope != 64 || c < 64 || (c - 64) % 8 != 0 || c - 64 > 512 || !fits32(vecs)) return none();
    const int inverse = PyObject_IsTrue(a[6]);
    Output out;
    if (inverse < 0) { PyErr_Clear();  return none(); }
    if (!out.take(a[7], at::kBFloat16, {rows, vecs, c}, x)) return none();
    p.n_rows = rows;  p.vecs_per_row = int(vecs);  p.c = int(c);  p.n_rope = 64;  p.inverse = inverse;
    p.x = ptr(x);  p.out = ptr(out.t);  p.positions = ptr<int32_t>(pos);  p.norm_weight = ptr(w);
    const int rc = launch(lib.rope_norm, &p, stream_of(x));
    return rc != 0 ? code(rc) : out.result();
}

bool cache_dest(PyObject* pool_, PyObject* table_, PyObject* pos_, PyObject* status_, int64_t B, Dsv4CacheDest* d) {
    const at::Tensor *pool = tensor(pool_, at::kByte, 3), *table = tensor(table_, at::kInt, 2), *pos = tensor(pos_, at::kInt, 1), *status;
    if (pool == nullptr || table == nullptr || pos == nullptr || !optional_tensor(status_, at::kInt, 1, &status)) return false;
    if (pool->size(1) != kPage || pool->size(2) != kEntry || table->size(0) != B || pos->size(0) != B || (status != nullptr && status->numel() < 4) || !fits32(table->size(1))) return false;
    *d = Dsv4CacheDest{};
    d->kv_pool = ptr(pool);  d->block_table = ptr<int32_t>(table);  d->insert_pos = ptr<int32_t>(pos);
    d->max_pages = int(table->size(1));  d->num_pages = pool->size(0);  d->status = ptr<int32_t>(status);
    return true;
}

// (rows, kv_pool, block_table, insert_pos, n_rows, status) -> True
PyObject* insert(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 6) return none();
    const at::Tensor *rows = tensor(a[0], at::kBFloat16, 3), *n_rows;
    Dsv4CacheDest d;
    if (rows == nullptr || !optional_tensor(a[4], at::kInt, 1, &n_rows)) return none();
    const int64_t B = rows->size(0), T = rows->size(1);
    if (rows->size(2) != kQk || !fits32(B) || !fits32(T) || !has_shape(n_rows, {B}) || !cache_dest(a[1], a[2], a[3], a[5], B, &d)) return none();
    Dsv4KvQuantizeInsertParams p{};
    p.B = int(B);  p.T = int(T);  p.rows = ptr(rows);  p.stride_b = T * kQk;  p.stride_t = kQk;  p.n_rows = ptr<int32_t>(n_rows);  p.dst = &d;
    const int rc = launch(lib.insert, &p, stream_of(rows));
    if (rc != 0) return code(rc);
    Py_RETURN_TRUE;
}

// (C_a, C_b, Z_a, Z_b, B_a, B_b, m, out)
PyObject* csa_compress(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 8) return none();
    const at::Tensor* t[6];
    for (int i = 0; i < 6; ++i) {
        t[i] = tensor(a[i], at::kBFloat16, i < 4 ? 3 : 2);
        if (t[i] == nullptr) return none();
    }
    int64_t m;
    if (!integer(a[6], &m) || m != 4) return none();
    const int64_t B = t[0]->size(0), rows = t[0]->size(1), c = t[0]->size(2);
    for (int i = 1; i < 4; ++i)
        if (t[i]->sizes() != t[0]->sizes()) return none();
    if (!has_shape(t[4], {m, c}) || !has_shape(t[5], {m, c}) || rows % m != 0 || !fits32(B) || !fits32(rows) || !fits32(c)) return none();
    if (a[7] != Py_None) return none();                             // (a caller's output is not checked by the slow path: leave it to it)
    Output out;
    out.take(a[7], at::kBFloat16, {B, rows / m, c}, t[0]);
    Dsv4CsaCompressReduceParams p{};
    p.B = int(B);  p.n = int(rows);  p.c_out = int(c);  p.m = int(m);
    p.C_a = ptr(t[0]);  p.C_b = ptr(t[1]);  p.Z_a = ptr(t[2]);  p.Z_b = ptr(t[3]);  p.B_a = ptr(t[4]);  p.B_b = ptr(t[5]);  p.out = ptr(out.t);
    p.stride_C_b = rows * c;  p.stride_C_n = c;  p.stride_out_b = (rows / m) * c;  p.stride_out_blk = c;
    const int rc = launch(lib.csa_compress, &p, stream_of(t[0]));
    return rc != 0 ? code(rc) : out.result();
}

// (C, Z, bias, m, out, kv_pool, block_table, insert_pos, status, want_out) -> out, or False where none was asked for
PyObject* hca_compress(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 10) return none();
    const at::Tensor *C = tensor(a[0], at::kBFloat16, 3), *Z = tensor(a[1], at::kBFloat16, 3), *bias = tensor(a[2], at::kBFloat16, 2);
    int64_t m;
    if (C == nullptr || Z == nullptr || bias == nullptr || C->sizes() != Z->sizes() || !integer(a[3], &m)) return none();
    const int64_t B = C->size(0), rows = C->size(1), c = C->size(2);
    if (m < 1 || !has_shape(bias, {m, c}) || rows % m != 0 || c % 8 != 0 || !fits32(B) || !fits32(rows) || !fits32(c)) return none();
    Dsv4CacheDest d;
    const bool insert = a[5] != Py_None;
    if (insert && (c != kQk || !cache_dest(a[5], a[6], a[7], a[8], B, &d))) return none();
    const int want = PyObject_IsTrue(a[9]);
    if (want < 0) { PyErr_Clear();  return none(); }
    if (!want && !insert) return none();
    Output out;
    const bool with_out = want || a[4] != Py_None;
    if (with_out && !out.take(a[4], at::kBFloat16, {B, rows / m, c}, C)) return none();
    Dsv4HcaCompressParams p{};
    p.B = int(B);  p.n = int(rows);  p.c = int(c);  p.m = int(m);  p.C = ptr(C);  p.Z = ptr(Z);  p.bias = ptr(bias);
    p.stride_b = rows * c;  p.stride_n = c;  p.out = ptr(out.t);  p.dst = insert ? &d : nullptr;
    const int rc = launch(lib.hca_compress, &p, stream_of(C));
    if (rc != 0) return code(rc);
    if (with_out) return out.result();
    Py_RETURN_FALSE;
}

// (q_fp8, q_weight, key_pages, block_table, n_vis, k, scores, out, status)
PyObject* indexer(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 9) return none();
    const at::Tensor *q = tensor(a[0], at::kByte, 4), *w = tensor(a[1], at::kFloat, 3), *keys = tensor(a[2], at::kByte, 2), *table = tensor(a[3], at::kInt, 2);
    const at::Tensor* vis = tensor(a[4], at::kInt, 2);
    int64_t k;
    if (q == nullptr || w == nullptr || keys == nullptr || table == nullptr || vis == nullptr || !integer(a[5], &k)) return none();
    const int64_t B = q->size(0), s_q = q->size(1), pages = table->size(1), stride = pages * 64;
    if (q->size(2) != 64 || q->size(3) != 128 || (s_q != 1 && s_q != 2) || !has_shape(w, {B, s_q, 64}) || keys->size(1) != 64 * 128 + 256 || table->size(0) != B ||
        !has_shape(vis, {B, s_q}) || k < 1 || !fits32(k) || !fits32(B) || !fits32(stride))
        return none();
    const at::Tensor* status = a[8] == Py_None ? nullptr : any_tensor(a[8]);
    if (a[8] != Py_None && status == nullptr) return none();
    Output scores, out;
    if (a[6] == Py_None) {
        scores.take(a[6], at::kFloat, {B * s_q, stride}, q);
    } else {
        scores.given = a[6];
        scores.t = tensor(a[6], at::kFloat, 2);
        if (scores.t == nullptr || scores.t->size(0) != B * s_q || scores.t->size(1) < stride) return none();
    }
    if (!out.take(a[7], at::kInt, {B, s_q, k}, q)) return none();
    Dsv4IndexerTopkParams p{};
    p.B = int(B);  p.s_q = int(s_q);  p.max_pages = int(pages);  p.k = int(k);  p.num_pages = keys->size(0);  p.score_stride = scores.t->size(1);
    p.q_fp8 = ptr(q);  p.q_weight = ptr<float>(w);  p.key_pages = ptr(keys);  p.block_table = ptr<int32_t>(table);  p.n_vis = ptr<int32_t>(vis);
    p.scores = ptr<float>(scores.t);  p.out_indices = ptr<int32_t>(out.t);  p.status = ptr<int32_t>(status);
    const int rc = launch(lib.indexer, &p, stream_of(q));
    return rc != 0 ? code(rc) : pair(out, scores);
}

// (kind, B, s_q, H, topk, num_splits, num_sms, topk_len, kv_len, win_len, sched) -> the library's code
PyObject* plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 11) return none();
    int64_t v[7];
    for (int i = 0; i < 7; ++i)
        if (!integer(a[i], &v[i])) return none();
    const at::Tensor* t[4];
    for (int i = 0; i < 4; ++i) {
        t[i] = a[7 + i] == Py_None ? nullptr : any_tensor(a[7 + i]);
        if (a[7 + i] != Py_None && t[i] == nullptr) return none();
    }
    if (t[3] == nullptr) return none();
    Dsv4PlanParams p{};
    p.kind = int(v[0]);  p.B = int(v[1]);  p.s_q = int(v[2]);  p.H = int(v[3]);  p.topk = int(v[4]);  p.num_splits = int(v[5]);  p.num_sms = int(v[6]);
    p.topk_len = ptr<int32_t>(t[0]);  p.kv_len = ptr<int32_t>(t[1]);  p.win_len = ptr<int32_t>(t[2]);
    p.sched = ptr(t[3]);  p.sched_bytes = int64_t(t[3]->nbytes());
    return code(launch(lib.plan, &p, stream_of(t[3])));
}

// (partial_o, partial_lse, attn_sink, out, lse)
PyObject* combine(PyObject*, PyObject* const* a, Py_ssize_t n) {
    if (n != 5) return none();
    const at::Tensor *po = tensor(a[0], at::kFloat, 4), *pl = tensor(a[1], at::kFloat, 3), *sink;
    if (po == nullptr || pl == nullptr || !optional_tensor(a[2], at::kFloat, 1, &sink)) return none();
    const int64_t S = po->size(0), N = po->size(1), H = po->size(2), D = po->size(3);
    if (D != kLatent || !has_shape(pl, {S, N, H}) || !fits32(S) || !fits32(N) || !fits32(H)) return none();
    Output out, lse;
    for (int i = 3; i < 5; ++i)
        if (a[i] != Py_None && any_tensor(a[i]) == nullptr) return none();
    if (a[3] == Py_None) out.take(a[3], at::kBFloat16, {N, H, D}, po);
    else { out.given = a[3];  out.t = any_tensor(a[3]); }           // taken as they are, as by the slow path
    if (a[4] == Py_None) lse.take(a[4], at::kFloat, {N, H}, po);
    else { lse.given = a[4];  lse.t = any_tensor(a[4]); }
    Dsv4CombineParams p{};
    p.N = int(N);  p.H = int(H);  p.D = int(D);  p.num_splits = int(S);
    p.partial_o = ptr<float>(po);  p.partial_lse = ptr<float>(pl);  p.out = ptr(out.t);  p.lse = ptr<float>(lse.t);  p.attn_sink = ptr<float>(sink);
    p.stride_po_split = N * H * D;  p.stride_po_n = H * D;  p.stride_po_h = D;  p.stride_pl_split = N * H;  p.stride_pl_n = H;
    p.stride_out_n = H * D;  p.stride_out_h = D;  p.stride_lse_n = H;
    const int rc = launch(lib.combine, &p, stream_of(po));
    return rc != 0 ? code(rc) : pair(out, lse);
}

// C++ exceptions (the allocator's out-of-memory error among them) become None: the slow path meets the same error and raises it.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
    try {
        return F(self, a, n);
    } catch (...) {
        PyErr_Clear();
        return none();
    }
}

// (addresses of the library's entry points, in the order of struct Library)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
    void** slot = reinterpret_cast<void**>(&lib);
    if (n * Py_ssize_t(sizeof(void*)) != Py_ssize_t(sizeof(Library))) {
        PyErr_SetString(PyExc_TypeError, "bind() takes one address per entry point");
        return nullptr;
    }
    for (Py_ssize_t i = 0; i < n; ++i) {
        slot[i] = PyLong_AsVoidPtr(a[i]);
        if (slot[i] == nullptr && PyErr_Occurred()) return nullptr;
    }
    Py_RETURN_NONE;
}

#define DSV4_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&guarded<name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(&bind)), METH_FASTCALL, nullptr},
    DSV4_FAST(csa), DSV4_FAST(hca), DSV4_FAST(packed), DSV4_FAST(planes), DSV4_FAST(rope_norm), DSV4_FAST(insert), DSV4_FAST(csa_compress),
    DSV4_FAST(hca_compress), DSV4_FAST(indexer), DSV4_FAST(plan), DSV4_FAST(combine),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
