// Host side of the Python entry points: torch tensors -> the C ABI of libommx_b200.so.
//
// What this replaces: filling the argument structs through ctypes cost 22 us (pack), 30 us (store step) and 45 us
// (decode) of Python per call, most of it one attribute read at a time - more than the kernels of a 16K-token decode
// take.  Here the same reads are a few nanoseconds each.
//
// The functions below serve a call or decline it.  `decode` and `pack_into` check what their Python callers document
// and return None without touching anything when a check fails; the caller then goes through the arguments one by
// one and raises the exception that says what is wrong.  Everything else raises here.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Device.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/object_ptr.h>

#include <cctype>
#include <cstdlib>
#include <cstring>
#include <string>

#include "../../include/ommx_b200.h"

// the torch and python this module is built for; the loader reads it from the file before it loads the module
extern "C" __attribute__((used, visibility("default"))) const char ommx_host_built_for[] = OMMX_HOST_BUILT_FOR;

namespace {

using at::Tensor;

// ---- small readers --------------------------------------------------------------------------------
const Tensor *as_tensor(PyObject *o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// int(o) for anything int() takes; false (and no Python error set) otherwise
bool as_long(PyObject *o, int64_t *out) {
    if (PyLong_CheckExact(o)) {
        int overflow = 0;
        *out = PyLong_AsLongLongAndOverflow(o, &overflow);
        return overflow == 0;
    }
    PyObject *n = PyNumber_Long(o);
    if (!n) { PyErr_Clear(); return false; }
    int overflow = 0;
    *out = PyLong_AsLongLongAndOverflow(n, &overflow);
    Py_DECREF(n);
    return overflow == 0;
}
bool as_double(PyObject *o, double *out) {
    if (PyFloat_CheckExact(o)) { *out = PyFloat_AS_DOUBLE(o); return true; }
    PyObject *n = PyNumber_Float(o);
    if (!n) { PyErr_Clear(); return false; }
    *out = PyFloat_AS_DOUBLE(n);
    Py_DECREF(n);
    return true;
}
bool as_bool(PyObject *o, bool *out) {
    const int t = PyObject_IsTrue(o);
    if (t < 0) { PyErr_Clear(); return false; }
    *out = t != 0;
    return true;
}
// the environment switch is on: set, and not one of the spellings of "off"
bool env_on(const char *name) {
    const char *v = getenv(name);
    if (!v) return false;
    while (isspace((unsigned char)*v)) ++v;
    size_t n = strlen(v);
    while (n && isspace((unsigned char)v[n - 1])) --n;
    if (n == 0) return false;
    for (const char *off : {"0", "false", "off", "no"})
        if (n == strlen(off) && strncasecmp(v, off, n) == 0) return false;
    return true;
}

// Whether any switch of this package is set: one pass over the environment where a getenv per switch takes one each (nine
// of them were 1.5 us of a decode call under 135 variables).
bool any_switch() {
    for (char **e = environ; e && *e; ++e)
        if (strncmp(*e, "OMMX", 4) == 0) return true;
    return false;
}

// a fresh tensor without the dispatcher's round (pack_block makes twelve)
Tensor fresh(at::IntArrayRef size, const at::TensorOptions &o) { return at::detail::empty_cuda(size, o); }

struct Names {                                        // interned dictionary keys and attribute names
    PyObject *k_base, *k_scale, *k_zp, *k_obmp, *k_oval, *k_fp4_mapscale, *k_fp4_mapcenter, *v_main, *v_scale, *v_zp;
    PyObject *planes, *k, *kv_outlier_map, *k_hist, *v_hist, *num_seqs, *ring_cap, *sink, *recent, *seq_dev,
        *req_to_token, *req_to_group, *P_per_seq, *G_per_seq, *k_tail, *v_tail, *max_tail_len, *b_seq, *b_tail, *status,
        *sel;
} N;

// ---- the plane descriptor -------------------------------------------------------------------------
struct PlaneSet {
    const Tensor *k_base, *k_scale, *k_zp, *k_idx, *k_oval, *k_ms, *k_mc, *v_main, *v_scale, *v_zp;
};
void *ptr(const Tensor *t) { return t ? t->data_ptr() : nullptr; }
void *ptr(const Tensor &t) { return t.defined() ? t.data_ptr() : nullptr; }
// memory a kernel may touch: a plain host tensor is declined, not handed to the GPU
bool reachable(const Tensor *t) { return !t || t->is_cuda() || t->is_pinned(); }

bool fill_planes(const PlaneSet &s, int64_t k, bool use_map, bool relidx7, ommx_kv_planes *p) {
    for (const Tensor *t : {s.k_base, s.k_scale, s.k_zp, s.v_main, s.v_scale, s.v_zp})
        if (!t || !t->is_contiguous() || !reachable(t)) return false;
    for (const Tensor *t : {s.k_idx, s.k_oval, s.k_ms, s.k_mc})
        if (t && (!t->is_contiguous() || !reachable(t))) return false;
    if (s.k_base->dim() != 4 || s.k_scale->dim() < 1) return false;
    const auto kind = s.k_scale->scalar_type();
    if (kind == at::kChar) p->scale_kind = OMMX_SCALE_INT8_EXP;
    else if (kind == at::kBFloat16) p->scale_kind = OMMX_SCALE_BF16;
    else if (kind == at::kFloat) p->scale_kind = OMMX_SCALE_F32;
    else return false;
    if (relidx7 && (!s.k_idx || s.k_idx->scalar_type() != at::kByte || s.k_idx->size(-1) != (7 * k + 7) / 8)) return false;
    p->n_kv_heads = (int32_t)s.k_base->size(2);
    p->head_dim = (int32_t)s.k_base->size(3) * 4;
    p->page_size = (int32_t)s.k_base->size(1);
    p->num_pages = (int32_t)s.k_base->size(0);
    p->num_group_slots = (int32_t)s.k_scale->size(0);
    p->outliers_per_vector = (int32_t)k;
    p->kv_outlier_map = use_map && k > 0 ? 1 : 0;
    p->k_base = ptr(s.k_base); p->k_scale = ptr(s.k_scale); p->k_zp = ptr(s.k_zp);
    p->k_obmp = ptr(s.k_idx); p->k_oval = ptr(s.k_oval); p->k_mapscale = ptr(s.k_ms); p->k_mapcenter = ptr(s.k_mc);
    p->v_main = ptr(s.v_main); p->v_scale = ptr(s.v_scale); p->v_zp = ptr(s.v_zp);
    p->outlier_index = relidx7 ? OMMX_OIDX_RELIDX7 : OMMX_OIDX_BITMASK;
    return true;
}
// the plane dict of the package (bitmask index)
bool read_plane_dict(PyObject *d, PlaneSet *s) {
    if (!PyDict_Check(d)) return false;
    struct { PyObject *key; const Tensor **to; } all[] = {
        {N.k_base, &s->k_base}, {N.k_scale, &s->k_scale}, {N.k_zp, &s->k_zp}, {N.k_obmp, &s->k_idx}, {N.k_oval, &s->k_oval},
        {N.k_fp4_mapscale, &s->k_ms}, {N.k_fp4_mapcenter, &s->k_mc}, {N.v_main, &s->v_main}, {N.v_scale, &s->v_scale}, {N.v_zp, &s->v_zp}};
    for (auto &e : all) {
        PyObject *v = PyDict_GetItem(d, e.key);       // borrowed
        *e.to = v ? as_tensor(v) : nullptr;
        if (v && !*e.to && v != Py_None) return false;
    }
    return true;
}

// other Python threads run meanwhile; restored on the way out of an exception too
struct NoGil {
    PyThreadState *state = PyEval_SaveThread();
    ~NoGil() { PyEval_RestoreThread(state); }
};

template <typename Fn> int launch(const at::Device &dev, Fn fn) {
    const c10::cuda::CUDAGuard guard(dev);
    void *stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    const NoGil no_gil;
    return fn(stream);
}

// the one value of a device tensor (synchronises)
int64_t read_int(const Tensor &t) {
    const NoGil no_gil;
    return t.item().toLong();
}

// ---- decode ---------------------------------------------------------------------------------------
enum DecodeArg { Q, K_BASE, K_SCALE, K_ZP, K_OIDX, K_OVAL, V_MAIN, V_SCALE, V_ZP, K_TAIL, V_TAIL, B_TAIL_LEN, O, LSE,
                 REQ_TO_TOKEN, REQ_TO_GROUP, B_SEQ_LEN, SM_SCALE, PAGE_SIZE, LOGIT_CAP, K_OUT, K_FORMAT, COMBINADIC, BITMAP,
                 K_OBMP, MAPSCALE, MAPCENTER, OUTLIER_MAP, SPLITS, MAX_SEQ, MAX_TAIL, ATTN_LOGITS, START_OFFSET, SEG_BASE,
                 STATUS, STAGE, STATIC_WS, HEAD_GATHER, N_DECODE_ARGS };
const char *const ABL_FLAGS[] = {"OMMX_ABL_NO_OUTLIER", "OMMX_ABL_V_NODEQUANT", "OMMX_ABL_K_NODEQUANT", "OMMX_ABL_NO_UNPACK", "OMMX_ABL_TEST_STALL"};

// None: declined.  Negative: what the C ABI returned.  Otherwise the ablation bits the call ran with (0 in service).
PyObject *py_decode(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != N_DECODE_ARGS) { PyErr_SetString(PyExc_TypeError, "decode: wrong argument count"); return nullptr; }
#define NEED(cond) do { if (!(cond)) Py_RETURN_NONE; } while (0)
    // ---- plain values ----
    int64_t page_size, k, start_offset, seg_base, stage, max_seq, max_tail, splits;
    bool combinadic, bitmap, use_map, static_ws;
    double sm_scale, logit_cap;
    NEED(as_long(a[PAGE_SIZE], &page_size) && page_size > 0 && as_long(a[K_OUT], &k) && as_long(a[STAGE], &stage));
    NEED(as_double(a[SM_SCALE], &sm_scale) && as_double(a[LOGIT_CAP], &logit_cap));
    NEED(as_bool(a[COMBINADIC], &combinadic) && as_bool(a[BITMAP], &bitmap) && as_bool(a[OUTLIER_MAP], &use_map) && as_bool(a[STATIC_WS], &static_ws));
    start_offset = seg_base = 0;
    if (a[START_OFFSET] != Py_None) NEED(as_long(a[START_OFFSET], &start_offset));
    if (a[SEG_BASE] != Py_None) NEED(as_long(a[SEG_BASE], &seg_base));
    NEED(PyUnicode_Check(a[K_FORMAT]));
    const char *fmt = PyUnicode_AsUTF8(a[K_FORMAT]);
    if (!fmt) return nullptr;
    NEED(strcasecmp(fmt, "i2f4") == 0 || strcasecmp(fmt, "itf4") == 0);
    const bool switches = any_switch();
    combinadic = combinadic || (switches && env_on("OMMX_VLLM_KV_COMBINADIC_READ"));
    bitmap = bitmap || (switches && env_on("OMMX_VLLM_KV_BITMAP_READ"));
    const bool relidx7 = k > 0 && !bitmap;
    NEED(!(bitmap && combinadic) && !(relidx7 && combinadic) && k <= 16);
    NEED(start_offset >= 0 && start_offset < page_size && seg_base >= 0 && seg_base <= INT32_MAX);
    NEED(stage >= 0 && stage <= 2 && !(static_ws && stage != 0));

    // ---- tensors ----
    const Tensor *q = as_tensor(a[Q]), *o = as_tensor(a[O]), *lse = as_tensor(a[LSE]), *r2t = as_tensor(a[REQ_TO_TOKEN]),
                 *r2g = as_tensor(a[REQ_TO_GROUP]), *b_seq = as_tensor(a[B_SEQ_LEN]), *b_tail = as_tensor(a[B_TAIL_LEN]),
                 *kt = as_tensor(a[K_TAIL]), *vt = as_tensor(a[V_TAIL]);
    PlaneSet s;
    s.k_base = as_tensor(a[K_BASE]); s.k_scale = as_tensor(a[K_SCALE]); s.k_zp = as_tensor(a[K_ZP]);
    s.v_main = as_tensor(a[V_MAIN]); s.v_scale = as_tensor(a[V_SCALE]); s.v_zp = as_tensor(a[V_ZP]);
    s.k_idx = relidx7 ? as_tensor(a[K_OIDX]) : (k > 0 ? as_tensor(a[K_OBMP]) : nullptr);
    s.k_oval = k > 0 ? as_tensor(a[K_OVAL]) : nullptr;
    use_map = use_map && k > 0;
    s.k_ms = use_map ? as_tensor(a[MAPSCALE]) : nullptr;
    s.k_mc = use_map ? as_tensor(a[MAPCENTER]) : nullptr;
    NEED(q && o && lse && r2t && r2g && b_seq && s.k_base && s.k_scale && s.v_main && s.v_scale);
    NEED(k <= 0 || (s.k_idx && s.k_oval));
    NEED(!use_map || (s.k_ms && s.k_mc));
    NEED(q->is_cuda() && q->dim() == 3 && o->dim() == 3 && lse->dim() == 2 && r2t->dim() >= 1 && r2g->dim() >= 1);
    ommx_decode_args d;
    memset(&d, 0, sizeof(d));
    NEED(fill_planes(s, k, use_map, relidx7, &d.planes));
    const int64_t pages = s.k_base->size(0), slots = s.k_scale->size(0), v_groups = s.v_scale->size(-1);
    NEED(s.k_base->size(1) == page_size && pages <= INT32_MAX && slots <= INT32_MAX);
    NEED(!(pages && slots) || (pages * page_size) / slots == 32);
    NEED(!v_groups || (s.v_main->size(-1) * 4) / v_groups == 32);
    if (pages)
        for (const Tensor *t : {s.k_base, s.v_main, s.v_scale, s.v_zp})
            NEED(t->dim() >= 2 && t->stride(0) == page_size * t->stride(1) && t->stride(-1) == 1);
    const int64_t batch = q->size(0), heads = q->size(1), kv_heads = d.planes.n_kv_heads, D = s.v_main->size(-1) * 4;
    NEED(kv_heads > 0 && heads >= kv_heads && heads % kv_heads == 0);
    const at::Device dev = q->device();
    for (const Tensor *t : {o, lse, b_seq, r2t, r2g}) NEED(t->device() == dev);
    for (const Tensor *t : {kt, vt, b_tail}) NEED(!t || t->device() == dev);
    NEED(q->scalar_type() == at::kBFloat16 && q->stride(2) == 1 && o->stride(2) == 1);
    NEED(o->size(0) >= batch && o->size(1) >= heads && o->size(2) == D);
    NEED(o->scalar_type() == at::kFloat || o->scalar_type() == at::kBFloat16);
    NEED(lse->size(0) >= batch && lse->size(1) >= heads && lse->stride(1) == 1 && lse->scalar_type() == at::kFloat);
    NEED((r2t->scalar_type() == at::kInt || r2t->scalar_type() == at::kLong) && r2g->scalar_type() == r2t->scalar_type());
    NEED(b_seq->scalar_type() == at::kInt && (!b_tail || b_tail->scalar_type() == at::kInt));

    // ---- lengths, splits, workspace ----
    if (a[MAX_SEQ] != Py_None) {
        NEED(as_long(a[MAX_SEQ], &max_seq));
        max_seq = pages ? std::max<int64_t>(1, max_seq) : 0;
    } else {
        max_seq = b_seq->numel() > 0 ? read_int(b_seq->max()) : 0;
    }
    if (a[MAX_TAIL] != Py_None) NEED(as_long(a[MAX_TAIL], &max_tail));
    else max_tail = b_tail && b_tail->numel() > 0 ? read_int(b_tail->max()) : 0;
    NEED(max_seq <= INT32_MAX && max_tail <= INT32_MAX);
    if (a[SPLITS] != Py_None) {
        NEED(as_long(a[SPLITS], &splits));
    } else {
        const char *forced = switches ? getenv("OMMX_ATTN_NUM_KV_SPLITS") : nullptr;
        while (forced && isspace((unsigned char)*forced)) ++forced;
        if (forced && *forced) {
            PyObject *mod = PyImport_ImportModule("open_ommx_serve_b200.attention.paged_decode");   // its strict reader
            PyObject *v = mod ? PyObject_CallMethod(mod, "_env_int", "si", "OMMX_ATTN_NUM_KV_SPLITS", 1) : nullptr;
            Py_XDECREF(mod);
            if (!v) return nullptr;
            const bool ok = as_long(v, &splits);
            Py_DECREF(v);
            NEED(ok);
        } else {
            const c10::cuda::CUDAGuard guard(dev);
            splits = ommx_b200_auto_num_kv_splits((int32_t)std::max<int64_t>(max_seq, 1), (int32_t)batch, (int32_t)kv_heads);
        }
    }
    splits = std::max<int64_t>(1, splits);
    NEED(splits <= INT32_MAX);
    Tensor own_logits;
    if (!static_ws) {
        const Tensor *al = as_tensor(a[ATTN_LOGITS]);
        if (!al) {
            NEED(a[ATTN_LOGITS] == Py_None);
            own_logits = fresh({batch, heads, splits + 1, D + 1}, q->options().dtype(at::kFloat));
            al = &own_logits;
        }
        NEED(al->scalar_type() == at::kFloat && al->device() == dev && al->dim() == 4 && al->size(0) >= batch && al->size(1) >= heads);
        NEED(al->size(3) == D + 1 && al->stride(3) == 1 && al->size(2) >= splits);
        d.attn_logits = (float *)al->data_ptr();
        d.al_stride_b = al->stride(0); d.al_stride_h = al->stride(1); d.al_stride_s = al->stride(2);
    }
    if (max_tail > 0) {
        NEED(kt && vt && b_tail && kt->dim() == 4 && kt->scalar_type() == at::kBFloat16 && vt->scalar_type() == at::kBFloat16);
        NEED(kt->strides() == vt->strides() && kt->stride(3) == 1);
        d.k_tail = kt->data_ptr(); d.v_tail = vt->data_ptr();
        d.tail_stride_b = kt->stride(0); d.tail_stride_t = kt->stride(1); d.tail_stride_h = kt->stride(2);
        d.b_tail_len = (const int32_t *)b_tail->data_ptr();
    }
    d.q = q->data_ptr(); d.q_dtype = OMMX_DT_BF16; d.batch = (int32_t)batch; d.n_q_heads = (int32_t)heads;
    d.q_stride_b = q->stride(0); d.q_stride_h = q->stride(1);
    d.b_seq_len = (const int32_t *)b_seq->data_ptr();
    d.req_to_token = r2t->data_ptr(); d.req_to_group = r2g->data_ptr();
    d.table_is_int64 = r2t->scalar_type() == at::kLong;
    d.r2t_stride_b = r2t->stride(0); d.r2g_stride_b = r2g->stride(0);
    d.o = o->data_ptr(); d.o_dtype = o->scalar_type() == at::kFloat ? OMMX_DT_F32 : OMMX_DT_BF16;
    d.o_stride_b = o->stride(0); d.o_stride_h = o->stride(1);
    d.lse = (float *)lse->data_ptr(); d.lse_stride_b = lse->stride(0);
    d.num_kv_splits = (int32_t)splits; d.max_seq_len = (int32_t)max_seq; d.max_tail_len = (int32_t)max_tail;
    d.seg_group_base = (int32_t)seg_base; d.packed_start_offset = (int32_t)start_offset;
    d.sm_scale = (float)sm_scale; d.logit_cap = (float)logit_cap;
    if (a[STATUS] != Py_None) {
        const Tensor *st = as_tensor(a[STATUS]);
        NEED(st && reachable(st));
        d.status = (int32_t *)st->data_ptr();
    }
    // differential-timing knobs: the caller records them, so a leaked export cannot pass as served
    for (size_t i = 0; switches && i < sizeof(ABL_FLAGS) / sizeof(ABL_FLAGS[0]); ++i)
        if (env_on(ABL_FLAGS[i])) d.abl_flags |= 1 << i;
    if (a[HEAD_GATHER] != Py_None) {
        NEED(stage != 1);
        PyObject *pd = THPDevice_New(dev);
        PyObject *g = pd ? PyObject_CallMethod(a[HEAD_GATHER], "check", "LLLO", (long long)batch, (long long)heads, (long long)D, pd) : nullptr;
        Py_XDECREF(pd);
        if (!g) return nullptr;
        d.gather = (const ommx_head_gather *)PyLong_AsVoidPtr(g);
        Py_DECREF(g);
    }
    const int rc = launch(dev, [&](void *stream) {
        if (static_ws) return ommx_b200_decode_static_ws(&d, stream);
        return stage == 0 ? ommx_b200_decode(&d, stream) : (stage == 1 ? ommx_b200_decode_stage1(&d, stream) : ommx_b200_decode_stage2(&d, stream));
    });
    return PyLong_FromLong(rc != 0 ? rc : d.abl_flags);
    END_HANDLE_TH_ERRORS
}

// ---- pack -----------------------------------------------------------------------------------------
bool dtype_code(const Tensor &t, int32_t *out) {
    switch (t.scalar_type()) {
        case at::kFloat: *out = OMMX_DT_F32; return true;
        case at::kBFloat16: *out = OMMX_DT_BF16; return true;
        case at::kHalf: *out = OMMX_DT_F16; return true;
        default: return false;
    }
}
bool index_table(PyObject *o, const int32_t **out) {
    *out = nullptr;
    if (o == Py_None) return true;
    const Tensor *t = as_tensor(o);
    if (!t || t->scalar_type() != at::kInt || !t->is_cuda() || !t->is_contiguous()) return false;
    *out = (const int32_t *)t->data_ptr();
    return true;
}

// K and V [32n, H, D] into `planes`.  False: declined.
bool pack_planes(const Tensor &K0, const Tensor &V0, const PlaneSet &s, const int32_t *pages, const int32_t *groups, int64_t k,
                 bool is_signed, bool use_pow2, bool use_map, int32_t *status, int *rc) {
    Tensor K = K0, V = V0;
    if (K.dim() != 3 || K.sizes() != V.sizes() || K.scalar_type() != V.scalar_type() || !K.is_cuda() || !reachable(&V)) return false;
    if (K.stride(2) != 1 || V.stride(2) != 1 || K.strides() != V.strides()) { K = K.contiguous(); V = V.contiguous(); }
    ommx_pack_args a;
    memset(&a, 0, sizeof(a));
    if (!dtype_code(K, &a.in_dtype) || K.size(0) > INT32_MAX) return false;
    if (!fill_planes(s, k, use_map, false, &a.planes)) return false;
    if (a.planes.n_kv_heads != K.size(1) || a.planes.head_dim != K.size(2)) return false;
    a.k = K.data_ptr(); a.v = V.data_ptr();
    a.num_tokens = (int32_t)K.size(0);
    a.stride_token = K.stride(0); a.stride_head = K.stride(1);
    a.dst_pages = pages; a.dst_groups = groups;
    a.outlier_select = is_signed; a.use_pow2 = use_pow2;
    a.status = status;
    *rc = launch(K.device(), [&](void *stream) { return ommx_b200_pack_kv(&a, stream); });
    return true;
}

// pack_into(K, V, planes, dst_pages, dst_groups, k, outlier_select, use_pow2, kv_outlier_map, status)
PyObject *py_pack_into(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 10) { PyErr_SetString(PyExc_TypeError, "pack_into: wrong argument count"); return nullptr; }
    const Tensor *K = as_tensor(a[0]), *V = as_tensor(a[1]), *st = as_tensor(a[9]);
    PlaneSet s;
    const int32_t *pages, *groups;
    int64_t k;
    bool use_pow2, use_map;
    NEED(K && V && read_plane_dict(a[2], &s) && index_table(a[3], &pages) && index_table(a[4], &groups) && as_long(a[5], &k));
    NEED(PyUnicode_Check(a[6]) && as_bool(a[7], &use_pow2) && as_bool(a[8], &use_map) && (st || a[9] == Py_None) && reachable(st));
    const char *sel = PyUnicode_AsUTF8(a[6]);
    if (!sel) return nullptr;
    const bool is_signed = strcasecmp(sel, "signed") == 0;
    NEED(is_signed || strcasecmp(sel, "abs") == 0);
    int rc = 0;
    NEED(pack_planes(*K, *V, s, pages, groups, k, is_signed, use_pow2, use_map, (int32_t *)ptr(st), &rc));
    return PyLong_FromLong(rc);
    END_HANDLE_TH_ERRORS
}

// pack_block(K, V, page_size, k, relidx7, signed, use_pow2, kv_outlier_map, scale_kind, check_finite) -> (planes, status bits)
// K, V contiguous-enough CUDA tensors of a length the caller has checked.  Every byte of every plane is written by the
// pack kernels (identity destinations), so nothing is cleared first.
PyObject *py_pack_block(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 10) { PyErr_SetString(PyExc_TypeError, "pack_block: wrong argument count"); return nullptr; }
    const Tensor *K = as_tensor(a[0]), *V = as_tensor(a[1]);
    int64_t ps, k, kind;
    bool relidx7, is_signed, use_pow2, use_map, check;
    NEED(K && V && K->is_cuda() && K->dim() == 3 && as_long(a[2], &ps) && as_long(a[3], &k) && as_bool(a[4], &relidx7) && as_bool(a[5], &is_signed) &&
         as_bool(a[6], &use_pow2) && as_bool(a[7], &use_map) && as_long(a[8], &kind) && as_bool(a[9], &check) && ps > 0 && k >= 0);
    const int64_t T = K->size(0), H = K->size(1), D = K->size(2), pages = T / ps, G = T / 32;
    const c10::cuda::CUDAGuard guard(K->device());
    const auto bytes = K->options().dtype(at::kByte), ints = K->options().dtype(at::kInt);
    const auto scale = K->options().dtype(kind == OMMX_SCALE_INT8_EXP ? at::kChar : (kind == OMMX_SCALE_BF16 ? at::kBFloat16 : at::kFloat));
    const auto zp = K->options().dtype(kind == OMMX_SCALE_F32 ? at::kFloat : at::kBFloat16);
    Tensor k_base = fresh({pages, ps, H, D / 4}, bytes), v_main = fresh({pages, ps, H, D / 4}, bytes);
    Tensor k_scale = fresh({G, H, D}, scale), k_zp = fresh({G, H, D}, zp);
    Tensor v_scale = fresh({pages, ps, H, D / 32}, scale), v_zp = fresh({pages, ps, H, D / 32}, zp);
    Tensor k_obmp, k_oval, k_ms, k_mc, k_oidx;
    if (k > 0) {
        k_obmp = fresh({G, H, D, 4}, bytes);
        k_oval = fresh({G, H, D, (k + 1) / 2}, bytes);
        if (use_map) { k_ms = fresh({G, H, D}, zp); k_mc = fresh({G, H, D}, zp); }
    }
    auto opt = [](const Tensor &t) { return t.defined() ? &t : nullptr; };
    const PlaneSet s{&k_base, &k_scale, &k_zp, opt(k_obmp), opt(k_oval), opt(k_ms), opt(k_mc), &v_main, &v_scale, &v_zp};
    Tensor status;
    if (check) status = fresh({1}, ints);
    Tensor r2t = fresh({1, pages}, ints), r2g = fresh({1, G}, ints);
    int rc = launch(K->device(), [&](void *stream) {
        return ommx_b200_identity_tables((int32_t *)r2t.data_ptr(), (int32_t)pages, (int32_t *)r2g.data_ptr(), (int32_t)G, (int32_t *)ptr(status), stream);
    });
    if (rc != 0) return PyLong_FromLong(rc);
    NEED(pack_planes(*K, *V, s, nullptr, nullptr, k, is_signed, use_pow2, use_map, check ? (int32_t *)status.data_ptr() : nullptr, &rc));
    if (rc == 0 && relidx7 && k > 0) {
        // same outlier set, other index encoding: k ascending 7-bit positions per frame (the value plane is shared)
        k_oidx = fresh({G, H, D, (7 * k + 7) / 8}, bytes);
        rc = launch(K->device(), [&](void *stream) {
            return ommx_b200_outlier_index_convert(k_obmp.data_ptr(), k_oidx.data_ptr(), G * H * D, (int32_t)k, 1, nullptr, stream);
        });
        k_obmp = Tensor();
    }
    if (rc != 0) return PyLong_FromLong(rc);
    THPObjectPtr d(PyDict_New());                          // made while the GPU packs; the status is read last
    if (!d) return nullptr;
    struct { const char *name; const Tensor *t; } out[] = {
        {"k_base", &k_base}, {"k_scale", &k_scale}, {"k_zp", &k_zp}, {"k_oidx", &k_oidx}, {"k_crank", nullptr}, {"k_obmp", &k_obmp}, {"k_oval", &k_oval},
        {"k_fp4_mapscale", &k_ms}, {"k_fp4_mapcenter", &k_mc}, {"v_main", &v_main}, {"v_scale", &v_scale}, {"v_zp", &v_zp},
        {"req_to_token", &r2t}, {"req_to_group", &r2g}};
    for (auto &e : out) {
        if (e.t && e.t->defined()) {
            PyObject *w = THPVariable_Wrap(*e.t);
            PyDict_SetItemString(d.get(), e.name, w);
            Py_XDECREF(w);
        } else {
            PyDict_SetItemString(d.get(), e.name, Py_None);
        }
    }
    int64_t bits = 0;
    if (check) bits = read_int(status);
    return Py_BuildValue("(NL)", d.release(), (long long)bits);
    END_HANDLE_TH_ERRORS
}

// ---- the pool's store step ------------------------------------------------------------------------
// Attribute readers that leave a Python error behind when the pool object is not what it should be.
struct PoolReader {
    PyObject *pool;
    bool ok = true;
    Tensor tensor(PyObject *name) {                    // a reference of our own: the attribute may be swapped meanwhile
        PyObject *v = ok ? PyObject_GetAttr(pool, name) : nullptr;
        const Tensor *t = v ? as_tensor(v) : nullptr;
        Tensor r = t ? *t : Tensor();
        if (!v) ok = false;
        else if (!t && v != Py_None) { PyErr_Format(PyExc_TypeError, "pool.%U is not a tensor", name); ok = false; }
        Py_XDECREF(v);
        return r;
    }
    int64_t integer(PyObject *name) {
        PyObject *v = ok ? PyObject_GetAttr(pool, name) : nullptr;
        int64_t r = 0;
        if (!v) ok = false;
        else if (!as_long(v, &r)) { PyErr_Format(PyExc_TypeError, "pool.%U is not an integer", name); ok = false; }
        Py_XDECREF(v);
        return r;
    }
};


// the pool descriptor; its tensors stay referenced by the pool object the caller holds
bool read_pool(PyObject *pool, ommx_kv_pool *p, at::Device *dev) {
    PoolReader r{pool};
    PyObject *planes = PyObject_GetAttr(pool, N.planes);
    if (!planes) return false;
    PlaneSet s;
    const int64_t k = r.integer(N.k), use_map = r.integer(N.kv_outlier_map);
    const bool ok = r.ok && read_plane_dict(planes, &s) && fill_planes(s, k, use_map != 0, false, &p->planes);
    if (ok) *dev = s.k_base->device();
    Py_DECREF(planes);
    if (!ok) {
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "the pool's planes must be contiguous tensors of the package's layout");
        return false;
    }
    p->k_hist = ptr(r.tensor(N.k_hist)); p->v_hist = ptr(r.tensor(N.v_hist));
    p->num_seqs = (int32_t)r.integer(N.num_seqs); p->ring_cap = (int32_t)r.integer(N.ring_cap);
    p->sink_tokens = (int32_t)r.integer(N.sink); p->recent_window = (int32_t)r.integer(N.recent);
    p->seq_len = (int32_t *)ptr(r.tensor(N.seq_dev));
    p->req_to_token = (const int32_t *)ptr(r.tensor(N.req_to_token)); p->req_to_group = (const int32_t *)ptr(r.tensor(N.req_to_group));
    p->pages_per_seq = (int32_t)r.integer(N.P_per_seq); p->groups_per_seq = (int32_t)r.integer(N.G_per_seq);
    return r.ok;
}

// New rows as the store kernels take them: bf16 on the pool's device, [B, H, D] or for one row [H, D], last dim contiguous
bool new_rows(const Tensor &K, const Tensor &V, const ommx_kv_pool &p, const at::Device &dev, int64_t batch, int64_t *sb, int64_t *sh) {
    const int64_t d = K.dim();
    if ((d != 3 && !(d == 2 && batch == 1)) || V.sizes() != K.sizes() || V.strides() != K.strides()) return false;
    if (K.scalar_type() != at::kBFloat16 || V.scalar_type() != at::kBFloat16 || K.device() != dev || V.device() != dev || K.stride(d - 1) != 1) return false;
    if (K.size(d - 1) != p.planes.head_dim || K.size(d - 2) != p.planes.n_kv_heads || (d == 3 && K.size(0) != batch)) return false;
    *sb = d == 3 ? K.stride(0) : 0;
    *sh = K.stride(d - 2);
    return true;
}

// kv_append(pool, batch, advance, K, V, slots, write_pos, outputs): K, V the new rows or None; slots / write_pos index tensors the
// caller has checked, or None (slots: the pool's selected ones).  None: K / V need the caller's conversions first.
PyObject *py_kv_append(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 8) { PyErr_SetString(PyExc_TypeError, "kv_append: wrong argument count"); return nullptr; }
    ommx_kv_append_args d;
    memset(&d, 0, sizeof(d));
    at::Device dev(at::kCUDA);
    if (!read_pool(a[0], &d.pool, &dev)) return nullptr;
    PoolReader r{a[0]};
    int64_t batch, advance;
    bool outputs;
    if (!as_long(a[1], &batch) || !as_long(a[2], &advance) || !as_bool(a[7], &outputs)) { PyErr_SetString(PyExc_TypeError, "kv_append: batch, advance, outputs"); return nullptr; }
    const Tensor *K = as_tensor(a[3]), *V = as_tensor(a[4]), *slots = as_tensor(a[5]), *wpos = as_tensor(a[6]);
    if (advance) {
        NEED(K && V && new_rows(*K, *V, d.pool, dev, batch, &d.new_stride_b, &d.new_stride_h));
        d.k_new = K->data_ptr(); d.v_new = V->data_ptr();
    }
    Tensor sel;
    if (!slots && !wpos) { sel = r.tensor(N.sel); d.slots = ptr(sel); }
    else {
        d.slots = ptr(slots); d.write_pos = ptr(wpos);
        d.index_is_int64 = (slots ? slots : wpos)->scalar_type() == at::kLong;
    }
    d.batch = (int32_t)batch; d.advance = (int32_t)advance; d.outlier_select = 1; d.use_pow2 = 1;
    if (outputs) {
        d.k_tail = ptr(r.tensor(N.k_tail)); d.v_tail = ptr(r.tensor(N.v_tail)); d.max_tail = (int32_t)r.integer(N.max_tail_len);
        d.b_seq_len = (int32_t *)ptr(r.tensor(N.b_seq)); d.b_tail_len = (int32_t *)ptr(r.tensor(N.b_tail));
    }
    d.status = (int32_t *)ptr(r.tensor(N.status));
    if (!r.ok) return nullptr;
    return PyLong_FromLong(launch(dev, [&](void *stream) { return ommx_b200_kv_append_decode(&d, stream); }));
    END_HANDLE_TH_ERRORS
}

// kv_append_block(pool, slot, K, V): prefill of one slot; None: K / V need the caller's conversions first
PyObject *py_kv_append_block(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 4) { PyErr_SetString(PyExc_TypeError, "kv_append_block: wrong argument count"); return nullptr; }
    ommx_kv_pool p;
    memset(&p, 0, sizeof(p));
    at::Device dev(at::kCUDA);
    if (!read_pool(a[0], &p, &dev)) return nullptr;
    PoolReader r{a[0]};
    const Tensor *K = as_tensor(a[2]), *V = as_tensor(a[3]);
    int64_t slot, st, sh;
    NEED(K && V && as_long(a[1], &slot) && K->dim() == 3 && new_rows(*K, *V, p, dev, K->size(0), &st, &sh));
    int32_t *status = (int32_t *)ptr(r.tensor(N.status));
    if (!r.ok) return nullptr;
    return PyLong_FromLong(launch(dev, [&](void *stream) {
        return ommx_b200_kv_append_block(&p, (int32_t)slot, K->data_ptr(), V->data_ptr(), st, sh, (int32_t)K->size(0), status, stream);
    }));
    END_HANDLE_TH_ERRORS
}

// kv_gather_tail(pool, sel, tail_idx, k_tail, v_tail, with_tables): tensors the caller has checked.  Returns the C ABI's code, or
// with_tables the two table rows of every selected sequence ([B, pages], [B, groups])
PyObject *py_kv_gather_tail(PyObject *, PyObject *const *a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 6) { PyErr_SetString(PyExc_TypeError, "kv_gather_tail: wrong argument count"); return nullptr; }
    ommx_kv_pool p;
    memset(&p, 0, sizeof(p));
    at::Device dev(at::kCUDA);
    if (!read_pool(a[0], &p, &dev)) return nullptr;
    PoolReader r{a[0]};
    const Tensor *sel = as_tensor(a[1]), *idx = as_tensor(a[2]), *kt = as_tensor(a[3]), *vt = as_tensor(a[4]);
    bool tables;
    if (!idx || !kt || !vt || !as_bool(a[5], &tables)) { PyErr_SetString(PyExc_TypeError, "kv_gather_tail: tensors expected"); return nullptr; }
    for (const Tensor *t : {sel, idx, kt, vt})
        if (!reachable(t)) { PyErr_SetString(PyExc_ValueError, "kv_gather_tail: sel, tail indices and residual buffers must be CUDA tensors"); return nullptr; }
    const Tensor sel_c = sel ? sel->contiguous() : Tensor(), idx_c = idx->contiguous();
    int32_t *status = (int32_t *)ptr(r.tensor(N.status));
    if (!r.ok) return nullptr;
    Tensor r2t, r2g;
    if (tables) {
        const c10::cuda::CUDAGuard guard(dev);
        r2t = at::empty({idx_c.size(0), p.pages_per_seq}, kt->options().dtype(at::kInt));
        r2g = at::empty({idx_c.size(0), p.groups_per_seq}, kt->options().dtype(at::kInt));
    }
    const int rc = launch(dev, [&](void *stream) {
        return ommx_b200_kv_gather_inputs(&p, ptr(sel_c), idx_c.data_ptr(), idx_c.scalar_type() == at::kLong, (int32_t)idx_c.size(0), (int32_t)idx_c.size(1),
                                          kt->data_ptr(), vt->data_ptr(), (int32_t *)ptr(r2t), (int32_t *)ptr(r2g), status, stream);
    });
    if (!tables || rc != 0) return PyLong_FromLong(rc);
    return Py_BuildValue("(NN)", THPVariable_Wrap(r2t), THPVariable_Wrap(r2g));
    END_HANDLE_TH_ERRORS
}

PyMethodDef METHODS[] = {
    {"decode", (PyCFunction)(void (*)())py_decode, METH_FASTCALL, "paged decode attention; None when an argument needs explaining"},
    {"pack_into", (PyCFunction)(void (*)())py_pack_into, METH_FASTCALL, "quantize and pack into given planes; None when an argument needs explaining"},
    {"pack_block", (PyCFunction)(void (*)())py_pack_block, METH_FASTCALL, "quantize and pack into fresh planes"},
    {"kv_append", (PyCFunction)(void (*)())py_kv_append, METH_FASTCALL, "decode-step store of a pool"},
    {"kv_append_block", (PyCFunction)(void (*)())py_kv_append_block, METH_FASTCALL, "prefill of one slot of a pool"},
    {"kv_gather_tail", (PyCFunction)(void (*)())py_kv_gather_tail, METH_FASTCALL, "residual rows by position"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef MODULE = {PyModuleDef_HEAD_INIT, "_host", "torch tensors -> the C ABI of libommx_b200.so", -1, METHODS, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
    struct { PyObject **to; const char *name; } all[] = {
        {&N.k_base, "k_base"}, {&N.k_scale, "k_scale"}, {&N.k_zp, "k_zp"}, {&N.k_obmp, "k_obmp"}, {&N.k_oval, "k_oval"}, {&N.k_fp4_mapscale, "k_fp4_mapscale"},
        {&N.k_fp4_mapcenter, "k_fp4_mapcenter"}, {&N.v_main, "v_main"}, {&N.v_scale, "v_scale"}, {&N.v_zp, "v_zp"}, {&N.planes, "planes"}, {&N.k, "k"},
        {&N.kv_outlier_map, "kv_outlier_map"}, {&N.k_hist, "k_hist"}, {&N.v_hist, "v_hist"}, {&N.num_seqs, "num_seqs"}, {&N.ring_cap, "ring_cap"},
        {&N.sink, "sink"}, {&N.recent, "recent"}, {&N.seq_dev, "seq_dev"}, {&N.req_to_token, "_req_to_token"}, {&N.req_to_group, "_req_to_group"},
        {&N.P_per_seq, "P_per_seq"}, {&N.G_per_seq, "G_per_seq"}, {&N.k_tail, "k_tail"}, {&N.v_tail, "v_tail"}, {&N.max_tail_len, "max_tail_len"},
        {&N.b_seq, "b_seq"}, {&N.b_tail, "b_tail"}, {&N.status, "status"}, {&N.sel, "_sel"}};
    for (auto &e : all)
        if (!(*e.to = PyUnicode_InternFromString(e.name))) return nullptr;
    return PyModule_Create(&MODULE);
}
