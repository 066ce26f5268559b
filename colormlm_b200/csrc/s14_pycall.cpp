// The Python mirror's per-token calls as CPython functions over the C ABI: they take the tensors as they are,
// read addresses and sizes, look up torch's current stream, fill the call's descriptor and release the
// interpreter lock around the call.  Through ctypes that took as long as the kernel launch behind it or longer
// (2.5 to 4 us of a 4.6 to 6 us call; here 0.6 us).  Every function returns the status of the C call; the Python side
// turns a status into S14Error.  Nothing is computed here, and no torch header is needed: a tensor's data_ptr,
// shape and dtype are asked for by name.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstring>

#include "../../include/polaris_s14_cuda.h"

namespace {

PyObject *n_data_ptr, *n_shape, *n_dtype, *n_numel, *n_expert_ids, *n_weights, *n_pages;  // interned names
PyObject *n_value, *n_as_parameter, *n_cuda_stream;
PyTypeObject *t_void_p;                   // ctypes.c_void_p
// What torch has to be asked, filled on the first call that needs it (a program that names its streams and uses host
// buffers does without torch): its dtypes, and the lookups of the current device and its current stream.
PyObject *t_float32, *t_bfloat16;
PyObject *f_device, *f_raw_stream;        // two C functions; where torch lacks them, f_stream: torch.cuda.current_stream
PyObject *f_stream;

struct Failed {};   // a Python error is set
struct Refused {};  // not a call the library could take: None is returned

// What ctypes passes as a void pointer beside ints: its own c_void_p, and objects that name one as their parameter
// (torch.cuda.Stream is one).
void *foreign_pointer(PyObject *v, int depth = 0) {
    PyObject *inner = nullptr;
    if (PyObject_TypeCheck(v, t_void_p)) inner = PyObject_GetAttr(v, n_value);
    else if (depth < 2 && PyObject_HasAttr(v, n_as_parameter)) inner = PyObject_GetAttr(v, n_as_parameter);
    else PyErr_Format(PyExc_TypeError, "an address or handle is needed, not %s", Py_TYPE(v)->tp_name);
    if (!inner) throw Failed{};
    void *p = nullptr;
    bool failed = false;
    if (PyLong_Check(inner)) {
        p = PyLong_AsVoidPtr(inner);
        failed = PyErr_Occurred() != nullptr;
    } else if (inner != Py_None) {
        try {
            p = foreign_pointer(inner, depth + 1);
        } catch (const Failed &) {
            failed = true;
        }
    }
    Py_DECREF(inner);
    if (failed) throw Failed{};
    return p;
}

void *address(PyObject *tensor) {
    PyObject *args[1] = {tensor};
    PyObject *v = PyObject_VectorcallMethod(n_data_ptr, args, 1 | PY_VECTORCALL_ARGUMENTS_OFFSET, nullptr);
    if (!v) throw Failed{};
    void *p = PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    if (PyErr_Occurred()) throw Failed{};
    return p;
}
void *address_or_null(PyObject *tensor) { return tensor == Py_None ? nullptr : address(tensor); }

void *pointer(PyObject *v) {  // a device address or handle held as an int, a ctypes.c_void_p, None, or what stands in for one
    if (v == Py_None) return nullptr;
    if (!PyLong_Check(v)) return foreign_pointer(v);
    void *p = PyLong_AsVoidPtr(v);
    if (PyErr_Occurred()) throw Failed{};
    return p;
}
uint32_t u32(PyObject *v) {
    const unsigned long r = PyLong_AsUnsignedLongMask(v);
    if (PyErr_Occurred()) throw Failed{};
    return (uint32_t)r;
}
float f32(PyObject *v) {
    const double r = PyFloat_AsDouble(v);
    if (PyErr_Occurred()) throw Failed{};
    return (float)r;
}

// The first n sizes of a tensor (or, `last`, its last one alone); returns its number of dimensions.
int sizes(PyObject *tensor, uint32_t *out, int n, bool last = false) {
    PyObject *s = PyObject_GetAttr(tensor, n_shape);
    if (!s) throw Failed{};
    const int dims = PyTuple_Check(s) ? (int)PyTuple_GET_SIZE(s) : -1;
    if (dims < n) {
        Py_DECREF(s);
        PyErr_Format(PyExc_IndexError, "a tensor of %d dimensions is needed", n);
        throw Failed{};
    }
    for (int i = 0; i < n; ++i) out[i] = (uint32_t)PyLong_AsUnsignedLongMask(PyTuple_GET_ITEM(s, last ? dims - 1 : i));
    Py_DECREF(s);
    return dims;
}
// tokens of a [hidden] or [tokens, hidden] tensor
uint32_t token_count(PyObject *x) {
    uint32_t n[1];
    return sizes(x, n, 1) == 1 ? 1u : n[0];
}

PyObject *attr_of(PyObject *o, const char *name) {
    if (!o) throw Failed{};
    PyObject *v = PyObject_GetAttrString(o, name);
    Py_DECREF(o);
    if (!v) throw Failed{};
    return v;
}
PyObject *torch_attr(const char *name) { return attr_of(PyImport_ImportModule("torch"), name); }
void ask_torch_types() {
    PyObject *f = torch_attr("float32"), *b = torch_attr("bfloat16");
    t_float32 = f, t_bfloat16 = b;
}
void ask_torch_streams() {
    PyObject *init = attr_of(torch_attr("cuda"), "init");  // the raw lookups do not initialise torch
    PyObject *done = PyObject_CallNoArgs(init);
    Py_DECREF(init);
    if (!done) throw Failed{};
    Py_DECREF(done);
    try {
        PyObject *d = attr_of(torch_attr("_C"), "_cuda_getDevice"), *r = attr_of(torch_attr("_C"), "_cuda_getCurrentRawStream");
        f_device = d, f_raw_stream = r;
    } catch (const Failed &) {
        PyErr_Clear();
        f_stream = attr_of(torch_attr("cuda"), "current_stream");
    }
}

// S14_STREAM_*; a tensor of another type ends the call with None, which the Python side reports
uint32_t stream_type(PyObject *tensor) {
    PyObject *d = PyObject_GetAttr(tensor, n_dtype);
    if (!d) throw Failed{};
    Py_DECREF(d);  // torch keeps its dtypes
    if (!t_bfloat16) ask_torch_types();
    if (d == t_bfloat16) return S14_STREAM_BF16;
    if (d == t_float32) return S14_STREAM_F32;
    throw Refused{};
}

// The caller's stream, or torch's current one; torch's default stream is passed by its own handle
// (cudaStreamLegacy), because the C ABI reads NULL as the context's own stream.
void *stream_of(PyObject *stream) {
    if (stream != Py_None) return pointer(stream);
    if (!f_raw_stream && !f_stream) ask_torch_streams();
    PyObject *raw;
    if (f_raw_stream) {
        PyObject *dev = PyObject_CallNoArgs(f_device);
        if (!dev) throw Failed{};
        raw = PyObject_CallOneArg(f_raw_stream, dev);
        Py_DECREF(dev);
    } else {
        PyObject *current = PyObject_CallNoArgs(f_stream);
        if (!current) throw Failed{};
        raw = PyObject_GetAttr(current, n_cuda_stream);
        Py_DECREF(current);
    }
    if (!raw) throw Failed{};
    void *p = PyLong_AsVoidPtr(raw);
    Py_DECREF(raw);
    if (PyErr_Occurred()) throw Failed{};
    return p ? p : (void *)1;
}

template <class Call>
PyObject *unlocked(Call call) {
    int32_t rc;
    Py_BEGIN_ALLOW_THREADS
    rc = call();
    Py_END_ALLOW_THREADS
    return PyLong_FromLong(rc);
}

#define S14_ARGS(name, count)                                                                            \
    if (nargs != (count)) return PyErr_Format(PyExc_TypeError, name ": %d arguments are needed", (count)); \
    try {
#define S14_DONE                               \
    }                                          \
    catch (const Failed &) { return nullptr; } \
    catch (const Refused &) { Py_RETURN_NONE; }

s14_ctx *ctx_of(PyObject *v) { return (s14_ctx *)pointer(v); }

s14_hc_params hc_params(PyObject *x, PyObject *fn, PyObject *scale, PyObject *base, uint32_t iters, float norm_eps, float hc_eps) {
    s14_hc_params p = {};
    uint32_t s[3];
    sizes(x, s, 3);
    p.n_tokens = s[0], p.hc = s[1], p.hidden = s[2];
    p.dtype = stream_type(x);
    p.sinkhorn_iters = iters, p.norm_eps = norm_eps, p.hc_eps = hc_eps;
    p.hc_fn = (const float *)address(fn), p.hc_scale = (const float *)address(scale), p.hc_base = (const float *)address(base);
    return p;
}

// (ctx, stream, x, hc_fn, hc_scale, hc_base, reduced, post, comb, iters, norm_eps, hc_eps)
PyObject *hc_pre(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("hc_pre", 12)
    const s14_hc_params p = hc_params(a[2], a[3], a[4], a[5], u32(a[9]), f32(a[10]), f32(a[11]));
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]), *x = address(a[2]), *red = address(a[6]), *post = address(a[7]), *comb = address(a[8]);
    return unlocked([&] { return s14_cmd_hc_pre(c, st, &p, x, red, (float *)post, (float *)comb); });
    S14_DONE
}

// (ctx, stream, x, hc_fn, hc_scale, hc_base, reduced, pre, norm_eps, hc_eps)
PyObject *hc_head_reduce(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("hc_head_reduce", 10)
    const s14_hc_params p = hc_params(a[2], a[3], a[4], a[5], 1u, f32(a[8]), f32(a[9]));
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]), *x = address(a[2]), *red = address(a[6]), *pre = address(a[7]);
    return unlocked([&] { return s14_cmd_hc_head_reduce(c, st, &p, x, red, (float *)pre); });
    S14_DONE
}

// (ctx, stream, branch, residual, post, comb, merged)
PyObject *hc_post(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("hc_post", 7)
    uint32_t s[3];
    sizes(a[3], s, 3);
    const uint32_t dt = stream_type(a[3]);
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]), *branch = address(a[2]), *res = address(a[3]), *post = address(a[4]), *comb = address(a[5]),
         *merged = address(a[6]);
    return unlocked([&] { return s14_cmd_hc_post(c, st, s[0], s[1], s[2], dt, branch, res, (const float *)post, (const float *)comb, merged); });
    S14_DONE
}

// (ctx, stream, x, weight, eps, out)
PyObject *rms_norm(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("rms_norm", 6)
    uint32_t s[2];
    sizes(a[2], s, 2);
    const uint32_t dt = stream_type(a[2]);
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]), *x = address(a[2]), *w = address(a[3]), *out = address(a[5]);
    const float eps = f32(a[4]);
    return unlocked([&] { return s14_cmd_rms_norm(c, st, s[0], s[1], dt, x, (const float *)w, eps, out); });
    S14_DONE
}

// (ctx, stream, x, weight_bf16, logits_out, n_rows or None)
PyObject *head_logits(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("head_logits", 6)
    uint32_t sw[2], so[1];
    const uint32_t n_tokens = token_count(a[2]);
    sizes(a[3], sw, 2);
    sizes(a[4], so, 1, true);
    const uint32_t rows = a[5] == Py_None ? sw[0] : u32(a[5]);
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]), *x = address(a[2]), *w = address(a[3]), *out = address(a[4]);
    return unlocked([&] { return s14_cmd_head_logits(c, st, (const float *)x, n_tokens, (const uint16_t *)w, rows, sw[1], (float *)out, so[0]); });
    S14_DONE
}

// (ctx, stream, logits, result)
PyObject *greedy_argmax(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("greedy_argmax", 4)
    PyObject *args[1] = {a[2]};
    PyObject *v = PyObject_VectorcallMethod(n_numel, args, 1 | PY_VECTORCALL_ARGUMENTS_OFFSET, nullptr);
    if (!v) return nullptr;
    const uint32_t n = (uint32_t)PyLong_AsUnsignedLongMask(v);
    Py_DECREF(v);
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]), *logits = address(a[2]), *res = address(a[3]);
    return unlocked([&] { return s14_cmd_greedy_argmax(c, st, (const float *)logits, n, (int64_t *)res); });
    S14_DONE
}

// (ctx, stream, state, hc_fn, hc_scale, hc_base, norm_weight, head_weight, logits_out, norm_eps, hc_eps)
PyObject *exec_head(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("exec_head", 11)
    const s14_hc_params p = hc_params(a[2], a[3], a[4], a[5], 1u, f32(a[9]), f32(a[10]));
    uint32_t sw[1];
    sizes(a[7], sw, 1);
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]), *state = address(a[2]), *nw = address(a[6]), *w = address(a[7]), *out = address(a[8]);
    return unlocked([&] {
        return s14_exec_hc_head_norm_full_logits(c, st, &p, (const float *)nw, (const uint16_t *)w, sw[0], (const uint16_t *)state, (float *)out);
    });
    S14_DONE
}

// The items of a short sequence (list, tuple, array).
struct Items {
    PyObject *fast;
    Py_ssize_t n;
    explicit Items(PyObject *seq) : fast(PySequence_Fast(seq, "a sequence is needed")), n(0) {
        if (!fast) throw Failed{};
        n = PySequence_Fast_GET_SIZE(fast);
    }
    Items(const Items &) = delete;
    ~Items() { Py_DECREF(fast); }
    PyObject *operator[](Py_ssize_t i) const { return PySequence_Fast_GET_ITEM(fast, i); }
};
struct Owned {
    PyObject *o;
    explicit Owned(PyObject *v) : o(v) {
        if (!o) throw Failed{};
    }
    Owned(const Owned &) = delete;
    ~Owned() { Py_DECREF(o); }
};
unsigned long long whole(PyObject *v) {
    if (PyLong_CheckExact(v)) {
        const unsigned long long r = PyLong_AsUnsignedLongLongMask(v);
        if (PyErr_Occurred()) throw Failed{};
        return r;
    }
    Owned i(PyNumber_Long(v));  // numpy integers and the like
    const unsigned long long r = PyLong_AsUnsignedLongLongMask(i.o);
    if (PyErr_Occurred()) throw Failed{};
    return r;
}

// A TokenRoute (expert_ids, weights, pages): at most six matching items.
void token_route(PyObject *route, s14_token_route &r) {
    Owned ids_o(PyObject_GetAttr(route, n_expert_ids)), w_o(PyObject_GetAttr(route, n_weights)), p_o(PyObject_GetAttr(route, n_pages));
    Items ids(ids_o.o), w(w_o.o), pages(p_o.o);
    if (ids.n > (Py_ssize_t)S14_EXPERTS_PER_TOKEN || w.n != ids.n || pages.n != ids.n) throw Refused{};
    std::memset(&r, 0, sizeof(r));
    r.n_routed = (uint32_t)ids.n;
    for (Py_ssize_t j = 0; j < ids.n; ++j) {
        r.expert_ids[j] = (uint16_t)whole(ids[j]);
        r.weights[j] = f32(w[j]);
        r.pages[j] = (const uint8_t *)(uintptr_t)whole(pages[j]);
    }
}

// (ctx, stream, ffn_input, residual, post, comb, route, shared_page, shared_kind, inter, state_out, branch_out or None)
PyObject *exec_moe(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("exec_moe", 12)
    s14_token_route route;
    token_route(a[6], route);
    s14_exec_moe_desc d = {};
    uint32_t s[1];
    sizes(a[2], s, 1, true);
    d.hidden = s[0], d.inter = u32(a[9]), d.shared_kind = u32(a[8]);
    d.route = &route;
    d.shared_page = (const uint8_t *)pointer(a[7]);
    d.ffn_input_bf16 = (const uint16_t *)address(a[2]), d.residual_bf16 = (const uint16_t *)address(a[3]);
    d.post = (const float *)address(a[4]), d.comb = (const float *)address(a[5]);
    d.state_out_bf16 = (uint16_t *)address(a[10]), d.moe_branch_out_bf16 = (uint16_t *)address_or_null(a[11]);
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]);
    return unlocked([&] { return s14_exec_routed_and_shared_moe_then_hc_post(c, st, &d); });
    S14_DONE
}

s14_routed_layer_desc routed_desc(PyObject *x, PyObject *wr, PyObject *bias, PyObject *table, PyObject *shared, PyObject *kind,
                                  PyObject *inter, PyObject *y, PyObject *ids, PyObject *weights, PyObject *score_fn, PyObject *top_k,
                                  PyObject *route_scale) {
    s14_routed_layer_desc d = {};
    uint32_t sw[2];
    d.router.n_tokens = token_count(x);
    sizes(wr, sw, 2);
    d.router.n_experts = sw[0], d.router.hidden = sw[1];
    d.router.top_k = u32(top_k), d.router.score_fn = u32(score_fn), d.router.route_scale = f32(route_scale);
    d.router.x = (const float *)address(x);
    d.router.router_weight_bf16 = (const uint16_t *)address(wr);
    d.router.bias = (const float *)address_or_null(bias);
    d.router.ids_out = (int32_t *)address_or_null(ids), d.router.weights_out = (float *)address_or_null(weights);
    d.inter = u32(inter), d.shared_kind = u32(kind);
    d.page_table = (const uint8_t *const *)address(table);
    d.shared_page = (const uint8_t *)pointer(shared);
    d.y = (float *)address(y);
    return d;
}

// (ctx, stream, x, wr, bias, page_table, shared_page, shared_kind, inter, y, ids, weights, score_fn, top_k, route_scale)
PyObject *routed_layer(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("routed_layer", 15)
    const s14_routed_layer_desc d = routed_desc(a[2], a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14]);
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]);
    return unlocked([&] { return s14_cmd_routed_moe_layer(c, st, &d); });
    S14_DONE
}

// (ctx, stream, block, x, wr, bias, page_table, shared_page, shared_kind, inter, y, ids, weights, score_fn, top_k, route_scale)
PyObject *routed_block(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("routed_block", 16)
    const s14_routed_layer_desc d = routed_desc(a[3], a[4], a[5], a[6], a[7], a[8], a[9], a[10], a[11], a[12], a[13], a[14], a[15]);
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]);
    s14_block *b = (s14_block *)pointer(a[2]);
    return unlocked([&] { return s14_cmd_routed_moe_block(c, st, b, &d); });
    S14_DONE
}

// (ctx, stream, stack, x, h_out)
PyObject *stack_decode(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("stack_decode", 5)
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]), *x = address(a[3]), *h = address(a[4]);
    s14_stack *k = (s14_stack *)pointer(a[2]);
    return unlocked([&] { return s14_cmd_stack_decode(c, st, k, (const float *)x, (float *)h); });
    S14_DONE
}

// The Python classes of the bound operators' records, in the order of set_records' arguments: two of them have the
// same size, so a record's bytes do not tell what it is.
enum RecordKind { kMxfp4, kFp8, kSwiglu, kRouteMix, kAccumulate, kRecordKinds };
PyTypeObject *record_types[kRecordKinds];

PyObject *set_records(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    if (nargs != kRecordKinds) return PyErr_Format(PyExc_TypeError, "set_records: %d classes are needed", (int)kRecordKinds);
    for (int i = 0; i < kRecordKinds; ++i)
        if (!PyType_Check(a[i])) return PyErr_Format(PyExc_TypeError, "set_records: a class is needed");
    for (int i = 0; i < kRecordKinds; ++i) {
        PyTypeObject *old = record_types[i];
        record_types[i] = (PyTypeObject *)Py_NewRef(a[i]);
        Py_XDECREF(old);
    }
    Py_RETURN_NONE;
}

// (ctx, stream, dispatch): a bound operator's record, read through the buffer protocol
template <RecordKind kKind, class Dispatch, int32_t (*kCall)(s14_ctx *, void *, const Dispatch *)>
PyObject *bound(PyObject *, PyObject *const *a, Py_ssize_t nargs) {
    S14_ARGS("a bound operator", 3)
    if (!record_types[kKind] || !PyObject_TypeCheck(a[2], record_types[kKind]))
        return PyErr_Format(PyExc_TypeError, "the dispatch record is a %s, not one of this operator", Py_TYPE(a[2])->tp_name);
    s14_ctx *c = ctx_of(a[0]);
    void *st = stream_of(a[1]);
    Py_buffer v;
    if (PyObject_GetBuffer(a[2], &v, PyBUF_SIMPLE) != 0) return nullptr;
    if (v.len != (Py_ssize_t)sizeof(Dispatch)) {
        PyBuffer_Release(&v);
        return PyErr_Format(PyExc_TypeError, "the dispatch record is not laid out as the library's");
    }
    PyObject *r = unlocked([&] { return kCall(c, st, (const Dispatch *)v.buf); });
    PyBuffer_Release(&v);
    return r;
    S14_DONE
}

#define S14_FAST(name, fn) {name, (PyCFunction)(void (*)(void))(fn), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    S14_FAST("set_records", set_records),
    S14_FAST("hc_pre", hc_pre),
    S14_FAST("hc_post", hc_post),
    S14_FAST("hc_head_reduce", hc_head_reduce),
    S14_FAST("rms_norm", rms_norm),
    S14_FAST("head_logits", head_logits),
    S14_FAST("greedy_argmax", greedy_argmax),
    S14_FAST("exec_head", exec_head),
    S14_FAST("exec_moe", exec_moe),
    S14_FAST("routed_layer", routed_layer),
    S14_FAST("routed_block", routed_block),
    S14_FAST("stack_decode", stack_decode),
    S14_FAST("mxfp4_matvec", (bound<kMxfp4, s14_mxfp4_dispatch, s14_cmd_mxfp4_matvec>)),
    S14_FAST("fp8_matvec", (bound<kFp8, s14_fp8_dispatch, s14_cmd_fp8_matvec>)),
    S14_FAST("swiglu_limit", (bound<kSwiglu, s14_swiglu_limit_dispatch, s14_cmd_swiglu_limit>)),
    S14_FAST("route_mix", (bound<kRouteMix, s14_route_mix_dispatch, s14_cmd_route_mix>)),
    S14_FAST("moe_accumulate", (bound<kAccumulate, s14_moe_accumulate_dispatch, s14_cmd_moe_accumulate>)),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_s14call", "Per-token calls of the Python mirror over the C ABI.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__s14call(void) {
    n_data_ptr = PyUnicode_InternFromString("data_ptr");
    n_shape = PyUnicode_InternFromString("shape");
    n_dtype = PyUnicode_InternFromString("dtype");
    n_numel = PyUnicode_InternFromString("numel");
    n_expert_ids = PyUnicode_InternFromString("expert_ids");
    n_weights = PyUnicode_InternFromString("weights");
    n_pages = PyUnicode_InternFromString("pages");
    n_value = PyUnicode_InternFromString("value");
    n_as_parameter = PyUnicode_InternFromString("_as_parameter_");
    n_cuda_stream = PyUnicode_InternFromString("cuda_stream");
    PyObject *ctypes = PyImport_ImportModule("ctypes");
    if (!ctypes) return nullptr;
    PyObject *void_p = PyObject_GetAttrString(ctypes, "c_void_p");
    Py_DECREF(ctypes);
    if (!void_p) return nullptr;
    if (!PyType_Check(void_p)) return PyErr_Format(PyExc_TypeError, "ctypes.c_void_p is not a class");
    t_void_p = (PyTypeObject *)void_p;
    return PyModule_Create(&module);
}
