// Native host path of the operators: tensors in, checked, outputs allocated, parameter blocks filled, one call of the
// C ABI on the current stream.  Everything here also exists as plain C (include/pikv_b200.h); this module only takes the
// per-call marshalling out of the interpreter, where it cost 40 to 70 us a call (attribute look-ups, a ctypes field and a
// tensor allocation at a time) - several times what the kernels of a decode step take.
//
// Conventions: arguments are positional (METH_FASTCALL); a cache is passed as its module's buffer dict and its geometry;
// None stands for an absent tensor.  Errors are raised as pikv_b200.PikvError, torch's own as what they are.
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/Exceptions.h>
#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/core/InferenceMode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAStream.h>

#include <cstdarg>
#include <exception>
#include <string>

#include "../../../include/pikv_b200.h"

namespace {

PyObject* g_error = nullptr;              // pikv_b200.PikvError

struct Raised : std::exception {};        // a Python error is set

[[noreturn]] void fail(const char* fmt, ...) {
    char text[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(text, sizeof(text), fmt, ap);
    va_end(ap);
    PyErr_SetString(g_error, text);
    throw Raised();
}

void check(int rc, const char* what) {
    if (rc != PIKV_OK) fail("%s failed with status %d: %s", what, rc, pikv_last_error());
}

using OptType = c10::optional<at::ScalarType>;

// a contiguous CUDA tensor of that type
at::Tensor req(PyObject* o, const char* name, OptType type = c10::nullopt) {
    if (!THPVariable_Check(o)) fail("%s must be a CUDA tensor (there is no CPU path)", name);
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda()) fail("%s must be a CUDA tensor (there is no CPU path)", name);
    if (type && t.scalar_type() != *type)
        fail("%s must be %s, got %s", name, c10::toString(*type), c10::toString(t.scalar_type()));
    return t.is_contiguous() ? t : t.contiguous();
}
at::Tensor opt(PyObject* o, const char* name, OptType type = c10::nullopt) { return o == Py_None ? at::Tensor() : req(o, name, type); }

// a tensor that is written: a contiguous copy would take the update and be dropped
at::Tensor written(PyObject* o, const char* name, OptType type) {
    if (o == Py_None) return at::Tensor();
    if (THPVariable_Check(o) && !THPVariable_Unpack(o).is_contiguous()) fail("%s is updated in place and must be contiguous", name);
    return req(o, name, type);
}

// an fp32 vector, converted if it has another type
at::Tensor f32(PyObject* o, const char* name) {
    at::Tensor t = opt(o, name);
    return !t.defined() || t.scalar_type() == at::kFloat ? t : t.to(at::kFloat);
}

// rows of x [..., K]
int rows_of(const at::Tensor& x, const char* name) {
    if (x.dim() < 1 || x.size(-1) < 1) fail("%s must have a last dimension of at least 1", name);
    return (int)(x.numel() / x.size(-1));
}

// the kernels read (or write) that many elements
const at::Tensor& holds(const at::Tensor& t, int64_t elements, const char* name) {
    if (t.defined() && t.numel() < elements) fail("%s has %lld elements, %lld are needed", name, (long long)t.numel(), (long long)elements);
    return t;
}

int dtype_code(const at::Tensor& t, const char* name) {
    if (t.scalar_type() == at::kFloat) return PIKV_F32;
    if (t.scalar_type() == at::kBFloat16) return PIKV_BF16;
    fail("%s: dtype %s not supported (float32 or bfloat16)", name, c10::toString(t.scalar_type()));
}

template <typename T = void>
T* ptr(const at::Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }

pikv_stream_t stream() { return static_cast<pikv_stream_t>(c10::cuda::getCurrentCUDAStream().stream()); }

at::TensorOptions on(const at::Tensor& like, at::ScalarType type) { return at::TensorOptions().device(like.device()).dtype(type); }

PyObject* wrap(const at::Tensor& t) {
    if (!t.defined()) Py_RETURN_NONE;
    return THPVariable_Wrap(t);
}

template <typename... Ts>
PyObject* tuple(const Ts&... ts) {
    PyObject* out = PyTuple_New(sizeof...(Ts));
    if (!out) throw Raised();
    Py_ssize_t i = 0;
    (PyTuple_SET_ITEM(out, i++, wrap(ts)), ...);
    return out;
}

long num(PyObject* o) {
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw Raised();
    return v;
}
float real(PyObject* o) {
    const double v = PyFloat_AsDouble(o);
    if (v == -1.0 && PyErr_Occurred()) throw Raised();
    return (float)v;
}
bool truth(PyObject* o) { return PyObject_IsTrue(o) == 1; }

// ---- small outputs ------------------------------------------------------------------------------------------
// at::empty on the device of `like`, straight from the caching allocator where nothing watches the dispatcher: a routing
// result is seven tensors of a few hundred bytes, and a decode batch's call is about as long as its host path (64 tokens:
// 16.4 us of host in a call of 16.5 us, 17.9 and 18.0 with at::empty).
struct Fresh {
    at::TensorOptions options;
    c10::Allocator* allocator = nullptr;
    explicit Fresh(const at::Tensor& like) : options(at::TensorOptions().device(like.device())) {
        if (like.device().index() == c10::cuda::current_device() && !c10::impl::TorchDispatchModeTLS::any_modes_set())
            allocator = c10::cuda::CUDACachingAllocator::get();
    }
    at::Tensor operator()(at::ScalarType type, at::IntArrayRef sizes) const {
        if (!allocator) return at::empty(sizes, options.dtype(type));
        return at::Tensor(at::detail::empty_generic(sizes, allocator, c10::DispatchKeySet(c10::DispatchKey::CUDA), type, c10::nullopt));
    }
};

// ---- caches ----------------------------------------------------------------------------------------------
PyObject *s_k_codes, *s_v_codes, *s_k_scale, *s_v_scale, *s_k_zp, *s_v_zp, *s_page_table, *s_length, *s_status;

// a buffer of the module (borrowed): Tensor, or undefined when it is absent or None
const at::Tensor& buffer(PyObject* dict, PyObject* key) {
    static const at::Tensor none;
    PyObject* o = PyDict_GetItemWithError(dict, key);
    if (!o) {
        if (PyErr_Occurred()) throw Raised();
        return none;
    }
    if (o == Py_None) return none;
    if (!THPVariable_Check(o)) fail("cache buffer is not a tensor");
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda() || !t.is_contiguous()) fail("the cache's buffers must be contiguous CUDA tensors (there is no CPU path)");
    return t;
}

struct Cache {
    PyObject* buffers;
    int num_seqs, n_kv, bits, symmetric, max_pages, num_pages;
    static constexpr int ARGS = 7;
    explicit Cache(PyObject* const* a)
        : buffers(a[0]), num_seqs((int)num(a[1])), n_kv((int)num(a[2])), bits((int)num(a[3])), symmetric(truth(a[4]) ? 1 : 0),
          max_pages((int)num(a[5])), num_pages((int)num(a[6])) {
        if (!PyDict_Check(buffers)) fail("a cache is passed as its buffer dict");
    }
    void* at(PyObject* key) const { return ptr(buffer(buffers, key)); }
    void fill(pikv_append_params& p) const {
        p.page_table = static_cast<const int32_t*>(at(s_page_table));
        p.num_seqs = num_seqs; p.max_pages = max_pages; p.num_pages = num_pages;
        p.bits = bits; p.symmetric = symmetric; p.n_kv = n_kv;
        p.k_codes = at(s_k_codes); p.v_codes = at(s_v_codes);
        p.k_scale = at(s_k_scale); p.v_scale = at(s_v_scale);
        p.k_zp = at(s_k_zp); p.v_zp = at(s_v_zp);
        p.status = static_cast<uint32_t*>(at(s_status));
    }
};

void kv_rows(const Cache& c, const at::Tensor& k, const at::Tensor& v, const char* what) {
    if (k.dim() != 2 || k.size(1) != (int64_t)c.n_kv * PIKV_HEAD_DIM || v.sizes() != k.sizes())
        fail("%s: k and v must both be [T, %d]", what, c.n_kv * PIKV_HEAD_DIM);
}

// append(cache..., k, v, dst_seq, slot)  /  append_rope(cache..., k, v, dst_seq, slot, cos, sin, positions)
PyObject* append(PyObject* const* a, Py_ssize_t n) {
    const Cache c(a);
    a += Cache::ARGS;
    const bool rope = n == Cache::ARGS + 7;
    if (rope && (c.bits != 8 || !c.symmetric)) fail("append_rope writes int8 symmetric caches");
    const at::Tensor k = req(a[0], "k", rope ? OptType(at::kBFloat16) : c10::nullopt), v = req(a[1], "v", k.scalar_type());
    kv_rows(c, k, v, "append");
    const at::Tensor dst = req(a[2], "dst_seq", at::kInt), slot = req(a[3], "slot", at::kInt);
    pikv_append_params p = {};
    c.fill(p);
    p.k = ptr(k); p.v = ptr(v); p.dtype = dtype_code(k, "k"); p.T = (int32_t)k.size(0);
    p.top_k = dst.dim() == 1 ? 1 : (int32_t)dst.size(1);
    if (dst.size(0) < k.size(0) || slot.numel() < k.size(0) * p.top_k) fail("append: dst_seq and slot must have a row per token");
    p.dst_seq = ptr<int32_t>(dst); p.slot = ptr<int32_t>(slot);
    if (!rope) {
        check(pikv_kv_append_quant(&p, stream()), "pikv_kv_append_quant");
        Py_RETURN_NONE;
    }
    const at::Tensor cos = req(a[4], "cos", at::kFloat), sin = req(a[5], "sin", at::kFloat), pos = opt(a[6], "positions", at::kInt);
    if (cos.dim() != 2 || cos.size(1) != PIKV_HEAD_DIM / 2 || sin.sizes() != cos.sizes()) fail("cos / sin must be [max_pos, %d]", PIKV_HEAD_DIM / 2);
    if (pos.defined() && pos.numel() < k.size(0)) fail("append_rope: positions must have one entry per token");
    check(pikv_kv_append_rope(&p, ptr<float>(cos), ptr<float>(sin), ptr<int32_t>(pos), (int32_t)cos.size(0), stream()), "pikv_kv_append_rope");
    Py_RETURN_NONE;
}

// ---- gates -------------------------------------------------------------------------------------------------
// The tensors of a gate result, in the order of ops.GateResult.
struct GateOut {
    at::Tensor probs, idx, w, slot, counts, psum, len, workspace;
    // from a tuple of a caller's result, or new
    GateOut(PyObject* given, const at::Tensor& like, int T, int E, int k, bool want_probs) {
        if (given != Py_None) {
            if (!PyTuple_Check(given) || PyTuple_GET_SIZE(given) != 8) fail("gate: a result has eight tensors");
            at::Tensor* to[8] = {&probs, &idx, &w, &slot, &counts, &psum, &len, &workspace};
            static const char* names[8] = {"probs", "topk_idx", "topk_w", "slot", "counts_k", "prob_sum", "new_len", "workspace"};
            const bool whole[8] = {false, true, false, true, true, false, true, false};
            const int64_t size[8] = {(int64_t)T * E, (int64_t)T * k, (int64_t)T * k, (int64_t)T * k, (int64_t)k * E, E, E, 0};
            for (int i = 0; i < 8; ++i) {
                PyObject* o = PyTuple_GET_ITEM(given, i);
                if (o == Py_None) continue;
                // raw pointers of them go to the kernels as outputs
                if (!THPVariable_Check(o)) fail("the result's %s must be a CUDA tensor", names[i]);
                const at::Tensor& t = THPVariable_Unpack(o);
                if (!t.is_cuda() || !t.is_contiguous() || (i < 7 && t.scalar_type() != (whole[i] ? at::kInt : at::kFloat)))
                    fail("the result's %s must be a contiguous CUDA tensor%s", names[i], i == 7 ? "" : whole[i] ? " of int32" : " of float32");
                *to[i] = holds(t, size[i], names[i]);
            }
            return;
        }
        // a storage each: a caller may keep, save or resize one without the others
        const Fresh fresh(like);
        if (want_probs) probs = fresh(at::kFloat, {T, E});
        idx = fresh(at::kInt, {T, k});
        w = fresh(at::kFloat, {T, k});
        slot = fresh(at::kInt, {T, k});
        counts = fresh(at::kInt, {k, E});
        psum = fresh(at::kFloat, {E});
        len = fresh(at::kInt, {E});
    }
    void fill(pikv_gate_params& g) const {
        g.probs = ptr<float>(probs); g.topk_idx = ptr<int32_t>(idx); g.topk_w = ptr<float>(w); g.slot = ptr<int32_t>(slot);
        g.counts_k = ptr<int32_t>(counts); g.prob_sum = ptr<float>(psum); g.new_len = ptr<int32_t>(len);
    }
    PyObject* result() const { return tuple(probs, idx, w, slot, counts, psum, len, workspace); }
};

// what the tail of every gate takes: top_k, expert_mask, mask_mode, correction, temperature, renorm_eps, capacity,
// slot_base, want_probs
struct GateTail {
    int k, mode, capacity;
    at::Tensor mask, corr, base;
    float temperature, eps;
    bool want_probs;
    static constexpr int ARGS = 9;
    explicit GateTail(PyObject* const* a)
        : k((int)num(a[0])), mode((int)num(a[2])), capacity((int)num(a[6])), mask(f32(a[1], "gate vector")), corr(f32(a[3], "gate vector")),
          base(opt(a[7], "slot_base", at::kInt)), temperature(real(a[4])), eps(real(a[5])), want_probs(truth(a[8])) {}
    void fill(pikv_gate_params& g) const {
        holds(mask, g.E, "expert_mask"); holds(corr, g.E, "correction"); holds(base, g.E, "slot_base");
        g.top_k = k;
        g.expert_mask = ptr<float>(mask);
        g.mask_mode = mask.defined() ? mode : PIKV_MASK_NONE;
        g.correction = ptr<float>(corr);
        g.temperature = temperature; g.renorm_eps = eps; g.capacity = capacity;
        g.slot_base = ptr<int32_t>(base);
    }
};

at::Tensor workspace(const at::Tensor& like, size_t bytes) { return at::empty({(int64_t)std::max<size_t>(bytes, 1)}, on(like, at::kByte)); }

// gate(act, w2, b2, logits, tail..., out, phase)
PyObject* gate(PyObject* const* a, Py_ssize_t) {
    pikv_gate_params g = {};
    at::Tensor act, w2, b2, logits;
    if (a[3] != Py_None) {
        logits = req(a[3], "logits", at::kFloat);
        if (logits.dim() != 2) fail("logits must be [T,E]");
        g.T = (int32_t)logits.size(0); g.E = (int32_t)logits.size(1);
        g.dtype = PIKV_F32;
        g.logits_in = ptr<float>(logits);
    } else {
        act = req(a[0], "act");
        w2 = req(a[1], "w2", act.scalar_type());
        b2 = f32(a[2], "gate vector");
        if (act.dim() != 2 || w2.dim() != 2 || w2.size(1) != act.size(1)) fail("act must be [T,H] and w2 [E,H] with the same H");
        g.T = (int32_t)act.size(0); g.H = (int32_t)act.size(1); g.E = (int32_t)w2.size(0);
        g.dtype = dtype_code(act, "act");
        g.act = ptr(act); g.w2 = ptr(w2); g.b2 = ptr<float>(holds(b2, g.E, "b2"));
    }
    const at::Tensor& like = logits.defined() ? logits : act;
    const GateTail tail(a + 4);
    PyObject *given = a[4 + GateTail::ARGS], *phase = a[5 + GateTail::ARGS];
    g.phase = (int32_t)num(phase);
    tail.fill(g);
    GateOut out(given, like, g.T, g.E, g.top_k, tail.want_probs);
    out.fill(g);
    const size_t need = pikv_gate_tail_workspace_bytes(g.T, g.E, g.top_k);
    at::Tensor ws = out.workspace;
    if (!ws.defined() || (size_t)ws.numel() < need) {
        if (g.phase == PIKV_GATE_SLOTS) fail("gate phase 2 needs the result (and workspace) of the phase 1 call");
        ws = workspace(like, need);
        if (g.phase != PIKV_GATE_WHOLE || out.workspace.defined()) out.workspace = ws;
    }
    g.workspace = ptr(ws); g.workspace_bytes = (size_t)ws.numel();
    check(pikv_gate_fused(&g, stream()), "pikv_gate_fused");
    return out.result();
}

// route_append(cache..., act, w2, b2, k, v, tail..., out)
PyObject* route_append(PyObject* const* a, Py_ssize_t) {
    const Cache c(a);
    a += Cache::ARGS;
    const at::Tensor act = req(a[0], "act"), w2 = req(a[1], "w2", act.scalar_type()), b2 = f32(a[2], "b2");
    const at::Tensor k = req(a[3], "k"), v = req(a[4], "v", k.scalar_type());
    if (act.dim() != 2 || w2.dim() != 2 || w2.size(1) != act.size(1)) fail("act must be [T,H] and w2 [E,H] with the same H");
    if (w2.size(0) != c.num_seqs) fail("the cache has %d sequences, the gate %d experts", c.num_seqs, (int)w2.size(0));
    kv_rows(c, k, v, "route_append");
    if (k.size(0) < act.size(0)) fail("route_append: %d tokens in act, %d in k", (int)act.size(0), (int)k.size(0));
    const GateTail tail(a + 5);
    pikv_gate_params g = {};
    g.act = ptr(act); g.w2 = ptr(w2); g.b2 = ptr<float>(holds(b2, c.num_seqs, "b2")); g.dtype = dtype_code(act, "act");
    g.T = (int32_t)act.size(0); g.H = (int32_t)act.size(1); g.E = c.num_seqs;
    tail.fill(g);
    GateOut out(a[5 + GateTail::ARGS], act, g.T, g.E, g.top_k, tail.want_probs);
    out.fill(g);
    const size_t need = pikv_gate_tail_workspace_bytes(g.T, g.E, g.top_k);
    // owned by the result, so calls on different streams never share gate scratch
    if (!out.workspace.defined() || (size_t)out.workspace.numel() < need) out.workspace = workspace(act, need);
    g.workspace = ptr(out.workspace); g.workspace_bytes = (size_t)out.workspace.numel();
    pikv_append_params p = {};
    c.fill(p);
    p.k = ptr(k); p.v = ptr(v); p.dtype = dtype_code(k, "k"); p.T = g.T; p.top_k = g.top_k;
    check(pikv_route_append(&g, &p, stream()), "pikv_route_append");
    return out.result();
}

// (dispatch, combine, aux) of rows capacity rows, and the descriptor the kernels take; arguments rows, position_mode,
// balance, coefficient
struct Dense {
    at::Tensor d, c, aux;
    pikv_dense_out o = {};
    Dense(PyObject* const* a, const at::Tensor& like, at::IntArrayRef tokens, int64_t E) {
        const int64_t rows = num(a[0]);
        std::vector<int64_t> shape(tokens.begin(), tokens.end());
        shape.push_back(E);
        shape.push_back(rows);
        d = at::empty(shape, on(like, at::kFloat));
        c = at::empty(shape, on(like, at::kFloat));
        aux = at::empty({}, on(like, at::kFloat));
        o.dispatch = ptr<float>(d); o.combine = ptr<float>(c); o.aux = ptr<float>(aux);
        o.capacity = (int32_t)rows; o.position_mode = (int32_t)num(a[1]); o.balance = (int32_t)num(a[2]); o.coefficient = real(a[3]);
    }
};

// gate_mlp(x, w1, b1, w2, b2, tail..., out, rows, position_mode, balance, coefficient); rows 0: no dense outputs.
// Returns the result, with (dispatch [..., E, rows], combine, aux) behind it when they were asked for.
PyObject* gate_mlp(PyObject* const* a, Py_ssize_t) {
    const at::Tensor x = req(a[0], "x", at::kBFloat16), w1 = req(a[1], "w1", at::kBFloat16), w2 = req(a[3], "w2", at::kBFloat16);
    at::Tensor b1 = opt(a[2], "bias"), b2 = opt(a[4], "bias");
    if (x.dim() < 2 || w1.dim() != 2 || w2.dim() != 2 || w1.size(1) != x.size(-1) || w2.size(1) != w1.size(0))
        fail("gate net: x [T,K], w1 [H,K] and w2 [E,H] do not fit");
    const bool half = (!b1.defined() || b1.scalar_type() == at::kBFloat16) && (!b2.defined() || b2.scalar_type() == at::kBFloat16);
    if (!half) {
        if (b1.defined()) b1 = b1.to(at::kFloat);
        if (b2.defined()) b2 = b2.to(at::kFloat);
    }
    const GateTail tail(a + 5);
    PyObject* given = a[5 + GateTail::ARGS];
    PyObject* const* da = a + 6 + GateTail::ARGS;
    pikv_gate_params g = {};
    g.T = rows_of(x, "x"); g.H = (int32_t)w1.size(0); g.E = (int32_t)w2.size(0);
    g.dtype = PIKV_BF16; g.w2 = ptr(w2);
    holds(b1, g.H, "b1"); holds(b2, g.E, "b2");
    tail.fill(g);
    GateOut out(given, x, g.T, g.E, g.top_k, tail.want_probs);
    out.fill(g);
    const size_t need = pikv_gate_workspace_bytes(g.T, g.E, g.top_k);
    at::Tensor ws = out.workspace;
    if (!ws.defined() || (size_t)ws.numel() < need) ws = workspace(x, need);
    g.workspace = ptr(ws); g.workspace_bytes = (size_t)ws.numel();
    const int bias = half ? PIKV_BF16 : PIKV_F32;
    const long rows = num(da[0]);
    if (!rows) {
        check(pikv_gate_mlp_dense(&g, ptr(x), (int32_t)x.size(-1), ptr(w1), ptr(b1), ptr(b2), bias, nullptr, stream()), "pikv_gate_mlp_dense");
        return out.result();
    }
    Dense dense(da, x, x.sizes().slice(0, x.dim() - 1), g.E);
    // the kernels clear whole 16-byte words
    const bool inside = (int64_t)g.T * g.E * rows % 4 == 0;
    check(pikv_gate_mlp_dense(&g, ptr(x), (int32_t)x.size(-1), ptr(w1), ptr(b1), ptr(b2), bias, inside ? &dense.o : nullptr, stream()),
          "pikv_gate_mlp_dense");
    if (!inside)
        check(pikv_dispatch_loss(g.topk_idx, g.topk_w, g.slot, g.counts_k, g.prob_sum, g.T, g.E, g.top_k, &dense.o, stream()), "pikv_dispatch_loss");
    return tuple(out.probs, out.idx, out.w, out.slot, out.counts, out.psum, out.len, out.workspace, dense.d, dense.c, dense.aux);
}

// dispatch_loss(topk_idx, topk_w, slot, counts_k, prob_sum, E, rows, position_mode, balance, coefficient); no loss without prob_sum
PyObject* dispatch_loss(PyObject* const* a, Py_ssize_t) {
    const at::Tensor idx = req(a[0], "topk_idx", at::kInt), w = req(a[1], "topk_w", at::kFloat), slot = opt(a[2], "slot", at::kInt),
                     counts = opt(a[3], "counts_k", at::kInt), psum = opt(a[4], "prob_sum", at::kFloat);
    if (idx.dim() != 2) fail("topk_idx must be [T,k]");
    const int T = (int)idx.size(0), k = (int)idx.size(1), E = (int)num(a[5]);
    holds(w, idx.numel(), "topk_w"); holds(slot, idx.numel(), "slot"); holds(counts, (int64_t)k * E, "counts_k"); holds(psum, E, "prob_sum");
    Dense dense(a + 6, idx, {T}, E);
    if (!psum.defined()) dense.o.aux = nullptr, dense.aux = at::Tensor();
    check(pikv_dispatch_loss(ptr<int32_t>(idx), ptr<float>(w), ptr<int32_t>(slot), ptr<int32_t>(counts), ptr<float>(psum), T, E, k, &dense.o, stream()),
          "pikv_dispatch_loss");
    return tuple(dense.d, dense.c, dense.aux);
}

// ---- decode attention --------------------------------------------------------------------------------------
at::Tensor lengths(const Cache& c, const at::Tensor& ids, PyObject* given) {
    if (given != Py_None) return req(given, "seq_len", at::kInt);
    const at::Tensor& len = buffer(c.buffers, s_length);
    if (!ids.defined()) return len;
    if (!len.defined() || len.scalar_type() != at::kInt || len.numel() < c.num_seqs) fail("the cache's length must be one int32 per sequence");
    // ids outside the cache are for the kernels to report: their length is 0
    at::Tensor out = at::empty({ids.numel()}, on(ids, at::kInt));
    if (ids.numel())
        check(pikv_seq_lengths(ptr<int32_t>(len), ptr<int32_t>(ids), (int32_t)ids.numel(), c.num_seqs, ptr<int32_t>(out), stream()), "pikv_seq_lengths");
    return out;
}

// decode(cache..., q, seq_ids, seq_len, want_lse, scores)  /  decode_h2o(cache..., q, seq_ids, seq_len, acc, probs, step_max)
PyObject* decode(PyObject* const* a, Py_ssize_t n) {
    const Cache c(a);
    a += Cache::ARGS;
    const bool h2o = n == Cache::ARGS + 6;
    const bool q8 = c.bits == 8 && c.symmetric;
    if (h2o && !q8) fail("decode_attention_h2o reads int8 symmetric caches");
    if (!q8 && !(c.bits == 4 && !c.symmetric)) fail("decode_attention reads int8 symmetric and 4-bit asymmetric caches");
    const at::Tensor q = req(a[0], "q", at::kBFloat16);
    if (q.dim() != 3 || q.size(2) != PIKV_HEAD_DIM) fail("q must be [B, n_q, %d]", PIKV_HEAD_DIM);
    const at::Tensor ids = opt(a[1], "seq_ids", at::kInt), len = lengths(c, ids, a[2]);
    pikv_decode_params p = {};
    p.B = (int32_t)q.size(0); p.n_q = (int32_t)q.size(1); p.n_kv = c.n_kv;
    if (len.numel() < p.B || (ids.defined() && ids.numel() < p.B)) fail("decode: seq_len and seq_ids must have one entry per query");
    at::Tensor acc, probs, step, scores;
    bool want_lse = true;
    if (h2o) {
        if (a[3] == Py_None) fail("acc must be a CUDA tensor");
        acc = written(a[3], "acc", at::kFloat);
        probs = req(a[4], "probs", at::kHalf);
        step = req(a[5], "step_max", at::kFloat);
        p.probs16 = ptr(probs); p.step_max = ptr<float>(step);
        p.probs_stride = (int32_t)probs.size(-1); p.step_stride = (int32_t)step.size(-1);
        holds(acc, (int64_t)p.B * p.n_kv * acc.size(-1), "acc");
        holds(probs, (int64_t)p.B * p.n_q * probs.size(-1), "the workspace's probabilities");
        holds(step, (int64_t)p.B * p.n_q * step.size(-1), "the workspace's step maxima");
    } else {
        scores = written(a[4], "scores", at::kFloat);
        want_lse = truth(a[3]) || scores.defined();
        p.scores = ptr<float>(scores);
        p.score_stride = scores.defined() ? (int32_t)scores.size(-1) : 0;
        holds(scores, (int64_t)p.B * p.n_q * p.score_stride, "scores");
    }
    // scratch sized for this call's batch
    const size_t scratch = pikv_decode_attn_workspace_bytes(p.B, p.n_q, p.n_kv, 0, 0);
    at::Tensor out = at::empty_like(q), lse, ws = workspace(q, scratch);
    if (want_lse) lse = at::empty({p.B, p.n_q}, on(q, at::kFloat));
    p.q = ptr(q); p.out = ptr(out); p.lse = ptr<float>(lse);
    p.seq_ids = ptr<int32_t>(ids); p.seq_len = ptr<int32_t>(len);
    p.page_table = static_cast<const int32_t*>(c.at(s_page_table));
    p.num_seqs = c.num_seqs; p.max_pages = c.max_pages; p.num_pages = c.num_pages;
    p.k_codes = c.at(s_k_codes); p.v_codes = c.at(s_v_codes); p.k_scale = c.at(s_k_scale); p.v_scale = c.at(s_v_scale);
    p.workspace = ptr(ws); p.workspace_bytes = scratch;
    p.status = static_cast<uint32_t*>(c.at(s_status));
    if (q8) {
        check(pikv_decode_attn_q8(&p, stream()), "pikv_decode_attn_q8");
    } else {
        p.k_zp = c.at(s_k_zp); p.v_zp = c.at(s_v_zp);
        check(pikv_decode_attn_q4(&p, stream()), "pikv_decode_attn_q4");
    }
    if (h2o) {
        check(pikv_h2o_accumulate_probs(p.probs16, p.probs_stride, p.step_max, p.step_stride, p.lse, p.seq_len, p.B, p.n_q, p.n_kv,
                                        ptr<float>(acc), (int32_t)acc.size(-1), stream()), "pikv_h2o_accumulate_probs");
        return wrap(out);
    }
    return want_lse ? tuple(out, lse) : wrap(out);
}

// ---- eviction ----------------------------------------------------------------------------------------------
// select(acc, ts, heavy, recent, seg_len, n, want_idx, as_bool); n < 0: whole rows
PyObject* select(PyObject* const* a, Py_ssize_t) {
    at::Tensor acc = req(a[0], "acc", at::kFloat), ts = req(a[1], "ts", at::kFloat);
    if (acc.dim() == 1) acc = acc.unsqueeze(0), ts = ts.unsqueeze(0);
    if (acc.dim() != 2 || ts.numel() != acc.numel()) fail("h2o_select: acc and ts must be [segments, stride]");
    const int S = (int)acc.size(0), stride = (int)acc.size(1), heavy = (int)num(a[2]), recent = (int)num(a[3]);
    const at::Tensor len = opt(a[4], "seg_len", at::kInt);
    if (len.defined() && len.numel() < S) fail("h2o_select: seg_len must have one entry per segment");
    const long n = num(a[5]);
    const int64_t ks = std::max<int64_t>(1, std::min<int64_t>(stride, (int64_t)heavy + recent));
    // the kernel writes 0 and 1, which are bool's bytes
    at::Tensor mask = at::empty({S, stride}, on(acc, truth(a[7]) ? at::kBool : at::kByte)), keep, count = at::empty({S}, on(acc, at::kInt));
    if (truth(a[6])) keep = at::empty({S, ks}, on(acc, at::kInt));
    check(pikv_h2o_select(ptr<float>(acc), ptr<float>(ts), S, stride, ptr<int32_t>(len), n < 0 ? stride : (int32_t)n, heavy, recent,
                          static_cast<uint8_t*>(mask.data_ptr()), ptr<int32_t>(keep), (int32_t)ks, ptr<int32_t>(count), stream()), "pikv_h2o_select");
    return tuple(mask, keep, count);
}

// compact(src cache..., dst cache..., keep_idx, kept_count, per_head, src_acc, src_ts, dst_acc, dst_ts)
PyObject* compact(PyObject* const* a, Py_ssize_t) {
    const Cache s(a), d(a + Cache::ARGS);
    a += 2 * Cache::ARGS;
    const at::Tensor keep = req(a[0], "keep_idx", at::kInt), count = req(a[1], "kept_count", at::kInt);
    if (keep.dim() != 2) fail("compact_into: keep_idx must be [segments, keep]");
    if (s.max_pages != d.max_pages) fail("compact_into: source and destination must share the page-table width");
    pikv_compact_params p = {};
    p.keep_idx = ptr<int32_t>(keep); p.kept_count = ptr<int32_t>(count); p.keep_stride = (int32_t)keep.size(1);
    p.num_seqs = s.num_seqs; p.n_kv = s.n_kv; p.per_head = truth(a[2]) ? 1 : 0; p.bits = s.bits;
    p.src_page_table = static_cast<const int32_t*>(s.at(s_page_table));
    p.dst_page_table = static_cast<const int32_t*>(d.at(s_page_table));
    p.max_pages = s.max_pages; p.num_pages = std::min(s.num_pages, d.num_pages);
    p.src_k_codes = s.at(s_k_codes); p.src_v_codes = s.at(s_v_codes); p.src_k_scale = s.at(s_k_scale); p.src_v_scale = s.at(s_v_scale);
    p.src_k_zp = s.at(s_k_zp); p.src_v_zp = s.at(s_v_zp);
    p.dst_k_codes = d.at(s_k_codes); p.dst_v_codes = d.at(s_v_codes); p.dst_k_scale = d.at(s_k_scale); p.dst_v_scale = d.at(s_v_scale);
    p.dst_k_zp = d.at(s_k_zp); p.dst_v_zp = d.at(s_v_zp);
    const int64_t segments = (int64_t)s.num_seqs * (p.per_head ? s.n_kv : 1);
    holds(keep, segments * keep.size(1), "keep_idx"); holds(count, segments, "kept_count");
    static const char* names[2] = {"acc", "ts"};
    at::Tensor from[2], to[2];
    for (int i = 0; i < 2; ++i) {
        if ((a[3 + i] == Py_None) != (a[5 + i] == Py_None)) fail("compact_into: give src_%s and dst_%s together", names[i], names[i]);
        from[i] = opt(a[3 + i], "src scores", at::kFloat);
        to[i] = written(a[5 + i], i ? "dst_ts" : "dst_acc", at::kFloat);
        if (!from[i].defined()) continue;
        if (from[i].numel() != segments * from[i].size(-1) || to[i].numel() != segments * to[i].size(-1))
            fail("compact_into: src_%s / dst_%s must have one row per segment (%lld)", names[i], names[i], (long long)segments);
        if (to[i].size(-1) < keep.size(1)) fail("compact_into: dst_%s rows are shorter than keep_idx rows", names[i]);
        p.score_stride = (int32_t)from[i].size(-1);
        p.dst_score_stride = (int32_t)to[i].size(-1);
    }
    if (from[0].defined() && from[1].defined() && (from[0].size(-1) != from[1].size(-1) || to[0].size(-1) != to[1].size(-1)))
        fail("compact_into: scores and timestamps must share their row lengths");
    p.src_acc = ptr<float>(from[0]); p.src_ts = ptr<float>(from[1]); p.dst_acc = ptr<float>(to[0]); p.dst_ts = ptr<float>(to[1]);
    p.status = static_cast<uint32_t*>(s.at(s_status));
    check(pikv_h2o_compact(&p, stream()), "pikv_h2o_compact");
    Py_RETURN_NONE;
}

// ---- compressors -------------------------------------------------------------------------------------------
// quant_pair(k, v, group_size, qmin, qmax, symmetric, params_in, sample_count, count_add) -> (dk, dv, mse), shapes as given
PyObject* quant_pair(PyObject* const* a, Py_ssize_t) {
    const at::Tensor k = req(a[0], "keys"), v = req(a[1], "values", k.scalar_type());
    if (k.dim() < 1 || v.sizes() != k.sizes()) fail("keys and values must have the same shape");
    const int N = rows_of(k, "keys"), H = (int)k.size(-1), gs = (int)num(a[2]);
    const at::Tensor params = opt(a[6], "params_in", at::kFloat);
    if (gs > 0) holds(params, 2 * (((int64_t)H + gs - 1) / gs), "params_in");
    const at::Tensor counter = opt(a[7], "sample_count", at::kFloat);
    const size_t bytes = pikv_quant_block_pair_workspace_bytes(N, H, gs);
    at::Tensor dk = at::empty_like(k), dv = at::empty_like(v), mse = at::empty({}, on(k, at::kFloat)), ws = workspace(k, bytes);
    check(pikv_quant_block_pair(ptr(k), ptr(v), dtype_code(k, "keys"), N, H, gs, (int32_t)num(a[3]), (int32_t)num(a[4]), truth(a[5]) ? 1 : 0,
                                ptr<float>(params), ptr(dk), ptr(dv), ptr<float>(mse), ptr<float>(counter), real(a[8]), ptr(ws), bytes, stream()),
          "pikv_quant_block_pair");
    return tuple(dk, dv, mse);
}

at::Tensor bias_of(PyObject* o) {
    const at::Tensor b = opt(o, "bias");
    return !b.defined() || b.scalar_type() == at::kFloat || b.scalar_type() == at::kBFloat16 ? b : b.to(at::kFloat);
}
at::Tensor half_of(PyObject* o, const char* name) {
    const at::Tensor w = req(o, name);
    return w.scalar_type() == at::kBFloat16 ? w : w.to(at::kBFloat16);
}
std::vector<int64_t> with_last(const at::Tensor& x, int64_t last) {
    std::vector<int64_t> s(x.sizes().begin(), x.sizes().end());
    s.back() = last;
    return s;
}

// lowrank(x, w, bias, relu, residual, out_f32) -> [..., N]
PyObject* lowrank(PyObject* const* a, Py_ssize_t) {
    const at::Tensor x = req(a[0], "x", at::kBFloat16), w = half_of(a[1], "w"), b = bias_of(a[2]), r = opt(a[4], "residual", at::kBFloat16);
    const int M = rows_of(x, "x");
    if (w.dim() != 2 || w.size(1) != x.size(-1)) fail("w must be [N,%lld]", (long long)x.size(-1));
    const int K = (int)x.size(-1), N = (int)w.size(0);
    const bool f = truth(a[5]);
    holds(b, N, "bias"); holds(r, (int64_t)M * N, "residual");
    at::Tensor y = at::empty(with_last(x, N), on(x, f ? at::kFloat : at::kBFloat16));
    check(pikv_lowrank_project_bias(ptr(x), ptr(w), ptr(b), b.defined() ? dtype_code(b, "bias") : PIKV_F32, ptr(r), ptr(y), f ? PIKV_F32 : PIKV_BF16,
                                    M, N, K, truth(a[3]) ? 1 : 0, stream()), "pikv_lowrank_project_bias");
    return wrap(y);
}

// lowrank_pair(x, x', w1, w1', b1, b1', w2, w2', b2, b2') -> (y, y')
PyObject* lowrank_pair(PyObject* const* a, Py_ssize_t) {
    at::Tensor x[2], w1[2], b1[2], w2[2], b2[2], y[2];
    const void *xp[2], *w1p[2], *b1p[2], *w2p[2], *b2p[2];
    void* yp[2];
    bool half = true;                          // the kernel takes one bias type: fp32 unless all are bf16 (exact either way)
    for (int i = 0; i < 2; ++i) {
        x[i] = req(a[i], "x", at::kBFloat16);
        w1[i] = half_of(a[2 + i], "w1"); b1[i] = bias_of(a[4 + i]);
        w2[i] = half_of(a[6 + i], "w2"); b2[i] = bias_of(a[8 + i]);
        if (x[i].sizes() != x[0].sizes() || w1[i].dim() != 2 || w2[i].dim() != 2 || w1[i].sizes() != w1[0].sizes() || w2[i].sizes() != w2[0].sizes() ||
            x[i].dim() < 1 || w1[i].size(1) != x[i].size(-1) || w2[i].size(1) != w1[i].size(0))
            fail("lowrank_pair: x, w1 and w2 do not fit");
        holds(b1[i], w1[i].size(0), "bias"); holds(b2[i], w2[i].size(0), "bias");
        for (const at::Tensor* b : {&b1[i], &b2[i]}) half = half && (!b->defined() || b->scalar_type() == at::kBFloat16);
    }
    for (int i = 0; i < 2; ++i) {
        if (!half) {
            if (b1[i].defined()) b1[i] = b1[i].to(at::kFloat);
            if (b2[i].defined()) b2[i] = b2[i].to(at::kFloat);
        }
        y[i] = at::empty(with_last(x[i], w2[i].size(0)), on(x[i], at::kBFloat16));
        xp[i] = ptr(x[i]); w1p[i] = ptr(w1[i]); b1p[i] = ptr(b1[i]); w2p[i] = ptr(w2[i]); b2p[i] = ptr(b2[i]); yp[i] = ptr(y[i]);
    }
    const int M = rows_of(x[0], "x"), K = (int)x[0].size(-1);
    check(pikv_lowrank_pair(xp, w1p, b1p, w2p, b2p, half ? PIKV_BF16 : PIKV_F32, yp, M, K, (int32_t)w1[0].size(0), (int32_t)w2[0].size(0), stream()),
          "pikv_lowrank_pair");
    return tuple(y[0], y[1]);
}

// linear_f32(x, w, bias) -> [..., N]
at::Tensor linear_f32(const at::Tensor& x, const at::Tensor& w, const float* bias) {
    const int M = rows_of(x, "x"), K = (int)x.size(-1), N = (int)w.size(0);
    at::Tensor y = at::empty(with_last(x, N), on(x, at::kFloat));
    const size_t bytes = pikv_linear_f32_workspace_bytes(M, N, K);
    const at::Tensor ws = workspace(x, bytes);
    check(pikv_linear_f32(ptr<float>(x), ptr<float>(w), bias, ptr<float>(y), M, N, K, ptr(ws), bytes, stream()), "pikv_linear_f32");
    return y;
}
PyObject* linear(PyObject* const* a, Py_ssize_t) {
    const at::Tensor x = req(a[0], "x", at::kFloat), w = req(a[1], "w", at::kFloat), b = opt(a[2], "bias", at::kFloat);
    if (x.dim() < 1 || w.dim() != 2 || w.size(1) != x.size(-1) || (b.defined() && b.numel() != w.size(0))) fail("linear_f32: x, w and bias do not fit");
    return wrap(linear_f32(x, w, ptr<float>(b)));
}

// ---- PiKVMoE -----------------------------------------------------------------------------------------------
// The forward's kernels take raw weights, so every module they stand for has to be what it was built as: walked on each
// call, about 70 modules in a few microseconds.  Whatever does not fit leaves as NotApplicable and the caller runs the modules.
struct NotApplicable : std::exception {};

PyObject* interned(const char* s) {
    PyObject* o = PyUnicode_InternFromString(s);
    if (!o) throw Raised();
    return o;
}
#define PIKV_NAME(text) ([]() { static PyObject* const name = interned(text); return name; }())

void need(bool ok) {
    if (!ok) throw NotApplicable();
}

struct Mod {
    PyObject* dict;                            // borrowed: the module owns it and is held by its parent
    // a module of exactly that class, without hooks and without a forward of its own
    Mod(PyObject* m, PyObject* types, int type) {
        need(m && (PyObject*)Py_TYPE(m) == PyTuple_GET_ITEM(types, type));
        dict = PyObject_GenericGetDict(m, nullptr);
        if (!dict) throw Raised();
        Py_DECREF(dict);
        need(empty(PIKV_NAME("_forward_hooks")) && empty(PIKV_NAME("_forward_pre_hooks")) && !PyDict_GetItem(dict, PIKV_NAME("forward")));
    }
    PyObject* get(PyObject* key) const {
        PyObject* o = PyDict_GetItem(dict, key);
        need(o);
        return o;
    }
    bool empty(PyObject* key) const {
        PyObject* o = PyDict_GetItem(dict, key);
        return o && PyDict_Check(o) && PyDict_GET_SIZE(o) == 0;
    }
    PyObject* in(PyObject* table, PyObject* key) const {
        PyObject* t = get(table);
        need(PyDict_Check(t));
        PyObject* o = PyDict_GetItem(t, key);
        need(o);
        return o;
    }
    PyObject* child(PyObject* key) const { return in(PIKV_NAME("_modules"), key); }
    long integer(PyObject* key) const {
        PyObject* o = get(key);
        need(PyLong_CheckExact(o));
        return num(o);
    }
    float number(PyObject* key) const {
        PyObject* o = get(key);
        need(PyFloat_Check(o) || PyLong_CheckExact(o));
        return real(o);
    }
    bool is_false(PyObject* key) const { return get(key) == Py_False; }
};

struct MoeWalk {
    PyObject* types;
    c10::Device device;
    enum { MOE, MODULES, EXPERT, LORA, LINEAR, DROPOUT, CACHE, COMPRESSOR, PYRAMID, ADAPTIVE, BALANCED, IMPORTANCE, SEQUENTIAL, RELU, SIGMOID, SOFTMAX,
           NTYPES };

    const at::Tensor& tensor(PyObject* o, at::IntArrayRef sizes, at::ScalarType type = at::kFloat) const {
        need(THPVariable_CheckExact(o));               // a subclass may have calls of its own
        const at::Tensor& t = THPVariable_Unpack(o);
        need(t.layout() == at::kStrided && t.device() == device && t.scalar_type() == type && t.sizes() == sizes && t.is_contiguous() &&
             (!t.is_inference() || c10::InferenceMode::is_enabled()) && !t.unsafeGetTensorImpl()->is_python_dispatch() &&
             reinterpret_cast<uintptr_t>(t.const_data_ptr()) % (type == at::kFloat ? 16 : 8) == 0);
        return t;
    }
    const float* param(const Mod& m, PyObject* key, at::IntArrayRef sizes) const {
        return static_cast<const float*>(tensor(m.in(PIKV_NAME("_parameters"), key), sizes).const_data_ptr());
    }
    const at::Tensor& buf(const Mod& m, PyObject* key, at::IntArrayRef sizes, at::ScalarType type = at::kFloat) const {
        return tensor(m.in(PIKV_NAME("_buffers"), key), sizes, type);
    }
    static PyObject* digit(int64_t i) {
        static PyObject* names[PIKV_MOE_MAX_EXPERTS] = {};
        need(i < PIKV_MOE_MAX_EXPERTS);
        if (!names[i]) names[i] = interned(std::to_string(i).c_str());
        return names[i];
    }
    Mod list(PyObject* m, int type, int64_t count) const {
        const Mod l(m, types, type);
        PyObject* c = l.get(PIKV_NAME("_modules"));
        need(PyDict_Check(c) && (count < 0 || PyDict_GET_SIZE(c) == count));
        return l;
    }
    void linear(PyObject* m, int64_t out, int64_t in, const float*& w, const float*& b) const {
        const Mod l(m, types, LINEAR);
        w = param(l, PIKV_NAME("weight"), {out, in});
        b = param(l, PIKV_NAME("bias"), {out});
    }
    void lora(PyObject* m, int64_t H, const float*& a, const float*& b, int32_t& rank, float& scale) const {
        const Mod l(m, types, LORA);
        const Mod drop(l.child(PIKV_NAME("dropout")), types, DROPOUT);
        need(drop.is_false(PIKV_NAME("training")) || drop.number(PIKV_NAME("p")) == 0.f);
        const long r = l.integer(PIKV_NAME("rank"));
        need(r > 0 && r <= 16);
        rank = (int32_t)r;
        scale = l.number(PIKV_NAME("scaling"));
        a = param(l, PIKV_NAME("lora_A"), {H, r});
        b = param(l, PIKV_NAME("lora_B"), {r, H});
    }
    void plain(PyObject* m, int type) const { Mod(m, types, type); }
    // Linear(H, hidden), ReLU, Linear(hidden, out)[, tail]
    void net(PyObject* m, int64_t H, int64_t hidden, int64_t out, int tail, const float*& w1, const float*& b1, const float*& w2, const float*& b2) const {
        const Mod s = list(m, SEQUENTIAL, tail < 0 ? 3 : 4);
        linear(s.child(digit(0)), hidden, H, w1, b1);
        plain(s.child(digit(1)), RELU);
        linear(s.child(digit(2)), out, hidden, w2, b2);
        if (tail >= 0) plain(s.child(digit(3)), tail);
        if (tail == SOFTMAX) {
            const Mod t(s.child(digit(3)), types, tail);
            PyObject* dim = t.get(PIKV_NAME("dim"));
            need(PyLong_CheckExact(dim) && num(dim) == -1);
        }
    }
};

// moe(module, x, ring positions, classes) -> (weighted expert sum, logits or None, three gate results), or None where the modules have to run
PyObject* moe(PyObject* const* a, Py_ssize_t) {
    PyObject *positions = a[2], *types = a[3];
    if (!THPVariable_CheckExact(a[1])) Py_RETURN_NONE;
    const at::Tensor& xin = THPVariable_Unpack(a[1]);
    if (!xin.is_cuda() || xin.dim() != 3 || xin.scalar_type() != at::kFloat || !xin.numel() ||
        xin.device().index() != c10::cuda::current_device() || !PyList_CheckExact(positions) || !PyTuple_CheckExact(types) ||
        PyTuple_GET_SIZE(types) != MoeWalk::NTYPES)
        Py_RETURN_NONE;
    at::Tensor x = xin.contiguous();
    if (reinterpret_cast<uintptr_t>(x.const_data_ptr()) % 16) x = x.clone();
    using W = MoeWalk;
    const W walk{types, x.device()};
    pikv_moe_params p = {};
    at::Tensor touched[3 * PIKV_MOE_MAX_EXPERTS + 1];
    int n_touched = 0, topk[3];
    float temperature[2];
    try {
        need(x.size(0) * x.size(1) <= (1 << 21));
        p.B = (int32_t)x.size(0); p.S = (int32_t)x.size(1); p.H = (int32_t)x.size(2);
        const int64_t H = p.H;
        need(H % 128 == 0 && H <= 1024);
        // Wide models with many tokens: the fused layers run at a third of fp32 FMA rate and save the modules' launches, cuBLAS
        // runs at two thirds.  Modules / fused, 4 experts: H = 1024, 5040 tokens 1.21 to 1.31 (one sequence, eight), 7128 tokens 1.06
        // to 1.17, 10080 tokens 0.93 to 1.01, 65536 tokens 0.72 to 0.77; H = 768, 8960 tokens 1.04 to 1.19, 17920 tokens 0.87 to 0.98.  At
        // H = 512 only a long single sequence loses (its sums are one CTA's): 28512 tokens 1.07, 65536 tokens 0.93, eight
        // sequences 1.16 at 40328.  H = 256: 1.3 to 1.6 at 161312 tokens.  More experts move the line up (16, H = 1024: 1.68 at 3536 tokens).
        const int64_t rows = H > 512 ? (int64_t)p.B * p.S : H > 256 ? p.S : 0;
        need(rows * H * H <= (H > 512 ? int64_t(1) << 33 : int64_t(11) << 30));
        const Mod m(a[0], types, W::MOE);
        const Mod experts = walk.list(m.child(PIKV_NAME("experts")), W::MODULES, -1), caches = walk.list(m.child(PIKV_NAME("kv_caches")), W::MODULES, -1);
        const int64_t E = PyDict_GET_SIZE(experts.get(PIKV_NAME("_modules")));
        need(E > 0 && E <= PIKV_MOE_MAX_EXPERTS && PyDict_GET_SIZE(caches.get(PIKV_NAME("_modules"))) >= E && PyList_GET_SIZE(positions) == E);
        need(!PyDict_GetItem(m.dict, PIKV_NAME("update_cache")));
        p.E = (int32_t)E;
        touched[n_touched++] = walk.buf(m, PIKV_NAME("cache_ptrs"), {E}, at::kLong);
        p.cache_ptrs = ptr<int64_t>(touched[0]);
        // router
        const Mod r(m.child(PIKV_NAME("router")), types, W::ADAPTIVE);
        walk.net(r.child(PIKV_NAME("router_selector")), H, H / 2, 2, W::SOFTMAX, p.sel_w1, p.sel_b1, p.sel_w2, p.sel_b2);
        const Mod lb(r.child(PIKV_NAME("load_balancing_router")), types, W::BALANCED), imp(r.child(PIKV_NAME("importance_router")), types, W::IMPORTANCE);
        const Mod* gates[2] = {&lb, &imp};
        pikv_moe_net* nets[2] = {&p.lb, &p.imp};
        for (int i = 0; i < 2; ++i) {
            const Mod& g = *gates[i];
            walk.net(g.child(PIKV_NAME("router")), H, H, E, -1, nets[i]->w1, nets[i]->b1, nets[i]->w2, nets[i]->b2);
            temperature[i] = nets[i]->temperature = g.number(PIKV_NAME("temperature"));
            topk[i] = (int)g.integer(PIKV_NAME("top_k"));
            need(g.integer(PIKV_NAME("num_experts")) == E && !PyDict_GetItem(g.dict, PIKV_NAME("_gate")));
        }
        topk[2] = (int)r.integer(PIKV_NAME("top_k"));
        need(r.integer(PIKV_NAME("num_experts")) == E);
        for (int k : topk) need(k >= 1 && k <= std::min<int64_t>(E, 8));
        walk.net(imp.child(PIKV_NAME("importance_predictor")), H, H / 2, 1, W::SIGMOID, p.pred.w1, p.pred.b1, p.pred.w2, p.pred.b2);
        // experts and their caches
        for (int64_t e = 0; e < E; ++e) {
            pikv_moe_expert& t = p.expert[e];
            const Mod x_(experts.child(W::digit(e)), types, W::EXPERT), c(caches.child(W::digit(e)), types, W::CACHE);
            walk.linear(x_.child(PIKV_NAME("dense")), H, H, t.w, t.b);
            walk.lora(x_.child(PIKV_NAME("lora")), H, t.lora_a, t.lora_b, t.rank, t.scale);
            need(c.is_false(PIKV_NAME("use_scheduling")) && !PyDict_GetItem(c.dict, PIKV_NAME("update")) && !PyDict_GetItem(c.dict, PIKV_NAME("get_all")));
            const long size = c.integer(PIKV_NAME("size"));
            need(size > 0 && size < (1 << 20));
            t.slots = (int32_t)size;
            PyObject* at = PyList_GET_ITEM(positions, e);
            need(PyLong_Check(at));
            t.slot = (int32_t)num(at);
            need(t.slot >= 0 && t.slot < size);
            const at::Tensor &k = walk.buf(c, PIKV_NAME("keys"), {size, H}), &v = walk.buf(c, PIKV_NAME("values"), {size, H}),
                             &w = walk.buf(c, PIKV_NAME("importance"), {size});
            for (int64_t q = 0; q < e; ++q) need(p.expert[q].values != ptr<float>(v));      // one cache under two names is read after it is written
            t.keys = ptr<float>(k); t.values = ptr<float>(v); t.importance = ptr<float>(w);
            touched[n_touched++] = k; touched[n_touched++] = v; touched[n_touched++] = w;
            const Mod outer(c.child(PIKV_NAME("compressor")), types, W::COMPRESSOR), pyramid(outer.child(PIKV_NAME("compressor")), types, W::PYRAMID);
            const Mod layers = walk.list(pyramid.child(PIKV_NAME("compression_layers")), W::MODULES, 2);
            const Mod first(layers.child(W::digit(0)), types, W::LINEAR);
            const long mid = first.integer(PIKV_NAME("out_features"));
            need(mid > 0 && mid % 4 == 0 && mid <= 1024);
            t.mid = (int32_t)mid;
            walk.linear(layers.child(W::digit(0)), mid, H, t.c1_w, t.c1_b);
            walk.linear(layers.child(W::digit(1)), H, mid, t.c2_w, t.c2_b);
            walk.lora(c.child(PIKV_NAME("value_lora")), H, t.v_a, t.v_b, t.v_rank, t.v_scale);
        }
    } catch (const NotApplicable&) {
        Py_RETURN_NONE;
    }
    const int T = p.B * p.S, E = p.E;
    at::Tensor out = at::empty_like(x), logits;
    // The vocabulary projection, unless it is hooked or of another kind, or has few rows: up to 32 of them read w once
    // whichever way, and splitting w first costs more (256 -> 50257: 32 rows 36 us split, 34 as a plain layer; 64: 36, 58).
    if (T > 32 && p.H <= 256) {
        try {
            const Mod m(a[0], types, W::MOE), v(m.child(PIKV_NAME("vocab_proj")), types, W::LINEAR);
            const long V = v.integer(PIKV_NAME("out_features"));
            need(V > 0 && V <= (1 << 24));
            walk.linear(m.child(PIKV_NAME("vocab_proj")), V, p.H, p.vocab_w, p.vocab_b);
            logits = at::empty({p.B, p.S, V}, on(x, at::kFloat));
            p.vocab_out = ptr<float>(logits);
            p.V = (int32_t)V;
        } catch (const NotApplicable&) {
        }
    }
    p.workspace_bytes = pikv_moe_workspace_bytes(p.B, p.S, p.H, E, p.V);
    const size_t row = ((size_t)T * E * 4 + 255) & ~size_t(255);
    size_t tail[3], total = ((p.workspace_bytes + 255) & ~size_t(255)) + 3 * row;
    for (int i = 0; i < 3; ++i) total += tail[i] = (pikv_gate_tail_workspace_bytes(T, E, topk[i]) + 255) & ~size_t(255);
    at::Tensor ws;                             // all experts' outputs among it, where the modules hold one at a time
    try {
        ws = workspace(x, total);
    } catch (const c10::OutOfMemoryError&) {
        Py_RETURN_NONE;
    }
    char* base = ptr<char>(ws);
    p.workspace = base;
    base += (p.workspace_bytes + 255) & ~size_t(255);
    float* raw[3];
    for (int i = 0; i < 3; ++i, base += row) raw[i] = reinterpret_cast<float*>(base);
    p.x = ptr<float>(x); p.out = ptr<float>(out);
    p.logits_lb = raw[0]; p.logits_imp = raw[1]; p.logits_mix = raw[2];
    check(pikv_moe_forward(&p, stream()), "pikv_moe_forward");
    for (int i = 0; i < n_touched; ++i)
        if (!touched[i].is_inference()) touched[i].unsafeGetTensorImpl()->bump_version();
    for (int e = 0; e < E; ++e) {
        PyObject* next = PyLong_FromLong((p.expert[e].slot + 1) % p.expert[e].slots);
        if (!next || PyList_SetItem(positions, e, next)) throw Raised();
    }
    pikv_gate_params g[3] = {};
    const pikv_gate_params* list[3] = {&g[0], &g[1], &g[2]};
    std::vector<GateOut> results;
    results.reserve(3);
    for (int i = 0; i < 3; ++i) {
        g[i].T = T; g[i].E = E; g[i].top_k = topk[i]; g[i].dtype = PIKV_F32; g[i].logits_in = raw[i];
        g[i].mask_mode = PIKV_MASK_NONE; g[i].temperature = i < 2 ? temperature[i] : 1.f;
        results.emplace_back(Py_None, x, T, E, topk[i], i < 2);
        results[i].fill(g[i]);
        g[i].workspace = base; g[i].workspace_bytes = tail[i];
        base += tail[i];
    }
    check(pikv_gate_logits(list, 3, stream()), "pikv_gate_logits");
    PyObject* result = PyTuple_New(5);
    if (!result) throw Raised();
    PyTuple_SET_ITEM(result, 0, wrap(out));
    PyTuple_SET_ITEM(result, 1, wrap(logits));
    for (int i = 0; i < 3; ++i) PyTuple_SET_ITEM(result, 2 + i, results[i].result());
    return result;
}

// ---- module ------------------------------------------------------------------------------------------------
using Fn = PyObject* (*)(PyObject* const*, Py_ssize_t);
template <Fn F, int N, int M = N>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != N && n != M) {
        PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", N, n);
        return nullptr;
    }
    try {
        c10::NoGradGuard no_grad;
        return F(args, n);
    } catch (const Raised&) {
    } catch (...) {                            // torch's own errors keep their types, the allocator's among them
        if (!PyErr_Occurred()) torch::translate_exception_to_python(std::current_exception());
    }
    return nullptr;
}
template <Fn F, int N, int M = N>
PyMethodDef method(const char* name) {
    return {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(entry<F, N, M>)), METH_FASTCALL, nullptr};
}

constexpr int C = Cache::ARGS, G = GateTail::ARGS;
PyMethodDef methods[] = {
    method<append, C + 4, C + 7>("append"),
    method<gate, 4 + G + 2>("gate"),
    method<gate_mlp, 5 + G + 5>("gate_mlp"),
    method<dispatch_loss, 10>("dispatch_loss"),
    method<route_append, C + 5 + G + 1>("route_append"),
    method<decode, C + 5, C + 6>("decode"),
    method<select, 8>("select"),
    method<compact, 2 * C + 7>("compact"),
    method<quant_pair, 9>("quant_pair"),
    method<lowrank, 6>("lowrank"),
    method<lowrank_pair, 10>("lowrank_pair"),
    method<linear, 3>("linear_f32"),
    method<moe, 4>("moe"),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
    PyObject* lib = PyImport_ImportModule("pikv_b200._lib");
    if (!lib) return nullptr;
    g_error = PyObject_GetAttrString(lib, "PikvError");
    Py_DECREF(lib);
    if (!g_error) return nullptr;
    if (pikv_abi_version() != PIKV_ABI_VERSION) {
        PyErr_Format(g_error, "libpikv_b200.so has ABI %d, the host module expects %d", pikv_abi_version(), PIKV_ABI_VERSION);
        return nullptr;
    }
    s_k_codes = PyUnicode_InternFromString("k_codes"); s_v_codes = PyUnicode_InternFromString("v_codes");
    s_k_scale = PyUnicode_InternFromString("k_scale"); s_v_scale = PyUnicode_InternFromString("v_scale");
    s_k_zp = PyUnicode_InternFromString("k_zp"); s_v_zp = PyUnicode_InternFromString("v_zp");
    s_page_table = PyUnicode_InternFromString("page_table"); s_length = PyUnicode_InternFromString("length");
    s_status = PyUnicode_InternFromString("status");
    return PyModule_Create(&module_def);
}
