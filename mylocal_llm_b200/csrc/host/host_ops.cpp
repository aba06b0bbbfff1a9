// Native host path: the operators' launch sequences without an interpreter between two launches.
//
// A decode step is a chain of short kernels; enqueued from Python each of them costs 10-20 us of host time (argument
// checks, ctypes conversion, several small allocations), more than most of the kernels take (a batch-16 step of the
// 1.7B Llama shape: 5 ms of host time for 3 ms of kernels). This extension module does the same checks, allocations
// (torch's caching allocator, so streams and CUDA-graph pools behave as before) and C ABI calls in C++. It contains no
// computation and no kernels of its own: every launch goes through the entry points of libb200q.so, whose addresses
// Python hands over once (bind). A call outside what it covers returns None and the Python layer, which raises the
// documented exceptions, takes over; the results are the same bits either way. (Token ids outside the vocabulary: NaN for
// their sequence here, a device-side assertion of the gather there.)
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "b200q.h"

namespace py = pybind11;

namespace {

struct Api {
#define FN(name) decltype(&b200q_##name) name = nullptr
    FN(last_error); FN(gemv); FN(gemm); FN(gemm_ws); FN(gemm_workspace_bytes); FN(gemm_supported); FN(rmsnorm);
    FN(residual_rmsnorm); FN(gemv_norm); FN(gemv_norm_supported); FN(router_logits_t); FN(router_topk_ex);
    FN(router_topk_plan_row); FN(shared_gate); FN(moe_plan_ex); FN(moe_token_image_bytes); FN(moe_token_images);
    FN(moe_gate_up); FN(moe_gate_up_images); FN(moe_down); FN(moe_hidden_image_bytes); FN(moe_gate_up_streams); FN(moe_down_streams); FN(moe_hidden_images); FN(moe_down_images); FN(moe_combine); FN(silu_mul); FN(rope_attention);
    FN(prefill_attention); FN(embed_tokens);
#undef FN
} api;
PyObject *b200q_error = nullptr;        // the package's exception for CUDA errors

void bind(const py::dict &addresses, py::object error_type) {
#define FN(name) api.name = reinterpret_cast<decltype(api.name)>(addresses["b200q_" #name].cast<uintptr_t>())
    FN(last_error); FN(gemv); FN(gemm); FN(gemm_ws); FN(gemm_workspace_bytes); FN(gemm_supported); FN(rmsnorm);
    FN(residual_rmsnorm); FN(gemv_norm); FN(gemv_norm_supported); FN(router_logits_t); FN(router_topk_ex);
    FN(router_topk_plan_row); FN(shared_gate); FN(moe_plan_ex); FN(moe_token_image_bytes); FN(moe_token_images);
    FN(moe_gate_up); FN(moe_gate_up_images); FN(moe_down); FN(moe_hidden_image_bytes); FN(moe_gate_up_streams); FN(moe_down_streams); FN(moe_hidden_images); FN(moe_down_images); FN(moe_combine); FN(silu_mul); FN(rope_attention);
    FN(prefill_attention); FN(embed_tokens);
#undef FN
    b200q_error = error_type.release().ptr();
}

// Non-zero return codes become the exceptions _lib.call raises. The launches run without the interpreter's lock, as they do
// through ctypes (a launch into a full queue waits for the GPU): the code travels as a C++ exception.
struct CallError {
    int rc;
    std::string text;
    void raise() const { PyErr_SetString(rc == 1 ? PyExc_ValueError : rc == 3 ? PyExc_NotImplementedError : b200q_error, text.c_str()); }
};
void check(int rc, const char *name) {
    if (rc) throw CallError{rc, std::string(name) + ": " + api.last_error()};
}
#define CALL(name, ...) check(api.name(__VA_ARGS__), "b200q_" #name)

// Environment switches are read at every call, as the Python layer does.
bool env_is(const char *name, const char *value) {
    const char *v = std::getenv(name);
    return v && std::strcmp(v, value) == 0;
}
bool env_set_other_than(const char *name, const char *value) {
    const char *v = std::getenv(name);
    return v && std::strcmp(v, value) != 0;
}

void *stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

int dtype_id(at::ScalarType t) {
    return t == at::kFloat ? B200Q_F32 : t == at::kHalf ? B200Q_F16 : t == at::kBFloat16 ? B200Q_BF16 : -1;
}
at::Tensor empty(at::IntArrayRef sizes, at::ScalarType t, const at::Device &device) {
    return at::empty(sizes, at::TensorOptions().dtype(t).device(device));
}
bool gguf_gemm_format(int fmt) { return fmt == B200Q_Q8_0 || fmt == B200Q_Q4_K || fmt == B200Q_Q5_K || fmt == B200Q_Q6_K; }

// Tokens from which BF16 calls on GGUF-layout weights take the GEMM, by format (0: never): quantized_linear.GEMM_MIN_TOKENS
// as it stands at the call (None: no entry).
int gemm_from(PyObject *tokens) {
    if (tokens == Py_None) return 0;
    int overflow = 0;
    const long v = PyLong_AsLongAndOverflow(tokens, &overflow);
    return overflow > 0 || v > 0x7fffffff ? 0x7fffffff : v < 1 ? 1 : static_cast<int>(v);
}
struct GemmRule {
    int q8_0 = 0, q4_k = 0, q5_k = 0, q6_k = 0;
    int of(int fmt) const {
        return fmt == B200Q_Q8_0 ? q8_0 : fmt == B200Q_Q4_K ? q4_k : fmt == B200Q_Q5_K ? q5_k : fmt == B200Q_Q6_K ? q6_k : 0;
    }
};

// y[m, n] = x[m, k] W^T by the rule of quantized_linear (GEMM for many BF16 tokens on a GGUF layout, else GEMV).
void linear_into(const void *x, int x_dtype, int m, const void *w, int fmt, int n, int k, void *y, int y_dtype,
                 int gemm_min_tokens, const at::Device &device) {
    if (gemm_min_tokens > 0 && m >= gemm_min_tokens && gguf_gemm_format(fmt) && x_dtype == B200Q_BF16 &&
        (reinterpret_cast<uintptr_t>(x) & 15) == 0 && reinterpret_cast<uintptr_t>(w) % (fmt == B200Q_Q8_0 ? 4 : 2) == 0 &&
        !env_is("B200Q_GEMM", "0") && !env_set_other_than("B200Q_KERNEL", "auto") && api.gemm_supported(fmt, n, k, x_dtype, m)) {
        const long long bytes = api.gemm_workspace_bytes(fmt, n, k, x_dtype, m);
        if (bytes && !env_is("B200Q_GEMM_SPLITK", "0")) {
            const at::Tensor scratch = empty({bytes}, at::kByte, device);
            CALL(gemm_ws, w, fmt, n, k, x, x_dtype, m, y, y_dtype, scratch.data_ptr(), bytes, stream());
        } else {
            CALL(gemm, w, fmt, n, k, x, x_dtype, m, y, y_dtype, stream());
        }
    } else {
        CALL(gemv, w, fmt, n, k, x, x_dtype, m, y, y_dtype, stream());
    }
}

// ------------------------------------------------------------------------------------------------ linear
// linear(x, data, fmt, n, k, out_dtype | None, GEMM from this many tokens on | None): the tensor, or None when the call needs the Python layer.
PyObject *linear_fast(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
    if (nargs != 7 || !THPVariable_Check(args[0]) || !THPVariable_Check(args[1])) Py_RETURN_NONE;
    HANDLE_TH_ERRORS
        const at::Tensor &x = THPVariable_Unpack(args[0]), &w = THPVariable_Unpack(args[1]);
        const int fmt = static_cast<int>(PyLong_AsLong(args[2])), n = static_cast<int>(PyLong_AsLong(args[3])),
                  k = static_cast<int>(PyLong_AsLong(args[4])), gemm_min = gemm_from(args[6]);
        if (PyErr_Occurred()) return nullptr;
        const int64_t nd = x.dim();
        const int dt = dtype_id(x.scalar_type());
        if (!x.is_cuda() || (nd != 2 && nd != 3) || x.size(nd - 1) != k || dt < 0 || !x.is_contiguous() || x.device() != w.device())
            Py_RETURN_NONE;
        at::ScalarType out_type = x.scalar_type();
        if (args[5] != Py_None) {
            if (!THPDtype_Check(args[5])) Py_RETURN_NONE;
            out_type = reinterpret_cast<THPDtype *>(args[5])->scalar_type;
        }
        const int ydt = dtype_id(out_type);
        const int64_t m = x.numel() / k;
        if (ydt < 0 || m == 0 || m > 0x7fffffff) Py_RETURN_NONE;
        at::Tensor y = nd == 2 ? empty({m, n}, out_type, x.device()) : empty({x.size(0), x.size(1), n}, out_type, x.device());
        try {
            py::gil_scoped_release unlocked;
            linear_into(x.data_ptr(), dt, static_cast<int>(m), w.data_ptr(), fmt, n, k, y.data_ptr(), ydt, gemm_min, x.device());
        } catch (const CallError &e) {
            e.raise();
            return nullptr;
        }
        return THPVariable_Wrap(std::move(y));
    END_HANDLE_TH_ERRORS
}
PyMethodDef linear_def = {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(linear_fast)), METH_FASTCALL, nullptr};

// ------------------------------------------------------------------------------------------------ MoE layer
// 256-byte aligned pieces of one scratch allocation.
struct Carver {
    size_t used = 0;
    size_t take(size_t bytes) {
        const size_t at = used;
        used = (used + bytes + 255) / 256 * 256;
        return at;
    }
};

constexpr int SEGMENT_CAP = 8;          // tokens of one expert per pass of the grouped kernels
constexpr int TOKEN_IMAGE_MIN_ROWS = 32;  // of moe_ops: images for the block-structured gate/up kernels

struct MoeLayer {
    at::Tensor router, bias, gate_vector;               // [E, D] FP32; bias / shared-expert gate may be undefined
    at::Tensor gate, up, down;                          // banks (addressed by stride when there are no tables)
    at::Tensor gate_table, up_table, down_table;        // pointer tables; undefined: banks
    int64_t gate_stride = 0, up_stride = 0, down_stride = 0;
    int gate_fmt = 0, up_fmt = 0, down_fmt = 0, experts = 0, top_k = 0, d = 0, f = 0;
    float floor = 0.f;
    bool aligned16 = false, with_shared = false, row_plan = true;

    // x [t, d] contiguous CUDA rows -> out [t, d] of out_type
    void run(const at::Tensor &x, int64_t t64, at::Tensor &out) const {
        const int t = static_cast<int>(t64), xdt = dtype_id(x.scalar_type()), odt = dtype_id(out.scalar_type());
        const int k = top_k + (with_shared ? 1 : 0), plan_experts = experts + (with_shared ? 1 : 0), total = t * k;
        const int max_segments = std::min(plan_experts, total) + total / SEGMENT_CAP;
        const bool q45 = gate_fmt == up_fmt && (gate_fmt == B200Q_Q4_K || gate_fmt == B200Q_Q5_K ||
                                                gate_fmt == B200Q_Q4_K_TILED || gate_fmt == B200Q_Q5_K_TILED);
        const bool images = !env_is("B200Q_TOKEN_IMAGES", "0");
        const int image_bytes = images && q45 && (t >= TOKEN_IMAGE_MIN_ROWS || api.moe_gate_up_streams(gate_fmt, f, d, xdt, max_segments))
                                    ? std::max(0, api.moe_token_image_bytes(d, xdt)) : 0;
        const int hidden_bytes = images && api.moe_down_streams(down_fmt, d, f, max_segments) ? api.moe_hidden_image_bytes(f) : 0;
        Carver c;
        const size_t o_logits = c.take(sizeof(float) * t * experts), o_weights = c.take(sizeof(float) * total),
                     o_ids = c.take(sizeof(int64_t) * total), o_scale = c.take(sizeof(float) * t),
                     o_counts = c.take(4 * plan_experts), o_offsets = c.take(4 * (plan_experts + 1)), o_order = c.take(4 * total),
                     o_inv = c.take(4 * total), o_seg = c.take(12 * static_cast<size_t>(max_segments)), o_misc = c.take(8),
                     o_hbuf = c.take(sizeof(float) * total * f), o_terms = c.take(sizeof(float) * total * d),
                     o_images = c.take(static_cast<size_t>(image_bytes) * t), o_hidden = c.take(static_cast<size_t>(hidden_bytes) * total);
        const at::Tensor scratch = empty({static_cast<int64_t>(c.used)}, at::kByte, x.device());
        uint8_t *base = static_cast<uint8_t *>(scratch.data_ptr());
        auto f32 = [&](size_t o) { return reinterpret_cast<float *>(base + o); };
        auto i32 = [&](size_t o) { return reinterpret_cast<int32_t *>(base + o); };
        float *logits = f32(o_logits), *weights = f32(o_weights), *hbuf = f32(o_hbuf), *terms = f32(o_terms);
        int64_t *ids = reinterpret_cast<int64_t *>(base + o_ids);
        int32_t *counts = i32(o_counts), *offsets = i32(o_offsets), *order = i32(o_order), *inv = i32(o_inv);
        int32_t *seg_expert = i32(o_seg), *seg_begin = seg_expert + max_segments, *seg_count = seg_begin + max_segments;
        int32_t *num_segments = i32(o_misc), *status = num_segments + 1;
        void *s = stream();
        CALL(router_logits_t, x.data_ptr(), xdt, t, d, router.data_ptr<float>(), bias.defined() ? bias.data_ptr<float>() : nullptr,
             experts, logits, s);
        const float *scale = nullptr;
        if (gate_vector.defined()) {
            CALL(shared_gate, x.data_ptr(), xdt, t, d, gate_vector.data_ptr<float>(), f32(o_scale), s);
            scale = f32(o_scale);
        }
        const int extra = with_shared ? experts : -1;
        if (t == 1 && row_plan && with_shared && experts <= 1024 && top_k <= 31) {
            CALL(router_topk_plan_row, logits, experts, top_k, 1, floor, extra, scale, weights, ids, plan_experts, counts, offsets,
                 order, inv, seg_expert, seg_begin, seg_count, num_segments, max_segments, status, s);
        } else {
            CALL(router_topk_ex, logits, t, experts, top_k, 1, floor, extra, scale, weights, ids, s);
            CALL(moe_plan_ex, ids, 1, t, k, plan_experts, -1, SEGMENT_CAP, counts, offsets, order, inv, seg_expert, seg_begin,
                 seg_count, num_segments, max_segments, status, s);
        }
        const bool tables = gate_table.defined();
        auto table = [&](const at::Tensor &v) { return tables ? static_cast<const uint64_t *>(v.data_ptr()) : nullptr; };
        auto bank = [&](const at::Tensor &v) { return tables ? nullptr : v.data_ptr(); };
        const int64_t gs = tables ? 0 : gate_stride, us = tables ? 0 : up_stride, ds = tables ? 0 : down_stride;
        if (image_bytes) {
            CALL(moe_token_images, x.data_ptr(), xdt, t, d, base + o_images, s);
            CALL(moe_gate_up_images, bank(gate), gs, gate_fmt, bank(up), us, up_fmt, table(gate_table), table(up_table), aligned16,
                 f, d, x.data_ptr(), xdt, base + o_images, k, order, seg_expert, seg_begin, seg_count, num_segments, max_segments,
                 hbuf, s);
        } else {
            CALL(moe_gate_up, bank(gate), gs, gate_fmt, bank(up), us, up_fmt, table(gate_table), table(up_table), aligned16, f, d,
                 x.data_ptr(), xdt, k, order, seg_expert, seg_begin, seg_count, num_segments, max_segments, hbuf, s);
        }
        if (hidden_bytes) {
            CALL(moe_hidden_images, hbuf, total, f, base + o_hidden, s);
            CALL(moe_down_images, bank(down), ds, down_fmt, table(down_table), aligned16, 0, d, f, hbuf, base + o_hidden, weights, order,
                 seg_expert, seg_begin, seg_count, num_segments, max_segments, terms, s);
        } else
            CALL(moe_down, bank(down), ds, down_fmt, table(down_table), aligned16, 0, d, f, hbuf, weights, order, seg_expert, seg_begin,
             seg_count, num_segments, max_segments, terms, s);
        CALL(moe_combine, terms, inv, t, k, d, nullptr, nullptr, out.data_ptr(), odt, s);
    }

    at::Tensor forward(const at::Tensor &hidden) const {
        at::Tensor out = at::empty_like(hidden);
        run(hidden, hidden.numel() / d, out);
        return out;
    }
};

// hidden -> MoE layers with residual-add + RMSNorm between them (PackedMoEStack.forward's chain).
struct MoeStack {
    std::vector<MoeLayer> layers;
    std::vector<at::Tensor> gammas;        // layers.size() + 1, one type
    float eps = 0.f;

    std::pair<at::Tensor, at::Tensor> forward(const at::Tensor &residual) const {
        const int d = layers[0].d;
        const int64_t rows = residual.numel() / d;
        const at::ScalarType type = gammas[0].scalar_type();
        const int gdt = dtype_id(type);
        at::Tensor hidden = empty(residual.sizes(), type, residual.device()), branch = empty(residual.sizes(), type, residual.device());
        at::Tensor res = residual, next;
        CALL(rmsnorm, residual.data_ptr(), B200Q_F32, gammas[0].data_ptr(), gdt, static_cast<int>(rows), d, eps, hidden.data_ptr(), gdt,
             stream());
        for (size_t i = 0; i < layers.size(); ++i) {
            layers[i].run(hidden, rows, branch);
            if (!next.defined()) next = at::empty_like(residual);      // (later layers update it in place)
            CALL(residual_rmsnorm, res.data_ptr<float>(), branch.data_ptr(), gdt, 1.0f, gammas[i + 1].data_ptr(), gdt,
                 static_cast<int>(rows), d, eps, next.data_ptr<float>(), hidden.data_ptr(), gdt, stream());
            res = next;
        }
        return {res, hidden};
    }
};

// ------------------------------------------------------------------------------------------------ Llama decoder
struct Matrix {
    at::Tensor data, native;               // decode layout; GGUF-layout copy for many-token calls (may be undefined)
    int fmt = 0, native_fmt = 0, n = 0, k = 0;
};
struct LlamaLayer {
    at::Tensor norm1, norm2;
    Matrix qkv, o, gate_up, down;
};

struct Llama {
    std::vector<LlamaLayer> layers;
    at::Tensor embed, final_norm, cos, sin;
    Matrix lm_head;
    int embed_fmt = 0, d = 0, f = 0, heads = 0, kv_heads = 0, head_dim = 0, vocab = 0;
    float eps = 0.f;
    at::ScalarType type = at::kBFloat16;

    int dt() const { return dtype_id(type); }
    // ExternalLlamaModel._linear: many BF16 rows read the GGUF copy, everything else the decode layout
    void linear(const at::Tensor &x, int64_t m, const Matrix &w, at::Tensor &y, const GemmRule &rule, bool choose = true) const {
        const int from = choose && w.native.defined() ? rule.of(w.native_fmt) : 0;
        const bool native = from > 0 && type == at::kBFloat16 && m >= from;
        linear_into(x.data_ptr(), dtype_id(x.scalar_type()), static_cast<int>(m), native ? w.native.data_ptr() : w.data.data_ptr(),
                    native ? w.native_fmt : w.fmt, w.n, w.k, y.data_ptr(), dtype_id(y.scalar_type()),
                    rule.of(native ? w.native_fmt : w.fmt), x.device());
    }
    at::Tensor embed_tokens(const at::Tensor &ids) const {
        at::Tensor r = empty({ids.numel(), d}, at::kFloat, ids.device());
        CALL(embed_tokens, embed.data_ptr(), embed_fmt, vocab, d, ids.data_ptr<int64_t>(), static_cast<int>(ids.numel()),
             r.data_ptr<float>(), stream());
        return r;
    }
    void norm(const at::Tensor &x, const at::Tensor &gamma, int64_t rows, at::Tensor &y) const {
        CALL(rmsnorm, x.data_ptr(), B200Q_F32, gamma.data_ptr(), dt(), static_cast<int>(rows), d, eps, y.data_ptr(), dt(), stream());
    }
    void add_norm(at::Tensor &residual, const at::Tensor &branch, const at::Tensor &gamma, int64_t rows, at::Tensor &y) const {
        CALL(residual_rmsnorm, residual.data_ptr<float>(), branch.data_ptr(), dt(), 1.0f, gamma.data_ptr(), dt(),
             static_cast<int>(rows), d, eps, residual.data_ptr<float>(), y.data_ptr(), dt(), stream());
    }
    void silu(const at::Tensor &gu, int64_t rows, at::Tensor &act) const {
        CALL(silu_mul, gu.data_ptr<float>(), static_cast<int>(rows), f, act.data_ptr(), dt(), stream());
    }

    // One token per sequence: ids [B], caches [layers, B, kv_heads, horizon, head_dim], position [1] int64 (device).
    at::Tensor decode(const at::Tensor &ids, const at::Tensor &kc, const at::Tensor &vc, const at::Tensor &position,
                      const GemmRule &rule) const {
        const int64_t b = ids.numel(), qd = static_cast<int64_t>(heads) * head_dim, kd = static_cast<int64_t>(kv_heads) * head_dim;
        const at::Device dev = ids.device();
        at::Tensor residual = embed_tokens(ids), hidden = empty({b, d}, type, dev), qkv = empty({b, qd + 2 * kd}, at::kFloat, dev),
                   ctx = empty({b, qd}, type, dev), branch = empty({b, d}, type, dev), gu = empty({b, 2 * static_cast<int64_t>(f)}, at::kFloat, dev),
                   act = empty({b, f}, type, dev), logits = empty({b, vocab}, at::kFloat, dev);
        at::Tensor other = b == 1 ? at::empty_like(residual) : at::Tensor();      // the fused norm + projection writes a new stream
        const float scale = static_cast<float>(std::pow(static_cast<double>(head_dim), -0.5));
        const int64_t layer_bytes = kc.stride(0) * kc.element_size();
        // residual += branch, y = norm(residual) W^T: one launch for a single row where the fused kernel covers it
        auto norm_linear = [&](const at::Tensor &gamma, const Matrix &w, at::Tensor &y) {
            if (b == 1 && w.k == d && api.gemv_norm_supported(w.fmt, w.n, w.k, dt(), 1)) {
                CALL(gemv_norm, w.data.data_ptr(), w.fmt, w.n, w.k, residual.data_ptr<float>(), branch.data_ptr(), dt(), 1.0f,
                     gamma.data_ptr(), dt(), eps, 1, other.data_ptr<float>(), y.data_ptr(), B200Q_F32, stream());
                std::swap(residual, other);
                return;
            }
            add_norm(residual, branch, gamma, b, hidden);
            linear(hidden, b, w, y, rule);
        };
        for (size_t i = 0; i < layers.size(); ++i) {
            const LlamaLayer &l = layers[i];
            if (i == 0) {
                norm(residual, l.norm1, b, hidden);
                linear(hidden, b, l.qkv, qkv, rule);
            } else {
                norm_linear(l.norm1, l.qkv, qkv);
            }
            float *q = qkv.data_ptr<float>();
            const int64_t row = qd + 2 * kd;
            CALL(rope_attention, q, q + qd, q + qd + kd, row, row, row, position.data_ptr<int64_t>(), cos.data_ptr<float>(),
                 sin.data_ptr<float>(), static_cast<int>(cos.size(0)), static_cast<int>(b), heads, kv_heads, head_dim,
                 static_cast<int>(kc.size(3)), static_cast<uint8_t *>(kc.data_ptr()) + i * layer_bytes,
                 static_cast<uint8_t *>(vc.data_ptr()) + i * layer_bytes, dt(), scale, ctx.data_ptr(), dt(), stream());
            linear(ctx, b, l.o, branch, rule, false);
            norm_linear(l.norm2, l.gate_up, gu);
            silu(gu, b, act);
            linear(act, b, l.down, branch, rule);
        }
        norm_linear(final_norm, lm_head, logits);
        return logits;
    }

    // The whole prompt from position 0 on: ids [B, T]; logits of the last position.
    at::Tensor prefill(const at::Tensor &ids, const at::Tensor &kc, const at::Tensor &vc, const GemmRule &rule) const {
        const int64_t b = ids.size(0), t = ids.size(1), rows = b * t, qd = static_cast<int64_t>(heads) * head_dim,
                      kd = static_cast<int64_t>(kv_heads) * head_dim;
        const at::Device dev = ids.device();
        at::Tensor residual = embed_tokens(ids), hidden = empty({rows, d}, type, dev), qkv = empty({rows, qd + 2 * kd}, at::kFloat, dev),
                   ctx = empty({rows, qd}, type, dev), branch = empty({rows, d}, type, dev),
                   gu = empty({rows, 2 * static_cast<int64_t>(f)}, at::kFloat, dev), act = empty({rows, f}, type, dev);
        const float scale = static_cast<float>(std::pow(static_cast<double>(head_dim), -0.5));
        const int64_t layer_bytes = kc.stride(0) * kc.element_size(), row = qd + 2 * kd;
        norm(residual, layers[0].norm1, rows, hidden);
        for (size_t i = 0; i < layers.size(); ++i) {
            const LlamaLayer &l = layers[i];
            linear(hidden, rows, l.qkv, qkv, rule);
            float *q = qkv.data_ptr<float>();
            CALL(prefill_attention, q, q + qd, q + qd + kd, row, row, row, cos.data_ptr<float>(), sin.data_ptr<float>(),
                 static_cast<int>(cos.size(0)), static_cast<int>(b), static_cast<int>(t), heads, kv_heads, head_dim,
                 static_cast<int>(kc.size(3)), static_cast<uint8_t *>(kc.data_ptr()) + i * layer_bytes,
                 static_cast<uint8_t *>(vc.data_ptr()) + i * layer_bytes, dt(), scale, ctx.data_ptr(), dt(), stream());
            linear(ctx, rows, l.o, branch, rule);
            add_norm(residual, branch, l.norm2, rows, hidden);
            linear(hidden, rows, l.gate_up, gu, rule);
            silu(gu, rows, act);
            linear(act, rows, l.down, branch, rule);
            add_norm(residual, branch, i + 1 < layers.size() ? layers[i + 1].norm1 : final_norm, rows, hidden);
        }
        const at::Tensor last = hidden.view({b, t, d}).select(1, t - 1).contiguous();
        at::Tensor logits = empty({b, vocab}, at::kFloat, dev);
        linear(last, b, lm_head, logits, rule, false);
        return logits;
    }
};

GemmRule gemm_rule(const py::list &v) {
    return {gemm_from(py::object(v[0]).ptr()), gemm_from(py::object(v[1]).ptr()), gemm_from(py::object(v[2]).ptr()), gemm_from(py::object(v[3]).ptr())};
}
at::Tensor or_undefined(const py::object &o) { return o.is_none() ? at::Tensor() : o.cast<at::Tensor>(); }

}  // namespace

PYBIND11_MODULE(_b200q_host, m) {
    using Unlocked = py::call_guard<py::gil_scoped_release>;
    py::register_local_exception_translator([](std::exception_ptr p) {
        try {
            if (p) std::rethrow_exception(p);
        } catch (const CallError &e) {
            e.raise();
        } catch (const c10::Error &) {
            torch::translate_exception_to_python(std::current_exception());
        }
    });
    m.def("bind", &bind);
    m.add_object("linear", py::reinterpret_steal<py::object>(PyCFunction_New(&linear_def, nullptr)));
    py::class_<MoeLayer>(m, "MoeLayer")
        .def(py::init([](at::Tensor router, py::object bias, py::object gate_vector, at::Tensor gate, at::Tensor up, at::Tensor down,
                         std::vector<int64_t> strides, std::vector<int> formats, py::object tables, bool aligned16, bool with_shared,
                         int experts, int top_k, int d, int f, double floor, bool row_plan) {
            MoeLayer l;
            l.router = router; l.bias = or_undefined(bias); l.gate_vector = or_undefined(gate_vector);
            l.gate = gate; l.up = up; l.down = down;
            l.gate_stride = strides.at(0); l.up_stride = strides.at(1); l.down_stride = strides.at(2);
            l.gate_fmt = formats.at(0); l.up_fmt = formats.at(1); l.down_fmt = formats.at(2);
            if (!tables.is_none()) {
                const auto t = tables.cast<std::vector<at::Tensor>>();
                l.gate_table = t.at(0); l.up_table = t.at(1); l.down_table = t.at(2);
            }
            l.aligned16 = aligned16; l.with_shared = with_shared; l.experts = experts; l.top_k = top_k; l.d = d; l.f = f;
            l.floor = static_cast<float>(floor); l.row_plan = row_plan;
            return l;
        }))
        .def("forward", &MoeLayer::forward, Unlocked());
    py::class_<MoeStack>(m, "MoeStack")
        .def(py::init([](std::vector<MoeLayer> layers, std::vector<at::Tensor> gammas, double eps) {
            MoeStack s;
            s.layers = std::move(layers); s.gammas = std::move(gammas); s.eps = static_cast<float>(eps);
            return s;
        }))
        .def("forward", &MoeStack::forward, Unlocked());
    py::class_<Llama>(m, "Llama")
        .def(py::init([](const py::dict &c) {
            auto matrix = [](const py::handle &h) {
                const auto t = py::cast<py::tuple>(h);              // (data, fmt, n, k, native | None, native_fmt)
                Matrix w;
                w.data = t[0].cast<at::Tensor>(); w.fmt = t[1].cast<int>(); w.n = t[2].cast<int>(); w.k = t[3].cast<int>();
                w.native = or_undefined(py::reinterpret_borrow<py::object>(t[4])); w.native_fmt = t[5].cast<int>();
                return w;
            };
            Llama l;
            l.embed = c["embed"].cast<at::Tensor>(); l.embed_fmt = c["embed_fmt"].cast<int>();
            l.final_norm = c["final_norm"].cast<at::Tensor>(); l.lm_head = matrix(c["lm_head"]);
            l.cos = c["cos"].cast<at::Tensor>(); l.sin = c["sin"].cast<at::Tensor>();
            l.d = c["d"].cast<int>(); l.f = c["f"].cast<int>(); l.heads = c["heads"].cast<int>();
            l.kv_heads = c["kv_heads"].cast<int>(); l.head_dim = c["head_dim"].cast<int>(); l.vocab = c["vocab"].cast<int>();
            l.eps = static_cast<float>(c["eps"].cast<double>());
            l.type = l.final_norm.scalar_type();
            for (const py::handle &h : c["layers"]) {
                const auto t = py::cast<py::tuple>(h);              // (norm1, norm2, qkv, o, gate_up, down)
                l.layers.push_back({t[0].cast<at::Tensor>(), t[1].cast<at::Tensor>(), matrix(t[2]), matrix(t[3]), matrix(t[4]), matrix(t[5])});
            }
            return l;
        }))
        .def("decode", [](const Llama &m, at::Tensor ids, at::Tensor k, at::Tensor v, at::Tensor position, const py::list &rule) {
            const GemmRule from = gemm_rule(rule);
            py::gil_scoped_release unlocked;
            return m.decode(ids, k, v, position, from);
        })
        .def("prefill", [](const Llama &m, at::Tensor ids, at::Tensor k, at::Tensor v, const py::list &rule) {
            const GemmRule from = gemm_rule(rule);
            py::gil_scoped_release unlocked;
            return m.prefill(ids, k, v, from);
        });
}
