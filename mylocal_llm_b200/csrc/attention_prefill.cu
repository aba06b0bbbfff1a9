// Prompt attention of the Llama path: rotate-half RoPE, the KV-cache store and causal attention over a prompt that
// starts at position 0 (BF16 caches), two launches per layer.
// Semantics follow the reference's inference attention (mini_llm/ops/attention_inference.py:255-277 for the rotation,
// scores q.k * scale, softmax over positions 0..i in FP32, values from the cache, grouped KV heads).
//
// The attention is FP32 throughout (queries, scores, probabilities; keys and values as the cache holds them) and every
// sum has one fixed order, the one of a plain chain of FP32 operators: a score is one chain of FMAs over the head
// dimension, a row's exponentials are added per residue of the position modulo 32 and then in a butterfly, every
// probability is divided before the value product, an output is one chain of FMAs over the positions. The results of a
// deep BF16 model depend on such orders far above the FP32 rounding (a last-bit difference flips BF16 roundings: the scale
// one unit in the last place up moves the logits of a 512-token prompt by 0 after one layer, 0.6 % after four, 1.8 % after
// twenty-four), so the kernel keeps the order of the operator chain it replaced, which rules out an online softmax and the
// tensor cores' own accumulation order. A row block's scores therefore stay in shared
// memory between the two products. Bound by the FP32 FMA rate (4 * 64 operations per query, key and head) and the
// shared-memory reads that feed it: 16 prompts of 512 tokens, 32 heads, 0.73 ms with the cache store = 11.9 T FMA/s of
// the causal half; the operator chain (full score matrix through HBM five times) took 2.7 ms.
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace b200q {

constexpr int PA_KEYS = 256;         // key positions per tile of the score product
constexpr int PA_VALUES = 64;        // positions per tile of the value product
constexpr int PA_SMEM_LIMIT = 232448;     // of every launch: one thread's prompt must not lower another's limit

__device__ __forceinline__ uint64_t pa_pack2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void pa_unpack2(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
// two independent FMAs, each rounded as the scalar one (half the issue slots)
__device__ __forceinline__ void pa_fma2(uint64_t &acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pa_rope_lo(float x0, float x1, float c, float s) {
    return __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
}
__device__ __forceinline__ float pa_rope_hi(float x0, float x1, float c, float s) {
    return __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
}

// Rotated keys and plain values of the prompt into the caches: one thread per (row, kv head, four dimensions and their
// partners half a head further), 16-byte loads, 8-byte stores.
__global__ void __launch_bounds__(256) prefill_kv_store_kernel(const float *k, const float *v, long long k_row,
                                                               long long v_row, const float *cos_t, const float *sin_t,
                                                               int b, int t, int hkv, int dh, int horizon,
                                                               __nv_bfloat16 *k_cache, __nv_bfloat16 *v_cache) {
    chain_trigger();
    chain_wait();         // the projections come from the preceding kernel
    const int quads = dh >> 3, half = dh >> 1;
    const long long total = static_cast<long long>(b) * t * hkv * quads;
    for (long long idx = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x; idx < total;
         idx += static_cast<long long>(gridDim.x) * 256) {
        const int i = static_cast<int>(idx % quads) * 4;
        long long rest = idx / quads;
        const int head = static_cast<int>(rest % hkv);
        rest /= hkv;                                          // = bb * t + tt
        const int tt = static_cast<int>(rest % t), bb = static_cast<int>(rest / t);
        const float *kp = k + rest * k_row + head * dh + i, *vp = v + rest * v_row + head * dh + i;
        const float4 k0 = *reinterpret_cast<const float4 *>(kp), k1 = *reinterpret_cast<const float4 *>(kp + half);
        const float4 v0 = *reinterpret_cast<const float4 *>(vp), v1 = *reinterpret_cast<const float4 *>(vp + half);
        const float4 c = *reinterpret_cast<const float4 *>(cos_t + static_cast<size_t>(tt) * half + i);
        const float4 s = *reinterpret_cast<const float4 *>(sin_t + static_cast<size_t>(tt) * half + i);
        const size_t dst = ((static_cast<size_t>(bb) * hkv + head) * horizon + tt) * dh + i;
        auto pack = [](float x, float y) {
            const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
            return *reinterpret_cast<const uint32_t *>(&p);
        };
        uint2 a;
        a.x = pack(pa_rope_lo(k0.x, k1.x, c.x, s.x), pa_rope_lo(k0.y, k1.y, c.y, s.y));
        a.y = pack(pa_rope_lo(k0.z, k1.z, c.z, s.z), pa_rope_lo(k0.w, k1.w, c.w, s.w));
        *reinterpret_cast<uint2 *>(k_cache + dst) = a;
        a.x = pack(pa_rope_hi(k0.x, k1.x, c.x, s.x), pa_rope_hi(k0.y, k1.y, c.y, s.y));
        a.y = pack(pa_rope_hi(k0.z, k1.z, c.z, s.z), pa_rope_hi(k0.w, k1.w, c.w, s.w));
        *reinterpret_cast<uint2 *>(k_cache + dst + half) = a;
        a.x = pack(v0.x, v0.y);
        a.y = pack(v0.z, v0.w);
        *reinterpret_cast<uint2 *>(v_cache + dst) = a;
        a.x = pack(v1.x, v1.y);
        a.y = pack(v1.z, v1.w);
        *reinterpret_cast<uint2 *>(v_cache + dst + half) = a;
    }
}

// e / sum correctly rounded, from the correctly rounded reciprocal `inv` of sum: Markstein's theorem (IBM J. Res. Dev.
// 34(1), 1990) - q = e * inv is within an ulp, its remainder is exact in an FMA, and the corrected quotient rounds
// correctly (sum is in [1, 2^31) here). Quotients too small for an exact remainder take the plain division.
__device__ __forceinline__ float pa_quotient(float e, float sum, float inv) {
    const float q = __fmul_rn(e, inv);
    const float p = __fmaf_rn(__fmaf_rn(-q, sum, e), inv, q);
    return (e > 1e-30f || e == 0.f) ? p : __fdiv_rn(e, sum);
}
__device__ __forceinline__ void pa_bf16x8_to_float(const uint4 &v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __uint_as_float(w[i] << 16);
        f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

// One CTA = ROWS query rows of one (batch, head), head_dim 64, 8 threads per row; CTAs are numbered longest first.
// Score product: a warp owns four rows, its lane tx the keys 4 tx.. and 128 + 4 tx.. of a 256-key tile (32 FMA chains,
// in pairs); the keys stay BF16 in shared memory (half the bytes per read, two ALU operations per pair to widen).
// Value product: the threads of the first half own four rows 4 ty.. and four dimensions 4 tx.. each (16 FMA chains, in
// pairs); the values stay BF16 as well. Shared memory: rotated queries [64][ROWS], one key tile [64][256] or value tile
// [64][64] in BF16, scores [ROWS][sp].
template <int ROWS>
__global__ void __launch_bounds__(ROWS * 8, 1) prefill_attention_kernel(
    const float *q, long long q_row, const __nv_bfloat16 *k_cache, const __nv_bfloat16 *v_cache, const float *cos_t,
    const float *sin_t, int b, int t, int h, int hkv, int horizon, float scale, int sp, __nv_bfloat16 *out) {
    constexpr int DH = 64, HALF = 32, THREADS = ROWS * 8;
    constexpr int KDIMS = DH * PA_KEYS / THREADS;            // dimensions of a key that one thread stages (32 or 64)
    extern __shared__ __align__(128) uint8_t smem[];
    float *qt_s = reinterpret_cast<float *>(smem);           // [DH][ROWS]
    float *v_s = qt_s + DH * ROWS;
    uint16_t *k_s = reinterpret_cast<uint16_t *>(v_s);       // [DH][PA_KEYS], then [PA_VALUES][DH], BF16
    float *s_s = v_s + DH * PA_KEYS / 2;                     // [ROWS][sp]
    chain_trigger();
    chain_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pairs = b * h;
    const int nqt = (t + ROWS - 1) / ROWS;
    const int qt = nqt - 1 - static_cast<int>(blockIdx.x) / pairs;
    const int bh = static_cast<int>(blockIdx.x) % pairs, bb = bh / h, head = bh - bb * h, kvh = head / (h / hkv);
    const int row0 = qt * ROWS, kend = min(row0 + ROWS, t);       // this block sees the positions 0..kend-1
    const size_t cache0 = (static_cast<size_t>(bb) * hkv + kvh) * horizon * DH;

    // key tile of the next iteration in registers
    const int kpos = tid & (PA_KEYS - 1), kd0 = (tid / PA_KEYS) * KDIMS;
    uint4 kreg[KDIMS / 8];
    auto fetch_keys = [&](int kt) {
        const int pos = kt * PA_KEYS + kpos;
        const uint4 *src = reinterpret_cast<const uint4 *>(k_cache + cache0 + static_cast<size_t>(pos) * DH + kd0);
#pragma unroll
        for (int i = 0; i < KDIMS / 8; ++i) kreg[i] = pos < kend ? src[i] : make_uint4(0u, 0u, 0u, 0u);
    };
    fetch_keys(0);
    {
        // one row and four dimensions with their partners per thread (consecutive lanes: consecutive rows)
        const int r = tid & (ROWS - 1), d = 4 * (tid / ROWS), row = min(row0 + r, t - 1);
        const float *qp = q + (static_cast<size_t>(bb) * t + row) * q_row + static_cast<size_t>(head) * DH + d;
        const float4 x0 = *reinterpret_cast<const float4 *>(qp), x1 = *reinterpret_cast<const float4 *>(qp + HALF);
        const float4 c = *reinterpret_cast<const float4 *>(cos_t + static_cast<size_t>(row) * HALF + d);
        const float4 s = *reinterpret_cast<const float4 *>(sin_t + static_cast<size_t>(row) * HALF + d);
        float *lo = qt_s + d * ROWS + r, *hi = lo + HALF * ROWS;
        lo[0] = pa_rope_lo(x0.x, x1.x, c.x, s.x);
        lo[ROWS] = pa_rope_lo(x0.y, x1.y, c.y, s.y);
        lo[2 * ROWS] = pa_rope_lo(x0.z, x1.z, c.z, s.z);
        lo[3 * ROWS] = pa_rope_lo(x0.w, x1.w, c.w, s.w);
        hi[0] = pa_rope_hi(x0.x, x1.x, c.x, s.x);
        hi[ROWS] = pa_rope_hi(x0.y, x1.y, c.y, s.y);
        hi[2 * ROWS] = pa_rope_hi(x0.z, x1.z, c.z, s.z);
        hi[3 * ROWS] = pa_rope_hi(x0.w, x1.w, c.w, s.w);
    }

    auto widen = [](uint32_t w) { return pa_pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); };

    // ---- scores
    const int ktiles = (kend + PA_KEYS - 1) / PA_KEYS;
    for (int kt = 0; kt < ktiles; ++kt) {
#pragma unroll
        for (int i = 0; i < KDIMS / 8; ++i) {
            const uint32_t w[4] = {kreg[i].x, kreg[i].y, kreg[i].z, kreg[i].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                k_s[(kd0 + 8 * i + 2 * e) * PA_KEYS + kpos] = static_cast<uint16_t>(w[e]);
                k_s[(kd0 + 8 * i + 2 * e + 1) * PA_KEYS + kpos] = static_cast<uint16_t>(w[e] >> 16);
            }
        }
        __syncthreads();
        if (kt + 1 < ktiles) fetch_keys(kt + 1);
        const bool upper = kt * PA_KEYS + PA_KEYS / 2 < kend;         // some row sees the second half of the tile
        uint64_t acc[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[r][i] = 0ull;
        const float *qp = qt_s + warp * 4;
        const uint16_t *kp = k_s + 4 * lane;
        auto product = [&](auto both) {
#pragma unroll 8
            for (int d = 0; d < DH; ++d) {
                const float4 qv = *reinterpret_cast<const float4 *>(qp + d * ROWS);
                const uint2 k0 = *reinterpret_cast<const uint2 *>(kp + d * PA_KEYS);
                const uint64_t ka = widen(k0.x), kb = widen(k0.y);
                uint64_t kc = 0ull, kd = 0ull;
                if (decltype(both)::value) {
                    const uint2 k1 = *reinterpret_cast<const uint2 *>(kp + d * PA_KEYS + PA_KEYS / 2);
                    kc = widen(k1.x);
                    kd = widen(k1.y);
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float qs = r == 0 ? qv.x : r == 1 ? qv.y : r == 2 ? qv.z : qv.w;
                    const uint64_t qq = pa_pack2(qs, qs);
                    pa_fma2(acc[r][0], qq, ka);
                    pa_fma2(acc[r][1], qq, kb);
                    if (decltype(both)::value) {
                        pa_fma2(acc[r][2], qq, kc);
                        pa_fma2(acc[r][3], qq, kd);
                    }
                }
            }
        };
        if (upper) product(std::true_type{});
        else product(std::false_type{});
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float *dst = s_s + (warp * 4 + r) * sp + kt * PA_KEYS + 4 * lane;
            *reinterpret_cast<ulonglong2 *>(dst) = make_ulonglong2(acc[r][0], acc[r][1]);
            if (upper) *reinterpret_cast<ulonglong2 *>(dst + PA_KEYS / 2) = make_ulonglong2(acc[r][2], acc[r][3]);
        }
        __syncthreads();
    }

    // first value tile on its way while the probabilities are formed
    constexpr int VPIECES = PA_VALUES * DH / 8 / THREADS;    // 16-byte pieces of a value tile per thread (1 or 2)
    uint4 vreg[VPIECES];
    auto fetch_values = [&](int vt) {
#pragma unroll
        for (int i = 0; i < VPIECES; ++i) {
            const int id = tid + i * THREADS, pos = vt * PA_VALUES + (id >> 3);
            vreg[i] = pos < kend ? *reinterpret_cast<const uint4 *>(v_cache + cache0 + static_cast<size_t>(pos) * DH + 8 * (id & 7))
                                 : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    fetch_values(0);

    // ---- probabilities, a warp per row
    const int vtiles = (kend + PA_VALUES - 1) / PA_VALUES;
    for (int r = warp; r < ROWS; r += THREADS / 32) {
        const int row = row0 + r;
        if (row >= t) break;
        float *sr = s_s + r * sp;
        float m = __int_as_float(0xff800000);
        for (int j0 = 0; j0 <= row; j0 += 128) {             // (any order: a maximum has no rounding)
            const int j = j0 + 4 * lane;
            const float4 x = *reinterpret_cast<const float4 *>(sr + j);
            if (j <= row) m = fmaxf(m, __fmul_rn(x.x, scale));
            if (j + 1 <= row) m = fmaxf(m, __fmul_rn(x.y, scale));
            if (j + 2 <= row) m = fmaxf(m, __fmul_rn(x.z, scale));
            if (j + 3 <= row) m = fmaxf(m, __fmul_rn(x.w, scale));
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        // the first 512 positions stay in registers between the two passes
        float sum = 0.f, kept[16];
        const int span = vtiles * PA_VALUES;
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) kept[i + u] = 0.f;
            if (32 * i <= row) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int j = 32 * (i + u) + lane;
                    const float e = expf(__fsub_rn(__fmul_rn(sr[j], scale), m));
                    kept[i + u] = j <= row ? e : 0.f;        // (adding a zero changes nothing)
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) sum = __fadd_rn(sum, kept[i + u]);
            }
        }
        for (int j = 512 + lane; j <= row; j += 32) {
            const float e = expf(__fsub_rn(__fmul_rn(sr[j], scale), m));
            sum = __fadd_rn(sum, e);
            sr[j] = e;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, o));
        const float inv = __frcp_rn(sum);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (32 * i < span) sr[32 * i + lane] = pa_quotient(kept[i], sum, inv);
        for (int j = 512 + lane; j < span; j += 32) sr[j] = j <= row ? pa_quotient(sr[j], sum, inv) : 0.f;
    }

    // ---- values: the first half of the threads, four rows and four dimensions each (sixteen chains per thread)
    const int tx = tid & 15, ty = tid >> 4;
    const bool owner = tid < THREADS / 2;
    uint64_t o2[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r) o2[r][0] = o2[r][1] = 0ull;
    for (int vt = 0; vt < vtiles; ++vt) {
        if (vt) __syncthreads();                             // everyone is done with the previous tile
#pragma unroll
        for (int i = 0; i < VPIECES; ++i) {
            const int id = tid + i * THREADS;
            *reinterpret_cast<uint4 *>(k_s + (id >> 3) * DH + 8 * (id & 7)) = vreg[i];
        }
        __syncthreads();                                     // (the first one also orders the probabilities)
        if (vt + 1 < vtiles) fetch_values(vt + 1);
        if (!owner) continue;
        const float *pp = s_s + 4 * ty * sp + vt * PA_VALUES;
        const uint16_t *vp = k_s + 4 * tx;
#pragma unroll 4
        for (int j = 0; j < PA_VALUES; j += 4) {
            float4 p[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) p[r] = *reinterpret_cast<const float4 *>(pp + r * sp + j);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint2 vw = *reinterpret_cast<const uint2 *>(vp + (j + u) * DH);
                const uint64_t va = widen(vw.x), vb = widen(vw.y);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float f = u == 0 ? p[r].x : u == 1 ? p[r].y : u == 2 ? p[r].z : p[r].w;
                    const uint64_t f2 = pa_pack2(f, f);
                    pa_fma2(o2[r][0], f2, va);
                    pa_fma2(o2[r][1], f2, vb);
                }
            }
        }
    }
    if (!owner) return;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int row = row0 + 4 * ty + r;
        if (row < t) {
            float f0, f1, f2, f3;
            pa_unpack2(o2[r][0], f0, f1);
            pa_unpack2(o2[r][1], f2, f3);
            const __nv_bfloat162 a = __floats2bfloat162_rn(f0, f1), c = __floats2bfloat162_rn(f2, f3);
            *reinterpret_cast<uint2 *>(out + (static_cast<size_t>(bb) * t + row) * h * DH + static_cast<size_t>(head) * DH + 4 * tx) =
                make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&c));
        }
    }
}

// Query rows per CTA: 32 while two such CTAs (256 threads, scores of t positions each) share an SM's shared memory,
// which overlaps one CTA's staging with the other's products (16 prompts of 512, 32 heads: 726 us against 737 with one
// 64-row CTA); 64 while one 64-row CTA fits; 32 again for longer prompts.
static int prefill_rows(int t) { return t <= 512 ? 32 : t <= 640 ? 64 : 32; }
static int prefill_score_stride(int t) { return (t + 127) / 128 * 128 + 4; }
static size_t prefill_smem(int t) {
    const int rows = prefill_rows(t);
    return (static_cast<size_t>(64) * rows + 32 * PA_KEYS + static_cast<size_t>(rows) * prefill_score_stride(t)) * 4;
}

}  // namespace b200q

using namespace b200q;

extern "C" {

int b200q_prefill_attention_supported(int heads, int kv_heads, int head_dim, int t, int horizon, int cache_dtype,
                                      int out_dtype) {
    return head_dim == 64 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && t > 0 && horizon >= t &&
           horizon <= 1024 && cache_dtype == B200Q_BF16 && out_dtype == B200Q_BF16;
}

int b200q_prefill_attention(const float *q, const float *k, const float *v, int64_t q_row_stride, int64_t k_row_stride,
                            int64_t v_row_stride, const float *cos_table, const float *sin_table, int table_rows, int batch,
                            int t, int heads, int kv_heads, int head_dim, int horizon, void *k_cache, void *v_cache,
                            int cache_dtype, float scale, void *out, int out_dtype, void *stream) {
    if (!q || !k || !v || !cos_table || !sin_table || !k_cache || !v_cache || !out)
        return fail(B200Q_EINVAL, "prefill_attention: NULL pointer");
    if (batch <= 0 || t <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || horizon < t || table_rows < t ||
        !dtype_valid(cache_dtype) || !dtype_valid(out_dtype) || q_row_stride < static_cast<int64_t>(heads) * head_dim ||
        k_row_stride < static_cast<int64_t>(kv_heads) * head_dim || v_row_stride < static_cast<int64_t>(kv_heads) * head_dim)
        return fail(B200Q_EINVAL, "prefill_attention: bad argument");
    if (!b200q_prefill_attention_supported(heads, kv_heads, head_dim, t, horizon, cache_dtype, out_dtype))
        return fail(B200Q_EUNSUPPORTED, "prefill_attention: needs head_dim 64, BF16 caches and a horizon up to 1024");
    const uintptr_t all = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
                          reinterpret_cast<uintptr_t>(cos_table) | reinterpret_cast<uintptr_t>(sin_table) |
                          reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache) |
                          reinterpret_cast<uintptr_t>(out);
    if ((all & 15) || ((q_row_stride | k_row_stride | v_row_stride) & 3))
        return fail(B200Q_EUNSUPPORTED, "prefill_attention: operands and row strides must be 16-byte aligned");
    const int rows = prefill_rows(t);
    const long long ctas = static_cast<long long>((t + rows - 1) / rows) * batch * heads;
    if (ctas > 0x7fffffffLL) return fail(B200Q_EUNSUPPORTED, "prefill_attention: too many tiles");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const long long items = static_cast<long long>(batch) * t * kv_heads * (head_dim / 8);
    const int blocks = static_cast<int>(std::min<long long>((items + 255) / 256, 16LL * sm_count()));
    __nv_bfloat16 *kc = static_cast<__nv_bfloat16 *>(k_cache), *vc = static_cast<__nv_bfloat16 *>(v_cache);
    launch_chained(prefill_kv_store_kernel, dim3(blocks), dim3(256), 0, s, k, v, static_cast<long long>(k_row_stride),
                   static_cast<long long>(v_row_stride), cos_table, sin_table, batch, t, kv_heads, head_dim, horizon, kc, vc);
    const size_t smem = prefill_smem(t);
    auto kernel = rows == 64 ? prefill_attention_kernel<64> : prefill_attention_kernel<32>;
    if (cudaFuncSetAttribute(reinterpret_cast<const void *>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             PA_SMEM_LIMIT) != cudaSuccess) {
        cudaGetLastError();
        return fail(B200Q_ECUDA, "prefill_attention: shared memory opt-in failed");
    }
    launch_chained(kernel, dim3(static_cast<unsigned>(ctas)), dim3(rows * 8), smem, s, q,
                   static_cast<long long>(q_row_stride), kc, vc, cos_table, sin_table, batch, t, heads, kv_heads, horizon,
                   scale, prefill_score_stride(t), static_cast<__nv_bfloat16 *>(out));
    return check_launch("prefill_attention");
}

}  // extern "C"
