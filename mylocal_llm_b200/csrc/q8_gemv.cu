// Integer-dot mode: Q8_1 activations against Q4_K weights (decode GEMV, 1..4 tokens per pass).
//
// The FP32-lane and FP16-fragment kernels turn every 4-bit code into a floating-point value before
// it meets the activation; at HBM speed that decode, not the memory system, bounds the Q4_K GEMV.
// With activations quantised to int8 (Q8_1: blocks of 32 values with an FP16 scale d and the FP16
// sum of the block, mini_llm/ops/q8_1_gpu.py:30-58 of the reference) a masked nibble word is
// already the operand of a 4-way integer dot (dp4a), so a weight costs about one instruction.
// Arithmetic per 256-value super-block and token, as in the reference's mixed Q8 kernels
// (mini_llm/ops/mixed_q8_gpu.py:86-139): per sub-block s
//     sd += dx_s * float(dot_s * sc_s),   sm += dx_s * float(sum_s * mn_s)
// with dot_s = integer dot of codes and activation codes, sum_s = integer sum of the activation
// codes, and the super-block contributes dw * sd - dmin * sm. Every integer quantity is exact; the
// FP32 partial sums are added in this kernel's own order (lane, K part), so results agree with the
// reference formula to FP32 rounding, not bit for bit. The mode changes numerics with respect to
// FP32 activations (int8 rounding of x: relative 1/254 of a block's largest value) and is therefore
// opt-in.
//
// Layout of the work: as the direct-load kernel (mma_direct.cuh). A CTA of 16 warps = rg row groups
// of 16 rows x kp parts of K; a warp streams the packed bytes of its rows' super-blocks with 128-bit
// loads (GGUF layout or the Q4_K tile layout), one item ahead in registers; lane (g, tig) handles
// rows g and g+8 and, of every sub-block, the values 4 tig.. and 16 + 4 tig.. (the words of SuperBlockRegs). The int8
// activations of the whole K range sit in shared memory, the sixteen words of a lane in a super-block side by side, with
// dx and dx * (sum of a block's codes) beside them.
#include "mma_direct.cuh"

namespace b200q {

constexpr int Q8G_WARPS = 16;
constexpr int Q8G_THREADS = Q8G_WARPS * 32;

struct Q8GemvArgs {
    const uint8_t *w;
    int tiled;
    int n, k, m;
    long long row_bytes;
    const uint8_t *xq;        // Q8_1 blocks [m, k/32] of 36 bytes
    void *y;
    int y_dtype;
    int kp, rg;               // K parts and row groups per CTA (kp * rg == 16)
};

// ---------------------------------------------------------------------------------------------
// Q8_1 quantiser: one warp per block of 32 values, IEEE arithmetic (the reference's "ieee" control:
// no fast-math). d32 = bounded(max|x| / 127); code = 0 for an all-zero block, else round-half-away
// (x / d32) clamped to +-127; stores half(d32), half(bounded(sum x)) with the sum taken by the
// xor butterfly 16, 8, 4, 2, 1 (lane 0's value), then the 32 codes.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float q8_bounded(float x) { return fabsf(x) > 65504.f ? copysignf(65504.f, x) : x; }

__global__ void q8_1_quantize_kernel(const void *x, int x_dtype, long long total, uint8_t *out) {
    chain_trigger();
    chain_wait();
    const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= total) return;                       // total is a multiple of 32: whole warps leave together
    const float v = load_as_float(x, x_dtype, static_cast<size_t>(i));
    float a = fabsf(v), s = v;
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, off));
        s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, off));
    }
    const float d = q8_bounded(__fdiv_rn(a, 127.f));
    float q = a == 0.f ? 0.f : roundf(__fdiv_rn(v, d));
    q = q > 127.f ? 127.f : q < -127.f ? -127.f : q;
    uint8_t *blk = out + (i >> 5) * 36;
    blk[4 + (i & 31)] = static_cast<uint8_t>(static_cast<int8_t>(q));
    if ((i & 31) == 0) {
        *reinterpret_cast<__half *>(blk) = __float2half_rn(q8_bounded(d));
        *reinterpret_cast<__half *>(blk + 2) = __float2half_rn(q8_bounded(s));
    }
}

// ---------------------------------------------------------------------------------------------
// GEMV kernel
// ---------------------------------------------------------------------------------------------
template <int MT, bool Q5>
__global__ void __launch_bounds__(Q8G_THREADS, 1) q4k_q8_gemv_kernel(const Q8GemvArgs a) {
    constexpr int QB = Q5 ? 176 : 144;                        // bytes of a native super-block
    constexpr int TILE = direct_tile_bytes<Q5>();              // bytes of a 16-row tile (b200q_q4k_retile / b200q_q5k_retile)
    chain_trigger();
    extern __shared__ __align__(16) uint8_t smem[];
    const int nblk = a.k >> 5, nsb = a.k >> 8;
    // shared memory: codes [MT][k] | dx [MT][nblk] | dxs [MT][nblk] | partial [2][16 warps][16 rows][MT]
    int8_t *qs_s = reinterpret_cast<int8_t *>(smem);
    float *dx_s = reinterpret_cast<float *>(smem + static_cast<size_t>(MT) * a.k);
    float *dxs_s = dx_s + MT * nblk;
    float *partial = dxs_s + MT * nblk;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int rgi = warp / a.kp, kpi = warp - rgi * a.kp;
    const int rows_per_block = 16 * a.rg;
    const int total_blocks = (a.n + rows_per_block - 1) / rows_per_block;
    const int blk_begin = static_cast<int>(static_cast<long long>(total_blocks) * blockIdx.x / gridDim.x);
    const int blk_end = static_cast<int>(static_cast<long long>(total_blocks) * (blockIdx.x + 1) / gridDim.x);

    auto issue = [&](int row0, int sb, SuperBlockRegs<Q5> &it) {
        if (a.tiled) {
            const int group = min((row0 >> 4) + rgi, (a.n >> 4) - 1);
            load_superblock_tiled<Q5>(it, a.w + (static_cast<size_t>(group) * nsb + sb) * TILE, lane);
        } else {
            load_superblock<Q5>(it, a.w + static_cast<size_t>(min(row0 + 16 * rgi + g, a.n - 1)) * a.row_bytes + sb * QB,
                                a.w + static_cast<size_t>(min(row0 + 16 * rgi + g + 8, a.n - 1)) * a.row_bytes + sb * QB, tig);
        }
    };
    const int sb_count = kpi < nsb ? (nsb - kpi + a.kp - 1) / a.kp : 0;     // this warp's super-blocks: kpi, kpi+kp, ..
    SuperBlockRegs<Q5> cur, nxt;
    if (blk_begin < blk_end && sb_count > 0) issue(blk_begin * rows_per_block, kpi, nxt);   // weights: before the wait

    chain_wait();                 // the activation blocks come from the preceding kernel (the quantiser)
    // stage the activations: 36-byte blocks -> 32-byte code blocks + scales
    for (int i = tid; i < MT * nblk; i += Q8G_THREADS) {
        const int t = i / nblk, b = i - t * nblk;
        const bool live = t < a.m;
        const uint8_t *src = a.xq + (static_cast<size_t>(t) * nblk + b) * 36;
        uint32_t wds[8];
        int sum = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            wds[j] = live ? *reinterpret_cast<const uint32_t *>(src + 4 + 4 * j) : 0u;
            sum = __dp4a(0x01010101, static_cast<int>(wds[j]), sum);
        }
        // block b & 7 of its super-block: words q and q + 4 belong to lane q of a quad
        uint8_t *dst = reinterpret_cast<uint8_t *>(qs_s) + static_cast<size_t>(t) * a.k + 256 * (b >> 3) + 8 * (b & 7);
#pragma unroll
        for (int q = 0; q < 4; ++q) *reinterpret_cast<uint2 *>(dst + 64 * q) = make_uint2(wds[q], wds[q + 4]);
        const float dx = live ? __half2float(*reinterpret_cast<const __half *>(src)) : 0.f;
        dx_s[i] = dx;
        dxs_s[i] = dx * static_cast<float>(sum);
    }
    __syncthreads();
    if (blk_begin >= blk_end) return;

    int pbuf = 0;
    for (int blk = blk_begin; blk < blk_end; ++blk) {
        const int row0 = blk * rows_per_block;
        float tot_a[MT], tot_b[MT];
#pragma unroll
        for (int t = 0; t < MT; ++t) tot_a[t] = tot_b[t] = 0.f;
        for (int it = 0; it < sb_count; ++it) {
            cur = nxt;
            if (it + 1 < sb_count) issue(row0, kpi + (it + 1) * a.kp, nxt);
            else if (blk + 1 < blk_end) issue(row0 + rows_per_block, kpi, nxt);
            const int sb = kpi + it * a.kp;
            if (!a.tiled) transpose_native<Q5>(cur, tig);
            // the eight scales of a row, and the minima of the two sub-blocks whose sums this lane adds (2 tig, 2 tig + 1)
            auto scales = [&](const uint4 &hd, uint32_t (&sc)[2], float (&mn)[2], float &d, float &dmin) {
                d = half_bits_to_float(hd.x & 0xffffu);
                dmin = half_bits_to_float(hd.x >> 16);
                sc[0] = hd.y & 0x3f3f3f3fu;
                sc[1] = (hd.w & 0x0f0f0f0fu) | ((hd.y >> 2) & 0x30303030u);
                const uint32_t m = ((tig & 2) ? ((hd.w >> 4) & 0x0f0f0f0fu) | ((hd.z >> 2) & 0x30303030u) : hd.z & 0x3f3f3f3fu) >> (16 * (tig & 1));
                mn[0] = static_cast<float>(m & 0xffu);
                mn[1] = static_cast<float>((m >> 8) & 0xffu);
            };
            uint32_t sc_a[2], sc_b[2];
            float mn_a[2], mn_b[2], d_a, dm_a, d_b, dm_b;
            scales(cur.hd[0], sc_a, mn_a, d_a, dm_a);
            scales(cur.hd[1], sc_b, mn_b, d_b, dm_b);
            const uint32_t wa[8] = {cur.q[0].x, cur.q[0].y, cur.q[0].z, cur.q[0].w, cur.q[1].x, cur.q[1].y, cur.q[1].z, cur.q[1].w};
            const uint32_t wb[8] = {cur.q[2].x, cur.q[2].y, cur.q[2].z, cur.q[2].w, cur.q[3].x, cur.q[3].y, cur.q[3].z, cur.q[3].w};
            const uint32_t ha[2] = {cur.h[0].x, cur.h[0].y}, hb[2] = {cur.h[1].x, cur.h[1].y};
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                float sd_a = 0.f, sd_b = 0.f;
                const uint4 *up = reinterpret_cast<const uint4 *>(qs_s + static_cast<size_t>(t) * a.k + 256 * sb + 64 * tig);
                const float4 *dp = reinterpret_cast<const float4 *>(dx_s + t * nblk + sb * 8);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const uint4 u = up[c];                                    // sub-block 2c: words j = 0, 1; then 2c + 1
                    const float4 dx4 = dp[c >> 1];
#pragma unroll
                    for (int nib = 0; nib < 2; ++nib) {
                        const int s = 2 * c + nib;
                        const int uw[2] = {static_cast<int>(nib ? u.z : u.x), static_cast<int>(nib ? u.w : u.y)};
                        int dot_a = 0, dot_b = 0;
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            uint32_t ua = (wa[2 * c + j] >> (4 * nib)) & 0x0f0f0f0fu, ub = (wb[2 * c + j] >> (4 * nib)) & 0x0f0f0f0fu;
                            if (Q5) {                          // bit s of the fifth-bit byte -> bit 4 of the code
                                ua |= ((ha[j] >> s) << 4) & 0x10101010u;
                                ub |= ((hb[j] >> s) << 4) & 0x10101010u;
                            }
                            dot_a = __dp4a(static_cast<int>(ua), uw[j], dot_a);
                            dot_b = __dp4a(static_cast<int>(ub), uw[j], dot_b);
                        }
                        const int sh = 8 * (s & 3);
                        const float dx = (s & 3) == 0 ? dx4.x : (s & 3) == 1 ? dx4.y : (s & 3) == 2 ? dx4.z : dx4.w;
                        // |dot * sc| <= 8 * 31 * 127 * 63 < 2^22: integer -> float by adding it to the bits of 1.5 * 2^23
                        const int va = dot_a * static_cast<int>((sc_a[s >> 2] >> sh) & 0xffu) + 0x4b400000;
                        const int vb = dot_b * static_cast<int>((sc_b[s >> 2] >> sh) & 0xffu) + 0x4b400000;
                        sd_a = fmaf(dx, __int_as_float(va) - 12582912.0f, sd_a);
                        sd_b = fmaf(dx, __int_as_float(vb) - 12582912.0f, sd_b);
                    }
                }
                const float2 dxs = *reinterpret_cast<const float2 *>(dxs_s + t * nblk + sb * 8 + 2 * tig);
                tot_a[t] += d_a * sd_a - dm_a * fmaf(dxs.x, mn_a[0], dxs.y * mn_a[1]);
                tot_b[t] += d_b * sd_b - dm_b * fmaf(dxs.x, mn_b[0], dxs.y * mn_b[1]);
            }
        }
        // the four lanes of a quad hold the four quarters of each sub-block pair: add them, then the K parts
#pragma unroll
        for (int t = 0; t < MT; ++t) {
            tot_a[t] += __shfl_xor_sync(0xffffffffu, tot_a[t], 1);
            tot_a[t] += __shfl_xor_sync(0xffffffffu, tot_a[t], 2);
            tot_b[t] += __shfl_xor_sync(0xffffffffu, tot_b[t], 1);
            tot_b[t] += __shfl_xor_sync(0xffffffffu, tot_b[t], 2);
        }
        // The K parts of a row group are added by that group's own warps behind a barrier of just those warps, with
        // the partial sums double-buffered: no CTA-wide stop per row block (a warp writes buffer b again only after
        // its group's next barrier, which every reader of b has reached by then).
        float *pb = partial + pbuf * (Q8G_WARPS * 16 * MT);
        if (tig == 0) {
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                pb[(warp * 16 + g) * MT + t] = tot_a[t];
                pb[(warp * 16 + g + 8) * MT + t] = tot_b[t];
            }
        }
        const int group_threads = a.kp * 32;
        if (a.kp == 1) __syncwarp();
        else named_barrier_sync(2 + rgi, group_threads);          // kp >= 2: at most 8 row groups, ids 2..9
        for (int o = kpi * 32 + lane; o < 16 * MT; o += group_threads) {
            const int t = o % MT, r = o / MT;
            const int orow = row0 + 16 * rgi + r;
            if (orow >= a.n || t >= a.m) continue;
            float sum = 0.f;
            for (int kq = 0; kq < a.kp; ++kq) sum += pb[((rgi * a.kp + kq) * 16 + r) * MT + t];
            store_from_float(a.y, a.y_dtype, static_cast<size_t>(t) * a.n + orow, sum);
        }
        pbuf ^= 1;
    }
}

}  // namespace b200q

using namespace b200q;

extern "C" int b200q_quantize_q8_1(const void *x, int x_dtype, int rows, int k, void *out, void *stream) {
    if (!x || !out) return fail(B200Q_EINVAL, "quantize_q8_1: NULL pointer");
    if (!dtype_valid(x_dtype) || rows <= 0 || k <= 0 || k % 32) return fail(B200Q_EINVAL, "quantize_q8_1: bad argument (K %% 32)");
    const long long total = static_cast<long long>(rows) * k;
    const unsigned blocks = static_cast<unsigned>((total + 255) / 256);
    launch_chained(q8_1_quantize_kernel, dim3(blocks), dim3(256), 0, static_cast<cudaStream_t>(stream), x, x_dtype, total,
                   static_cast<uint8_t *>(out));
    return check_launch("quantize_q8_1");
}

extern "C" int b200q_gemv_q8_1(const void *w, int fmt, int n, int k, const void *xq, int m, void *y, int y_dtype,
                               void *stream) {
    if (!w || !xq || !y) return fail(B200Q_EINVAL, "gemv_q8_1: NULL pointer");
    const bool tiled = fmt == B200Q_Q4_K_TILED || fmt == B200Q_Q5_K_TILED;
    const bool q5 = fmt == B200Q_Q5_K || fmt == B200Q_Q5_K_TILED;
    if (fmt != B200Q_Q4_K && fmt != B200Q_Q5_K && !tiled)
        return fail(B200Q_EUNSUPPORTED, "gemv_q8_1: the integer-dot mode reads Q4_K / Q5_K (GGUF or tile layout)");
    if (!dtype_valid(y_dtype) || n <= 0 || m <= 0 || k <= 0 || k % 256) return fail(B200Q_EINVAL, "gemv_q8_1: bad shape n=%d k=%d m=%d", n, k, m);
    if (tiled && n % 16) return fail(B200Q_EINVAL, "gemv_q8_1: the tile layout needs rows in multiples of 16");
    if ((reinterpret_cast<uintptr_t>(w) & 15) || (reinterpret_cast<uintptr_t>(xq) & 3))
        return fail(B200Q_EUNSUPPORTED, "gemv_q8_1: weights must be 16-byte and activation blocks 4-byte aligned");
    const int nsb = k / 256;
    for (int t0 = 0; t0 < m;) {
        const int mt = m - t0 >= 4 ? 4 : m - t0 >= 2 ? 2 : 1;        // tokens of this pass (1, 2 or 4)
        Q8GemvArgs a{};
        a.w = static_cast<const uint8_t *>(w); a.tiled = tiled ? 1 : 0; a.n = n; a.k = k;
        a.m = mt;
        a.row_bytes = static_cast<long long>(nsb) * (q5 ? 176 : 144);
        a.xq = static_cast<const uint8_t *>(xq) + static_cast<size_t>(t0) * (k / 32) * 36;
        a.y = static_cast<uint8_t *>(y) + static_cast<size_t>(t0) * n * dtype_size(y_dtype);
        a.y_dtype = y_dtype;
        // K parts: as few as still give every SM about six row blocks (see the direct-load kernel)
        int kp = 1;
        auto blocks_for = [&](int parts) { return (static_cast<long long>(n) + 16 * (Q8G_WARPS / parts) - 1) / (16 * (Q8G_WARPS / parts)); };
        while (kp * 2 <= Q8G_WARPS && kp * 2 <= nsb && blocks_for(kp) < 6LL * sm_count()) kp *= 2;
        a.kp = kp; a.rg = Q8G_WARPS / kp;
        const size_t smem = static_cast<size_t>(mt) * k + static_cast<size_t>(mt) * (k / 32) * 8 + 2 * Q8G_WARPS * 16 * mt * 4;
        if (smem > 200 * 1024) return fail(B200Q_EUNSUPPORTED, "gemv_q8_1: K=%d too large for the activation tile", k);
        auto fn = q5 ? (mt == 4 ? q4k_q8_gemv_kernel<4, true> : mt == 2 ? q4k_q8_gemv_kernel<2, true> : q4k_q8_gemv_kernel<1, true>)
                     : (mt == 4 ? q4k_q8_gemv_kernel<4, false> : mt == 2 ? q4k_q8_gemv_kernel<2, false> : q4k_q8_gemv_kernel<1, false>);
        cudaError_t err = cudaFuncSetAttribute(reinterpret_cast<const void *>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (err != cudaSuccess) {
            cudaGetLastError();
            return fail(B200Q_ECUDA, "gemv_q8_1: shared memory opt-in failed: %s", cudaGetErrorString(err));
        }
        int grid = sm_count();
        const long long blocks = blocks_for(kp);
        if (blocks < grid) grid = static_cast<int>(blocks);
        launch_chained(fn, dim3(grid), dim3(Q8G_THREADS), smem, static_cast<cudaStream_t>(stream), a);
        int rc = check_launch("gemv_q8_1");
        if (rc) return rc;
        t0 += mt;
    }
    return B200Q_OK;
}
