// Grouped gate/up and down projections over token images (grouped_stream.cuh): kernels, the hidden-activation images and
// the launches.
#include <cstdlib>
#include <cstring>

#include "grouped_stream.cuh"
#include "mma_host.h"

namespace b200q {

// Gate/up + SwiGLU over Q4_K / Q5_K tiles: hbuf[sorted assignment, row].
template <bool Q5, int NTERMS>
__global__ void __launch_bounds__(GS_THREADS, 1) grouped_gate_up_kernel(const GroupedArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    chain_trigger();
    chain_wait();                 // plan and images come from preceding kernels
    constexpr int TILE = direct_tile_bytes<Q5>();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int team = warp / a.kp, kpi = warp - team * a.kp;
    float *partial = reinterpret_cast<float *>(smem + GS_CTRL_BYTES);
    const int plane = a.nsb * 512, sums_off = NTERMS * plane, scale_off = sums_off + a.nsb * 32;
    int pbuf = 0;
    auto work = [&](int seg, int group, const uint8_t *buf, TileStream<TILE, true> &stream) -> bool {
        const int begin = a.seg_begin[seg], count = min(a.seg_count[seg], 8);
        const uint8_t *image = buf + g * a.smem_stride;
        const uint8_t *fp = image + tig * 8 + kpi * 512, *xp = image + sums_off + tig * 4 + kpi * 32;
        float tg[1][4] = {{0.f, 0.f, 0.f, 0.f}}, tu[1][4] = {{0.f, 0.f, 0.f, 0.f}};
        auto frag = [&](int, int fi, int p) { return *reinterpret_cast<const uint2 *>(fp + fi * 32 + p * plane); };
        auto sums = [&](int, int term) { return *reinterpret_cast<const uint32_t *>(xp + term * 16); };
        bool ok = true;
        for (int sb = kpi; sb < a.nsb; sb += a.kp) {
            SuperBlockRegs<Q5> ra, rb;
            const uint8_t *tile;
            if (!(ok = stream.next(tile))) break;
            read_superblock_tile<Q5>(ra, rb, tile, lane);
            stream.refill(lane);
            superblock_mma<Q5, NTERMS, 1>(ra, rb, frag, sums, tig, tg);
            if (!(ok = stream.next(tile))) break;
            read_superblock_tile<Q5>(ra, rb, tile, lane);
            stream.refill(lane);
            superblock_mma<Q5, NTERMS, 1>(ra, rb, frag, sums, tig, tu);
            fp += a.kp * 512;
            xp += a.kp * 32;
        }
        float v[8] = {tg[0][0], tg[0][1], tg[0][2], tg[0][3], tu[0][0], tu[0][1], tu[0][2], tu[0][3]};
        if (!add_parts(v, partial, pbuf, a.kp, team, kpi, warp, lane) || !ok) return ok;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = 2 * tig + e;
            if (t < count) {
                const float inv = *reinterpret_cast<const float *>(buf + t * a.smem_stride + scale_off + 4);
                float *dst = a.y + static_cast<size_t>(begin + t) * a.n + group * 16 + g;
                dst[0] = swiglu_f32(v[e] * inv, v[4 + e] * inv);
                dst[8] = swiglu_f32(v[2 + e] * inv, v[6 + e] * inv);
            }
        }
        return true;
    };
    grouped_walk<false, TILE, true>(a, smem, work);
}

// Down projection over Q6_K / Q8_0 tiles of FP32 hidden activations (two FP16 planes), times the route weight.
template <typename T>
__global__ void __launch_bounds__(GS_THREADS, 1) grouped_down_kernel(const GroupedArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    chain_trigger();
    chain_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int team = warp / a.kp, kpi = warp - team * a.kp;
    float *partial = reinterpret_cast<float *>(smem + GS_CTRL_BYTES);
    const int plane = a.nsb * 512, scale_off = 2 * plane;
    int pbuf = 0;
    auto work = [&](int seg, int group, const uint8_t *buf, TileStream<T::BYTES, false> &stream) -> bool {
        const int begin = a.seg_begin[seg], count = min(a.seg_count[seg], 8);
        // the lane's two tokens: route weight and output row (used at the end)
        float route[2] = {0.f, 0.f};
        float *out[2] = {nullptr, nullptr};
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = 2 * tig + e;
            if (t < count) {
                const int flat = a.order[begin + t];
                route[e] = a.route[flat];
                out[e] = term_row_pointer(a.y, a.y_table, a.rows_per_rank, a.n, a.flat_rows ? flat : begin + t);
            }
        }
        const uint8_t *fp = buf + g * a.smem_stride + tig * 16 + kpi * 512;
        float tot[1][4] = {{0.f, 0.f, 0.f, 0.f}};
        auto frag = [&](int, int pair, int p) { return fp + pair * 64 + p * plane; };
        bool ok = true;
        for (int sb = kpi; sb < a.nsb; sb += a.kp) {
            typename T::Regs r;
            const uint8_t *tile;
            if (!(ok = stream.next(tile))) break;
            T::read(r, tile, lane);
            stream.refill(lane);
            T::template mma<2, 1, 8>(r, frag, tot);
            fp += a.kp * 512;
        }
        if (!add_parts(tot[0], partial, pbuf, a.kp, team, kpi, warp, lane) || !ok) return ok;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = 2 * tig + e;
            if (t < count) {
                const float inv = *reinterpret_cast<const float *>(buf + t * a.smem_stride + scale_off + 4);
                float *dst = out[e] + group * 16 + g;
                dst[0] = tot[0][e] * inv * route[e];
                dst[8] = tot[0][2 + e] * inv * route[e];
            }
        }
        return true;
    };
    grouped_walk<true, T::BYTES, false>(a, smem, work);
}

// Image of one row of FP32 hidden activations, a warp per row: the power-of-two scale and the two FP16 planes of
// prepare_fragments, pairs of fragments of the four lanes of a quad side by side (64 bytes), then scale and inverse.
__global__ void __launch_bounds__(256) hidden_image_kernel(const float *h, int rows, int k, uint8_t *images, int image_bytes) {
    chain_trigger();
    chain_wait();
    const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const float *src = h + static_cast<size_t>(row) * k;
    uint8_t *dst = images + static_cast<size_t>(row) * image_bytes;
    constexpr int KEEP = 8;                              // chunks of four values per lane kept between the passes
    float4 kept[KEEP];
    float amax = 0.f;
    const int chunks = k >> 2;
#pragma unroll
    for (int i = 0; i < KEEP; ++i) {
        const int c = lane + 32 * i;
        kept[i] = c < chunks ? *reinterpret_cast<const float4 *>(src + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    auto grow = [&](const float4 &v) {
        // integer maxima of the magnitudes' bits: a NaN stays the largest, as in prepare_fragments
        const uint32_t m = max(max(__float_as_uint(fabsf(v.x)), __float_as_uint(fabsf(v.y))), max(__float_as_uint(fabsf(v.z)), __float_as_uint(fabsf(v.w))));
        amax = __uint_as_float(max(__float_as_uint(amax), m));
    };
#pragma unroll
    for (int i = 0; i < KEEP; ++i) grow(kept[i]);
    for (int c = lane + 32 * KEEP; c < chunks; c += 32) grow(*reinterpret_cast<const float4 *>(src + 4 * c));
    amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(amax)));
    float s = 1.0f;
    if (amax > 0.f && amax < __int_as_float(0x7f800000)) {
        int e;
        frexpf(amax, &e);
        s = ldexpf(1.0f, min(14 - e, 100));
    }
    const int plane = k * 2;
    auto put = [&](int c, const float4 &v4) {
        const float v[4] = {v4.x, v4.y, v4.z, v4.w};
        unsigned short hi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float sv = v[i] * s;
            const __half hv = __float2half_rn(sv);
            hi[i] = __half_as_ushort(hv);
            lo[i] = __half_as_ushort(__float2half_rn(sv - __half2float(hv)));
        }
        // positions 4c..: pair c >> 3, quad lane c & 3, fragment (c >> 2) & 1
        uint8_t *at = dst + (c >> 3) * 64 + (c & 3) * 16 + ((c >> 2) & 1) * 8;
        *reinterpret_cast<uint2 *>(at) = make_uint2(hi[0] | (static_cast<uint32_t>(hi[2]) << 16), hi[1] | (static_cast<uint32_t>(hi[3]) << 16));
        *reinterpret_cast<uint2 *>(at + plane) = make_uint2(lo[0] | (static_cast<uint32_t>(lo[2]) << 16), lo[1] | (static_cast<uint32_t>(lo[3]) << 16));
    };
#pragma unroll
    for (int i = 0; i < KEEP; ++i)
        if (lane + 32 * i < chunks) put(lane + 32 * i, kept[i]);
    for (int c = lane + 32 * KEEP; c < chunks; c += 32) put(c, *reinterpret_cast<const float4 *>(src + 4 * c));
    if (lane == 0) *reinterpret_cast<float4 *>(dst + 2 * plane) = make_float4(s, 1.0f / s, 0.f, 0.f);
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
// Warps per 16-row group (parts of K). A CTA deals its row groups to 16 / kp teams: the last round is on average half
// empty, which costs 1 / (2 kp) of a round, while every doubling of kp adds a meeting of the team per group (about 2 % of a
// group of eight super-blocks). About 65 % of the bound are segments that exist (measured 62-73 % for 16 to 256 tokens over
// 512 experts).
static int grouped_kp(int n, int nsb, int max_segments) {
    const double groups = 0.65 * max_segments * (n / 16) / sm_count();
    int best = 1;
    double cost = 1e30;
    for (int kp = 1; kp <= 8 && kp <= nsb; kp *= 2) {
        const double c = (groups * kp / GS_WARPS + 0.5) / kp * (1.0 + 0.16 * (kp - 1) / nsb);
        if (c < cost) {
            cost = c;
            best = kp;
        }
    }
    return best;
}

// Shared memory of a launch: false when two segment buffers and two tiles per warp do not fit; what is left goes to the
// tile rings first. row_bytes: what the four lanes of a token read side by side.
static bool grouped_plan(int kp, int image_bytes, int row_bytes, int tile_bytes, GroupedArgs &a, size_t &smem) {
    a.kp = kp;
    a.image_bytes = image_bytes;
    a.smem_stride = (image_bytes + 127 - row_bytes) / 128 * 128 + row_bytes;
    a.off_ring = GS_CTRL_BYTES + (kp > 1 ? GS_PART_BYTES : 0);
    const int room = MM_SMEM_LIMIT - a.off_ring, buf_bytes = 8 * a.smem_stride, ring_bytes = GS_WARPS * tile_bytes;
    a.ring = (room - 2 * buf_bytes) / ring_bytes;
    if (a.ring > GS_MAX_RING) a.ring = GS_MAX_RING;
    if (room < 2 * buf_bytes || a.ring < 2) return false;
    a.bufs = (room - a.ring * ring_bytes) / buf_bytes;
    if (a.bufs > GS_MAX_BUFS) a.bufs = GS_MAX_BUFS;
    a.off_bufs = a.off_ring + a.ring * ring_bytes;
    smem = a.off_bufs + static_cast<size_t>(a.bufs) * 8 * a.smem_stride;
    return true;
}

static bool plan_gate_up(int fmt, int n, int k, int x_dtype, int max_segments, GroupedArgs &a, size_t &smem) {
    const int image_bytes = direct_token_image_bytes(k, x_dtype);
    return image_bytes && n % 16 == 0 &&
           grouped_plan(grouped_kp(n, k / 256, max_segments), image_bytes, 32, fmt == B200Q_Q5_K ? Q5T_TILE_BYTES : Q4T_TILE_BYTES, a, smem);
}
static bool plan_down(int fmt, int n, int k, int max_segments, GroupedArgs &a, size_t &smem) {
    const int image_bytes = hidden_image_bytes(k);
    return image_bytes && n % 16 == 0 &&
           grouped_plan(grouped_kp(n, k / 256, max_segments), image_bytes, 64, fmt == B200Q_Q8_0_TILED ? Q8T_TILE_BYTES : Q6T_TILE_BYTES, a, smem);
}

// Where streaming, the images' conversion included, is the faster one (device time of the two launches against the
// block-structured kernel's, 148 SMs; nine shapes of 64-512 experts, 2-512 tokens):
//   gate/up from 113 segments and 162 tiles of each matrix per SM on: 512 experts of 512 x 2048, top 11, BF16: 8 tokens
//     (99 segments) 1.02, 16 (198) 0.90, 64 0.91, 256 0.93; 64 of 2048 x 2048: 84 segments 1.06, 125 0.93; 128 of
//     512 x 1024: 169 segments (146 tiles) 1.06, 189 (163) 0.91.
//   down from 41 segments on, up to 1024 columns: 512 of 1024 x 512 (Q6_K): 37 segments 1.21, 49 0.86, 688 0.88; 64 of
//     2048 x 1024: 45 segments 0.85; wider rows leave two tiles per warp and lose (64 of 1024 x 1536: 1.07-1.15).
//   Q8_0 (tiles a third larger, less to decode) with one super-block per row 0.92-1.06, with two above 256 segments
//     0.96-1.04: left to the block-structured kernel; 512 of 2048 x 512: 198 segments 0.83, 128 of 2048 x 768: 0.70-0.99.
// B200Q_GROUPED_STREAM=1 / 0: wherever a plan fits / never (tests, A/B measurements), read at every call.
static int stream_override() {
    const char *v = std::getenv("B200Q_GROUPED_STREAM");
    return v && (v[0] == '0' || v[0] == '1') ? v[0] - '0' : -1;
}
int grouped_gate_up_kp(int fmt, int n, int k, int x_dtype, int max_segments) {
    GroupedArgs a{};
    size_t smem = 0;
    const int forced = stream_override();
    if (forced == 0) return 0;
    if (forced < 0 && (max_segments <= 112 || static_cast<long long>(max_segments) * (n / 16) * (k / 256) < 162LL * sm_count())) return 0;
    return plan_gate_up(fmt, n, k, x_dtype, max_segments, a, smem) ? a.kp : 0;
}
int grouped_down_kp(int fmt, int n, int k, int max_segments) {
    GroupedArgs a{};
    size_t smem = 0;
    const int forced = stream_override();
    if (forced == 0) return 0;
    if (forced < 0 && (max_segments <= 40 || k > 1024)) return 0;
    if (forced < 0 && fmt == B200Q_Q8_0_TILED && (k < 512 || (k == 512 && max_segments > 256))) return 0;
    return plan_down(fmt, n, k, max_segments, a, smem) ? a.kp : 0;
}

int hidden_image_bytes(int k) { return k > 0 && k % 256 == 0 && k <= 8192 ? k * 4 + 16 : 0; }

int hidden_images(const float *h, int rows, int k, void *images, cudaStream_t stream) {
    if (hidden_image_bytes(k) == 0 || ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(images)) & 15))
        return fail(B200Q_EUNSUPPORTED, "hidden images: f must be a multiple of 256, buffers 16-byte aligned");
    launch_chained(hidden_image_kernel, dim3((rows + 7) / 8), dim3(256), 0, stream, h, rows, k, static_cast<uint8_t *>(images),
                   hidden_image_bytes(k));
    return check_launch("hidden images");
}

static bool grouped_args(const MmaRequest &q, GroupedArgs &a) {
    a.wa = q.wa; a.wb = q.wb; a.stride_a = q.stride_a; a.stride_b = q.stride_b;
    a.table_a = q.table_a; a.table_b = q.table_b;
    a.n = q.n; a.nsb = q.k / 256;
    a.images = static_cast<const uint8_t *>(q.images);
    a.topk = q.topk; a.order = q.order; a.seg_expert = q.seg_expert; a.seg_begin = q.seg_begin; a.seg_count = q.seg_count;
    a.num_segments = q.num_segments; a.max_segments = q.max_segments; a.y = static_cast<float *>(q.y); a.route = q.route;
    a.flat_rows = q.flat_rows; a.y_table = q.y_table; a.rows_per_rank = q.rows_per_rank;
    a.status = device_status_word();
    return a.status != nullptr;
}

static int launch_grouped(void (*fn)(const GroupedArgs), const GroupedArgs &a, size_t smem, cudaStream_t stream, const char *what) {
    if (cudaFuncSetAttribute(reinterpret_cast<const void *>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize, MM_SMEM_LIMIT) != cudaSuccess) {
        cudaGetLastError();
        return fail(B200Q_ECUDA, "%s: shared memory opt-in failed", what);
    }
    launch_chained(fn, dim3(sm_count()), dim3(GS_THREADS), smem, stream, a);
    return check_launch(what);
}

int grouped_gate_up_launch(const MmaRequest &q, cudaStream_t stream, bool *launched) {
    *launched = false;
    if (!q.images || !q.tiled || (reinterpret_cast<uintptr_t>(q.images) & 15) ||
        !grouped_gate_up_kp(q.fmt_a, q.n, q.k, q.x_dtype, q.max_segments))
        return B200Q_OK;
    GroupedArgs a{};
    size_t smem = 0;
    if (!plan_gate_up(q.fmt_a, q.n, q.k, q.x_dtype, q.max_segments, a, smem) || !grouped_args(q, a)) return B200Q_OK;
    const bool two = q.x_dtype == B200Q_F32, q5 = q.fmt_a == B200Q_Q5_K;
    auto fn = q5 ? (two ? grouped_gate_up_kernel<true, 2> : grouped_gate_up_kernel<true, 1>)
                 : (two ? grouped_gate_up_kernel<false, 2> : grouped_gate_up_kernel<false, 1>);
    *launched = true;
    return launch_grouped(fn, a, smem, stream, "grouped gate/up");
}

int grouped_down_launch(const MmaRequest &q, cudaStream_t stream, bool *launched) {
    *launched = false;
    if (!q.images || (reinterpret_cast<uintptr_t>(q.images) & 15) || !grouped_down_kp(q.fmt_a, q.n, q.k, q.max_segments)) return B200Q_OK;
    GroupedArgs a{};
    size_t smem = 0;
    if (!plan_down(q.fmt_a, q.n, q.k, q.max_segments, a, smem) || !grouped_args(q, a)) return B200Q_OK;
    *launched = true;
    return launch_grouped(q.fmt_a == B200Q_Q8_0_TILED ? grouped_down_kernel<Q8Tile> : grouped_down_kernel<Q6Tile>, a, smem, stream,
                          "grouped down");
}

}  // namespace b200q
