// Direct-load tensor-core GEMV for Q4_K / Q5_K (sm_100a), 8 tokens per token tile, one or two
// token tiles per pass over the weights.
//
// Q4_K / Q5_K super-blocks are 16-byte multiples, so every lane can fetch exactly the packed
// bytes it needs with 128-bit global loads (four lanes cover 64 contiguous bytes of a row, eight
// rows per instruction) - no shared-memory staging of weights, no producer warp, no barrier on
// the weight path. 16 warps per SM, each with the next super-block already in flight, keep about
// 48 KB of loads outstanding per SM.
//
// Arithmetic per super-block (256 weights of one row):
//   * the lanes of a quad hold interleaved 4-byte words of a row's codes (word w of a 32-byte chunk belongs to lane
//     w & 3), so the sixteen codes of one mma step come from one sub-block in every lane;
//   * a masked nibble pair is used as it stands: 0..15 in the low (or bits 4..7 of the) mantissa bits of an FP16 is the
//     subnormal q * 2^-24 (16 q * 2^-24), which the tensor cores multiply exactly - one AND per pair (plus one shift per
//     word) instead of a byte permute and a packed FMA (Q5_K ORs the fifth bit in above the nibble);
//   * two mma.m16n8k16 per sub-block, then one FP32 FMA per accumulator with the sub-block's 6-bit scale;
//   * the minima go through one more mma: A = the eight 6-bit mins, B = per-sub-block activation
//     sums (FP16 high + remainder), giving sum(mn * sum_x);
//   * y += d * acc - dmin * acc_min in FP32, the powers of two folded into d and dmin.
// Every product is exact; roundings are the FP32 accumulations, as in the FP32-lane kernels.
// What bounds it: instruction issue (about 230 per 16 x 256 tile of Q4_K, 394 with the packed FMA form; at HBM speed a
// tile may take 400 issue slots of its scheduler).
//
// Activations are prepared once per CTA (or per expert segment) exactly as in mma_gemv.cuh:
// power-of-two scaling per token, FP16 high (+ remainder for FP32 inputs), stored as B fragments.
#pragma once

#include "mma_gemv.cuh"

namespace b200q {

constexpr int MD_WARPS = 16;
constexpr int MD_THREADS = MD_WARPS * 32;
constexpr int MD_CTRL_BYTES = 1024;
constexpr int MD_PART_FLOATS = MD_WARPS * 256;          // [warp][16 rows][8 tokens][2 streams]
constexpr int MD_PART_BYTES = 2 * MD_PART_FLOATS * 4;   // double buffered
constexpr float MD_XS_SCALE = 0.015625f;                // activation sums are stored divided by 64

struct DirectArgs {
    const uint8_t *wa;
    const uint8_t *wb;
    long long stride_a, stride_b;
    const unsigned long long *table_a, *table_b;   // optional per-expert pointer tables
    int rb;              // packed bytes per weight row (both streams share the format)
    int tiled;           // weights in the 16-row tile layout of their format (see load_superblock_tiled)
    int n, k, m;
    int kp, rg;          // warps along K and row groups per CTA pass (kp * rg == 16)
    int nterms;
    int off_bfrag, off_xsfrag;
    const void *x;
    int x_dtype;
    void *y;
    int y_dtype;
    int topk;
    const int32_t *order;
    const int32_t *seg_expert;
    const int32_t *seg_begin;
    const int32_t *seg_count;
    const int32_t *num_segments;
    int max_segments;
    const float *route;
    int flat_rows;       // mode 3: term rows stored at the flat assignment index
    const uint64_t *y_table;   // mode 3, optional: per-rank base addresses of the term buffers (peer memory)
    int rows_per_rank;   // flat rows owned by each rank when y_table is set
    const uint8_t *images;   // mode 2, optional: token images (token_image_kernel), image_stride bytes per row of x
    int image_stride;
};

// The pointers of a launch that a persistent multi-stage kernel changes between calls of a stage body (the
// kernels fill it from their arguments; the shapes and the split of the work stay in the argument block).
struct StagePointers {
    const void *x;
    void *y;
    const unsigned long long *table_a, *table_b;
    const int32_t *order, *seg_expert, *seg_begin, *seg_count, *num_segments;
    const float *route;
    int prepared_row;      // grouped gate/up: the row of x whose fragments the caller has already prepared in the
                           // CTA's buffers (-1: none); a first segment of just that row then needs no preparation
};

__device__ __forceinline__ uint4 ldg128(const uint8_t *p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

// The first product of a chain: no accumulator to clear and read.
__device__ __forceinline__ void mma_f16_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                              uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// Packed bytes of two rows' (g, g + 8) super-block as seen by one lane. q[0..1] / q[2..3]: the code words of row g /
// g + 8, word (c, j) of chunk c = bytes [32c + 16j + 4tig, +4) of the row's 128 code bytes, two chunks per uint4 in the
// order (c, 0), (c, 1), (c + 1, 0), (c + 1, 1). h: Q5_K's fifth-bit bytes [16j + 4tig, +4), j = 0, 1, of the two rows.
template <bool Q5>
struct SuperBlockRegs {
    uint4 hd[2];    // d, dmin, 12 scale/min bytes of each row
    uint4 q[4];
    uint2 h[2];
};

// In GGUF rows a lane's words lie 16 bytes apart: four lanes load 64 contiguous bytes (16 each) and exchange words, a
// 4 x 4 transpose inside the quad.
__device__ __forceinline__ void quad_exchange(uint32_t &lo, uint32_t &hi, bool upper, int mask) {
    const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? lo : hi, mask);
    if (upper) lo = got;
    else hi = got;
}
__device__ __forceinline__ uint4 quad_transpose(uint4 v, int tig) {
    quad_exchange(v.x, v.y, tig & 1, 1);
    quad_exchange(v.z, v.w, tig & 1, 1);
    quad_exchange(v.x, v.z, tig & 2, 2);
    quad_exchange(v.y, v.w, tig & 2, 2);
    return v;
}

// The transpose of a native block's words is left to the consumer (transpose_native): the shuffles would wait for the
// loads here.
template <bool Q5>
__device__ __forceinline__ void load_superblock(SuperBlockRegs<Q5> &r, const uint8_t *row_a, const uint8_t *row_b, int tig) {
    constexpr int CODES = Q5 ? 48 : 16;
    r.hd[0] = ldg128(row_a);
    r.hd[1] = ldg128(row_b);
    r.q[0] = ldg128(row_a + CODES + 16 * tig);
    r.q[1] = ldg128(row_a + CODES + 64 + 16 * tig);
    r.q[2] = ldg128(row_b + CODES + 16 * tig);
    r.q[3] = ldg128(row_b + CODES + 64 + 16 * tig);
    if (Q5) {
        const uint32_t *ha = reinterpret_cast<const uint32_t *>(row_a + 16 + 4 * tig), *hb = reinterpret_cast<const uint32_t *>(row_b + 16 + 4 * tig);
        r.h[0] = make_uint2(__ldg(ha), __ldg(ha + 4));
        r.h[1] = make_uint2(__ldg(hb), __ldg(hb + 4));
    }
}
template <bool Q5>
__device__ __forceinline__ void transpose_native(SuperBlockRegs<Q5> &r, int tig) {
#pragma unroll
    for (int i = 0; i < 4; ++i) r.q[i] = quad_transpose(r.q[i], tig);
}

// Q4_K tile layout (device-side re-ordering of the GGUF bytes, same size): a tile holds the 16
// super-blocks of 16 consecutive rows at one K position (2304 bytes):
//   [0, 256)     the 16 rows' first 16 bytes (d, dmin, scales/mins), row r at 16*r
//   [256, 2304)  four planes of 512 bytes with one 16-byte piece per lane (lane*16): planes 0/1 = the words q[0] / q[1]
//                above of row g, planes 2/3 those of row g+8: what a lane of the native layout holds after its exchange
// Tiles are ordered (row group, super-block): a warp instruction reads 512 contiguous bytes.
constexpr int Q4T_TILE_BYTES = 2304;
// Q5_K the same way (2816 bytes, the size of 16 native blocks): the 16 headers, then two planes of 256 bytes with the
// rows' fifth-bit words (lane*8: words j = 0, 1 of row g, then of row g + 8), then the four quant planes:
//   [0, 256) headers | [256, 768) fifth bits | [768, 2816) planes 0/1 (row g), 2/3 (row g + 8), lane * 16 each
constexpr int Q5T_TILE_BYTES = 2816;
template <bool Q5>
__host__ __device__ constexpr int direct_tile_bytes() { return Q5 ? Q5T_TILE_BYTES : Q4T_TILE_BYTES; }

__device__ __forceinline__ uint2 ldg64(const uint8_t *p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

template <bool Q5>
__device__ __forceinline__ void load_superblock_tiled(SuperBlockRegs<Q5> &r, const uint8_t *tile, int lane) {
    constexpr int CODES = Q5 ? 768 : 256;
    const int g = lane >> 2;
    r.hd[0] = ldg128(tile + 16 * g);
    r.hd[1] = ldg128(tile + 16 * (g + 8));
#pragma unroll
    for (int i = 0; i < 4; ++i) r.q[i] = ldg128(tile + CODES + 512 * i + lane * 16);
    if (Q5) {
        r.h[0] = ldg64(tile + 256 + lane * 8);
        r.h[1] = ldg64(tile + 512 + lane * 8);
    }
}

// The same from a tile in shared memory.
template <bool Q5>
__device__ __forceinline__ void read_superblock_tile(SuperBlockRegs<Q5> &r, const uint8_t *tile, int lane) {
    constexpr int CODES = Q5 ? 768 : 256;
    const int g = lane >> 2;
    r.hd[0] = *reinterpret_cast<const uint4 *>(tile + 16 * g);
    r.hd[1] = *reinterpret_cast<const uint4 *>(tile + 16 * (g + 8));
#pragma unroll
    for (int i = 0; i < 4; ++i) r.q[i] = *reinterpret_cast<const uint4 *>(tile + CODES + 512 * i + lane * 16);
    if (Q5) {
        r.h[0] = *reinterpret_cast<const uint2 *>(tile + 256 + lane * 8);
        r.h[1] = *reinterpret_cast<const uint2 *>(tile + 512 + lane * 8);
    }
}

// Scales of one row: the eight 6-bit sub-block scales as FP16 subnormal pairs widened to FP32 (sc * 2^-24), the lane's
// pair of minima as FP16 subnormals (A operand of the min product), d and dmin with the powers of two that undo both
// subnormal forms (2^24 of the codes, 2^24 of the scales; 2^24 of the minima and the 64 of MD_XS_SCALE).
struct RowScales {
    float sc[8];
    uint32_t mins;      // (mn[2*tig], mn[2*tig+1])
    float d, dmin;
};

__device__ __forceinline__ RowScales decode_scales(const uint4 &hd, int tig) {
    RowScales s;
    const __half2 dd = *reinterpret_cast<const __half2 *>(&hd.x);
    s.d = __low2float(dd) * 281474976710656.0f;       // 2^48
    s.dmin = __high2float(dd) * 1073741824.0f;        // 2^30
    const uint32_t sc_lo = hd.y & 0x3f3f3f3fu;                                       // sub-blocks 0..3
    const uint32_t sc_hi = (hd.w & 0x0f0f0f0fu) | ((hd.y >> 2) & 0x30303030u);        // sub-blocks 4..7
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t pair = __byte_perm(i < 2 ? sc_lo : sc_hi, 0u, (i & 1) ? 0x4342 : 0x4140);
        const __half2 h = *reinterpret_cast<const __half2 *>(&pair);
        s.sc[2 * i] = __low2float(h);
        s.sc[2 * i + 1] = __high2float(h);
    }
    const uint32_t mn = (tig & 2) ? ((hd.w >> 4) & 0x0f0f0f0fu) | ((hd.z >> 2) & 0x30303030u) : hd.z & 0x3f3f3f3fu;
    s.mins = __byte_perm(mn, 0u, (tig & 1) ? 0x4342 : 0x4140);
    return s;
}


// ---------------------------------------------------------------------------------------------
// Activation fragments for the direct kernel, in natural order: fragment f holds positions 16f .. 16f + 15; for lane
// (g = lane>>2, tig = lane&3) token g at positions 16f + 4 tig + {0,2 -> b0 ; 1,3 -> b1}, the positions of the codes in
// that lane's word. The two fragments of a sub-block lie side by side (one 16-byte load): uint2 entry
// ((f >> 1) * 32 + lane) * 2 + (f & 1).
// xsfrag (sb, term) holds (sum_x[sub 2*tig], sum_x[sub 2*tig+1]) / 64 for token g.
// ---------------------------------------------------------------------------------------------
// Four consecutive activations starting at element index e (a multiple of 4) as floats.
// `vec_ok` tells whether the tensor allows aligned vector loads.
__device__ __forceinline__ void load4(const void *x, int x_dtype, size_t e, bool vec_ok, float (&v)[4]) {
    if (x_dtype == B200Q_F32) {
        if (vec_ok) {
            const float4 t = *reinterpret_cast<const float4 *>(static_cast<const float *>(x) + e);
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = static_cast<const float *>(x)[e + i];
        }
    } else {
        uint2 raw;
        if (vec_ok) raw = *reinterpret_cast<const uint2 *>(static_cast<const uint16_t *>(x) + e);
        else {
            const uint16_t *p = static_cast<const uint16_t *>(x) + e;
            raw.x = p[0] | (static_cast<uint32_t>(p[1]) << 16);
            raw.y = p[2] | (static_cast<uint32_t>(p[3]) << 16);
        }
        if (x_dtype == B200Q_F16) {
            v[0] = __half2float(__ushort_as_half(static_cast<unsigned short>(raw.x & 0xffffu)));
            v[1] = __half2float(__ushort_as_half(static_cast<unsigned short>(raw.x >> 16)));
            v[2] = __half2float(__ushort_as_half(static_cast<unsigned short>(raw.y & 0xffffu)));
            v[3] = __half2float(__ushort_as_half(static_cast<unsigned short>(raw.y >> 16)));
        } else {  // bf16: the upper 16 bits of an FP32
            v[0] = __uint_as_float(raw.x << 16);
            v[1] = __uint_as_float(raw.x & 0xffff0000u);
            v[2] = __uint_as_float(raw.y << 16);
            v[3] = __uint_as_float(raw.y & 0xffff0000u);
        }
    }
}

// Every thread owns whole chunks of four consecutive activations (chunk c of token t covers
// positions 4c..4c+3, which is exactly one fragment entry): one pass loads them and finds the
// per-token maximum, the second converts from registers (chunks beyond KEEP per thread are
// loaded again). Entries of tokens >= m_tokens are left as they are: a column of B only feeds the
// same column of the product, and those columns are never stored.

// (THREADS consecutive threads tid = 0..THREADS-1 take part and meet at named barrier BARRIER; the result does
// not depend on THREADS, which must be a multiple of 32.)
template <int NTERMS, int KEEP, int THREADS = MD_THREADS, int BARRIER = 1, typename RowFn>
__device__ __forceinline__ void prepare_direct(RowFn row_of, int m_tokens, int k, const void *x, int x_dtype,
                                               uint2 *bfrag, uint32_t *xsfrag, float *tok_scale, int tid) {
    const int lane = tid & 31;
    const int nsb = k >> 8;
    const int nfrag = nsb * 16;
    const size_t esize = x_dtype == B200Q_F32 ? 4 : 2;
    const bool vec_ok = (reinterpret_cast<uintptr_t>(x) % (4 * esize)) == 0;   // rows are multiples of 256 elements
    unsigned int *amax_bits = reinterpret_cast<unsigned int *>(tok_scale + 16);   // [8], non-negative floats as ints
    if (tid < 8) amax_bits[tid] = 0u;
    named_barrier_sync(BARRIER, THREADS);
    const int chunks_per_token = k >> 2;            // a multiple of 64: a warp's 32 chunks share one token
    const int total = m_tokens * chunks_per_token;
    float kept[KEEP][4];
    const int first = tid & ~31;
    // 1. load, per-token maximum magnitude
    auto load_chunk = [&](int c0, float (&v)[4]) {
        const int t = c0 / chunks_per_token;
        load4(x, x_dtype, static_cast<size_t>(row_of(t)) * k + static_cast<size_t>(c0 + lane - t * chunks_per_token) * 4,
              vec_ok, v);
        float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
        for (int o = 16; o; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        // NaN/Inf inputs: keep the scale at 1 (the bit pattern compares above every finite value)
        if (lane == 0) atomicMax(&amax_bits[t], __float_as_uint(amax));
    };
#pragma unroll
    for (int sl = 0; sl < KEEP; ++sl)
        if (first + sl * THREADS < total) load_chunk(first + sl * THREADS, kept[sl]);
    for (int c0 = first + KEEP * THREADS; c0 < total; c0 += THREADS) {
        float v[4];
        load_chunk(c0, v);
    }
    named_barrier_sync(BARRIER, THREADS);
    if (tid < 8) {
        const float amax = __uint_as_float(amax_bits[tid]);
        float s = 1.0f;
        if (amax > 0.f && amax < __int_as_float(0x7f800000)) {
            int e;
            frexpf(amax, &e);
            s = ldexpf(1.0f, min(14 - e, 100));   // scaled maximum in [2^13, 2^14)
        }
        tok_scale[tid] = s;
        tok_scale[8 + tid] = 1.0f / s;
    }
    named_barrier_sync(BARRIER, THREADS);
    // 2. scale, split, store: the chunk at position p of token t is the entry of fragment f = p>>4, lane 4t + ((p>>2)&3)
    auto store_chunk = [&](int c0, const float (&v)[4]) {
        const int t = c0 / chunks_per_token;
        const int p = (c0 + lane - t * chunks_per_token) * 4;
        const float s = tok_scale[t];
        __half hi[4], lo[4];
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float sv = v[i] * s;
            hi[i] = __float2half_rn(sv);
            sum += __half2float(hi[i]);
            if (NTERMS == 2) {
                lo[i] = __float2half_rn(sv - __half2float(hi[i]));
                sum += __half2float(lo[i]);
            }
        }
        const int sb = p >> 8, sub = (p >> 5) & 7;
        const int entry = ((p >> 5) * 32 + 4 * t + ((p >> 2) & 3)) * 2 + ((p >> 4) & 1);
        uint2 out;
        out.x = static_cast<uint32_t>(__half_as_ushort(hi[0])) | (static_cast<uint32_t>(__half_as_ushort(hi[2])) << 16);
        out.y = static_cast<uint32_t>(__half_as_ushort(hi[1])) | (static_cast<uint32_t>(__half_as_ushort(hi[3])) << 16);
        bfrag[entry] = out;
        if (NTERMS == 2) {
            out.x = static_cast<uint32_t>(__half_as_ushort(lo[0])) | (static_cast<uint32_t>(__half_as_ushort(lo[2])) << 16);
            out.y = static_cast<uint32_t>(__half_as_ushort(lo[1])) | (static_cast<uint32_t>(__half_as_ushort(lo[3])) << 16);
            bfrag[nfrag * 32 + entry] = out;
        }
        // sub-block sum: its eight chunks sit in eight consecutive lanes
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        if ((lane & 7) == 0) {
            const float scaled = sum * MD_XS_SCALE;
            const __half h = __float2half_rn(scaled);
            const __half l = __float2half_rn(scaled - __half2float(h));
            // operand of the min product: lane 4*t + (sub>>1) holds sub-blocks (sub & ~1, sub | 1)
            const int lane_t = 4 * t + (sub >> 1);
            reinterpret_cast<unsigned short *>(xsfrag + (sb * 2 + 0) * 32 + lane_t)[sub & 1] = __half_as_ushort(h);
            reinterpret_cast<unsigned short *>(xsfrag + (sb * 2 + 1) * 32 + lane_t)[sub & 1] = __half_as_ushort(l);
        }
    };
#pragma unroll
    for (int sl = 0; sl < KEEP; ++sl)
        if (first + sl * THREADS < total) store_chunk(first + sl * THREADS, kept[sl]);
    for (int c0 = first + KEEP * THREADS; c0 < total; c0 += THREADS) {
        const int t = c0 / chunks_per_token;
        float v[4];
        load4(x, x_dtype, static_cast<size_t>(row_of(t)) * k + static_cast<size_t>(c0 + lane - t * chunks_per_token) * 4,
              vec_ok, v);
        store_chunk(c0, v);
    }
    named_barrier_sync(BARRIER, THREADS);
}

// Four consecutive activations as they lie in memory: FP32 inputs (NTERMS = 2) or 16-bit ones.
template <int NTERMS>
struct RawChunk {
    uint32_t w[NTERMS == 2 ? 4 : 2];
};
// The chunk at element index e (a multiple of 4); `vec_ok` tells whether the tensor allows aligned vector loads.
template <int NTERMS>
__device__ __forceinline__ void load_chunk(const void *x, size_t e, bool vec_ok, RawChunk<NTERMS> &r) {
    if constexpr (NTERMS == 2) {
        const float *p = static_cast<const float *>(x) + e;
        if (vec_ok) {
            const uint4 v = *reinterpret_cast<const uint4 *>(p);
            r.w[0] = v.x; r.w[1] = v.y; r.w[2] = v.z; r.w[3] = v.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) r.w[i] = __float_as_uint(p[i]);
        }
    } else {
        const uint16_t *p = static_cast<const uint16_t *>(x) + e;
        if (vec_ok) {
            const uint2 v = *reinterpret_cast<const uint2 *>(p);
            r.w[0] = v.x; r.w[1] = v.y;
        } else {
            r.w[0] = p[0] | (static_cast<uint32_t>(p[1]) << 16);
            r.w[1] = p[2] | (static_cast<uint32_t>(p[3]) << 16);
        }
    }
}
// Bits of the largest magnitude of a chunk, in the type's own width: magnitudes order like their bits, Inf and NaN last.
template <int NTERMS>
__device__ __forceinline__ uint32_t chunk_amax(const RawChunk<NTERMS> &r) {
    if constexpr (NTERMS == 2) {
        return max(max(r.w[0] & 0x7fffffffu, r.w[1] & 0x7fffffffu), max(r.w[2] & 0x7fffffffu, r.w[3] & 0x7fffffffu));
    } else {
        const uint32_t m = __vmaxu2(r.w[0] & 0x7fff7fffu, r.w[1] & 0x7fff7fffu);
        return max(m & 0xffffu, m >> 16);
    }
}
template <int NTERMS>
__device__ __forceinline__ void chunk_values(const RawChunk<NTERMS> &r, bool f16, float (&v)[4]) {
    if constexpr (NTERMS == 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r.w[i]);
    } else if (f16) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            v[2 * i] = __half2float(__ushort_as_half(static_cast<unsigned short>(r.w[i] & 0xffffu)));
            v[2 * i + 1] = __half2float(__ushort_as_half(static_cast<unsigned short>(r.w[i] >> 16)));
        }
    } else {  // bf16: the upper 16 bits of an FP32
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            v[2 * i] = __uint_as_float(r.w[i] << 16);
            v[2 * i + 1] = __uint_as_float(r.w[i] & 0xffff0000u);
        }
    }
}

// The same preparation, the same bits, for many chunks per thread (dense launches of several tokens). What bounds it is
// the latency of the reads - every CTA reads all of x from L2 - so BATCH chunks are requested before the first is looked
// at, and the second pass starts with the batch that the first left in registers; above, the conversion behind every load
// waits for it. Launches of 8 tokens: Q4_K [8192 x 2048] 11.7 -> 8.7 us, Q8_0 [2048 x 8192] 27.7 -> 14.6 us; 16 tokens,
// Q8_0 [2048 x 2048] 14.6 -> 8.8 us. Up to MD_FEW_CHUNKS chunks per thread the short code above is the faster one: these copies of a chunk's
// code cost about 1 us of instruction fetch in a launch that uses one or two of them.
// SUMS: also the activation sums of the sub-blocks.
constexpr int MD_FEW_CHUNKS = 4;
template <int NTERMS, int BATCH, bool SUMS, int THREADS, int BARRIER, typename RowFn>
__device__ __forceinline__ void prepare_tokens(RowFn row_of, int m_tokens, int k, const void *x, int x_dtype,
                                               uint2 *bfrag, uint32_t *xsfrag, float *tok_scale, int tid) {
    const int lane = tid & 31;
    const int nfrag = k >> 4;
    const bool vec_ok = (reinterpret_cast<uintptr_t>(x) % (NTERMS == 2 ? 16 : 8)) == 0;   // rows are multiples of 256 elements
    const bool f16 = x_dtype == B200Q_F16;
    unsigned int *amax_bits = reinterpret_cast<unsigned int *>(tok_scale + 16);   // [8]
    if (tid < 8) amax_bits[tid] = 0u;
    named_barrier_sync(BARRIER, THREADS);
    const int chunks_per_token = k >> 2;            // a multiple of 64: a warp's 32 chunks share one token
    const int total = m_tokens * chunks_per_token, first = tid & ~31;
    // c / chunks_per_token for c <= 8 * chunks_per_token < 2^17 by a multiplication: the error of the rounded-up
    // reciprocal, c / 2^32 at most, is below the distance 1 / chunks_per_token to the next whole number
    const uint32_t recip = 0xffffffffu / static_cast<uint32_t>(chunks_per_token) + 1u;
    auto token_of = [&](int c) { return static_cast<int>(__umulhi(static_cast<uint32_t>(c), recip)); };
    RawChunk<NTERMS> raw[BATCH];
    auto load_batch = [&](int base) {
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const int c0 = base + i * THREADS;
            if (c0 >= total) break;
            const int t = token_of(c0);
            load_chunk<NTERMS>(x, static_cast<size_t>(row_of(t)) * k + static_cast<size_t>(c0 + lane - t * chunks_per_token) * 4,
                               vec_ok, raw[i]);
        }
    };
    // 1. per-token maximum magnitude
    int kept = first;                               // base of the batch in registers
    for (int base = first; base < total; base += BATCH * THREADS) {
        kept = base;
        load_batch(base);
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            const int c0 = base + i * THREADS;
            if (c0 >= total) break;
            const uint32_t m = __reduce_max_sync(0xffffffffu, chunk_amax<NTERMS>(raw[i]));
            if (lane == 0) atomicMax(&amax_bits[token_of(c0)], m);
        }
    }
    named_barrier_sync(BARRIER, THREADS);
    if (tid < 8) {
        const uint32_t bits = amax_bits[tid];
        float amax;
        if (NTERMS == 2) amax = __uint_as_float(bits);
        else amax = f16 ? __half2float(__ushort_as_half(static_cast<unsigned short>(bits))) : __uint_as_float(bits << 16);
        float s = 1.0f;                             // (stays 1 where the maximum is Inf or NaN)
        if (amax > 0.f && amax < __int_as_float(0x7f800000)) {
            int e;
            frexpf(amax, &e);
            s = ldexpf(1.0f, min(14 - e, 100));   // scaled maximum in [2^13, 2^14)
        }
        tok_scale[tid] = s;
        tok_scale[8 + tid] = 1.0f / s;
    }
    named_barrier_sync(BARRIER, THREADS);
    // 2. scale, split, store: the chunk at position p of token t is the entry of fragment f = p>>4, lane 4t + ((p>>2)&3)
    auto store_chunk = [&](int c0, const RawChunk<NTERMS> &r) {
        const int t = token_of(c0);
        const int p = (c0 + lane - t * chunks_per_token) * 4;
        const float s = tok_scale[t];
        float v[4];
        chunk_values<NTERMS>(r, f16, v);
        unsigned short hi[4], lo[4];
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float sv = v[i] * s;
            const __half h = __float2half_rn(sv);
            hi[i] = __half_as_ushort(h);
            if (SUMS) sum += __half2float(h);
            if (NTERMS == 2) {
                const __half l = __float2half_rn(sv - __half2float(h));
                lo[i] = __half_as_ushort(l);
                if (SUMS) sum += __half2float(l);
            }
        }
        const int entry = ((p >> 5) * 32 + 4 * t + ((p >> 2) & 3)) * 2 + ((p >> 4) & 1);
        bfrag[entry] = make_uint2(hi[0] | (static_cast<uint32_t>(hi[2]) << 16), hi[1] | (static_cast<uint32_t>(hi[3]) << 16));
        if (NTERMS == 2)
            bfrag[nfrag * 32 + entry] = make_uint2(lo[0] | (static_cast<uint32_t>(lo[2]) << 16), lo[1] | (static_cast<uint32_t>(lo[3]) << 16));
        if (SUMS) {
            // sub-block sum: its eight chunks sit in eight consecutive lanes
            const int sb = p >> 8, sub = (p >> 5) & 7;
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            sum += __shfl_xor_sync(0xffffffffu, sum, 4);
            if ((lane & 7) == 0) {
                const float scaled = sum * MD_XS_SCALE;
                const __half h = __float2half_rn(scaled);
                const __half l = __float2half_rn(scaled - __half2float(h));
                // operand of the min product: lane 4*t + (sub>>1) holds sub-blocks (sub & ~1, sub | 1)
                const int lane_t = 4 * t + (sub >> 1);
                reinterpret_cast<unsigned short *>(xsfrag + (sb * 2 + 0) * 32 + lane_t)[sub & 1] = __half_as_ushort(h);
                reinterpret_cast<unsigned short *>(xsfrag + (sb * 2 + 1) * 32 + lane_t)[sub & 1] = __half_as_ushort(l);
            }
        }
    };
    for (int base = kept;;) {
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            if (base + i * THREADS >= total) break;
            store_chunk(base + i * THREADS, raw[i]);
        }
        base = base == kept ? first : base + BATCH * THREADS;       // the batches before the kept one, again from memory
        if (base >= kept) break;
        load_batch(base);
    }
    named_barrier_sync(BARRIER, THREADS);
}

// ---------------------------------------------------------------------------------------------
// Token images. In the grouped gate/up launch every expert segment needs the fragments of its tokens, and
// a token routed to k experts would be converted k times (at 64 tokens: 704 conversions of 64 distinct
// rows, each a chain of dependent loads, a reduction and three barriers). token_image_kernel runs
// prepare_tokens once per token - same code, so the same bits - and stores what it wrote for token slot 0:
//   [NTERMS * nfrag * 32 bytes]  the slot's four lanes (tig 0..3, 16 bytes each) of every pair of fragments
//   [nsb * 2 * 16 bytes]         the slot's four words of every activation-sum row
//   [16 bytes]                   scale, inverse scale
// gather_token_images copies the images of a segment's tokens into the slots of the CTA's buffers with
// independent 16-byte loads.
// ---------------------------------------------------------------------------------------------
__host__ __device__ constexpr int token_image_units(int nterms, int nsb) {      // 16-byte units per token
    return nterms * nsb * 16 * 2 + nsb * 2 + 1;
}

template <int NTERMS>
__global__ void __launch_bounds__(MD_THREADS, 1) token_image_kernel(const void *x, int x_dtype, int k, uint8_t *images) {
    extern __shared__ __align__(128) uint8_t smem[];
    chain_trigger();
    chain_wait();                 // x comes from the preceding kernel
    const int nsb = k >> 8, nfrag = nsb * 16;
    float *tok_scale = reinterpret_cast<float *>(smem);
    uint2 *bfrag = reinterpret_cast<uint2 *>(smem + MD_CTRL_BYTES);
    uint32_t *xsfrag = reinterpret_cast<uint32_t *>(smem + MD_CTRL_BYTES + NTERMS * nfrag * 256);
    const int row = blockIdx.x, tid = threadIdx.x;
    prepare_direct<NTERMS, 4>([row](int) { return row; }, 1, k, x, x_dtype, bfrag, xsfrag, tok_scale, tid);
    const int nb = NTERMS * nfrag * 2, units = token_image_units(NTERMS, nsb);
    uint4 *dst = reinterpret_cast<uint4 *>(images + static_cast<size_t>(row) * units * 16);
    for (int u = tid; u < units; u += MD_THREADS) {
        uint4 v;
        if (u < nb) v = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(bfrag) + (u >> 2) * 512 + (u & 3) * 16);
        else if (u < units - 1) v = *reinterpret_cast<const uint4 *>(reinterpret_cast<const uint8_t *>(xsfrag) + (u - nb) * 128);
        else v = make_uint4(__float_as_uint(tok_scale[0]), __float_as_uint(tok_scale[8]), 0u, 0u);
        dst[u] = v;
    }
}

// Slots 0..m_tokens-1 of the CTA's buffers <- the images of rows order[seg_begin + t] / topk. The caller
// brackets the call with CTA barriers.
__device__ __forceinline__ void gather_token_images(const uint8_t *images, int image_stride, const int32_t *order,
                                                    int seg_begin, int topk, int m_tokens, int nterms, int nsb,
                                                    uint2 *bfrag, uint32_t *xsfrag, float *tok_scale, int tid) {
    const int nb = nterms * nsb * 32, units = token_image_units(nterms, nsb);
    const int t = (tid >> 5) & 7;                 // two warps per token slot, all their loads independent
    if (t < m_tokens) {
        const int row = order[seg_begin + t] / topk;
        const uint4 *src = reinterpret_cast<const uint4 *>(images + static_cast<size_t>(row) * image_stride);
#pragma unroll 5
        for (int u = (tid >> 8) * 32 + (tid & 31); u < units; u += 64) {
            const uint4 v = src[u];
            if (u < nb) *reinterpret_cast<uint4 *>(reinterpret_cast<uint8_t *>(bfrag) + (u >> 2) * 512 + t * 64 + (u & 3) * 16) = v;
            else if (u < units - 1) *reinterpret_cast<uint4 *>(reinterpret_cast<uint8_t *>(xsfrag) + (u - nb) * 128 + t * 16) = v;
            else {
                tok_scale[t] = __uint_as_float(v.x);
                tok_scale[8 + t] = __uint_as_float(v.y);
            }
        }
    }
}

// One super-block of rows (g, g+8): tot += d * sum_s sc_s * (codes_s . x_s) - dmin * sum_s mn_s * sum_x_s.
// With NT token tiles (8 tokens each; their fragments `btile` / `xtile` entries apart) every decoded
// A operand is multiplied into each tile, so the decode cost is paid once per 8*NT tokens; the
// arithmetic of one token does not depend on NT.
// frag(nt, s, plane): the lane's 16 bytes of sub-block s (its two fragments) in plane 0 (FP16 high parts) or 1
// (remainders) of token tile nt; sums(nt, term): the lane's word of the activation sums.
template <bool Q5, int NTERMS, int NT, typename FragFn, typename SumFn>
__device__ __forceinline__ void superblock_mma(const SuperBlockRegs<Q5> &r, const FragFn frag, const SumFn sums, int tig,
                                               float (&tot)[NT][4]) {
    const RowScales sa = decode_scales(r.hd[0], tig), sbk = decode_scales(r.hd[1], tig);
    // even sub-blocks (low nibbles) and odd ones (high nibbles, 16 times the code) in accumulators of their own
    float even[NT][4], odd[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) even[nt][i] = odd[nt][i] = 0.f;
    const uint32_t wa[8] = {r.q[0].x, r.q[0].y, r.q[0].z, r.q[0].w, r.q[1].x, r.q[1].y, r.q[1].z, r.q[1].w};
    const uint32_t wb[8] = {r.q[2].x, r.q[2].y, r.q[2].z, r.q[2].w, r.q[3].x, r.q[3].y, r.q[3].z, r.q[3].w};
    const uint32_t ha[2] = {r.h[0].x, r.h[0].y}, hb[2] = {r.h[1].x, r.h[1].y};
    // fifth bits of sub-block s, bytes 0 and 2 (byte = 0) or 1 and 3 (byte = 1) of a high-bit word, at bit 4 (odd
    // sub-blocks: bit 8, above a nibble in bits 4..7)
    auto fifth = [](uint32_t h, int s, int byte) {
        const int to = (s & 1) ? 8 : 4, from = s + 8 * byte;
        const uint32_t v = from >= to ? h >> (from - to) : h << (to - from);
        return v & ((s & 1) ? 0x01000100u : 0x00100010u);
    };
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const uint32_t a[2] = {wa[2 * c], wa[2 * c + 1]}, b[2] = {wb[2 * c], wb[2 * c + 1]};
        const uint32_t a8[2] = {a[0] >> 8, a[1] >> 8}, b8[2] = {b[0] >> 8, b[1] >> 8};
#pragma unroll
        for (int nib = 0; nib < 2; ++nib) {
            const int s = 2 * c + nib;
            const uint32_t mask = nib ? 0x00f000f0u : 0x000f000fu;
            uint32_t f[2][4];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                f[j][0] = a[j] & mask;
                f[j][1] = b[j] & mask;
                f[j][2] = a8[j] & mask;
                f[j][3] = b8[j] & mask;
                if (Q5) {
                    f[j][0] |= fifth(ha[j], s, 0);
                    f[j][1] |= fifth(hb[j], s, 0);
                    f[j][2] |= fifth(ha[j], s, 1);
                    f[j][3] |= fifth(hb[j], s, 1);
                }
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                float acc[4];
                const uint4 v = frag(nt, s, 0);
                mma_f16_first(acc, f[0][0], f[0][1], f[0][2], f[0][3], v.x, v.y);
                mma_f16(acc, f[1][0], f[1][1], f[1][2], f[1][3], v.z, v.w);
                if (NTERMS == 2) {
                    const uint4 u = frag(nt, s, 1);
                    mma_f16(acc, f[0][0], f[0][1], f[0][2], f[0][3], u.x, u.y);
                    mma_f16(acc, f[1][0], f[1][1], f[1][2], f[1][3], u.z, u.w);
                }
                float (&dst)[4] = nib ? odd[nt] : even[nt];
                dst[0] = fmaf(sa.sc[s], acc[0], dst[0]);
                dst[1] = fmaf(sa.sc[s], acc[1], dst[1]);
                dst[2] = fmaf(sbk.sc[s], acc[2], dst[2]);
                dst[3] = fmaf(sbk.sc[s], acc[3], dst[3]);
            }
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        float accm[4];
        mma_f16_first(accm, sa.mins, sbk.mins, 0u, 0u, sums(nt, 0), 0u);
        mma_f16(accm, sa.mins, sbk.mins, 0u, 0u, sums(nt, 1), 0u);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float sum = fmaf(0.0625f, odd[nt][i], even[nt][i]);
            tot[nt][i] = fmaf(i < 2 ? sa.d : sbk.d, sum, fmaf(i < 2 ? -sa.dmin : -sbk.dmin, accm[i], tot[nt][i]));
        }
    }
}


// ---------------------------------------------------------------------------------------------
// Kernel. MODE as in stream_gemv.cuh: 0 linear, 1 SwiGLU, 2 grouped gate/up, 3 grouped down.
// Work item of a warp = (row block, super-block of its K part, stream); the packed bytes of the
// next item are requested before the current one is computed.
// ---------------------------------------------------------------------------------------------
// NT (modes 0 and 1 only) is the number of 8-token tiles served by one pass over the weights: tile
// nt holds tokens 8nt..8nt+7 with its own scales (MD_TOK_STRIDE floats further on), fragments and
// activation sums.
constexpr int MD_TOK_STRIDE = 128;     // floats between the token tiles' scale blocks (inside the control bytes)
// The work of CTA `block` of `nblocks` (MD_THREADS threads, all of them call): the kernel below is this body
// for (blockIdx.x, gridDim.x); a persistent kernel that walks several stages calls it with its own.
// `smem`: 128-byte aligned, direct-kernel layout (control bytes, partial sums, fragments at a.off_bfrag).
template <bool Q5, int MODE, int NTERMS, int NT = 1>
__device__ __forceinline__ void mma_direct_body(const DirectArgs &a, const StagePointers &gp, uint8_t *smem, const int block,
                                                const int nblocks) {
    constexpr bool DUAL = (MODE == 1 || MODE == 2);
    constexpr bool GROUPED = (MODE >= 2);
    constexpr int QB = Q5 ? 176 : 144;
    static_assert(NT == 1 || !GROUPED, "several token tiles only in the dense modes");
    float *tok_scale = reinterpret_cast<float *>(smem);           // [8] scale, [8] inverse
    float *route_w = reinterpret_cast<float *>(smem + 128);       // [8]
    int *seg_tokens = reinterpret_cast<int *>(smem + 192);        // [8]
    float **out_ptr = reinterpret_cast<float **>(smem + 256);     // [8] mode 3 output row pointers
    float *partial = reinterpret_cast<float *>(smem + MD_CTRL_BYTES);
    uint2 *bfrag = reinterpret_cast<uint2 *>(smem + a.off_bfrag);
    uint32_t *xsfrag = reinterpret_cast<uint32_t *>(smem + a.off_xsfrag);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, tig = lane & 3;
    const int rgi = warp / a.kp, kpi = warp - rgi * a.kp;
    const int nsb = a.k >> 8;
    const int nfrag = nsb * 16;
    const int btile = NTERMS * nfrag * 32, xtile = nsb * 64;     // fragment / sum entries of one token tile

    const int rows_per_block = 16 * a.rg;
    const int blocks_per_unit = (a.n + rows_per_block - 1) / rows_per_block;
    long long units = 1;
    if (GROUPED) {
        int nseg = *gp.num_segments;
        if (nseg > a.max_segments) nseg = a.max_segments;
        units = nseg;
    }
    const long long total_blocks = units * blocks_per_unit;
    const long long blk_begin = total_blocks * block / nblocks;
    const long long blk_end = total_blocks * (block + 1) / nblocks;
    if (!GROUPED) {
        // the CTA's row blocks are one contiguous byte range of the matrix (rows, or 16-row tiles)
        if (blk_begin < blk_end) {
            size_t first, last;
            if (a.tiled) {
                first = static_cast<size_t>(blk_begin) * a.rg * nsb * direct_tile_bytes<Q5>();
                last = static_cast<size_t>(min(static_cast<long long>(a.n >> 4), blk_end * a.rg)) * nsb * direct_tile_bytes<Q5>();
            } else {
                first = static_cast<size_t>(blk_begin) * rows_per_block * a.rb;
                last = static_cast<size_t>(min(static_cast<long long>(a.n), blk_end * rows_per_block)) * a.rb;
            }
            const size_t cap = DUAL ? CHAIN_PREFETCH_BYTES / 2 : CHAIN_PREFETCH_BYTES;
            prefetch_l2_range(a.wa + first, last - first, cap, tid, MD_THREADS);
            if (DUAL) prefetch_l2_range(a.wb + first, last - first, cap, tid, MD_THREADS);
        }
        chain_wait();     // activations come from the preceding kernel
    }
    if (blk_begin >= blk_end) return;

    // items of this warp inside one row block: its super-blocks x streams
    const int sb_count = kpi < nsb ? (nsb - kpi + a.kp - 1) / a.kp : 0;
    const int items_per_block = sb_count * (DUAL ? 2 : 1);

    // Row pointers of a row block for this lane (rows g and g+8 of its row group, both streams);
    // rows past the end are clamped to the last row (loaded, never stored).
    struct BlockPtrs {
        const uint8_t *a_lo, *a_hi, *b_lo, *b_hi;
    };
    auto block_ptrs = [&](int unit, int row0) {
        BlockPtrs p;
        const int expert = GROUPED ? gp.seg_expert[unit] : 0;
        size_t off_lo, off_hi;
        if (a.tiled) {   // tile of (row group, super-block kpi); n is a multiple of 16 here
            const int group = min((row0 >> 4) + rgi, (a.n >> 4) - 1);
            off_lo = off_hi = (static_cast<size_t>(group) * nsb + kpi) * direct_tile_bytes<Q5>();
        } else {
            off_lo = static_cast<size_t>(min(row0 + 16 * rgi + g, a.n - 1)) * a.rb + static_cast<size_t>(kpi) * QB;
            off_hi = static_cast<size_t>(min(row0 + 16 * rgi + g + 8, a.n - 1)) * a.rb + static_cast<size_t>(kpi) * QB;
        }
        const uint8_t *base_a = expert_matrix(a.wa, a.stride_a, gp.table_a, expert);
        p.a_lo = base_a + off_lo;
        p.a_hi = base_a + off_hi;
        p.b_lo = p.b_hi = nullptr;
        if (DUAL) {
            const uint8_t *base_b = expert_matrix(a.wb, a.stride_b, gp.table_b, expert);
            p.b_lo = base_b + off_lo;
            p.b_hi = base_b + off_hi;
        }
        return p;
    };
    // item -> byte offset from the block pointers, and stream
    const int sb_step_bytes = a.kp * (a.tiled ? direct_tile_bytes<Q5>() : QB);
    auto issue_item = [&](const BlockPtrs &p, int item, SuperBlockRegs<Q5> &r) {
        const int stream = DUAL ? (item & 1) : 0;
        const size_t off = static_cast<size_t>(DUAL ? (item >> 1) : item) * sb_step_bytes;
        if (a.tiled) {
            load_superblock_tiled<Q5>(r, (stream ? p.b_lo : p.a_lo) + off, lane);
            return;
        }
        load_superblock<Q5>(r, (stream ? p.b_lo : p.a_lo) + off, (stream ? p.b_hi : p.a_hi) + off, tig);
    };

    int unit_i = static_cast<int>(blk_begin / blocks_per_unit);
    int bi = static_cast<int>(blk_begin - static_cast<long long>(unit_i) * blocks_per_unit);
    BlockPtrs cur_p = block_ptrs(unit_i, bi * rows_per_block), nxt_p = cur_p;

    SuperBlockRegs<Q5> cur, nxt;
    if (items_per_block > 0) issue_item(cur_p, 0, nxt);

    int m_tokens = a.m;
    int seg_begin = 0, cur_unit = -1, last_single = (MODE == 2) ? gp.prepared_row : -1;
    if (!GROUPED) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const auto row_of = [nt](int t) { return 8 * nt + t; };
            const int tokens = max(min(a.m - 8 * nt, 8), 0);
            if (NT == 2 || tokens * (a.k >> 2) > MD_FEW_CHUNKS * MD_THREADS)
                prepare_tokens<NTERMS, 8, true, MD_THREADS, 1>(row_of, tokens, a.k, gp.x, a.x_dtype, bfrag + nt * btile,
                                                               xsfrag + nt * xtile, tok_scale + nt * MD_TOK_STRIDE, tid);
            else
                prepare_direct<NTERMS, MD_FEW_CHUNKS>(row_of, tokens, a.k, gp.x, a.x_dtype, bfrag + nt * btile,
                                                      xsfrag + nt * xtile, tok_scale + nt * MD_TOK_STRIDE, tid);
        }
    }

    int pbuf = 0;
    for (long long blk = blk_begin; blk < blk_end; ++blk) {
        const int unit = unit_i;
        const int row0 = bi * rows_per_block;
        // advance the (unit, block-in-unit) counters and look up the next block's pointers
        if (++bi == blocks_per_unit) { bi = 0; ++unit_i; }
        const bool has_next = blk + 1 < blk_end;
        if (has_next) nxt_p = block_ptrs(unit_i, bi * rows_per_block);
        if (GROUPED && unit != cur_unit) {
            cur_unit = unit;
            seg_begin = gp.seg_begin[unit];
            m_tokens = min(gp.seg_count[unit], 8);
            int single = -1;
            if (MODE == 2 && m_tokens == 1) single = gp.order[seg_begin] / a.topk;
            const bool reuse = (single >= 0 && single == last_single);
            last_single = single;
            if (!reuse && MODE == 2 && a.images) {
                named_barrier_sync(1, MD_THREADS);       // every warp is done with the previous segment's fragments
                gather_token_images(a.images, a.image_stride, gp.order, seg_begin, a.topk, m_tokens, NTERMS, nsb, bfrag,
                                    xsfrag, tok_scale, tid);
                named_barrier_sync(1, MD_THREADS);
            } else if (!reuse) {
                named_barrier_sync(1, MD_THREADS);
                if (tid < m_tokens) {
                    const int flat = gp.order[seg_begin + tid];
                    seg_tokens[tid] = (MODE == 2) ? flat / a.topk : seg_begin + tid;
                    if (MODE == 3) {
                        route_w[tid] = gp.route[flat];
                        out_ptr[tid] = term_row_pointer(static_cast<float *>(gp.y), a.y_table, a.rows_per_rank, a.n, a.flat_rows ? flat : seg_begin + tid);
                    }
                }
                named_barrier_sync(1, MD_THREADS);
                prepare_direct<NTERMS, 2>([&](int t) { return seg_tokens[t]; }, m_tokens, a.k, gp.x, a.x_dtype, bfrag,
                                       xsfrag, tok_scale, tid);
            }
        }

        float tot_a[NT][4], tot_b[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) tot_a[nt][i] = tot_b[nt][i] = 0.f;
        for (int item = 0; item < items_per_block; ++item) {
            // (copying the prefetched registers measured faster than alternating two register sets)
            cur = nxt;
            // request the next item (same block, or the first item of the next block)
            if (item + 1 < items_per_block) issue_item(cur_p, item + 1, nxt);
            else if (has_next) issue_item(nxt_p, 0, nxt);
            if (!a.tiled) transpose_native<Q5>(cur, tig);
            const int stream = DUAL ? (item & 1) : 0;
            const int sb = kpi + (DUAL ? (item >> 1) : item) * a.kp;
            const uint4 *bf = reinterpret_cast<const uint4 *>(bfrag) + sb * 256 + lane;
            const uint32_t *xf = xsfrag + sb * 64 + lane;
            auto frag = [&](int nt, int s, int plane) { return bf[nt * (btile >> 1) + plane * nfrag * 16 + s * 32]; };
            auto sums = [&](int nt, int term) { return xf[nt * xtile + term * 32]; };
            if (stream == 0) superblock_mma<Q5, NTERMS, NT>(cur, frag, sums, tig, tot_a);
            else superblock_mma<Q5, NTERMS, NT>(cur, frag, sums, tig, tot_b);
        }

        // combine the kp partial sums of each row group in fixed order:
        // partial[warp][token tile][16 rows][8 tokens][2 streams]
        float *pb = partial + pbuf * (NT * MD_PART_FLOATS) + warp * (NT * 256);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            float *pt = pb + nt * 256;
            pt[(g * 8 + 2 * tig) * 2 + 0] = tot_a[nt][0];
            pt[(g * 8 + 2 * tig + 1) * 2 + 0] = tot_a[nt][1];
            pt[((g + 8) * 8 + 2 * tig) * 2 + 0] = tot_a[nt][2];
            pt[((g + 8) * 8 + 2 * tig + 1) * 2 + 0] = tot_a[nt][3];
            if (DUAL) {
                pt[(g * 8 + 2 * tig) * 2 + 1] = tot_b[nt][0];
                pt[(g * 8 + 2 * tig + 1) * 2 + 1] = tot_b[nt][1];
                pt[((g + 8) * 8 + 2 * tig) * 2 + 1] = tot_b[nt][2];
                pt[((g + 8) * 8 + 2 * tig + 1) * 2 + 1] = tot_b[nt][3];
            }
        }
        const int group_threads = a.kp * 32;
        if (a.kp == 1) __syncwarp();
        else named_barrier_sync(2 + rgi, group_threads);   // rg <= 8 here: barrier ids 2..9
        for (int o = kpi * 32 + lane; o < NT * 128; o += group_threads) {
            const int nt = o >> 7, r = (o >> 3) & 15, tl = o & 7, t = 8 * nt + tl;
            const int orow = row0 + 16 * rgi + r;
            if (orow >= a.n || t >= m_tokens) continue;
            const float *src = partial + pbuf * (NT * MD_PART_FLOATS) + (rgi * a.kp) * (NT * 256) + o * 2;
            float pa = 0.f, pbv = 0.f;
            for (int kq = 0; kq < a.kp; ++kq) {
                pa += src[kq * (NT * 256)];
                if (DUAL) pbv += src[kq * (NT * 256) + 1];
            }
            const float inv = tok_scale[nt * MD_TOK_STRIDE + 8 + tl];
            pa *= inv;
            pbv *= inv;
            if (MODE == 0) store_from_float(gp.y, a.y_dtype, static_cast<size_t>(t) * a.n + orow, pa);
            else if (MODE == 1)
                store_from_float(gp.y, a.y_dtype, static_cast<size_t>(t) * a.n + orow, swiglu_f32(pa, pbv));
            else if (MODE == 2)
                static_cast<float *>(gp.y)[static_cast<size_t>(seg_begin + t) * a.n + orow] = swiglu_f32(pa, pbv);
            else
                out_ptr[t][orow] = pa * route_w[t];
        }
        pbuf ^= 1;
        cur_p = nxt_p;
    }
}

template <bool Q5, int MODE, int NTERMS, int NT = 1>
__global__ void __launch_bounds__(MD_THREADS, 1) mma_direct_kernel(const DirectArgs a) {
    chain_trigger();      // the next kernel of the stream may be scheduled; it waits for this grid itself
    if (MODE >= 2) chain_wait();      // the segment list comes from the plan kernel
    extern __shared__ __align__(128) uint8_t smem[];
    const StagePointers gp{a.x, a.y, a.table_a, a.table_b, a.order, a.seg_expert, a.seg_begin, a.seg_count, a.num_segments, a.route, -1};
    mma_direct_body<Q5, MODE, NTERMS, NT>(a, gp, smem, blockIdx.x, gridDim.x);
}

}  // namespace b200q
