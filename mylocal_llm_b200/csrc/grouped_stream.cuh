// Grouped expert projections for plans of many segments (sm_100a): every warp streams its own tiles.
//
// The block-structured grouped kernels (mma_direct.cuh, q6k_tiled.cuh) stop the whole CTA whenever a segment (a run of up
// to eight tokens of one expert) ends: two barriers, a dependent look-up and the conversion or gather of the next
// segment's activations, 2-4 us each, and their blocks of 64-128 rows leave CTAs with nine or ten of them. Here
//   * the unit of work is one 16-row group of one segment (times a part of K, kp warps per group, where a plan is small);
//     a CTA owns a contiguous run of them and deals them to its warps in turn, so the warps of the chip finish within one
//     group of each other;
//   * the tokens' fragments are ready-made images (one per row of the input: mma_direct.cuh's token images, or
//     hidden_image_kernel for the hidden activations) that one bulk copy per token brings into a ring of segment buffers,
//     two segments ahead; a warp that enters a segment waits for its buffer's mbarrier and for nothing else;
//   * weights come by one bulk copy per tile into a ring of the warp's own (two to four tiles of 2.3-4.4 KB), refilled as
//     soon as a tile is in registers: 100-200 KB per SM are on their way at any time (two register sets in turn kept 37 KB
//     in flight and the warps waited for memory: 3.3 stalled per issue).
// Image rows lie behind one another in shared memory, 32 (token images, 8 bytes per lane and fragment) or 64 bytes (hidden
// images, pairs of fragments, 16 bytes per lane) more than a multiple of 128 apart, so the tokens of one wavefront read
// different banks.
// The sums are those of the block-structured kernels with the same kp, bit for bit.
// Bound by instruction issue (256 tokens, 512 experts, gate/up and down: 0.67 of the slots, ALU pipe 0.61 / 0.58, DRAM 3.5 /
// 3.3 TB/s; 428 and 679 instructions per 16 x 256 tile): positions in the run of row groups are kept by steps instead of
// divisions, and the copies are predicated, not branched around (3 % of an 8-layer step of 64 tokens). Block-structured ->
// streaming: 8-layer step of 64 tokens 2158 -> 2082 us, layer of 256 tokens 437 -> 378, of 16 tokens 143 -> 136.
#pragma once

#include "q6k_tiled.cuh"

namespace b200q {

constexpr int GS_WARPS = 16;
constexpr int GS_THREADS = GS_WARPS * 32;
constexpr int GS_MAX_BUFS = 3;                                 // segment buffers: bufs - 1 segments are requested ahead
constexpr int GS_MAX_RING = 4;                                 // tiles of a warp's ring
constexpr int GS_CTRL_BYTES = 1024;                            // mbarriers: [0, 64) segments, [64, 576) tiles
constexpr int GS_PART_BYTES = 2 * GS_WARPS * 32 * 8 * 4;       // K parts: [2][warp][lane][8]
constexpr int STATUS_GROUPED_WAIT = 121;                       // gave up waiting for a segment's activations
constexpr int STATUS_GROUPED_FREE = 122;                       // gave up waiting for a segment buffer
constexpr int STATUS_GROUPED_TILE = 123;                       // gave up waiting for a weight tile

struct GroupedArgs {
    const uint8_t *wa, *wb;
    long long stride_a, stride_b;
    const unsigned long long *table_a, *table_b;
    int n, nsb, kp;                // rows and super-blocks per row of an expert's matrix; warps per row group
    const uint8_t *images;         // one image per row of x (gate/up) or per sorted assignment (down)
    int image_bytes, smem_stride;  // bytes of an image; distance between two in shared memory
    int bufs, off_bufs;
    int ring, off_ring;            // tiles per warp ring; start of the rings in shared memory
    int topk;
    const int32_t *order, *seg_expert, *seg_begin, *seg_count, *num_segments;
    int max_segments;
    float *y;
    const float *route;
    int flat_rows;
    const uint64_t *y_table;
    int rows_per_rank;
    int *status;
};

// The CTA's ring of segment buffers as a warp sees it.
struct SegmentRing {
    uint64_t *full, *empty;
    int first, last;               // segments of this CTA: first .. last (inclusive)
    int bufs;
    int issued;                    // producer warp: next segment to request
};

// Requests the images of segment `seg` (all lanes of the producer warp); false = gave up waiting for the buffer.
template <bool SORTED>
__device__ __forceinline__ bool request_segment(const GroupedArgs &a, SegmentRing &ring, int seg, uint8_t *bufs, int lane) {
    const int at = seg - ring.first, buf = at % ring.bufs, use = at / ring.bufs;
    bool ok = true;
    if (use > 0) ok = __all_sync(0xffffffffu, mbar_wait_bounded(&ring.empty[buf], (use - 1) & 1, a.status, STATUS_GROUPED_FREE));
    if (!ok) return false;
    const int begin = a.seg_begin[seg], count = min(a.seg_count[seg], 8);
    if (lane == 0) mbar_arrive_expect_tx(&ring.full[buf], static_cast<uint32_t>(count) * a.image_bytes);
    __syncwarp();
    if (lane < count) {
        const int row = SORTED ? begin + lane : a.order[begin + lane] / a.topk;
        bulk_copy_g2s(bufs + static_cast<size_t>(buf) * 8 * a.smem_stride + lane * a.smem_stride,
                      a.images + static_cast<size_t>(row) * a.image_bytes, a.image_bytes, &ring.full[buf]);
    }
    return true;
}

// Position in the CTA's run of row groups, advanced a round of teams at a time (a division per item costs as much as a
// tile's loads).
struct GroupCursor {
    int item, seg, group;
    __device__ __forceinline__ void step(int teams, int groups_per_seg) {
        item += teams;
        group += teams;
        while (group >= groups_per_seg) {
            group -= groups_per_seg;
            ++seg;
        }
    }
};

// One bulk copy into the ring, announced on its barrier; issued by the lane that `issue` names, without a branch.
__device__ __forceinline__ void request_tile(bool issue, uint64_t *bar, uint8_t *dst, const uint8_t *src, uint32_t bytes) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %0, 0;\n\t"
        "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %4;\n\t"
        "@p cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%2], [%3], %4, [%1];\n\t}" ::"r"(
            static_cast<int>(issue)),
        "r"(smem_u32(bar)), "r"(smem_u32(dst)), "l"(src), "r"(bytes)
        : "memory");
}

// A warp's stream of weight tiles: the tiles of its row groups in order (DUAL: gate and up alternating), fetched by bulk
// copies a ring ahead of their use. All lanes keep the cursor, lane 0 issues.
template <int TILE, bool DUAL>
struct TileStream {
    const GroupedArgs &a;
    uint8_t *slots;                // this warp's ring
    uint64_t *full;                // its mbarriers
    int slot, phase;               // next tile to consume
    int item, end, teams, kpi;     // fetch cursor: row group, its tile, stream; end of the CTA's range
    GroupCursor ahead;             // the row group after that: na, nb are its matrices
    int groups_per_seg, sb, upper;
    const uint8_t *wa, *wb, *na, *nb;

    __device__ __forceinline__ void bases(const GroupCursor &at, const uint8_t *&pa, const uint8_t *&pb) const {
        if (at.item >= end) return;
        const int expert = a.seg_expert[at.seg];
        const size_t off = (static_cast<size_t>(at.group) * a.nsb + kpi) * TILE;
        pa = expert_matrix(a.wa, a.stride_a, a.table_a, expert) + off;
        if (DUAL) pb = expert_matrix(a.wb, a.stride_b, a.table_b, expert) + off;
    }
    __device__ __forceinline__ void start(const GroupCursor &first, int lane) {
        item = first.item;
        ahead = first;
        sb = kpi;
        upper = 0;
        slot = phase = 0;
        wa = wb = na = nb = nullptr;
        bases(first, wa, wb);
        ahead.step(teams, groups_per_seg);
        bases(ahead, na, nb);
        for (int i = 0; i < a.ring; ++i) fetch(i, lane);
    }
    // requests the tile at the cursor into slot `into` and moves on
    __device__ __forceinline__ void fetch(int into, int lane) {
        if (item >= end) return;
        request_tile(lane == 0, &full[into], slots + into * TILE, (DUAL && upper) ? wb : wa, TILE);
        if (DUAL) {
            upper ^= 1;
            if (upper) return;
        }
        sb += a.kp;
        wa += a.kp * TILE;
        if (DUAL) wb += a.kp * TILE;
        if (sb >= a.nsb) {
            item += teams;
            sb = kpi;
            wa = na;
            wb = nb;
            ahead.step(teams, groups_per_seg);
            bases(ahead, na, nb);
        }
    }
    // the next tile in shared memory (false: gave up); after its last read the caller calls refill()
    __device__ __forceinline__ bool next(const uint8_t *&tile) {
        tile = slots + slot * TILE;
        return __all_sync(0xffffffffu, mbar_wait_bounded(&full[slot], phase, a.status, STATUS_GROUPED_TILE)) != 0;
    }
    __device__ __forceinline__ void refill(int lane) {
        __syncwarp();
        fetch(slot, lane);
        if (++slot == a.ring) {
            slot = 0;
            phase ^= 1;
        }
    }
};

// Sums the K parts of a team's row group in ascending order: every warp but the first stores its eight sums, the team
// meets, the first warp adds. Two buffers in turn: a warp stores into a buffer again only after the team's next meeting,
// which the first warp reaches with its reads of that buffer done. Returns true in the warp that holds the total. A warp whose
// wait gave up comes here too: the meeting has no limit of its own.
template <int COUNT>
__device__ __forceinline__ bool add_parts(float (&v)[COUNT], float *partial, int &pbuf, int kp, int team, int kpi, int warp, int lane) {
    if (kp == 1) return true;
    float *buf = partial + pbuf * (GS_WARPS * 32 * 8);
    pbuf ^= 1;
    if (kpi) {
#pragma unroll
        for (int i = 0; i < COUNT; ++i) buf[(warp * 8 + i) * 32 + lane] = v[i];
    }
    named_barrier_sync(1 + team, kp * 32);
    if (kpi) return false;
    for (int q = 1; q < kp; ++q)
#pragma unroll
        for (int i = 0; i < COUNT; ++i) v[i] += buf[((warp + q) * 8 + i) * 32 + lane];
    return true;
}

// Warp-level walk over the CTA's work. SORTED: image rows are sorted assignments. The functor
// `work(seg, group, images, stream)` computes one row group from the images of its segment and the stream's next tiles;
// it returns false when a wait gave up, after it has met its team. A warp that gave up meets its team once for each of its
// remaining groups as well, so that the others get past it to their own limits.
template <bool SORTED, int TILE, bool DUAL, typename WorkFn>
__device__ __forceinline__ void grouped_walk(const GroupedArgs &a, uint8_t *smem, const WorkFn work) {
    uint64_t *full = reinterpret_cast<uint64_t *>(smem), *empty = full + 4;
    uint8_t *bufs = smem + a.off_bufs;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int groups_per_seg = a.n >> 4;
    const int nseg = min(*a.num_segments, a.max_segments);
    const long long total = static_cast<long long>(nseg) * groups_per_seg;
    const int begin = static_cast<int>(total * blockIdx.x / gridDim.x), end = static_cast<int>(total * (blockIdx.x + 1) / gridDim.x);
    if (begin >= end) return;
    SegmentRing ring{full, empty, begin / groups_per_seg, (end - 1) / groups_per_seg, a.bufs, 0};
    uint64_t *tile_bars = reinterpret_cast<uint64_t *>(smem + 64) + warp * GS_MAX_RING;
    if (tid == 0) {
        for (int b = 0; b < a.bufs; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&empty[b], GS_WARPS);
        }
    }
    if (lane == 0)
        for (int i = 0; i < GS_MAX_RING; ++i) mbar_init(&tile_bars[i], 1);
    fence_barrier_init();
    __syncthreads();
    const int teams = GS_WARPS / a.kp, team = warp / a.kp, kpi = warp - team * a.kp;
    GroupCursor at{begin, ring.first, begin - ring.first * groups_per_seg};     // this warp's row group
    at.step(team, groups_per_seg);
    int seg = ring.first, buf = 0, phase = 0;              // segment this warp is in, its buffer and that buffer's round
    TileStream<TILE, DUAL> stream{a, smem + a.off_ring + static_cast<size_t>(warp) * a.ring * TILE, tile_bars};
    stream.end = end;
    stream.teams = teams;
    stream.kpi = kpi;
    stream.groups_per_seg = groups_per_seg;
    stream.start(at, lane);
    ring.issued = ring.first;
    bool ok = true;
    const int ahead = a.bufs - 1;
    if (warp == 0)
        while (ok && ring.issued <= min(ring.first + ahead, ring.last)) ok = request_segment<SORTED>(a, ring, ring.issued++, bufs, lane);

    bool entered = false;                                  // this warp has waited for segment `seg`
    auto wait_full = [&](int b, int ph) {
        return __all_sync(0xffffffffu, mbar_wait_bounded(&full[b], ph, a.status, STATUS_GROUPED_WAIT)) != 0;
    };
    // Leaves the segments before `upto` in order, each after its activations have landed (also those this warp has no
    // group in: a buffer's next round can then not be released before this one). The producer requests the segments that
    // now fit only on its next entry (below): it would wait here for warps that are still in the segment it left.
    auto advance = [&](int upto) {
        while (ok && seg < upto) {
            if (!entered) ok = wait_full(buf, phase);
            if (ok && lane == 0) mbar_arrive(&empty[buf]);
            ++seg;
            if (++buf == a.bufs) {
                buf = 0;
                phase ^= 1;
            }
            entered = false;
            if (warp == 0)
                while (ok && ring.issued <= min(seg + ahead - 1, ring.last)) ok = request_segment<SORTED>(a, ring, ring.issued++, bufs, lane);
        }
    };
    while (ok && at.item < end) {
        advance(at.seg);
        if (ok && !entered) {
            ok = wait_full(buf, phase);
            entered = true;
        }
        if (!ok) break;
        ok = work(seg, at.group, bufs + static_cast<size_t>(buf) * 8 * a.smem_stride, stream);
        at.step(teams, groups_per_seg);
        // after its first group of a segment the producer asks for the one whose buffer the others have left by now
        if (warp == 0 && ok && ring.issued <= min(seg + ahead, ring.last)) ok = request_segment<SORTED>(a, ring, ring.issued++, bufs, lane);
    }
    if (!ok && a.kp > 1)
        for (; at.item < end; at.step(teams, groups_per_seg)) named_barrier_sync(1 + team, a.kp * 32);
    advance(ring.last + 1);
    if (!ok) {
        // gave up: copies may still be on their way into this CTA's shared memory - let each of them land (bounded)
        if (warp == 0)
            for (int s = max(ring.first, ring.issued - a.bufs); s < ring.issued; ++s)
                wait_full((s - ring.first) % a.bufs, ((s - ring.first) / a.bufs) & 1);
        for (int i = 0; i < a.ring; ++i) {
            mbar_wait_bounded(&tile_bars[stream.slot], stream.phase, a.status, STATUS_GROUPED_TILE);
            if (++stream.slot == a.ring) {
                stream.slot = 0;
                stream.phase ^= 1;
            }
        }
    }
}

}  // namespace b200q
