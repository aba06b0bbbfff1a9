"""The control flow of the streaming grouped kernels (``csrc/grouped_stream.cuh``) when a wait's limit runs out, on the CPU:
the header's own text, a thread per warp, barriers that count. Whichever warp gives up at whichever wait, every warp has to
come to its end: the team's meeting has no limit of its own, so a warp that leaves without it would hold the others for
good."""

import re
import shutil
import subprocess
from pathlib import Path

import pytest

import mylocal_llm_b200

CSRC = Path(mylocal_llm_b200.__file__).parent / "csrc"

STUBS = r"""
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>
using std::max; using std::min;
#define __device__
#define __forceinline__ inline
struct Dim { int x; };
thread_local Dim threadIdx;
static Dim blockIdx{0}, gridDim{1};
constexpr int STATUS = 0;
static std::mutex mu;
static std::condition_variable cv;
static std::atomic<bool> hung{false};
static int fail_warp = -1, fail_at = -1, gave_up = 0;
thread_local int waits = 0;
struct Bar { int expected = 0, arrived = 0, phase = 0; };
static Bar &bar(uint64_t *b) { return *reinterpret_cast<Bar *>(*b); }
static void mbar_init(uint64_t *b, int n) { Bar *p = new Bar; p->expected = n; *b = reinterpret_cast<uint64_t>(p); }
static void mbar_arrive(uint64_t *b) {
    std::lock_guard<std::mutex> l(mu);
    Bar &x = bar(b);
    if (++x.arrived == x.expected) { x.arrived = 0; x.phase ^= 1; cv.notify_all(); }
}
static void mbar_arrive_expect_tx(uint64_t *b, uint32_t) { mbar_arrive(b); }       // (copies land at once)
static bool mbar_wait_bounded(uint64_t *b, uint32_t parity, int *status, int code) {
    std::unique_lock<std::mutex> l(mu);
    const bool refuse = threadIdx.x / 32 == fail_warp && waits++ == fail_at;
    // (the first give-up is the planted one; from then on every wait has 40 ms, those that had begun included)
    for (int slices = 0; !refuse && (!gave_up || slices < 2); slices += gave_up > 0)
        if (cv.wait_for(l, std::chrono::milliseconds(20), [&] { return bar(b).phase != (int)parity; })) return true;
    ++gave_up;
    *status = code;
    return false;
}
struct Meet { int arrived = 0, round = 0; };
static Meet meets[17];
static void named_barrier_sync(int id, int threads) {                              // no limit on the GPU
    std::unique_lock<std::mutex> l(mu);
    Meet &m = meets[id];
    const int round = m.round;
    if (++m.arrived == threads / 32) { m.arrived = 0; ++m.round; cv.notify_all(); return; }
    if (!cv.wait_for(l, std::chrono::seconds(10), [&] { return m.round != round; })) { hung = true; m.arrived = 0; ++m.round; cv.notify_all(); }
}
static std::mutex sync_mu;
static void __syncthreads();
static void __syncwarp() {}
static int __all_sync(unsigned, int v) { return v; }
static void fence_barrier_init() {}
static void bulk_copy_g2s(void *, const void *, uint32_t, uint64_t *) {}
static const uint8_t *expert_matrix(const uint8_t *base, long long stride, const unsigned long long *, int e) { return base + e * stride; }
"""

MAIN = r"""
using namespace b200q;
static Meet everyone;
static void __syncthreads() {
    std::unique_lock<std::mutex> l(mu);
    const int round = everyone.round;
    if (++everyone.arrived == GS_WARPS) { everyone.arrived = 0; ++everyone.round; cv.notify_all(); return; }
    cv.wait(l, [&] { return everyone.round != round; });
}
int main(int argc, char **argv) {
    const int kp = atoi(argv[1]);
    fail_warp = atoi(argv[2]); fail_at = atoi(argv[3]);
    constexpr int SEGMENTS = 7, N = 16 * 24, NSB = 8;
    std::vector<int32_t> order(SEGMENTS * 8), expert(SEGMENTS), begin(SEGMENTS), count(SEGMENTS, 3);
    for (int i = 0; i < SEGMENTS; ++i) { expert[i] = i; begin[i] = 8 * i; }
    int32_t segments = SEGMENTS;
    int status = 0;
    std::vector<uint8_t> smem(1 << 20);
    GroupedArgs a{};
    a.n = N; a.nsb = NSB; a.kp = kp; a.image_bytes = 64; a.smem_stride = 96; a.bufs = 2; a.off_bufs = 1 << 18; a.ring = 3;
    a.off_ring = 1 << 17; a.topk = 1; a.order = order.data(); a.seg_expert = expert.data(); a.seg_begin = begin.data();
    a.seg_count = count.data(); a.num_segments = &segments; a.max_segments = SEGMENTS; a.status = &status;
    std::vector<float> partial(2 * GS_WARPS * 32 * 8);
    std::atomic<int> groups{0};
    std::vector<std::thread> warps;
    for (int w = 0; w < GS_WARPS; ++w)
        warps.emplace_back([&, w] {
            threadIdx.x = 32 * w;
            int pbuf = 0;
            const int team = w / kp, kpi = w - team * kp;
            grouped_walk<false, 64, true>(a, smem.data(), [&](int, int, const uint8_t *, TileStream<64, true> &stream) -> bool {
                bool ok = true;
                for (int sb = kpi; sb < NSB && ok; sb += kp)
                    for (int m = 0; m < 2 && ok; ++m) {
                        const uint8_t *tile;
                        if (!(ok = stream.next(tile))) break;
                        stream.refill(0);
                    }
                float v[8] = {};
                if (!add_parts(v, partial.data(), pbuf, kp, team, kpi, w, 0) || !ok) return ok;
                ++groups;
                return true;
            });
        });
    for (auto &t : warps) t.join();
    printf("%d %d %d %d\n", (int)hung.load(), status, groups.load(), gave_up);
}
"""


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no C++ compiler")
    text = (CSRC / "grouped_stream.cuh").read_text()
    text = re.sub(r"#pragma once|#include .*|#pragma unroll", "", text)
    # the one function of PTX: its two instructions by name
    text, n = re.subn(r"(void request_tile\([^{]*\{).*?\n\}\n", r"\1 (void)dst; (void)src; if (issue) mbar_arrive_expect_tx(bar, bytes); }\n",
                      text, flags=re.S)
    assert n == 1
    path = tmp_path_factory.mktemp("walk")
    (path / "walk.cpp").write_text(STUBS + text + MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-w", "walk.cpp", "-o", "walk"], cwd=path, check=True)
    return path / "walk"


def run(walk, kp, warp, at):
    out = subprocess.run([str(walk), str(kp), str(warp), str(at)], capture_output=True, text=True, timeout=100, check=True).stdout
    return [int(v) for v in out.split()]


@pytest.mark.parametrize("kp", [1, 2, 8])
def test_every_group_is_computed(walk, kp):
    assert run(walk, kp, -1, -1) == [0, 0, 7 * 24, 0]


@pytest.mark.parametrize("kp", [1, 2, 4, 8])
@pytest.mark.parametrize("warp,at", [(0, 0), (0, 1), (0, 9), (1, 0), (1, 1), (1, 6), (3, 2), (7, 11), (14, 4)])
def test_a_wait_that_gives_up_ends_the_kernel(walk, kp, warp, at):
    hung, status, groups, gave_up = run(walk, kp, warp, at)
    assert not hung and gave_up and status in (121, 122, 123) and groups < 7 * 24
