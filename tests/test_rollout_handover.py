"""The rollout kernels' loops over steps, compiled for the host with a thread of
the system for each thread of a block: no thread may still be reading a step's
record when thread 0 hands over to the next one.  One thread is held back after
the barrier that ends a step, and every record whose step has not run holds an
error word, as freshly allocated memory may."""
import pathlib
import re
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "phys-engine_gb300" / "csrc"
THREADS = 4

PRELUDE = r"""
#include <algorithm>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>
#include "ad_world.cuh"
#define __host__
#define __device__
#define __global__
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)
#define __grid_constant__
#define __shared__ static
struct Dim { unsigned x; };
thread_local Dim threadIdx;
static const Dim blockDim{THREADS};
using std::min;
static std::mutex g_mutex;
static std::condition_variable g_cv;
static unsigned g_waiting, g_turn;
static unsigned char s_dyn[64];
// A barrier of the block; ends the process when its threads do not all come.
static void __syncthreads() {
    std::unique_lock<std::mutex> lock(g_mutex);
    const unsigned turn = g_turn;
    if (++g_waiting == THREADS) {
        g_waiting = 0;
        ++g_turn;
        g_cv.notify_all();
    } else if (!g_cv.wait_for(lock, std::chrono::seconds(10), [&] { return g_turn != turn; })) {
        std::puts("a thread never came to a barrier");
        std::fflush(stdout);
        std::_Exit(3);
    }
}
static uint32_t atomicAdd(uint32_t *p, uint32_t v) { return __atomic_fetch_add(p, v, __ATOMIC_RELAXED); }
static uint32_t atomicOr(uint32_t *p, uint32_t v) { return __atomic_fetch_or(p, v, __ATOMIC_RELAXED); }
"""

# A step: its record's counters are its own, then the block's barrier, after
# which one thread is late.
STEP = r"""
static unsigned g_forward[THREADS], g_reverse[THREADS];
static void late() {
    if (threadIdx.x == THREADS - 1) std::this_thread::sleep_for(std::chrono::milliseconds(30));
}
static void forwardStepBlock(BlockWorld &bw, bool) {
    if (threadIdx.x == 0)
        for (int k = 0; k < 4; ++k) bw.sc.counts[k] = 0;
    ++g_forward[threadIdx.x];
    __syncthreads();
    late();
}
static void backwardStepBlock(const BlockWorld &bw, bool) {
    ++g_reverse[threadIdx.x];
    if (bw.sc.counts[3]) std::puts("a step is reversed that has not run");
    __syncthreads();
    late();
}
"""

MAIN = r"""
} // namespace
} // namespace pe
int main() {
    using namespace pe;
    constexpr uint32_t n = 2, steps = 5, every = 3, worlds = 2;
    const uint32_t start[worlds + 1] = {0, n, 2 * n}, order[worlds] = {0, 1};
    std::vector<float> ones(16 * n * worlds, 1.0f), out(16 * n * worlds);
    std::vector<uint8_t> flags(n * worlds, 0);
    uint32_t head = 0, err[worlds] = {0, 0};
    Args a{};
    a.nCk = (steps + every - 1) / every + 1;
    a.quarterPerBody = 8;
    a.iterations = 1;
    const size_t bytes = makeLayout(n, worldMaxPairs(n), worldMaxManifolds(n, 8), 1, a.nCk + every + 1, every).stride;
    std::vector<unsigned long long> arena(worlds * (bytes / 8 + 2), ~0ull);
    const unsigned long long off[worlds] = {0, (bytes + 15) / 16 * 16};
    a.arena = reinterpret_cast<unsigned char *>(arena.data());
    a.worldOff = off;
    a.order = order;
    a.bodyStart = start;
    a.shape = a.isStatic = flags.data();
    a.dims = a.iinv = a.mass = a.mu = a.rest = ones.data();
    a.worlds = worlds;
    a.steps = steps;
    a.ckEvery = every;
    a.queueHead = &head;
    a.err = err;
    std::vector<std::thread> block;
    for (unsigned t = 0; t < THREADS; ++t)
        block.emplace_back([&, t] {
            threadIdx.x = t;
            float *in = ones.data(), *o = out.data();
            CALL;
        });
    for (auto &t : block) t.join();
    bool ok = err[0] == 0 && err[1] == 0;
    for (unsigned t = 0; t < THREADS; ++t) ok = ok && g_forward[t] == worlds * steps && g_reverse[t] == REVERSED;
    std::printf("errors %u %u, steps of the threads", err[0], err[1]);
    for (unsigned t = 0; t < THREADS; ++t) std::printf(" %u+%u", g_forward[t], g_reverse[t]);
    std::puts("");
    return ok ? 0 : 1;
}
"""


@pytest.mark.parametrize("kernel", ["forward", "backward"])
def test_no_thread_reads_a_step_record_that_is_handed_over(kernel, tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    rollout, block = (CSRC / "rollout.cu").read_text(), (CSRC / "ad_block.cuh").read_text()
    loops = rollout[rollout.index("using namespace ad;"):rollout.index("// Block size and register budget.")]
    loops = loops.replace("extern __shared__ __align__(16) unsigned char s_dyn[];", "")
    record = re.search(r"struct BlockWorld \{.*?\n\};\n", block, re.S).group(0)
    extra = re.search(r"constexpr int kAdjointExtra = \d+;", block).group(0)
    call, reversed_ = {
        "forward": ("k_rollout_forward<THREADS, 1>(a, in, in, in, in, o, o, o, o)", "0"),
        "backward": ("k_rollout_backward<THREADS, 1>(a, in, in, in, in, o, o, o, o, o, o, o)", "worlds * steps"),
    }[kernel]
    src = tmp_path / "handover.cpp"
    src.write_text("\n".join([
        f"#define THREADS {THREADS}", PRELUDE, "namespace pe { namespace ad { using F = float;", record, extra,
        "} namespace { using namespace ad;", STEP, loops.replace("using namespace ad;", "", 1),
        f"#define CALL {call}", f"#define REVERSED {reversed_}", MAIN]))
    exe = tmp_path / "handover"
    subprocess.run([cxx, "-std=c++20", "-O1", "-w", "-pthread", f"-I{CSRC}", str(src), "-o", str(exe)], check=True,
                   timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
