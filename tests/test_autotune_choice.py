"""The batch's choice of kernel variants, compiled for the host against a clock:
one launch held up by the host, wherever it falls, must not change the choice."""
import pathlib
import re
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "phys-engine_gb300" / "csrc"

HARNESS = r"""
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <vector>
#define PE_CHECK(expr) expr
constexpr int kBatchVariantCount = 5;
struct BatchView {};
struct BatchBucket {
    std::vector<uint32_t> worlds = std::vector<uint32_t>(8);
    std::vector<double> candidateMs;
    uint32_t maxN = 0, maxM = 0, blocks = 0;
    int variant = 2;
    double tunedMs = 0.0;
};
// Variants' times alone and within a step: in the second bucket variant 3 is the
// fastest alone and variant 1 the one that leaves room for the first bucket.
static const double kAlone[2][5] = {{5.0, 4.0, 4.5, 6.0, 7.0}, {9.0, 6.0, 8.0, 5.0, 7.0}};
static const double kStep[2][5] = {{3.0, 2.0, 2.5, 4.0, 5.0}, {6.0, 3.0, 5.0, 3.4, 4.0}};
static double g_now, g_t[2];
static int g_calls, g_late = -1;
static void spend(double ms) { g_now += ms + (g_calls++ == g_late ? 5.0 : 0.0); }
static void launchBatchBucket(const BatchView &, int v, uint32_t bucket, int) { spend(kAlone[bucket][v]); }
static size_t batchSharedBytes(uint32_t, uint32_t) { return 0; }
static uint32_t batchMaxBlocks(int, size_t) { return 8; }
static void cudaSetDevice(int) {}
static void cudaMemsetAsync(void *, int, size_t, int) {}
static void cudaStreamSynchronize(int) {}
static void cudaEventRecord(int e, int) { g_t[e] = g_now; }
static void cudaEventElapsedTime(float *ms, int a, int b) { *ms = (float)(g_t[b] - g_t[a]); }
struct Words { uint32_t *ptr = nullptr; };
struct Batch {
    int device_ = 0, stream_ = 0, t0_ = 0, t1_ = 1;
    uint32_t parity_ = 0, err = 0, *hostErr_ = &err;
    Words queueHead_, batchErr_;
    std::vector<BatchBucket> buckets_ = std::vector<BatchBucket>(2);
    BatchView view(const BatchBucket &, float, uint32_t) const { return {}; }
    void launchAll(float, uint32_t) { spend(kStep[0][buckets_[0].variant] + kStep[1][buckets_[1].variant]); }
    bool finishStep() { return true; }
    void dropGraphs() {}
    void setVariant(BatchBucket &bk, int v) { bk.variant = v; }
    void autotune(float dt, int reps);
};
"""

MAIN = r"""
int main() {
    int bad = 0, total = 0;
    for (int reps : {1, 3}) {
        Batch quiet;
        g_calls = 0;
        g_late = -1;
        quiet.autotune(0.01f, reps);
        total = g_calls;
        if (quiet.buckets_[0].variant != 1 || quiet.buckets_[1].variant != 1) ++bad;
        for (g_late = 0; reps > 1 && g_late < total; ++g_late) {
            Batch b;
            g_calls = 0;
            b.autotune(0.01f, reps);
            if (b.buckets_[0].variant != 1 || b.buckets_[1].variant != 1) ++bad;
        }
    }
    std::printf("%d wrong choices, %d launches\n", bad, total);
    return bad != 0;
}
"""


def test_one_late_launch_does_not_change_the_variants(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    text = (CSRC / "batch.cu").read_text()
    at = text.index("void Batch::autotune(")
    body = text[at:text.index("\n}\n", at) + 3]
    # the bucket's index goes to the stub in place of its number of blocks
    body, n = re.subn(r"launchBatchBucket\(view, v, blocks, stream_\)", "launchBatchBucket(view, v, (uint32_t)bi, stream_)", body)
    assert n == 1
    src = tmp_path / "tune.cpp"
    src.write_text(HARNESS + body + MAIN)
    exe = tmp_path / "tune"
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", str(src), "-o", str(exe)], check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
