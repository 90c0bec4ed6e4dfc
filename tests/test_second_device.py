"""The launchers of kernels with more dynamic shared memory than a kernel has by
default, compiled for the host against a CUDA runtime of two devices that
remembers each kernel's limit on each device: a process that steps worlds on
both must raise it on both."""
import pathlib
import re
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "phys-engine_gb300" / "csrc"
CUDA = pathlib.Path("/usr/local/cuda/include")

RUNTIME = r"""
#include <cstdio>
#include <map>
#include <utility>
#include "pe_stages.h"
static int g_device;
static std::map<std::pair<int, const void *>, size_t> g_limit;
static int g_refused, g_launches;
extern "C" cudaError_t CUDARTAPI cudaGetDevice(int *d) { return *d = g_device, cudaSuccess; }
extern "C" cudaError_t CUDARTAPI cudaGetLastError() { return cudaSuccess; }
extern "C" const char *CUDARTAPI cudaGetErrorString(cudaError_t) { return ""; }
extern "C" cudaError_t CUDARTAPI cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int v) {
    g_limit[{g_device, f}] = (size_t)v;
    return cudaSuccess;
}
template <class... A> static cudaError_t cudaFuncSetAttribute(void (*f)(A...), cudaFuncAttribute a, int v) {
    return cudaFuncSetAttribute((const void *)f, a, v);
}
template <class K> static void launch(K *kernel, size_t bytes) {
    ++g_launches;
    const auto it = g_limit.find({g_device, (const void *)kernel});
    if (bytes > (it == g_limit.end() ? 48u * 1024u : it->second)) ++g_refused;
}
namespace pe {
unsigned long long g_kernelLaunches;
constexpr uint32_t kRegSortThreads = 1024, kSapBlockMax = 4096, kSapBlockPairs = 8192;
"""


def function(text, name):
    """The launcher `name` (with its template head), its launches as calls."""
    at = re.search(r"^(template <[^\n]*>\s*)?(static )?(void|bool) " + name + r"\(", text, re.M).start()
    body = text[at:text.index("\n}\n", at) + 3]
    return re.sub(r"(\w+(?:<[\w, ]+>)?)<<<[^,]*, [^,]*, (\w+), s>>>\(.*?\);", r"launch(\1, \2);", body, flags=re.S)


def test_shared_memory_limits_are_raised_on_every_device(tmp_path):
    cxx = shutil.which("g++")
    if not cxx or not (CUDA / "cuda_runtime.h").exists():
        pytest.skip("no g++ or no CUDA headers")
    broad, tree = (CSRC / "k_broad.cu").read_text(), (CSRC / "k_lbvh.cu").read_text()
    front = re.search(r"constexpr size_t frontBytes.*?\n", tree).group(0)
    sap = re.search(r"template <uint32_t N> constexpr bool kSapScratchInBuffer.*?\n}\n", broad, re.S).group(0)
    src = tmp_path / "devices.cpp"
    src.write_text("\n".join([
        RUNTIME, front, sap,
        "template <uint32_t T, int E> void k_sap_block() {}", "template <int E> void k_lbvh_front() {}",
        "void k_pairs_lists() {}", "bool sapFinalizesPairs(const BroadInput &, const PairBuffers &) { return true; }",
        function(broad, "launchSapBlock"), function(broad, "launchPairsLists"), function(tree, "launchFront"), "}",
        r"""
int main() {
    using namespace pe;
    BroadInput in{};
    PairBuffers pb{};
    LbvhBuffers lb{};
    PairMapping map{};
    for (int turn = 0; turn < 4; ++turn) {
        g_device = turn & 1;
        launchSapBlock<128, 1>(in, nullptr, nullptr, pb, nullptr, nullptr, nullptr, nullptr);
        launchSapBlock<1024, 4>(in, nullptr, nullptr, pb, nullptr, nullptr, nullptr, nullptr);
        launchPairsLists(in, map, pb, nullptr, nullptr);
        launchFront<1>(in, lb, 10, nullptr);
        launchFront<4>(in, lb, 12, nullptr);
    }
    std::printf("%d of %d launches refused, %zu limits\n", g_refused, g_launches, g_limit.size());
    return g_refused != 0 || g_launches != 20 || g_limit.size() != 10;
}
"""]))
    exe = tmp_path / "devices"
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", f"-I{CSRC}", f"-I{CUDA}", str(src), "-o", str(exe)], check=True,
                   timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_no_kernel_limit_is_kept_for_the_process():
    for f in sorted(CSRC.glob("*.cu")):
        for kept in re.findall(r"static (?:bool|int) \w+ = (?:false|-1);", f.read_text()):
            raise AssertionError(f"{f.name}: {kept}")
