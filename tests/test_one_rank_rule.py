"""The rule for a solve on one rank of the cluster, compiled for the host: the
bytes of any count of manifolds and points against the shared memory."""
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "phys-engine_gb300" / "csrc"
CUDA = pathlib.Path("/usr/local/cuda/include")


def test_one_rank_rule_for_any_count(tmp_path):
    cxx = shutil.which("g++")
    if not cxx or not (CUDA / "cuda_runtime.h").exists():
        pytest.skip("no g++ or no CUDA headers")
    src = tmp_path / "rule.cpp"
    src.write_text(r"""
#include <cstdio>
#include "pe_stages.h"
int main() {
    unsigned m, p, b;
    while (std::scanf("%u %u %u", &b, &m, &p) == 3)
        std::printf("%d\n", (int)pe::clusterFitsOneRank(b, pe::blockStageSlots(b), m, p));
}
""")
    exe = tmp_path / "rule"
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", f"-I{CSRC}", f"-I{CUDA}", str(src), "-o", str(exe)], check=True,
                   timeout=300)
    cases = [(b, m, p) for b in (64, 1024, 4096) for m in (0, 64, 900, 5_000_000, 134_217_728, 2**32 - 1)
             for p in (0, 64, 700, 24_403_223, 24_403_224, 2**32 // 176 * 2 + 5, 2**32 - 1)]
    r = subprocess.run([str(exe)], input="\n".join("%u %u %u" % c for c in cases), capture_output=True, text=True,
                       check=True, timeout=60)
    for (b, m, p), got in zip(cases, r.stdout.split()):
        slots = min(2 * b, 3072)
        want = (b * 20 + slots * 36 + 15) // 16 * 16 + 32 * m + 176 * p <= 224 * 1024
        assert bool(int(got)) == want, (b, m, p)
