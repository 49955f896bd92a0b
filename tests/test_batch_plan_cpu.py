"""How an lvl02 call's batch is divided over launches (plan_batch in
csrc/pbs_common.cuh), compiled for the host: every plan covers the batch
exactly once, a two-part plan starts with whole passes of its shape, and no
plan is estimated slower than any single launch."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "cufhedb_b200", "csrc")
SMS, BMAX = 148, 4000
SHAPES = (3, 2, 1)
DEFAULT = (16.60, 10.89, 5.72)

PROG = r"""
#include "pbs_common.cuh"
#include <cstdio>
#include <cstdlib>
int main(int argc, char **argv)
{
    const float ms[3] = {(float)atof(argv[1]), (float)atof(argv[2]), (float)atof(argv[3])};
    for (int B = 1; B <= %d; ++B) {
        const cfdb::BatchPlan p = cfdb::plan_batch(B, %d, cfdb::PBS02_SHAPES, ms, cfdb::PBS02_B200_MS);
        std::printf("%%d", p.parts);
        for (int k = 0; k < p.parts; ++k) std::printf(" %%d %%d", p.part[k].n, p.part[k].w);
        std::printf("\n");
    }
    return 0;
}
""" % (BMAX, SMS)


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cu").write_text(PROG)
    subprocess.run([nvcc, "-std=c++17", "-I", CSRC, "-o", str(d / "plan"), str(d / "plan.cu")], check=True,
                   capture_output=True, timeout=300)
    return str(d / "plan")


@pytest.mark.parametrize("ms", [(1.0, 1.0, 1.0), (18.0, 11.2, 6.5), (17.7, 13.8, 10.3), (0.001, 1000.0, 1000.0),
                                (1000.0, 1000.0, 0.001)])
def test_plans_cover_the_batch_and_beat_single_launches(exe, ms):
    out = subprocess.run([exe, *map(repr, ms)], check=True, capture_output=True, text=True).stdout.split("\n")
    t = dict(zip(SHAPES, DEFAULT if ms == (1.0, 1.0, 1.0) else ms))
    cost = lambda n, w: -(-(-(-n // w)) // SMS) * t[w]
    for B in range(1, BMAX + 1):
        f = [int(x) for x in out[B - 1].split()]
        parts = list(zip(f[1::2], f[2::2]))
        assert len(parts) == f[0] <= 2 and sum(n for n, _ in parts) == B and all(n > 0 for n, _ in parts)
        assert all(w in t for _, w in parts)
        if len(parts) == 2:
            assert parts[0][0] % (parts[0][1] * SMS) == 0
        planned = sum(cost(n, w) for n, w in parts)
        assert planned <= min(cost(B, w) for w in t) * (1 + 1e-5), (B, parts)
