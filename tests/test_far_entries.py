"""Single nuclear entries between points far apart on an axis, and the table of
live strips that their K ranges index.

An axis holds the two points of a single entry, any distance apart, and the
contraction's K range covers the span between them: 6 gap + 99 lattice positions
at tol 1e-8 for G10, in chunks of 16.  Up to a gap of 666 that is at most 256
chunks, what a block's table holds; from 667 on it is more.

Tolerance: the parity bar of the other nuclear tests (1e-12 relative + 1e-14)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from _common import HERE, assert_parity, g10
from oracle_binding import Oracle

REPO = os.path.dirname(HERE)
CSRC = os.path.join(REPO, "gausslectronitegrate_b200", "csrc")
DEBUG_LIB = os.path.join(REPO, "gausslectronitegrate_b200", "libgli_b200_debug.so")

TABLE_PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "dmma.cuh"
using namespace gli;
int main() {
    srand(7);
    const int sizes[] = {1, 2, 255, 256, 257, 258, 300, 1000, 40000, 70000};
    for (int nk : sizes)
        for (int turn = 0; turn < 20; ++turn) {
            constexpr int STRIPS = 8;
            int first[STRIPS], last[STRIPS], run[STRIPS];
            for (int t = 0; t < STRIPS; ++t) {
                const int a = rand() % nk, b = rand() % nk;
                const bool empty = rand() % 5 == 0;
                first[t] = empty ? 0 : a < b ? a : b;
                last[t] = empty ? -1 : turn == 0 ? nk - 1 : a < b ? b : a;
                run[t] = dm_strip_run(first[t], last[t]);
            }
            for (int kc = 0; kc < nk; kc = kc < 600 ? kc + 1 : kc + 61) {
                const int e = dm_run_entry(kc);
                if (e < 0 || e >= DM_MAX_CHUNKS || e >= nk) return printf("chunk %d of %d reads entry %d\n", kc, nk, e), 1;
                for (int g = 0; g < 2; ++g) {
                    const unsigned live = dm_live_run<STRIPS>(run, g, e), lo = live & 0xff, hi = live >> 8;
                    unsigned want_lo = STRIPS / 2, want_hi = 0;
                    for (int t = 0; t < STRIPS / 2; ++t)
                        if (first[2 * t + g] <= kc && kc <= last[2 * t + g]) {
                            if (want_lo > (unsigned)t) want_lo = t;
                            want_hi = t + 1;
                        }
                    const bool covers = want_hi <= want_lo || (lo <= want_lo && want_hi <= hi);
                    const bool equal = want_hi <= want_lo ? live == 0 : lo == want_lo && hi == want_hi;
                    if (!covers || hi > STRIPS / 2 || (nk <= DM_MAX_CHUNKS && !equal))
                        return printf("chunk %d of %d, parity %d: %u..%u\n", kc, nk, g, lo, hi), 1;
                }
            }
        }
    puts("table ok");
    return 0;
}
"""


def test_strip_table_covers_any_k_range(tmp_path):
    # the table's arithmetic on the host: no chunk reads past it, every live strip is covered
    src, exe = tmp_path / "table.cu", tmp_path / "table"
    src.write_text(TABLE_PROGRAM)
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC, "-I",
                    os.path.join(REPO, "include"), "-o", str(exe), str(src)], check=True, timeout=600)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "table ok" in r.stdout, r.stdout + r.stderr


POS = np.array([[0.3, -0.2, 0.1], [20.0, 0.0, -1.0]])
Q = [1, 7]


def check_gaps():
    import gausslectronitegrate_b200 as gli
    oracle = Oracle()
    for axis in range(3):
        for gap in (1, 6, 18, 666, 667, 1500):
            p = [[0, 1, 0], [1, 0, 0]]
            p[0][axis], p[1][axis] = -1, gap - 1
            got = gli.compute_nuclear_gausslet_integral(g10(), [tuple(x) for x in p], POS, Q, 1e-8)
            ref = oracle.nuclear_single(g10(), p, POS, Q, 1e-8)
            assert (ref != 0) == (gap < 17), (gap, ref)
            assert_parity(np.array([got]), np.array([ref]), what=f"gap {gap} on axis {axis}")


@pytest.mark.gpu
def test_far_entries_against_oracle():
    check_gaps()


@pytest.mark.gpu
def test_far_entries_in_the_bounds_checked_build():
    code = (f"import sys; sys.path[:0] = [{REPO!r}, {HERE!r}, {os.path.join(REPO, 'oracle')!r}]\n"
            "import test_far_entries as t, gausslectronitegrate_b200 as gli\n"
            "assert gli._abi.LIB_PATH.endswith('libgli_b200_debug.so')\n"
            "t.check_gaps(); print('gaps ok')\n")
    env = dict(os.environ, GLI_B200_LIBRARY=DEBUG_LIB)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env=env, timeout=900)
    assert r.returncode == 0 and "gaps ok" in r.stdout, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("gap", [(700, 700, 700), (1, 100_000, 0), (1_000_000, -1_000_000, 1_000_000)])
def test_entries_far_apart_are_zero(gap):
    # the lattice box between such points takes terabytes: no factor reaches, nothing is tabulated
    import gausslectronitegrate_b200 as gli
    got = gli.compute_nuclear_gausslet_integral(g10(), [(0, 0, 0), gap], POS, Q, 1e-8)
    assert not np.any(Oracle().factors(g10(), max(map(abs, gap)), 0.0)[0])
    assert got == 0.0
