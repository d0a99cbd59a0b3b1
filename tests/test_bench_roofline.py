"""bench.py's FP64 roofline, on the CPU: evaluations whose keys reach only part
of the lattice get an effective rate and no fraction, however low the rate."""
import os
import sys

import numpy as np
import pytest

from _common import HERE, g10

sys.path.insert(0, os.path.dirname(HERE))
import bench  # noqa: E402

STAGES = {"A": 0.15, "B": 0.1, "C_product": 0.02, "C_class": 0.01}


@pytest.mark.parametrize("dom", ["A", "B", "C_product", "C_class"])
@pytest.mark.parametrize("kind,L,U,banded", [("erida", 129, 465, True), ("erida", 33, 177, False), ("eri", 7, 141, False)])
def test_fraction_only_where_the_whole_lattice_is_executed(dom, kind, L, U, banded):
    reach = bench.mean_key_reach(kind, g10(), L, 1e-16)
    product = 0 if dom == "C_class" else 370_177
    r = bench.roofline((0, 0, 0), dom, STAGES, (L, 1000, L, product), U, 366_145, 37.0, reach)
    assert (r["frac"] is None) == banded
    assert ("effective" in r["flops_counted"]) == banded
    assert r["achieved"] is not None


def test_mean_reach_equals_the_folded_weights():
    # weights built entry by entry, 9 coefficients
    b, L, tol = np.array([0.01, -0.2, 0.5, 1.0, 2.0, 1.0, 0.5, -0.2, 0.01]), 4, 1e-3
    P = 2 * np.pi / 9 * np.convolve(b, b[::-1])
    P[np.abs(P) <= tol] = 0
    at = np.flatnonzero(P) - 8
    U = 3 * (L - 1) + np.abs(at).max() + 1
    spans = []
    for key in range(L):
        W = np.zeros(U)
        for m in at:
            W[abs(3 * key + m)] += P[m + 8]
        live = np.flatnonzero(W)
        spans.append(live[-1] - live[0] + 1)
    assert bench.mean_key_reach("erida", b, L, tol) == pytest.approx(np.mean(spans) / U)
