"""The sliced stage A on wide ERIDA grids: tiles whose K loop covers only the
positions that their keys reach, and tiles that no pair reads. Whole and partial
lists of the 129^3 grid (A keys in one column tile, two, the second nearly
empty; keys without weights at a large tol) against the FP64 form of the same
list, which the other reach tests hold to the oracle.

Tolerance: the mixed form's 1e-8 on every value."""
import ctypes as C

import numpy as np
import pytest

from _common import sym_grid
from test_reach import _radius, _values, gli  # noqa: F401

pytestmark = pytest.mark.gpu
L = 129


@pytest.fixture(scope="module")
def idx(gli):  # noqa: F811
    return gli.compute_sparse_erida_gausslet_integrals(np.load("tests/golden/reference_fixtures.npz")["g10"], sym_grid(L),
                                                       1e-3).indices


@pytest.mark.parametrize("part,tol", [("all", 1e-16), ("all", 1e-4), ("shell", 1e-16), ("near", 1e-16), ("far", 1e-16),
                                      ("rank", 1e-8)])
def test_sliced_stage(gli, idx, part, tol):  # noqa: F811
    r = _radius(L, idx)
    pick = {"all": r >= 0, "shell": (r >= 60) & (r < 64), "near": r <= 40, "far": r >= np.sort(r)[-4000],
            "rank": (np.arange(idx.size) >= idx.size // 3) & (np.arange(idx.size) < idx.size // 2)}[part]
    sub = np.ascontiguousarray(idx[pick])
    ref = _values(gli, L, sub, tol, 0)
    for _ in range(3):  # the first evaluation and the replays
        got = _values(gli, L, sub, tol, 1)
        paths = (C.c_int * 3)()
        gli.lib().gli_b200_last_paths(paths)
        assert paths[0] == 1  # stage A on the int8 tensor cores
        assert np.max(np.abs(got - ref)) <= 1e-8
