"""Projections with an infinite orbital coefficient: results that hold the
orbital are not finite (infinite on one point, where the sum is one positive
product), the others are as without it.  Every class has the value 1, so that
the sums are products of the orbitals' own sums.

Tolerance: as the other projections', 1e-12 of the largest result."""
import numpy as np
import pytest

from _common import g10, sym_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,M", [(1, 1), (1, 2), (3, 3), (5, 2)])
def test_infinite_coefficient(L, M):
    import gausslectronitegrate_b200 as gli
    rng = np.random.default_rng(L)
    spec = sym_grid(L)
    idx = gli.compute_sparse_eri_gausslet_integrals(g10(), spec, 1e-10).indices
    s = gli.SparseERI._make(g10(), spec, idx, np.ones(idx.size), 1e-10)
    B = rng.uniform(0.5, 1.5, (L ** 3, M))
    ref = s.project(B)
    B[L ** 3 // 2, M - 1] = np.inf
    got = s.project(B)
    holds = np.zeros((M,) * 4, dtype=bool)
    for axis in range(4):
        holds[(slice(None),) * axis + (M - 1,)] = True
    assert np.all(got[holds] == np.inf) if L == 1 else not np.any(np.isfinite(got[holds]))
    if M > 1:
        assert np.max(np.abs(got[~holds] - ref[~holds])) <= 1e-12 * np.max(np.abs(ref[~holds]))
