"""Nuclear matrices at the edges of the contraction's and the scatter's shapes
against the oracle: boxes with axes of one and two points, odd matrix sizes
(rows off the 16-byte grid), a z axis beyond the shared-memory scatter (64
points), keys whose factor vanishes at a large tol, several instances of
unequal size in one batch, and the single-entry form's two-point axes.

Tolerance: the parity bar of the other nuclear tests (1e-12 relative + 1e-14)."""
import numpy as np
import pytest

from _common import assert_parity, g10
from oracle_binding import Oracle

pytestmark = pytest.mark.gpu

POS = np.array([[0.3, -0.2, 0.1], [1.0, 0.0, -1.0]])
Q = [1, 7]


@pytest.fixture(scope="module")
def gli():
    import gausslectronitegrate_b200 as m
    if m.lib().gli_b200_device_count() == 0:
        pytest.fail("no CUDA device: the gpu tests need a B200")
    return m


@pytest.mark.parametrize("n", [(1, 1, 1), (2, 1, 2), (1, 3, 5), (3, 2, 3), (1, 1, 65), (1, 2, 17), (20, 1, 1)])
@pytest.mark.parametrize("tol", [1e-3, 1e-2])
def test_boxes_against_oracle(gli, n, tol):
    grid = [(-(k // 2), k) for k in n]
    got = gli.compute_nuclear_gausslet_integrals(g10(), grid, POS, Q, tol)
    assert_parity(got, Oracle().nuclear_matrix(g10(), grid, POS, Q, tol), what=f"{n} tol {tol}")


def test_unequal_batch_equals_its_instances(gli):
    grids = [[(-2, 5), (0, 1), (-1, 3)], [(-3, 7)] * 3, [(0, 1)] * 3, [(-1, 2), (-4, 9), (0, 2)]]
    pos, q = [POS, POS + 0.25, POS[:1], POS], [Q, Q, [3], Q]
    for form in ("fp64", "mixed"):
        outs = gli.compute_nuclear_gausslet_integrals_batch(g10(), grids, pos, q, 1e-6, form=form)
        for k, out in enumerate(outs):
            one = gli.compute_nuclear_gausslet_integrals(g10(), grids[k], pos[k], q[k], 1e-6)
            if form == "fp64":
                assert_parity(out, one, what=f"instance {k}")
            else:
                assert np.max(np.abs(out - one)) <= 5e-9


@pytest.mark.parametrize("a,b", [((0, 0, 0), (0, 0, 0)), ((0, 1, 0), (5, 1, -3)), ((2, -9, 0), (-9, 9, 0))])
def test_single_entries_against_oracle(gli, a, b):
    got = gli.compute_nuclear_gausslet_integral(g10(), [a, b], POS, Q, 1e-3)
    lo = [min(x, y) for x, y in zip(a, b)]
    grid = [(l, max(x, y) - l + 1) for l, x, y in zip(lo, a, b)]
    at = lambda p: np.ravel_multi_index([x - l for x, l in zip(p, lo)], [m for _, m in grid])  # noqa: E731
    ref = gli.compute_nuclear_gausslet_integrals(g10(), grid, POS, Q, 1e-3)[at(a), at(b)]
    assert_parity(np.array([got]), np.array([ref]), what="single entry")


def test_far_and_coincident_nuclei(gli):
    # a nucleus on a lattice point (the field's limit) and one far outside the box
    grid, pos = [(-1, 2), (-1, 3), (0, 2)], np.array([[0.0, 0.0, 0.0], [300.0, 0.5, -40.0]])
    got = gli.compute_nuclear_gausslet_integrals(g10(), grid, pos, [1, 2], 1e-3)
    assert_parity(got, Oracle().nuclear_matrix(g10(), grid, pos, [1, 2], 1e-3), what="far nucleus")
