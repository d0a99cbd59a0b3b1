"""Projections and applies by pair classes beyond 125 points: two 16-row tiles a
warp (129 points and up), blocks of 16 warps (257 points and up, and column
counts whose tables fill the shared memory), the diagonal plane's tiles that
start within a plane, and applies in several turns over the states.

References.  A projection onto more than 32 orbitals takes the general
contraction (slabs of the tensor, a product per point pair): the orbitals are
projected there with others appended.  An apply is held to dense entries of
sub-boxes, looked up class by class (fill_tensor), with states supported on the
sub-box's point pairs.

Tolerance: as the other projections', 1e-12 of the largest result (sums of up
to N^4 terms of both signs in FP64)."""
import numpy as np
import pytest

from _common import g10, sym_grid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gli():
    import gausslectronitegrate_b200 as m
    if m.lib().gli_b200_device_count() == 0:
        pytest.fail("no CUDA device: the gpu tests need a B200")
    return m


@pytest.fixture(scope="module")
def eri7(gli):
    return gli.compute_sparse_eri_gausslet_integrals(g10(), sym_grid(7), 1e-10)


def _rows(L, box):
    xs = [np.arange(s, s + n) + L // 2 for s, n in box]
    X, Y, Z = np.meshgrid(*xs, indexing="ij")
    return ((X * L + Y) * L + Z).ravel()


def _check(got, ref):
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("box", [[(-3, 5), (-2, 5), (-3, 6)], [(-3, 6), (-3, 6), (-2, 5)], [(-3, 7), (-3, 6), (-3, 6)],
                                 [(-3, 7), (-3, 7), (-3, 6)], [(-3, 7)] * 3, [(0, 3), (-3, 7), (-3, 7)],
                                 [(-3, 7), (-3, 7), (0, 3)]])
def test_project_large_boxes(eri7, box):
    rows = _rows(7, box)
    basis = np.zeros((343, 33))
    basis[rows] = np.random.default_rng(rows.size).standard_normal((rows.size, 33))
    ref = eri7.project(basis)
    for M in (1, 8, 20, 25, 32):
        _check(eri7.project(basis[:, :M].copy()), ref[:M, :M, :M, :M])


@pytest.mark.parametrize("box", [[(-3, 3), (-2, 4), (0, 4)], [(-3, 7), (0, 3), (2, 2)], [(1, 2), (-3, 3), (-3, 7)]])
def test_apply_at_343_points(eri7, box):
    # 7 states: two turns of contributions; every column for itself: one
    rows, rng = _rows(7, box), np.random.default_rng(3)
    n = rows.size
    V = eri7.fill_tensor(box).reshape(n, n, n, n)
    x = np.zeros((343, 343, 7))
    x[np.ix_(rows, rows)] = rng.standard_normal((n, n, 7))
    got = eri7.apply(x.reshape(343 * 343, 7)).reshape(343, 343, 7)
    ref = np.einsum("ijkl,jls->iks", V, x[np.ix_(rows, rows)], optimize=True)
    _check(got[np.ix_(rows, rows)], ref)
    one = eri7.apply(x[:, :, 6].reshape(343 * 343, 1)).reshape(343, 343)
    _check(one, got[:, :, 6])


def test_apply_of_full_states_at_343_points(eri7):
    # E[p q r s] = sum_ik B_ip B_kr (apply of b_q b_s)_ik against the projection
    rng = np.random.default_rng(5)
    B = rng.standard_normal((343, 3))
    E = eri7.project(B)
    states = np.stack([np.outer(B[:, q], B[:, s]).ravel() for q in range(3) for s in range(3)], axis=1)
    got = eri7.apply(states).reshape(343, 343, 9)
    _check(np.einsum("ip,ikc,kr->prc", B, got, B, optimize=True),
           np.stack([E[:, q, :, s] for q in range(3) for s in range(3)], axis=2))
