"""Projections and applies of complete ERI lists by pair classes, at the edges
of the kernel's tiles: boxes from one point to 5 x 5 x 5 (rows beyond a
16-row tile, x planes that are no multiple of the 4-wide k step), 1 to 32
orbitals (column tiles of 8), orbitals on points that are no box, and 1 to 9
states; against dense contractions of the filled tensor in numpy.

Tolerance: sums of N^2 to N^4 terms of one sign pattern or another in FP64,
as the projection tests' 1e-12 of the largest result."""
import numpy as np
import pytest

from _common import g10, sym_grid
from oracle_binding import project_factored

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tensors():
    import gausslectronitegrate_b200 as gli
    if gli.lib().gli_b200_device_count() == 0:
        pytest.fail("no CUDA device: the gpu tests need a B200")
    return {L: gli.compute_sparse_eri_gausslet_integrals(g10(), sym_grid(L), 1e-10) for L in (1, 3, 5)}


def _rows(L, box):
    xs = [np.arange(s, s + n) + L // 2 for s, n in box]
    X, Y, Z = np.meshgrid(*xs, indexing="ij")
    return ((X * L + Y) * L + Z).ravel()


def _check(got, ref):
    scale = np.max(np.abs(ref))
    assert np.max(np.abs(got - ref)) <= 1e-12 * scale


@pytest.mark.parametrize("L,box", [(1, [(0, 1)] * 3), (3, [(-1, 3)] * 3), (3, [(-1, 2), (0, 1), (-1, 3)]),
                                   (5, [(-2, 5), (-1, 2), (0, 3)]), (5, [(-2, 4)] * 3), (5, [(0, 1), (-2, 5), (-2, 5)])])
@pytest.mark.parametrize("M", [1, 7, 8, 9, 20, 25, 32])
def test_project_boxes(tensors, L, box, M):
    rng = np.random.default_rng(M)
    s, rows = tensors[L], _rows(L, box)
    basis = np.zeros((L ** 3, M))
    basis[rows] = rng.standard_normal((rows.size, M))
    _check(s.project(basis), project_factored(s.fill_tensor(box), basis[rows]))


@pytest.mark.parametrize("drop", [1, 20, 50])
def test_project_points_that_are_no_box(tensors, drop):
    # 64 points of a box without some of them: within twice the active points
    # (zero rows of the box), and beyond (the general contraction)
    rng = np.random.default_rng(drop)
    s, box = tensors[5], [(-2, 4)] * 3
    rows = _rows(5, box)
    basis = np.zeros((125, 6))
    basis[rows] = rng.standard_normal((64, 6))
    basis[rng.choice(rows, drop, replace=False)] = 0.0
    _check(s.project(basis), project_factored(s.fill_tensor(box), basis[rows]))


@pytest.mark.parametrize("L,ns", [(1, 1), (3, 1), (3, 2), (3, 5), (3, 9), (5, 1), (5, 3), (5, 4)])
def test_apply_states(tensors, L, ns):
    rng = np.random.default_rng(ns)
    s, N = tensors[L], L ** 3
    x = rng.standard_normal((N * N, ns))
    V = s.fill_tensor([(-(L // 2), L)] * 3)
    ref = np.empty((N, N, ns))
    for i in range(N):  # (i k) = sum_jl V[i j k l] x[j l]
        ref[i] = np.tensordot(V[i], x.reshape(N, N, ns), axes=([0, 2], [0, 1]))
    _check(s.apply(x).reshape(N, N, ns), ref)


def test_apply_keeps_columns_apart(tensors):
    # infinities in one state leave the others as they are, and its own
    # entries infinite or undefined, none finite
    rng = np.random.default_rng(1)
    x = rng.standard_normal((27 * 27, 3))
    ref = tensors[3].apply(x)
    x[5, 1] = np.inf
    got = tensors[3].apply(x)
    assert np.array_equal(got[:, [0, 2]], ref[:, [0, 2]])
    assert not np.isfinite(got[:27, 1]).any()
