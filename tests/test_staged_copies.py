"""Host copies through the ring of page-locked pieces: class lists and values of
more pieces than the ring has slots (96 MB in, 64 slots of 1 MB), sizes off the
piece boundaries, and dense results out of one piece to more than the ring."""
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


@pytest.mark.parametrize("entries", [262_145, 3_000_001, 6_000_003])
def test_long_lists_arrive_whole(gli, entries):
    # the classes of a 17^3 grid scattered in a long list of other indices: every
    # dense entry is found by the device's search with its own value
    rng = np.random.default_rng(entries)
    spec = sym_grid(17)
    real = gli.compute_sparse_erida_gausslet_integrals(g10(), spec, 1e-3).indices
    idx = np.unique(np.concatenate([real, rng.integers(0, 17 ** 6, 2 * entries)]))
    drop = rng.choice(np.setdiff1d(np.arange(idx.size), np.searchsorted(idx, real)), idx.size - entries, replace=False)
    idx = np.delete(idx, drop)
    s = gli.SparseERIDA._make(g10(), spec, idx, rng.standard_normal(idx.size), 1e-3)
    grid = [(-2, 5), (0, 2), (-1, 3)]
    pts = [(x, y, z) for x in range(-2, 3) for y in range(2) for z in range(-1, 2)]
    ref = np.array([[s.integral_value([p, q]) for q in pts] for p in pts])
    assert np.array_equal(s.fill_matrix(grid), ref)


@pytest.mark.parametrize("n", [(8, 8, 8), (9, 8, 8), (13, 16, 15)])
def test_dense_results_arrive_whole(gli, n):
    # 2.1, 2.7 and 78 MB
    b = g10()
    k = gli.compute_kinetic_gausslet_integrals(b, [(0, m) for m in n])
    one = [gli.compute_kinetic_gausslet_integrals(b, [(0, m), (0, 1), (0, 1)]) for m in n]
    eye = [np.eye(m) for m in n]
    c = one[0][0, 0]  # each axis' matrix holds the three axes' diagonal: leave one
    axis = [o - 2.0 / 3.0 * c * e for o, e in zip(one, eye)]
    ref = sum(np.kron(np.kron(axis[0] if a == 0 else eye[0], axis[1] if a == 1 else eye[1]),
                      axis[2] if a == 2 else eye[2]) for a in range(3))
    assert np.max(np.abs(k - ref)) <= 1e-13 * abs(c)
