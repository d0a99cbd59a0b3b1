"""Evaluations that follow the weights' reaches (lattice keys nonzero on part
of the positions: ERIDA grids from about 49 points per axis) against the
oracle: whole and partial class lists (one displacement shell, the farthest
classes, a rank's range, a single class), grids whose last column tile or
64-row tile is nearly empty, large tol (short reaches, keys without weights)
and both forms, and the same list evaluated twice (kept plan).

Tolerance: the parity bar (1e-12 relative + 1e-14); mixed form: within its
screening bound and the 1e-8 of the other mixed tests."""
import ctypes as C

import numpy as np
import pytest

from _common import assert_parity, g10, sym_grid
from oracle_binding import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gli():
    import gausslectronitegrate_b200 as m
    if m.lib().gli_b200_device_count() == 0:
        pytest.fail("no CUDA device: the gpu tests need a B200")
    return m


def _values(gli, L, idx, tol, form):
    b = np.ascontiguousarray(g10())
    g = gli._abi.GaussletData()
    g.coefficients = b.ctypes.data_as(gli._abi.dptr)
    g.indices.num, g.indices.istart = b.size, -(b.size - 1) // 2
    out = np.full(idx.size, np.nan)
    rc = gli.lib().gli_b200_sparse_values(0, C.byref(g), C.byref(gli._grid_struct(sym_grid(L))),
                                          idx.ctypes.data_as(gli._abi.lptr), idx.size, tol, form,
                                          out.ctypes.data_as(gli._abi.dptr))
    assert rc == 0, gli.lib().gli_b200_last_error_message().decode()
    return out


def _radius(L, idx):
    N = L ** 3
    i, j = idx // N, idx % N
    d = [np.abs(i // s % L - j // s % L) for s in (L * L, L, 1)]
    return np.sqrt(sum(x.astype(float) ** 2 for x in d))


@pytest.fixture(scope="module")
def lists(gli):
    made = {}

    def get(L):
        if L not in made:
            made[L] = gli.compute_sparse_erida_gausslet_integrals(g10(), sym_grid(L), 1e-3).indices
        return made[L]
    return get


@pytest.mark.parametrize("L,tol", [(33, 1e-5), (49, 1e-16), (65, 1e-16), (81, 1e-10), (97, 1e-16), (97, 1e-3), (129, 1e-8)])
def test_whole_lists(gli, lists, L, tol):
    idx = lists(L)
    rng = np.random.default_rng(L)
    at = np.unique(np.concatenate([rng.integers(0, idx.size, 150), np.arange(5), np.arange(idx.size - 5, idx.size)]))
    ref = Oracle().values("erida", g10(), sym_grid(L), idx[at], tol)
    first = _values(gli, L, idx, tol, 0)
    assert_parity(first[at], ref, what=f"{L} tol {tol}")
    for _ in range(2):  # the replays of the kept plan
        assert np.array_equal(_values(gli, L, idx, tol, 0), first)
    mixed = _values(gli, L, idx, tol, 1)
    assert np.max(np.abs(mixed - first)) <= 1e-8


@pytest.mark.parametrize("part", ["shell", "far", "near", "rank", "one"])
def test_partial_lists(gli, lists, part):
    L, tol = 81, 1e-14
    idx = lists(L)
    r = _radius(L, idx)
    pick = {"shell": (r >= 40) & (r < 41), "far": r >= np.sort(r)[-70], "near": r <= 6,
            "rank": (np.arange(idx.size) >= idx.size // 3) & (np.arange(idx.size) < idx.size // 2),
            "one": r == r.max()}[part]
    sub = np.ascontiguousarray(idx[pick])
    at = np.random.default_rng(3).integers(0, sub.size, min(sub.size, 120))
    got = _values(gli, L, sub, tol, 0)
    assert np.all(np.isfinite(got))
    assert_parity(got[at], Oracle().values("erida", g10(), sym_grid(L), sub[at], tol), what=part)


def test_no_weights_left(gli, lists):
    # every product below tol: all values are zero
    assert np.array_equal(_values(gli, 65, lists(65), 1e3, 0), np.zeros(lists(65).size))
