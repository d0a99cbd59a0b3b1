"""The key table of a complete ERI list is made while the list is compared with
the canonical one: a list of the canonical length with one class replaced (by an
index that is no canonical class) is expanded by lookups instead, whether the
comparison's answer is read before the contraction (projection) or after it
(apply).  The replaced class is then absent, its entries of the tensor zero.
Against dense contractions in numpy of the filled tensor.

Tolerance: as the projection tests', 1e-12 of the largest result."""
import numpy as np
import pytest

from _common import g10, sym_grid
from oracle_binding import project_factored

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lists():
    import gausslectronitegrate_b200 as gli
    if gli.lib().gli_b200_device_count() == 0:
        pytest.fail("no CUDA device: the gpu tests need a B200")
    return {L: gli.compute_sparse_eri_gausslet_integrals(g10(), sym_grid(L), 1e-10) for L in (3, 5)}


def _places(s):
    """classes whose index has no class after it: the first, a middle and the last"""
    gaps = np.flatnonzero(np.diff(s._indices) > 1)
    return [int(gaps[0]), int(gaps[gaps.size // 2]), s._indices.size - 1]


@pytest.mark.parametrize("L", [3, 5])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_replaced_class(lists, L, which):
    rng = np.random.default_rng(which)
    s, N, full = lists[L], L ** 3, [(-(L // 2), L)] * 3
    at, moved = _places(s)[which], s._indices.copy()
    moved[at] += 1
    t = type(s)._make(s._coeffs, s._spec, moved, s._values, s._tol)
    V, complete = t.fill_tensor(full), s.fill_tensor(full)
    absent = V != complete
    assert absent.any() and not V[absent].any() and absent.flat[s._indices[at]]
    x, basis = rng.standard_normal((N * N, 3)), rng.standard_normal((N, 5))
    ref = np.empty((N, N, 3))
    for i in range(N):  # (i k) = sum_jl V[i j k l] x[j l]
        ref[i] = np.tensordot(V[i], x.reshape(N, N, 3), axes=([0, 2], [0, 1]))
    got = t.apply(x).reshape(N, N, 3)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
    got, ref = t.project(basis), project_factored(V, basis)
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
