"""Results out through the ring of page-locked pieces at the edges of its rules:
8 MB (the smallest staged result), repeated until the pieces have gone round the
ring, sizes off the piece boundaries, and either side of 64 MB, where the pieces
grow to 4 MB.  The kinetic matrix in host memory equals, bit for bit, the same
kernel's matrix left on the device."""
import ctypes as C

import numpy as np
import pytest

from _common import g10

pytestmark = pytest.mark.gpu


# 7.98, 8 and 11.6 MB; 25, 63.99 and 64.07 MB; 135 MB
@pytest.mark.parametrize("n,turns", [((1, 1, 1023), 2), ((8, 16, 8), 9), ((7, 11, 16), 13), ((2, 907, 1), 3),
                                     ((1, 4, 724), 3), ((6, 21, 23), 3),
                                     ((13, 18, 18), 2)])
def test_results_arrive_whole(n, turns):
    import torch

    import gausslectronitegrate_b200 as gli
    b, grid = g10(), [(0, m) for m in n]
    N = n[0] * n[1] * n[2]
    db = torch.tensor(b, device="cuda")
    out = torch.empty((N, N), dtype=torch.float64, device="cuda")
    rc = gli.lib().gli_b200_kinetic_matrix_noalloc(C.c_void_p(db.data_ptr()), b.size, C.byref(gli._grid_struct(grid)),
                                                   C.c_void_p(out.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    ref = out.cpu().numpy()
    for _ in range(turns):
        assert np.array_equal(gli.compute_kinetic_gausslet_integrals(b, grid), ref)
