"""The one-launch Arnoldi column of the device FGMRES at the vector lengths where its
plan changes: one part, one block of 16 parts, a last block with one, 296 parts with 1,
2, 4, 8, 12 and 24 elements a thread, the column held in shared memory, and the launched
form beyond; against the oracle's FGMRES.

The operator is diagonal in [1, 2] plus a cyclic shift of 0.1 (condition below 2.5), so
the iterates carry the rounding of the sums only: a dot product of n terms is within
sqrt(n) eps = 5e-13 of its value in any order, for x and the history alike; 1e-11 leaves a
factor for the dozen columns."""

import numpy as np
import pytest

from oracle import solver as osol

pytestmark = pytest.mark.gpu

ROW = 296 * 256  # elements of all parts, one a thread


@pytest.mark.parametrize("n", [1, 2, 257, 4096, 4097, ROW, ROW + 1, 2 * ROW, 2 * ROW + 1, 4 * ROW, 4 * ROW + 1,
                               8 * ROW, 8 * ROW + 1, 12 * ROW + 1, 24 * ROW, 24 * ROW + 1, 54 * ROW, 54 * ROW + 1])
def test_column_plans_match_oracle(cuda, n):
    torch = cuda
    from gpu_fem.multigrid_v4 import _cupy_fgmres

    rng = np.random.default_rng(n)
    d, b = 1.0 + rng.random(n), rng.standard_normal(n)
    dt, bt = torch.as_tensor(d, device="cuda"), torch.as_tensor(b, device="cuda")
    hist, ref_hist = [], []
    x, it, conv = _cupy_fgmres(lambda v: dt * v + 0.1 * torch.roll(v, 1), bt, lambda v: 0.75 * v, tol=1e-9, maxiter=30,
                               restart=5, history=hist)
    xr, itr, convr = osol.fgmres(lambda v: d * v + 0.1 * np.roll(v, 1), b, lambda v: 0.75 * v, tol=1e-9, maxiter=30,
                                 restart=5, history=ref_hist)
    assert (it, conv) == (itr, convr)
    assert len(hist) == len(ref_hist)
    np.testing.assert_allclose(hist, ref_hist, rtol=0, atol=1e-11)
    np.testing.assert_allclose(x.cpu().numpy(), xr, rtol=0, atol=1e-11 * np.abs(xr).max())
