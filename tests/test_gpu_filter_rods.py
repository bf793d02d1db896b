"""The cone filter on rods and walls, whose tiles (csrc/simp.cu: filter_tile) are cut for
their shared memory.

The filter sums at most 179 positive weights per output and divides once: 1e-13 of the
largest entry.
"""

import numpy as np
import pytest

from oracle import solver as osol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,rmin", [((2100, 1, 1), 2.5), ((2100, 1, 1), 3.5), ((700, 3, 1), 3.2), ((300, 8, 1), 3.5),
                                       ((300, 1, 8), 3.0), ((1, 2100, 1), 3.5), ((1, 1, 700), 3.5)])
def test_filter_rods(cuda, dims, rmin):
    from gpu_fem.simp_loop import cone_filter

    H = osol.density_filter(*dims, rmin)
    x = np.random.default_rng(sum(dims)).random(int(np.prod(dims)))
    xd = cuda.as_tensor(x, device="cuda")
    for t, ref in ((False, H @ x), (True, H.T @ x)):
        got = cone_filter(xd, dims, rmin, transpose=t).cpu().numpy()
        assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max(), t
