"""The tiled cone filter and the one-launch OC bisection at the sizes where their
tiling changes (csrc/simp.cu): rows of one, 64 and 65 elements, axes no longer than
the filter's reach, radii up to 3.5; designs of one element, of one block, of
several blocks, and more elements than the blocks keep in shared memory.

Tolerances: the filter sums at most 179 positive weights per output and divides
once, so 1e-13 of the largest entry is some hundred roundings; the bisection's
multiplier is defined to its last bracket (1e-9) and the update follows it.
"""

import numpy as np
import pytest

from oracle import solver as osol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,rmin", [((1, 1, 1), 1.5), ((2, 3, 1), 2.5), ((5, 2, 3), 3.5), ((9, 4, 64), 1.5),
                                       ((9, 4, 65), 1.5), ((33, 17, 5), 2.2), ((12, 10, 7), 3.5), ((3, 70, 2), 1.0),
                                       ((40, 1, 130), 1.3)])
def test_filter_tiles(cuda, dims, rmin):
    from gpu_fem.simp_loop import cone_filter

    H = osol.density_filter(*dims, rmin)
    x = np.random.default_rng(sum(dims)).random(int(np.prod(dims)))
    xd = cuda.as_tensor(x, device="cuda")
    for t, ref in ((False, H @ x), (True, H.T @ x)):
        got = cone_filter(xd, dims, rmin, transpose=t).cpu().numpy()
        assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max(), t


@pytest.mark.parametrize("n", [1, 511, 1024, 1025, 60_001, 1_400_003])
@pytest.mark.parametrize("with_dv", [False, True])
def test_oc_bisection_sizes(cuda, n, with_dv):
    from gpu_fem.simp_loop import OCUpdater

    rng = np.random.default_rng(n)
    rho = np.clip(0.3 + 0.2 * rng.standard_normal(n), 1e-3, 1.0)
    dc = -np.exp(1.5 * rng.standard_normal(n))
    dv = 0.5 + rng.random(n) if with_dv else np.ones(n)
    vw = 0.5 + rng.random(n)

    def candidate(lm):
        r = rho * np.sqrt(-np.minimum(dc, -1e-12) / (lm * np.maximum(dv, 1e-12)))
        return np.clip(np.clip(r, rho - 0.2, rho + 0.2), 1e-3, 1.0)

    l1, l2, steps = 0.0, 1e9, 0
    while steps < 100:
        lm = 0.5 * (l1 + l2)
        steps += 1
        if (vw * candidate(lm)).sum() > 0.3 * n:
            l1 = lm
        else:
            l2 = lm
        if l2 - l1 < 1e-9:
            break
    t = [cuda.as_tensor(v, device="cuda") for v in (rho, dc, vw, dv)]
    got, change, lm_g, steps_g = OCUpdater()(t[0], t[1], t[2], 0.3, 0.2, dv_design=t[3] if with_dv else None)
    assert steps_g == steps and abs(lm_g - lm) <= 2e-9 * max(1.0, lm)
    ref = candidate(lm)
    np.testing.assert_allclose(got.cpu().numpy(), ref, rtol=0, atol=1e-8)
    assert change == pytest.approx(np.abs(ref - rho).max(), abs=1e-8)
