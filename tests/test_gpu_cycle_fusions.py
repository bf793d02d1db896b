"""The cycle's fused transfers (csrc/stencil.cu): the restriction that also makes the
coarse level's first smoothing step, and the prolongation added into the iterate, on
grids whose levels have odd, even and single-element extents (parents missing on one
side), over the cycle options that take or bypass them; FP64 applies against the
oracle's cycle.  The apply is linear with a condition number of some hundreds, so
roundings of 1e-16 stay below 1e-12: 1e-11."""

import numpy as np
import pytest

from oracle.gmg import GMG
from oracle.solver import Operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(4, 2, 2), (9, 5, 3), (16, 7, 6), (21, 10, 11)])
@pytest.mark.parametrize("kw", [
    dict(smoother_type="jacobi"),
    dict(smoother_type="chebyshev"),
    dict(smoother_type="jacobi", cycle_type="w"),
    dict(smoother_type="chebyshev", cycle_type="w"),
    dict(smoother_type="jacobi", coarse_correction_policy="residual_line_search"),
    dict(smoother_type="chebyshev", cycle_type="w", coarse_correction_policy="residual_line_search"),
    dict(smoother_type="jacobi", coarse_smooth_iters=1),
    dict(smoother_type="jacobi", root_enrichment_mode="weighted_gap_second"),
])
def test_apply_matches_oracle(cuda, dims, kw):
    torch = cuda
    from gpu_fem.bc_generator import generate_bc
    from gpu_fem.multigrid_v4 import GalerkinMatFreeGMG
    from gpu_fem.presets import cantilever_spec
    from gpu_fem.pub_simp_solver import KE_UNIT_3D, _edof_table_3d
    from gpu_fem.solver_v2 import MatrixFreeKff

    bc = generate_bc(cantilever_spec(*dims))
    free = bc.free_dofs.astype(np.int32)
    edof = torch.as_tensor(_edof_table_3d(*dims), device="cuda")
    mf = MatrixFreeKff(edof, torch.as_tensor(KE_UNIT_3D, device="cuda"), torch.as_tensor(free, device="cuda"),
                       len(free), bc.ndof, grid_dims=dims)
    kw = dict(kw, n_levels=3, fine_smoother="fp64")
    gmg = GalerkinMatFreeGMG(mf_op=mf, free=free, free_gpu=free, nelx=dims[0], nely=dims[1], nelz=dims[2],
                             KE_UNIT=KE_UNIT_3D, **kw)
    rng = np.random.default_rng(sum(dims))
    E = 0.5 + rng.random(int(np.prod(dims)))
    r = rng.standard_normal(len(free))
    ref = GMG(Operator(*dims, free), **kw)
    ref.setup(E)
    gmg.setup(torch.as_tensor(E, device="cuda"))
    zr = ref.apply(r)
    for _ in range(2):  # the second apply finds the levels' vectors as the first left them
        z = gmg.apply(torch.as_tensor(r, device="cuda")).cpu().numpy()
        assert np.linalg.norm(z - zr) <= 1e-11 * np.linalg.norm(zr)
