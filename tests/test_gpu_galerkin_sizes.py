"""The coarse-operator kernels (csrc/stencil.cu: level1_assemble_kernel, rap_kernel) at
the extents where their index sets change: coarse levels one element thick, odd fine
extents (a fine node or element past the last pair), node counts at multiples of the
blocks' 32 and 128 nodes and one beyond; against the oracle's dense triple product
through the hierarchy's preconditioner.

Four-level hierarchies on E in [0.5, 1.5]: levels 1 to 3 enter the apply through their
smoothing, residuals and the coarsest solve.  Roundings of 1e-16 stay below 1e-12 of a
linear map with a condition number of some hundreds: 1e-11."""

import numpy as np
import pytest

from oracle.gmg import GMG
from oracle.solver import Operator

pytestmark = pytest.mark.gpu


# level-1 nodes: 8, 24, 128, 135, 192, 288, 378
@pytest.mark.parametrize("dims", [(2, 2, 2), (5, 3, 7), (14, 6, 6), (17, 9, 5), (15, 11, 6), (22, 14, 5), (13, 17, 11)])
def test_apply_matches_oracle(cuda, dims):
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
    gmg = GalerkinMatFreeGMG(mf_op=mf, free=free, free_gpu=free, nelx=dims[0], nely=dims[1], nelz=dims[2],
                             KE_UNIT=KE_UNIT_3D, n_levels=4, smoother_type="jacobi", fine_smoother="fp64")
    rng = np.random.default_rng(sum(dims))
    E = 0.5 + rng.random(int(np.prod(dims)))
    r = rng.standard_normal(len(free))
    ref = GMG(Operator(*dims, free), n_levels=4, smoother_type="jacobi", fine_smoother="fp64")
    ref.setup(E)
    gmg.setup(torch.as_tensor(E, device="cuda"))
    zr = ref.apply(r)
    z = gmg.apply(torch.as_tensor(r, device="cuda")).cpu().numpy()
    assert np.linalg.norm(z - zr) <= 1e-11 * np.linalg.norm(zr)
