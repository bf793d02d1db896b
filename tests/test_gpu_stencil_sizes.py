"""The coarse-level stencil kernels (csrc/stencil.cu) at the node counts where their
tiling has edges: FP64 blocks of 32 nodes, BF16 groups of three nodes packed 30 to a
block.  The smoothed level has 8 to 540 nodes, among them exactly 30, 32 and 36, one
below and above multiples of three, and levels one element thick.

Three-level hierarchies on E in [0.5, 1.5], one preconditioner apply.  In FP64 it is
linear in its input with a condition number of some hundreds, so a rounding of 1e-16
stays below 1e-12: 1e-11 against the oracle.  The mixed cycle stores the coarse
operators in BF16 (relative rounding 2^-9 an entry, no row larger than the diagonal's
share): 5e-2 of the largest entry, where a misplaced coefficient or neighbour is of
order one."""

import numpy as np
import pytest

from oracle.gmg import GMG
from oracle.solver import Operator

pytestmark = pytest.mark.gpu


def _gmg(torch, dims, **kw):
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
    return free, GalerkinMatFreeGMG(mf_op=mf, free=free, free_gpu=free, nelx=dims[0], nely=dims[1], nelz=dims[2],
                                    KE_UNIT=KE_UNIT_3D, n_levels=3, **kw)


# smoothed level: 8, 32, 30, 36, 40, 81, 168, 190, 540 nodes
@pytest.mark.parametrize("dims", [(2, 2, 2), (14, 2, 2), (8, 4, 2), (6, 4, 4), (8, 6, 2), (4, 4, 16), (12, 10, 6),
                                  (37, 9, 2), (17, 11, 18)])
@pytest.mark.parametrize("smoother", ["jacobi", "chebyshev"])
def test_apply_matches_oracle(cuda, dims, smoother):
    torch = cuda
    rng = np.random.default_rng(sum(dims))
    E = 0.5 + rng.random(int(np.prod(dims)))
    free, gmg = _gmg(torch, dims, smoother_type=smoother, fine_smoother="fp64")
    _, mixed = _gmg(torch, dims, smoother_type=smoother, fine_smoother="fp32", cycle_precision="fp32")
    r = rng.standard_normal(len(free))
    ref = GMG(Operator(*dims, free), n_levels=3, smoother_type=smoother, fine_smoother="fp64")
    ref.setup(E)
    zr = ref.apply(r)
    for g in (gmg, mixed):
        g.setup(torch.as_tensor(E, device="cuda"))
    z = gmg.apply(torch.as_tensor(r, device="cuda")).cpu().numpy()
    assert np.linalg.norm(z - zr) <= 1e-11 * np.linalg.norm(zr)
    zm = mixed.apply(torch.as_tensor(r, device="cuda")).cpu().numpy()
    assert np.abs(zm - zr).max() <= 5e-2 * np.abs(zr).max()
