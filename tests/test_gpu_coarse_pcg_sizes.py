"""The one-launch coarse PCG (csrc/linalg.cu: pcg_coop_kernel) over the sizes where
its layout changes: one block, more blocks than exchange directly with one another
(32), one to three rows a lane group, and a system too large for it (the launched
form).

Two-level hierarchies on E in [0.5, 1.5] with 25 coarse iterations: the solve is
well conditioned (Jacobi-scaled condition number of a few hundred) and every system
has more than 25 unknowns (beyond its exact end a CG divides noise by noise), so 25
CG iterations in 64 bits carry a rounding of 1e-16 to at most some 1e-12, and one
preconditioner apply is compared with the oracle's to 1e-10.  The FP32 cycle's
apply agrees with the FP64 one to FP32 and BF16 storage accuracy (2e-2, the
coarse stencils' eight bits); replays of a captured cycle are bitwise the direct
launches.
"""

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
                                    KE_UNIT=KE_UNIT_3D, n_levels=2, dense_chol_max=0, coarse_pcg_iters=25,
                                    smoother_type="jacobi", **kw)


@pytest.mark.parametrize("dims", [(8, 4, 4), (17, 9, 5), (40, 20, 20), (48, 24, 24), (60, 30, 30), (64, 40, 32)])
def test_apply_matches_oracle(cuda, dims):
    torch = cuda
    rng = np.random.default_rng(sum(dims))
    E = 0.5 + rng.random(int(np.prod(dims)))
    free, gmg = _gmg(torch, dims, fine_smoother="fp64")
    gmg.setup(torch.as_tensor(E, device="cuda"))
    assert gmg.coarse_mode == "iterative"
    r = rng.standard_normal(len(free))
    z = gmg.apply(torch.as_tensor(r, device="cuda")).cpu().numpy()
    ref = GMG(Operator(*dims, free), n_levels=2, dense_chol_max=0, coarse_pcg_iters=25, smoother_type="jacobi",
              fine_smoother="fp64")
    ref.setup(E)
    zr = ref.apply(r)
    assert np.linalg.norm(z - zr) <= 1e-10 * np.linalg.norm(zr)


def test_fp32_cycle_and_captured_replay(cuda):
    torch = cuda
    dims = (40, 20, 20)
    rng = np.random.default_rng(1)
    E = torch.as_tensor(0.5 + rng.random(int(np.prod(dims))), device="cuda")
    out = {}
    for tag, kw in (("fp64", dict(fine_smoother="fp64")), ("fp32", dict(fine_smoother="fp32", cycle_precision="fp32")),
                    ("graph", dict(fine_smoother="fp32", cycle_precision="fp32", use_graphs=True))):
        free, gmg = _gmg(torch, dims, **kw)
        gmg.setup(E)
        r = torch.as_tensor(np.random.default_rng(2).standard_normal(len(free)), device="cuda")
        out[tag] = [gmg.apply(r).clone() for _ in range(4)]
    z = out["fp64"][0]
    assert float(torch.linalg.norm(out["fp32"][0] - z) / torch.linalg.norm(z)) <= 2e-2
    for tag in out:
        assert all(torch.equal(v, out[tag][0]) for v in out[tag]), tag
    assert torch.equal(out["graph"][0], out["fp32"][0])
