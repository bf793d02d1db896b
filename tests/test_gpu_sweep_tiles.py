"""The fine-operator sweep (csrc/fine.cu: sweep_kernel) where its tiles and variants
change: grids of one element, one row or one plane, extents around the parts the z
and y axes are cut into, random supports (node planes wholly free, wholly fixed and
partly free take different paths of the compact operator), the tile before and after
tuning, and a stiffness without the isotropic pattern of the Walsh blocks.

FP64: the product has at most 24 x 8 terms per DOF, 1e-13 of the result's norm as
the operator's other tests; FP32 operands and arithmetic 1e-5; BF16 operands with
FP32 accumulation against the oracle with the same operand rounding 1e-5.
"""

import os
import subprocess
import sys

import numpy as np
import pytest

from oracle.solver import Operator, fused_matvec_full

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

GRIDS = [(1, 1, 1), (2, 1, 3), (3, 40, 1), (1, 5, 130), (25, 3, 62), (7, 33, 16), (24, 12, 6), (9, 10, 63)]


@pytest.mark.parametrize("dims", GRIDS)
@pytest.mark.parametrize("support", ["random", "planes"])
def test_compact_product(cuda, dims, support):
    from gpu_fem import _lib
    from gpu_fem._native import to_numpy
    from gpu_fem.pub_simp_solver import KE_UNIT_3D, _edof_table_3d
    from gpu_fem.solver_v2 import MatrixFreeKff

    rng = np.random.default_rng(sum(dims))
    nx, ny, nz = dims
    ndof = 3 * (nx + 1) * (ny + 1) * (nz + 1)
    keep = rng.random(ndof) < 0.7
    if support == "planes":  # plane 0 fixed, the last one partly, the others free
        per = ndof // (nx + 1)
        keep = np.concatenate([np.zeros(per, bool), np.ones(ndof - 2 * per, bool), rng.random(per) < 0.6])
    keep[-1] = True
    free = np.flatnonzero(keep).astype(np.int32)
    E, u = 0.1 + rng.random(nx * ny * nz), rng.standard_normal(free.size)
    op = MatrixFreeKff(cuda.as_tensor(_edof_table_3d(*dims), device="cuda"), KE_UNIT_3D,
                       cuda.as_tensor(free.astype(np.int64), device="cuda"), free.size, ndof, grid_dims=dims)
    ref = Operator(nx, ny, nz, free).matvec(u, E)
    ud, Ed = cuda.as_tensor(u, device="cuda"), cuda.as_tensor(E, device="cuda")
    for tuned in (False, True):
        if tuned:
            _lib.call("simpfem_mesh_tune", op.mesh.handle, _lib.stream_ptr())
        y = to_numpy(op.matvec(ud, Ed))
        assert np.linalg.norm(y - ref) <= 1e-13 * np.linalg.norm(ref)
        y32 = to_numpy(op.matvec(ud.float(), Ed.float()))
        assert np.linalg.norm(y32 - ref) <= 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("dims", GRIDS)
def test_bf16_product(cuda, dims):
    from gpu_fem.cuda_fused_matvec import FusedMatvec
    from gpu_fem.pub_simp_solver import KE_UNIT_3D, _edof_table_3d

    nx, ny, nz = dims
    ndof = 3 * (nx + 1) * (ny + 1) * (nz + 1)
    rng = np.random.default_rng(ndof)
    E, u = (0.1 + rng.random(nx * ny * nz)).astype(np.float32), rng.standard_normal(ndof).astype(np.float32)
    edof = _edof_table_3d(*dims)
    op = FusedMatvec(cuda.as_tensor(edof, device="cuda"), cuda.as_tensor(KE_UNIT_3D, device="cuda"), ndof)
    y = op.matvec_full(cuda.as_tensor(u, device="cuda"), cuda.as_tensor(E, device="cuda"), dtype="bf16").cpu().numpy()
    ref = fused_matvec_full(nx, ny, nz, u, E, KE_UNIT_3D, dtype="bf16")
    assert np.linalg.norm(y - ref) <= 1e-5 * np.linalg.norm(ref)


_DENSE = r"""
import sys
import numpy as np
import torch
sys.path[:0] = [{root!r}, {pkg!r}]
from gpu_fem import _lib
from gpu_fem._native import NativeMesh
from oracle.solver import edof_table
rng = np.random.default_rng(5)
W = np.array([[(-1.0) ** bin(s & q).count("1") for q in range(8)] for s in range(8)])
M = np.zeros((8, 3, 8, 3))
e = [4, 2, 1]
for b in range(8):
    A = rng.standard_normal((3, 3))
    A = A @ A.T
    for r in range(3):
        for c in range(3):
            M[b ^ e[r], r, b ^ e[c], c] = A[r, c]
K = np.einsum("sq,sctd,tr->qcrd", W, M, W).reshape(24, 24)
ref_nodes = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
perm = [3 * (4 * a + 2 * b + c) + d for (a, b, c) in ref_nodes for d in range(3)]
K = K[np.ix_(perm, perm)]
for dims in ((5, 3, 4), (9, 10, 20)):
    nx, ny, nz = dims
    ndof = 3 * (nx + 1) * (ny + 1) * (nz + 1)
    free = np.arange(3 * (ny + 1) * (nz + 1), ndof, dtype=np.int32)
    m = NativeMesh(dims, free, K)
    E, u = 0.1 + rng.random(nx * ny * nz), np.zeros(ndof)
    u[free] = rng.standard_normal(free.size)
    ed = edof_table(nx, ny, nz)
    y = np.zeros(ndof)
    np.add.at(y, ed, (K @ u[ed].T * E[None, :]).T)
    for dt, tdt, tol in ((_lib.F64, torch.float64, 1e-13), (_lib.F32, torch.float32, 1e-5)):
        Et = torch.as_tensor(E, device="cuda").to(tdt)
        ut = torch.as_tensor(u[free], device="cuda").to(tdt)
        yt = torch.empty_like(ut)
        _lib.call("simpfem_matvec", m.handle, dt, _lib.ptr(Et), _lib.ptr(ut), _lib.ptr(yt), _lib.stream_ptr())
        err = np.linalg.norm(yt.double().cpu().numpy() - y[free]) / np.linalg.norm(y[free])
        assert err <= tol, (dims, dt, err)
    del m
print("ok")
"""


def test_stiffness_without_the_isotropic_pattern(cuda):
    """In a fresh process: all meshes alive on a device share one stiffness."""
    pkg = os.path.join(ROOT, "solver-admissibility-and-guarded-floor-selection_b200")
    r = subprocess.run([sys.executable, "-c", _DENSE.format(root=ROOT, pkg=pkg)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stderr[-2000:]
