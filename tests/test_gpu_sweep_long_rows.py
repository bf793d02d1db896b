"""The fine operator on grids with long rows along z, and on rods: every grid has tiles
(csrc/gmg.cu: sweep_candidates) to choose from.

The FP64 product has at most 24 x 8 terms per DOF: 1e-13 of the norm; FP32 1e-5.
"""

import re
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_TUNED = r"""
import os, sys
import numpy as np
import torch
sys.path[:0] = {path!r}
from gpu_fem import _lib
from gpu_fem._native import get_mesh
from gpu_fem.pub_simp_solver import KE_UNIT_3D
from oracle.solver import Operator
os.environ["SIMPFEM_TUNE_VERBOSE"] = "1"
nx, ny, nz = {dims!r}
free = np.arange(3 * (ny + 1) * (nz + 1), 3 * (nx + 1) * (ny + 1) * (nz + 1), dtype=np.int32)
rng = np.random.default_rng(nz)
E, u = 0.1 + rng.random(nx * ny * nz), rng.standard_normal(free.size)
ref = Operator(nx, ny, nz, free).matvec(u, E)
mesh = get_mesh((nx, ny, nz), free, KE_UNIT_3D)
for tuned in (False, True):
    if tuned:
        _lib.call("simpfem_mesh_tune", mesh.handle, _lib.stream_ptr())
    for dt, tdt, tol in ((_lib.F64, torch.float64, 1e-13), (_lib.F32, torch.float32, 1e-5)):
        Et, ut = (torch.as_tensor(v, device="cuda").to(tdt) for v in (E, u))
        y = torch.empty_like(ut)
        _lib.call("simpfem_matvec", mesh.handle, dt, _lib.ptr(Et), _lib.ptr(ut), _lib.ptr(y), _lib.stream_ptr())
        assert np.linalg.norm(y.double().cpu().numpy() - ref) <= tol * np.linalg.norm(ref), (dt, tuned)
print("ok")
"""


@pytest.mark.parametrize("dims", [(3, 5, 62), (3, 5, 63), (6, 4, 251), (6, 4, 252), (2, 3, 700), (700, 1, 2)])
def test_product_of_long_rows(cuda, dims):
    """Every grid has tiles to choose from, and blocks of at least one warp among them."""
    r = subprocess.run([sys.executable, "-c", _TUNED.format(path=sys.path, dims=dims)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stderr[-2000:]
    tiles = [int(a) * int(b) for a, b in re.findall(r"bj=(\d+) bk=(\d+)", r.stderr)]
    assert tiles and (max(tiles) >= 32 or dims == (700, 1, 2)), r.stderr[-500:]
