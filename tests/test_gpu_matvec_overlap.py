"""The FP64 operator product through the C interface with a result that shares memory
with its vector or its moduli: all of them are read before the result is written.  The
product has at most 24 x 8 terms per DOF, 1e-13 of the result's norm as the operator's
other tests."""

import numpy as np
import pytest

from oracle.solver import Operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shares,shift", [("u", 0), ("u", 1), ("u", -700), ("E", 0), ("E", -3)])
def test_shared_result(cuda, shares, shift):
    from gpu_fem import _lib
    from gpu_fem._native import get_mesh, to_numpy
    from gpu_fem.pub_simp_solver import KE_UNIT_3D

    nx, ny, nz = 24, 12, 6
    free = np.arange(3 * (ny + 1) * (nz + 1), 3 * (nx + 1) * (ny + 1) * (nz + 1), dtype=np.int32)
    rng = np.random.default_rng(shift + 1000)
    E, u = 0.1 + rng.random(nx * ny * nz), rng.standard_normal(free.size)
    mesh = get_mesh((nx, ny, nz), free, KE_UNIT_3D)
    shared = u if shares == "u" else E
    buf = cuda.zeros(2 * free.size + 2000, dtype=cuda.float64, device="cuda")
    at = 1000  # the result starts here, the shared operand at at - shift
    op = buf[at - shift:at - shift + shared.size]
    op.copy_(cuda.as_tensor(shared, device="cuda"))
    y = buf[at:at + free.size]
    ud = op if shares == "u" else cuda.as_tensor(u, device="cuda")
    Ed = op if shares == "E" else cuda.as_tensor(E, device="cuda")
    _lib.call("simpfem_matvec", mesh.handle, _lib.F64, _lib.ptr(Ed), _lib.ptr(ud), _lib.ptr(y), _lib.stream_ptr())
    ref = Operator(nx, ny, nz, free).matvec(u, E)
    assert np.linalg.norm(to_numpy(y) - ref) <= 1e-13 * np.linalg.norm(ref)
