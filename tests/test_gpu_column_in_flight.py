"""The Arnoldi column's form goes by the solves in flight (csrc/linalg.cu:
arnoldi_one_launch): alone a solve takes one launch a column, of several of 450,765 unknowns
some take the launched form, and every one keeps the bits of the solve alone."""

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_solves_in_flight_keep_their_bits(cuda):
    torch = cuda
    from gpu_fem import _lib
    from gpu_fem._native import mesh_namespace
    from gpu_fem.bc_generator import generate_bc
    from gpu_fem.multigrid_v4 import GalerkinMatFreeGMG
    from gpu_fem.presets import cantilever_spec
    from gpu_fem.pub_simp_solver import KE_UNIT_3D, _edof_table_3d
    from gpu_fem.solver_v2 import MatrixFreeKff

    dims, workers, repeats = (104, 52, 26), 6, 3
    bc = generate_bc(cantilever_spec(*dims))
    free = bc.free_dofs.astype(np.int32)
    edof = torch.as_tensor(_edof_table_3d(*dims), device="cuda")
    rng = np.random.default_rng(7)
    E = torch.as_tensor(0.5 + rng.random(int(np.prod(dims))), device="cuda")
    b = torch.as_tensor(rng.standard_normal(len(free)), device="cuda")

    def make(tag):
        with mesh_namespace(tag):
            mf = MatrixFreeKff(edof, torch.as_tensor(KE_UNIT_3D, device="cuda"), torch.as_tensor(free, device="cuda"),
                               len(free), bc.ndof, grid_dims=dims)
            g = GalerkinMatFreeGMG(mf_op=mf, free=free, free_gpu=free, nelx=dims[0], nely=dims[1], nelz=dims[2],
                                   KE_UNIT=KE_UNIT_3D, fine_smoother="fp32", cycle_precision="fp32",
                                   smoother_type="jacobi")
            g.setup(E)
            return g

    gs = [make(("in flight", k)) for k in range(workers)]
    for g in gs[1:]:  # workspaces
        g._native_fgmres(b, None, 1e-6, 40, 40, None)
    ref, it, conv = gs[0]._native_fgmres(b, None, 1e-6, 40, 40, None)
    count = _lib.lib().simpfem_launch_count()
    again = gs[0]._native_fgmres(b, None, 1e-6, 40, 40, None)
    alone = _lib.lib().simpfem_launch_count() - count
    assert conv and again[1] == it and torch.equal(again[0], ref)
    streams = [torch.cuda.Stream() for _ in gs]
    torch.cuda.synchronize()
    out, start = [[] for _ in gs], threading.Barrier(workers)

    def work(k):
        with torch.cuda.stream(streams[k]):
            start.wait()
            for _ in range(repeats):
                out[k].append(gs[k]._native_fgmres(b, None, 1e-6, 40, 40, None))
            streams[k].synchronize()

    count = _lib.lib().simpfem_launch_count()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(workers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    launches = _lib.lib().simpfem_launch_count() - count
    for k in range(workers):
        assert len(out[k]) == repeats
        for x, i, c in out[k]:
            assert (i, c) == (it, True) and torch.equal(x, ref), k
    assert launches > workers * repeats * alone  # some columns were launched step by step
