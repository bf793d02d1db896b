"""Exchanges over a grid that run out of their wait (csrc/gridcomm.cuh), made to by limits of a
few polls: the call ends with an error status or an unconverged solve, and the next call on the
same handle or workspace is bit for bit that of a fresh one.  A first block that gives up alone
lets the others, of which up to 32 exchange directly, go one exchange further and leave its
parts in the slots.  Every limit bounds a kernel at milliseconds; nothing waits on a flag that
another launch would set."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (polls, polls_first): nobody waits; the first block alone does not; the others alone do not
LIMITS = [(0, 0), (2000, 0), (0, 2000)]


def _opts(polls, first):
    from gpu_fem import _lib

    o = _lib.GridOpts()
    _lib.lib().simpfem_grid_default_opts(ctypes.byref(o))
    assert o.polls == o.polls_first == 1 << 21
    o.polls, o.polls_first = polls, first
    return o


def _set(gmg, o):
    from gpu_fem import _lib

    _lib.lib().simpfem_gmg_set_grid_opts(gmg._h, ctypes.byref(o) if o is not None else None)


def _gmg(torch, dims, **kw):
    from gpu_fem.bc_generator import generate_bc
    from gpu_fem.multigrid_v4 import GalerkinMatFreeGMG
    from gpu_fem.presets import cantilever_spec
    from gpu_fem.pub_simp_solver import KE_UNIT_3D, _edof_table_3d
    from gpu_fem.solver_v2 import MatrixFreeKff

    bc = generate_bc(cantilever_spec(*dims))
    free = bc.free_dofs.astype(np.int32)
    mf = MatrixFreeKff(torch.as_tensor(_edof_table_3d(*dims), device="cuda"), torch.as_tensor(KE_UNIT_3D, device="cuda"),
                       torch.as_tensor(free, device="cuda"), len(free), bc.ndof, grid_dims=dims)
    gmg = GalerkinMatFreeGMG(mf_op=mf, free=free, free_gpu=free, nelx=dims[0], nely=dims[1], nelz=dims[2],
                             KE_UNIT=KE_UNIT_3D, fine_smoother="fp64", smoother_type="jacobi", **kw)
    rng = np.random.default_rng(sum(dims))
    gmg.setup(torch.as_tensor(0.5 + rng.random(int(np.prod(dims))), device="cuda"))
    return gmg, torch.as_tensor(rng.standard_normal(len(free)), device="cuda")


# blocks of the Arnoldi column: a few, and more than exchange directly; the coarsest solve is dense
@pytest.mark.parametrize("dims", [(16, 8, 8), (60, 30, 20)])
@pytest.mark.parametrize("limits", LIMITS)
def test_arnoldi_column(cuda, dims, limits):
    torch = cuda
    gmg, b = _gmg(torch, dims, n_levels=3)
    ref = gmg._native_fgmres(b, None, 1e-8, 60, 30, None)
    assert ref[2]
    for _ in range(3):
        _set(gmg, _opts(*limits))
        x, it, conv = gmg._native_fgmres(b, None, 1e-8, 60, 30, None)
        assert not conv and bool(torch.isfinite(x).all())
        _set(gmg, None)
        x, it, conv = gmg._native_fgmres(b, None, 1e-8, 60, 30, None)
        assert (it, conv) == ref[1:] and torch.equal(x, ref[0])


# coarse systems of 8 and of 37 blocks with one row a lane group
@pytest.mark.parametrize("dims", [(16, 8, 4), (32, 16, 16)])
@pytest.mark.parametrize("limits", LIMITS)
def test_coarse_pcg(cuda, dims, limits):
    torch = cuda
    gmg, r = _gmg(torch, dims, n_levels=2, dense_chol_max=0, coarse_pcg_iters=25)
    assert gmg.coarse_mode == "iterative"
    ref = gmg.apply(r)
    for _ in range(3):
        _set(gmg, _opts(*limits))
        assert bool(torch.isnan(gmg.apply(r)).any())
        _set(gmg, None)
        assert torch.equal(gmg.apply(r), ref)


@pytest.mark.parametrize("n", [5000, 400_000])
@pytest.mark.parametrize("limits", LIMITS)
def test_oc_bisection(cuda, n, limits):
    torch = cuda
    from gpu_fem import _lib

    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    rho = torch.rand(n, dtype=torch.float64, device="cuda", generator=g).clamp_min(1e-3)
    dc = -torch.exp(torch.randn(n, dtype=torch.float64, device="cuda", generator=g))
    vw = 0.5 + torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    nbytes = int(_lib.lib().simpfem_oc_work_bytes())
    work = torch.empty(nbytes // 8, dtype=torch.float64, device="cuda")
    out = torch.empty_like(rho)

    def run(o):
        ch, lm, st, status = ctypes.c_double(), ctypes.c_double(), ctypes.c_int(), ctypes.c_int(-1)
        _lib.lib().simpfem_oc_update_opts(n, _lib.ptr(rho), _lib.ptr(dc), None, _lib.ptr(vw), 0.3, 0.2, _lib.ptr(out),
                                          _lib.ptr(work), nbytes, ctypes.byref(ch), ctypes.byref(lm), ctypes.byref(st),
                                          ctypes.byref(o) if o is not None else None, _lib.stream_ptr(),
                                          ctypes.byref(status))
        return status.value, ch.value, lm.value, st.value

    ref = run(None)
    first = out.clone()
    assert ref[0] == 0
    for _ in range(3):
        assert run(_opts(*limits))[0] == 9  # SIMPFEM_EINTERNAL
        assert b"wait" in _lib.lib().simpfem_last_error()
        assert run(None) == ref and torch.equal(out, first)
