"""What runs where a device cannot hold a whole grid at once (the option one_launch = 0 takes
it): the Arnoldi column step by step gives the bits of the one launch; the coarse PCG adds in
another order, 25 well-conditioned iterations in 64 bits apart by 1e-10 at most; the OC
bisection takes the same steps to a multiplier within its last bracket (1e-9, twice for the two
ends), and the update follows it."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _set(gmg, one_launch):
    from gpu_fem import _lib

    o = _lib.GridOpts()
    _lib.lib().simpfem_grid_default_opts(ctypes.byref(o))
    assert o.one_launch == 1
    o.one_launch = one_launch
    _lib.lib().simpfem_gmg_set_grid_opts(gmg._h, ctypes.byref(o))


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


def _launches(fn):
    from gpu_fem import _lib

    before = _lib.lib().simpfem_launch_count()
    out = fn()
    return out, _lib.lib().simpfem_launch_count() - before


# 1, 2, 4, 6 and 22 elements a thread (the launched dot products take four in a pass)
@pytest.mark.parametrize("dims", [(16, 8, 8), (60, 30, 20), (76, 40, 24), (104, 52, 26), (160, 80, 40)])
def test_arnoldi_column(cuda, dims):
    gmg, b = _gmg(cuda, dims, n_levels=3 if dims[0] < 70 else 4)
    (x, it, conv), one = _launches(lambda: gmg._native_fgmres(b, None, 1e-8, 60, 30, None))
    _set(gmg, 0)
    (xl, itl, convl), many = _launches(lambda: gmg._native_fgmres(b, None, 1e-8, 60, 30, None))
    assert conv and (itl, convl) == (it, conv) and cuda.equal(xl, x)
    # column j: j + 2 dot products and updates, the rotation and the new vector against one launch
    assert many - one == sum(j + 4 - 1 for j in range(it))


@pytest.mark.parametrize("dims", [(16, 8, 4), (50, 26, 24)])
def test_coarse_pcg(cuda, dims):
    gmg, r = _gmg(cuda, dims, n_levels=2, dense_chol_max=0, coarse_pcg_iters=25)
    z, one = _launches(lambda: gmg.apply(r))
    _set(gmg, 0)
    zl, many = _launches(lambda: gmg.apply(r))
    assert many > one + 25
    assert float((z - zl).norm() / z.norm()) <= 1e-10
    _set(gmg, 1)
    assert cuda.equal(gmg.apply(r), z)


@pytest.mark.parametrize("n", [1, 5000, 400_003])
@pytest.mark.parametrize("with_dv", [False, True])
def test_oc_bisection(cuda, n, with_dv):
    torch = cuda
    from gpu_fem import _lib

    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    rho = torch.rand(n, dtype=torch.float64, device="cuda", generator=g).clamp_min(1e-3)
    dc = -torch.exp(torch.randn(n, dtype=torch.float64, device="cuda", generator=g))
    vw = 0.5 + torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    dv = 0.5 + torch.rand(n, dtype=torch.float64, device="cuda", generator=g) if with_dv else None
    nbytes = int(_lib.lib().simpfem_oc_work_bytes())
    work = torch.empty(nbytes // 8, dtype=torch.float64, device="cuda")
    o = _lib.GridOpts()
    _lib.lib().simpfem_grid_default_opts(ctypes.byref(o))

    def run(one_launch):
        o.one_launch = one_launch
        out = torch.empty_like(rho)
        ch, lm, st, status = ctypes.c_double(), ctypes.c_double(), ctypes.c_int(), ctypes.c_int(-1)
        _lib.lib().simpfem_oc_update_opts(n, _lib.ptr(rho), _lib.ptr(dc), _lib.ptr(dv) if with_dv else None,
                                          _lib.ptr(vw), 0.3, 0.2, _lib.ptr(out), _lib.ptr(work), nbytes,
                                          ctypes.byref(ch), ctypes.byref(lm), ctypes.byref(st), ctypes.byref(o),
                                          _lib.stream_ptr(), ctypes.byref(status))
        assert status.value == 0
        return out, ch.value, lm.value, st.value

    (x, ch, lm, st), one = _launches(lambda: run(1))
    (xl, chl, lml, stl), many = _launches(lambda: run(0))
    assert one == 1 and many == 2 * (st + 1)
    assert stl == st and abs(lml - lm) <= 2e-9 * max(1.0, lm)
    assert float((x - xl).abs().max()) <= 1e-8 and abs(ch - chl) <= 1e-8
