"""simpfem_oc_update's workspace is an array of doubles: one that starts between two 16-byte
boundaries gives the bits that one on a boundary gives, and nothing is written outside it."""

import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 60_001])
def test_workspace_at_any_double(cuda, n):
    torch = cuda
    from gpu_fem import _lib

    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    rho = torch.rand(n, dtype=torch.float64, device="cuda", generator=g).clamp_min(1e-3)
    dc = -torch.exp(torch.randn(n, dtype=torch.float64, device="cuda", generator=g))
    vw = 0.5 + torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    nbytes = int(_lib.lib().simpfem_oc_work_bytes())
    words = nbytes // 8
    assert 8 * words == nbytes

    def run(off):
        buf = torch.full((words + off + 4,), 7.0, dtype=torch.float64, device="cuda")
        out = torch.empty_like(rho)
        ch, lm, st = ctypes.c_double(), ctypes.c_double(), ctypes.c_int()
        _lib.call("simpfem_oc_update", n, _lib.ptr(rho), _lib.ptr(dc), None, _lib.ptr(vw), 0.3, 0.2, _lib.ptr(out),
                  _lib.ptr(buf) + 8 * off, nbytes, ctypes.byref(ch), ctypes.byref(lm), ctypes.byref(st),
                  _lib.stream_ptr())
        assert bool((buf[:off] == 7.0).all()) and bool((buf[off + words:] == 7.0).all())
        return out, ch.value, lm.value, st.value

    ref = run(0)
    got = run(1)
    assert torch.equal(got[0], ref[0]) and got[1:] == ref[1:]
