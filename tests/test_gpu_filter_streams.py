"""Cone filters of different radii in flight at the same time (csrc/simp.cu: the neighbours are a
kernel argument): launches of two radii alternating on two streams without a wait between them
give what each gives by itself, bit for bit."""

import pytest

pytestmark = pytest.mark.gpu


def test_two_radii_on_two_streams(cuda):
    torch = cuda
    from gpu_fem.simp_loop import cone_filter

    dims = (160, 80, 40)
    x = torch.rand(dims[0] * dims[1] * dims[2], dtype=torch.float64, device="cuda")
    radii = (1.5, 3.5)
    ref = [cone_filter(x, dims, r) for r in radii]
    streams = [torch.cuda.Stream() for _ in radii]
    torch.cuda.synchronize()
    out = [[], []]
    for _ in range(20):
        for k, r in enumerate(radii):
            with torch.cuda.stream(streams[k]):
                out[k].append(cone_filter(x, dims, r))
    torch.cuda.synchronize()
    for k in range(2):
        assert all(torch.equal(v, ref[k]) for v in out[k]), radii[k]
