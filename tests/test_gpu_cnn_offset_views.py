"""The proposer's training step and forward on views of any float alignment: x is copied into
shared memory by 16-byte asynchronous copies where it starts on 16 bytes and float by float
elsewhere, so a view one to three floats into a buffer gives the aligned copy's bits."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 5])
def test_offset_views_give_the_aligned_bits(cuda, batch):
    torch = cuda
    from gpu_fem.floor_proposer import FloorProposerNet

    g = torch.Generator(device="cuda")
    g.manual_seed(batch)
    net = FloorProposerNet(max_batch=batch, seed=3)
    x = torch.rand((batch, 4096), device="cuda", generator=g)
    f = torch.rand((batch, 2), device="cuda", generator=g)
    y = torch.arange(batch, device="cuda", dtype=torch.int32) % 3
    loss, grad = net.loss_grad(x, f, y, want_grad=True)
    p = net.forward(x, f)
    for off in (1, 2, 3):
        buf = torch.empty(batch * 4096 + 8, device="cuda")
        xv = buf[off:off + batch * 4096].view(batch, 4096)
        xv.copy_(x)
        fb = torch.empty(batch * 2 + 8, device="cuda")
        fv = fb[off:off + batch * 2].view(batch, 2)
        fv.copy_(f)
        yb = torch.empty(batch + 8, device="cuda", dtype=torch.int32)
        yv = yb[off:off + batch]
        yv.copy_(y)
        assert xv.data_ptr() % 16 == 4 * off
        loss_v, grad_v = net.loss_grad(xv, fv, yv, want_grad=True)
        assert np.float32(loss_v) == np.float32(loss)
        assert np.array_equal(grad_v, grad), off
        assert torch.equal(net.forward(xv, fv), p), off
