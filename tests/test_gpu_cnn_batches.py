"""The floor proposer's tiled convolution kernels (csrc/cnn.cu) at batches where
their blocks are partly empty: two and four samples share a block of the data
gradients, four and 32 a step of the weight gradients, whose ring holds four steps.

Small batches: float32 sums of at most 34 * 27 (forward, data) or 4096 * 31 terms
(weight gradients, added in partial sums) against the float64 oracle:
probabilities and loss to 2e-5, each parameter tensor's gradient to 1e-3 of its
largest entry.  Batches beyond 148 samples: some hidden unit out of millions lies
within a float32 rounding of its ReLU's kink, where the derivative jumps and the
oracle's choice is not the kernels' (149 samples: one unit at 6.5e-8 moves a tensor
by 1.1e-3 of its largest entry), so the gradient is compared with the sum over
sub-batches of 31, whose units take the same sides: float32 sums in another order,
2e-5 of the tensor's largest entry.
"""

import numpy as np
import pytest

from oracle import cnn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31])
def test_partial_blocks(cuda, n):
    from gpu_fem.floor_proposer import FloorProposerNet

    rng = np.random.default_rng(n)
    theta = cnn.init_params(n).astype(np.float32)
    theta += (0.02 * rng.standard_normal(theta.size)).astype(np.float32)
    x = rng.random((n, 1, 16, 16, 16)).astype(np.float32)
    f = (rng.standard_normal((n, 2)) * 0.5).astype(np.float32)
    lab = rng.integers(0, 3, n).astype(np.int32)
    net = FloorProposerNet(max_batch=200, params=theta)
    xd, fd = cuda.as_tensor(x, device="cuda"), cuda.as_tensor(f, device="cuda")
    prob = net.forward(xd, fd).cpu().numpy()
    logits, _ = cnn.forward(theta, x, f)
    e = np.exp(logits - logits.max(axis=1, keepdims=True))
    np.testing.assert_allclose(prob, e / e.sum(axis=1, keepdims=True), atol=2e-5, rtol=0)
    loss, g = net.loss_grad(xd, fd, cuda.as_tensor(lab, device="cuda"), want_grad=True)
    ref_loss, ref_g = cnn.loss_and_grad(theta, x, f, lab)
    assert abs(loss - ref_loss) <= 2e-5 * max(1.0, abs(ref_loss))
    offs = np.cumsum([0] + [int(np.prod(s)) for s in cnn.param_shapes()])
    for i in range(len(offs) - 1):
        ref = ref_g[offs[i]:offs[i + 1]]
        assert np.abs(g[offs[i]:offs[i + 1]] - ref).max() <= 1e-3 * np.abs(ref).max(), i


@pytest.mark.parametrize("n", [149, 200])
def test_blocks_of_several_samples(cuda, n):
    from gpu_fem.floor_proposer import FloorProposerNet

    rng = np.random.default_rng(n)
    theta = cnn.init_params(n).astype(np.float32)
    theta += (0.02 * rng.standard_normal(theta.size)).astype(np.float32)
    xd = cuda.as_tensor(rng.random((n, 16 ** 3)).astype(np.float32), device="cuda")
    fd = cuda.as_tensor((rng.standard_normal((n, 2)) * 0.5).astype(np.float32), device="cuda")
    yd = cuda.as_tensor(rng.integers(0, 3, n).astype(np.int32), device="cuda")
    net = FloorProposerNet(max_batch=200, params=theta)
    loss, g = net.loss_grad(xd, fd, yd, want_grad=True)
    ref, ref_loss = np.zeros(theta.size), 0.0
    for a in range(0, n, 31):
        b = min(n, a + 31)
        part_loss, part = net.loss_grad(xd[a:b], fd[a:b], yd[a:b], want_grad=True)
        ref += part.astype(np.float64) * (b - a) / n
        ref_loss += part_loss * (b - a) / n
    assert abs(loss - ref_loss) <= 2e-5 * max(1.0, abs(ref_loss))
    offs = np.cumsum([0] + [int(np.prod(s)) for s in cnn.param_shapes()])
    for i in range(len(offs) - 1):
        r = ref[offs[i]:offs[i + 1]]
        assert np.abs(g[offs[i]:offs[i + 1]] - r).max() <= 2e-5 * np.abs(r).max(), i
