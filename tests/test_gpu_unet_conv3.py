"""The mma.sync convolution at every channel count that its kernel is compiled for
(1 to 4 chunks of 16 channels, and any number), on the mma.sync path (forward and
backward) and on the tcgen05 path (backward), at the smallest grid, where every tile
of 4 x 8 x 8 cells is cut, and at one with whole and cut tiles.

Every output channel has one weight of +1 or -1 at a random tap and input channel,
so a convolution only moves values and both sides hold the same BF16 numbers; what
is left are values whose scale, average or sum of eight lies at a rounding boundary.
Loss and gradients against the CPU oracle: such a value is off by 2^-8, and it can
happen at the features, three poolings, three upsamplings' backward and the head,
eight times on a way through the network: 2^-5 of the norm. A wrong cell, tap or
channel changes a layer's gradient as a whole."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(8, 3), (24, 1)])
@pytest.mark.parametrize("tc", [False, True])
def test_moves(n, batch, tc):
    torch = pytest.importorskip("torch")
    from flip3d_gb300 import gpu
    from oracle import unet_oracle as U
    rng = np.random.default_rng(n)
    shape = (batch, n, n, n)
    A = (rng.random(shape) < 0.7).astype(np.uint8)
    b, x0, r0, x = (rng.normal(0, 1, shape).astype(np.float32) for _ in range(4))
    net = gpu.UNet(seed=7)
    net.set_tensor_path(tc)
    woff, boff, hoff, total = U.layout()
    p = np.zeros(total, np.float32)
    for l, (ci, co, _) in enumerate(U.CONVS):
        w = np.zeros((27, ci, co), np.float32)
        # the input layer reads its four real channels, the others all of theirs in turn
        src = rng.permutation(np.arange(max(co, ci)) % (4 if l == 0 else ci))[:co]
        w[rng.integers(0, 27, co), src, np.arange(co)] = rng.choice([-1.0, 1.0], co)
        p[woff[l]:woff[l] + 27 * ci * co] = w.ravel()
    p[hoff:hoff + 16] = rng.choice([-1.0, 1.0], 16)
    net.set_params(p)
    t = [torch.tensor(a.reshape(-1), device="cuda") for a in (A, b, x0, r0, x)]
    torch.cuda.synchronize()
    loss, g = net.gradients(n, batch, *(a.data_ptr() for a in t))
    want, og, _ = U.loss_and_grads(p.astype(np.float64), A, b, x0, r0, x, round_bf16=True)
    tol = 2.0 ** -5
    assert abs(loss - want) <= tol * abs(want)
    for l, (ci, co, _) in enumerate(U.CONVS):
        a, e = woff[l], boff[l] + co
        assert np.linalg.norm(g[a:e] - og[a:e]) <= tol * np.linalg.norm(og[a:e]), l
    assert np.linalg.norm(g[hoff:] - og[hoff:]) <= tol * np.linalg.norm(og[hoff:])
