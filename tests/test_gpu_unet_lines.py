"""The tcgen05 convolution's lines per unit (2, 4 or 8 on 128-cell segments): the
autotuner's choice and the default give the same bits, with one and with two
segments a line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 256])
def test_lines_give_the_same_bits(n):
    torch = pytest.importorskip("torch")
    from flip3d_gb300 import gpu
    rng = np.random.default_rng(n)
    m = n ** 3
    A = torch.tensor((rng.random(m, dtype=np.float32) < 0.7).astype(np.uint8), device="cuda")
    b, x0, r0 = (torch.tensor(rng.standard_normal(m, dtype=np.float32), device="cuda")
                 for _ in range(3))
    net = gpu.UNet(seed=4)
    outs = []
    try:
        for mode in (1, 0):
            gpu.set_autotune(-1)
            gpu.set_autotune(mode)
            d = torch.zeros(m, dtype=torch.float32, device="cuda")
            torch.cuda.synchronize()
            net.predict(n, 1, A.data_ptr(), b.data_ptr(), x0.data_ptr(), r0.data_ptr(),
                        d.data_ptr())
            torch.cuda.synchronize()
            outs.append(d.cpu().numpy())
    finally:
        gpu.set_autotune(1)
    assert np.isfinite(outs[0]).all() and np.abs(outs[0]).max() > 0
    assert np.array_equal(outs[0], outs[1])
