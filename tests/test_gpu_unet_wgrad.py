"""Weight gradients at the edges of their tiles: x-runs shorter than 16 cells,
of 16 cells and a remainder, longer than 64 (two runs), marches of one row and
of several, one volume and several. Against the numpy oracle; the tolerance
is the one of tests/test_gpu_unet.py (BF16 activations that sit near a
rounding boundary; a wrong tap, channel or run gives O(1))."""
import numpy as np
import pytest

from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 4, 4, 4), (2, 4, 20, 12), (1, 8, 4, 68), (3, 4, 12, 16),
                                   (1, 4, 8, 128)])
def test_gradients_match_oracle(nusif_lib, shape):
    import torch

    from nusif import UNet
    rng = np.random.default_rng(4)
    flat = U.init_params(4)
    x = rng.standard_normal(shape + (2,)).astype(np.float32)
    t = rng.standard_normal(shape).astype(np.float32)
    onet = U.UNet(flat)
    loss, dout = U.mse(onet.forward(x), t)
    gref = onet.backward(dout)
    with UNet() as net:
        net.set_params(flat)
        gl = net.train_step(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda(), update=False)
        g = net.grads()
    assert gl == pytest.approx(loss, rel=2e-2)
    o = 0
    for name, ci, co, _ in U.LAYERS:
        for n, what in ((27 * ci * co, ""), (co, " bias")):
            a, b = g[o:o + n].astype(np.float64), gref[o:o + n]
            assert np.linalg.norm(a - b) < 5e-2 * np.linalg.norm(b), name + what
            o += n
