"""Weight and bias gradients against exact sums: a network whose activations
are all 1 and whose output gradients are small integers times powers of two of
many sizes, exact in BF16, at every layer, so that a gradient is a sum of
positive numbers over the cells and what is left of its error is the order and
the rounding of that sum.

Every layer's weights are 0 but those of the centre tap to its first output
channel, which are 1; biases bring each channel back to 1. The targets are
constant over 4 x 4 x 4 cells, so sums over children stay exact as well."""
import numpy as np
import pytest

from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu

# layer -> level and multiple of the target in its (masked) output gradient
GRADS = {"out": (0, 1), "d0b": (0, 1), "d0a": (0, 1), "d1b": (1, 8), "d1a": (1, 8), "e2a": (2, 64),
         "e1b": (1, 16), "e1a": (1, 16), "e0b": (0, 3), "e0a": (0, 3)}


def _ones_network():
    flat = []
    for name, ci, co, _ in U.LAYERS:
        w = np.zeros((27, co, ci), np.float32)
        b = np.ones(co, np.float32)
        if name == "out":
            w[13] = 1.0
            b[:] = -ci
        elif name != "e0a":
            w[13, 0] = 1.0
            b[0] = 1.0 - ci
        flat += [w.ravel(), b]
    return np.concatenate(flat)


def _sums(shape, seed):
    """(gradients of the network, {layer: (exact weight sums [27], exact bias sum)}), shape
    [B, Z, Y, X] of a power of two cells."""
    import torch

    from nusif import UNet
    b, z, y, x = shape
    n = b * z * y * x
    assert n & (n - 1) == 0
    rng, blocks = np.random.default_rng(seed), (b, z // 4, y // 4, x // 4)
    k = rng.integers(1, 86, blocks) * 2.0 ** -rng.integers(0, 16, blocks)  # 3 k has 8 bits
    up = [np.kron(k, np.ones((1, s, s, s))) * (2.0 / n) for s in (4, 2, 1)]  # of each level
    with UNet() as net:
        net.set_params(_ones_network())
        ones = torch.ones(shape + (2,), device="cuda")
        t = torch.from_numpy((-np.kron(k, np.ones((1, 4, 4, 4)))).astype(np.float32)).cuda()
        assert float(net.forward(ones).abs().max()) == 0.0
        net.train_step(ones, t, update=False)
        grads = net.grads().astype(np.float64)
    exact = {}
    for name, (level, m) in GRADS.items():
        g = m * up[level]
        taps = []
        for dz, dy, dx in U.TAPS:
            s = [slice(max(0, -d), e - max(0, d)) for d, e in zip((dz, dy, dx), g.shape[1:])]
            taps.append(g[:, s[0], s[1], s[2]].sum())
        exact[name] = np.array(taps), g.sum()
    return grads, exact


def _errors(shape, seed=1):
    """{layer: (largest relative error of its weight gradients, of its bias gradients)}"""
    grads, exact = _sums(shape, seed)
    out, o = {}, 0
    for name, ci, co, _ in U.LAYERS:
        w = grads[o:o + 27 * co * ci].reshape(27, co * ci)
        o += 27 * co * ci
        bias = grads[o:o + co]
        o += co
        ew, eb = exact[name]
        out[name] = (np.abs(w / ew[:, None] - 1.0).max(), np.abs(bias / eb - 1.0).max())
    return out


SHAPES = [(1, 128, 128, 128), (2, 256, 128, 64), (1, 32, 64, 128), (4, 64, 32, 16)]


@pytest.mark.parametrize("shape", SHAPES)
def test_bias_gradients_are_rounded_sums(nusif_lib, shape):
    """A row's cells (64 at most, four steps of the tensor core, which drops up to
    2^-23 of the sum in each), then rounded FP32 additions of the rows and of the
    blocks' sums, 250 of them here at most: 2^-22 + 2 sqrt(250) 2^-24 = 2.1e-6."""
    errors = _errors(shape)
    assert max(bias for _, bias in errors.values()) < 2.1e-6, errors


@pytest.mark.parametrize("shape", SHAPES)
def test_weight_gradients_drift_with_short_chains_only(nusif_lib, shape):
    """A chain of the tensor core is at most a 256th of a layer's cells (or 64), 16
    cells a step, each dropping half of a unit in the last place of a sum that
    grows to the chain's: steps / 2 times 0.36 2^-23 of it. Half as much again
    for the sums' unevenness, and the bound of the rounded additions above."""
    errors = _errors(shape)
    for name, (level, _) in GRADS.items():
        cells = np.prod(shape) / 8 ** level
        steps = max(64, cells / 256) / 16
        bound = 1.5 * steps / 2 * 0.36 * 2.0 ** -23 + 2.1e-6
        assert errors[name][0] < (2.1e-6 if name in ("e0a", "out") else bound), (name, errors)
