"""Weight and bias gradients of the network, a block per nine taps and voxel range, against FP64 sums over the
activations and gradients that the device itself holds: grids whose voxel ranges leave remainders of a tile of
128, one sample and several, every channel combination."""

import numpy as np
import pytest

from mumag_matrixfree2_gb300 import learned
from oracle import unet as ou

pytestmark = pytest.mark.gpu

# layer: (its input, its output)
TENSORS = {"d0b": ("d0a", "out"), "d0a": ("h0", "d0a"), "d1b": ("d1a", "d1b"), "d1a": ("h1", "d1a"),
           "d2b": ("d2a", "d2b"), "d2a": ("h2", "d2a"), "b3c": ("b3b", "b3c"), "b3b": ("b3a", "b3b"),
           "b3a": ("p2", "b3a"), "e2b": ("e2a", "s2"), "e2a": ("p1", "e2a"), "e1b": ("e1a", "s1"),
           "e1a": ("p0", "e1a"), "e0b": ("e0a", "s0"), "e0a": ("x", "e0a")}


@pytest.mark.parametrize("grid, batch", [(16, 1), (24, 3), (40, 2)])
def test_weight_gradients_are_the_sums_over_voxels(cuda_ok, grid, batch):
    rng = np.random.default_rng(grid)
    net = learned.UNet(grid, batch, learned.init_params(3))
    net.forward(rng.standard_normal((batch, grid, grid, grid, 4)).astype(np.float32))
    net.backward(rng.standard_normal((batch, grid, grid, grid)).astype(np.float32))
    grads = net.get_grads()
    for name, (xin, out) in TENSORS.items():
        w = b = wa = ba = 0.0
        for s in range(batch):
            x = net.read(xin, s).astype(np.float64)
            d = net.read(out, s, grad=True).astype(np.float64)
            if name != "d0b":
                assert not np.any(d[net.read(out, s) <= 0.0]), name  # masked by the ReLU
            w = w + ou.conv3d_wgrad(x, d)
            wa = wa + ou.conv3d_wgrad(np.abs(x), np.abs(d))
            b = b + d.sum((0, 1, 2))
            ba = ba + np.abs(d).sum((0, 1, 2))
        if name == "e0a":  # padded input channels never learn
            w[:, 4:] = wa[:, 4:] = 0.0
        # at most 64 accumulations in a row in FP32, each off by one unit of 2^-23 of the sum of |terms|
        assert np.all(np.abs(grads[name + ".w"] - w) <= 64 * 2.0**-23 * wa + 1e-30), name
        assert np.all(np.abs(grads[name + ".b"] - b) <= 64 * 2.0**-23 * ba + 1e-30), name


def _splits(grid, batch):
    """The split of each voxel of a sample in the weight gradient of a layer with 16 x 16 channels, and their number:
    tiles of 128 of the padded planes that hold the grid, three blocks an SM."""
    P = grid + 2
    tiles = -(-P * P * grid // 128)
    ns = max(1, min(64, tiles, 456 // (3 * batch)))
    per = -(-tiles // ns)
    z, y, x = np.meshgrid(*[np.arange(grid)] * 3, indexing="ij")
    return (z * P * P + (y + 1) * P + x + 1) // (128 * per), -(-tiles // per)


def test_gradient_sums_past_the_range_of_floats(cuda_ok):
    """Bias partials whose sum passes FP32's range on the way and ends inside it, and partials that are infinite: an FP64
    sum of them is finite, or infinite, and never NaN.  A block's eight threads an element take every eighth partial,
    so the signs go by that: six threads of one, two of the other."""
    grid, batch = 16, 4
    net = learned.UNet(grid, batch, learned.init_params(3))
    x = np.random.default_rng(7).standard_normal((batch, grid, grid, grid, 4)).astype(np.float32)
    split, ns = _splits(grid, batch)
    part = np.arange(batch)[:, None, None, None] * ns + split[None]
    net.forward(x)
    net.backward(np.where(part % 8 < 6, -3e38, 3e38).astype(np.float32))
    d = np.stack([net.read("out", s, grad=True)[..., 0] for s in range(batch)]).astype(np.float64)
    of_thread = np.array([d[part % 8 == j].sum() for j in range(8)])
    big = np.finfo(np.float32).max
    assert np.abs(np.cumsum(of_thread)).max() > big > abs(d.sum())
    # at most 100 FP32 additions in a row: two of a tile's voxels by each of 96 threads, for two tiles, then the threads
    assert abs(net.get_grads()["d0b.b"][0] - d.sum()) <= 101 * 2.0**-24 * np.abs(d).sum()
    # one voxel of each of two samples without a bound, of one sign
    t = np.zeros((batch, grid, grid, grid), np.float32)
    t[0, 1, 2, 3] = t[1, 3, 2, 1] = -np.inf
    net.forward(x)
    net.backward(t)
    assert net.get_grads()["d0b.b"][0] == np.inf


def test_weight_gradients_at_the_training_size(cuda_ok):
    """32^3, eight samples: at most 17 tiles of 128 voxels a block.  A weight's partial is a chain of 4 multiplications of 16 voxels
    for each tile, of which an addend can be cut off at 2^-24 of the largest (17 of them), then the two halves; a bias's
    is 2 additions a tile and 96 threads' sums."""
    grid, batch = 32, 8
    rng = np.random.default_rng(grid)
    net = learned.UNet(grid, batch, learned.init_params(3))
    net.forward(rng.standard_normal((batch, grid, grid, grid, 4)).astype(np.float32))
    net.backward(rng.standard_normal((batch, grid, grid, grid)).astype(np.float32))
    grads = net.get_grads()
    for name in ("d0b", "d1a", "e2b"):
        xin, out = TENSORS[name]
        w = b = wa = ba = 0.0
        for s in range(batch):
            x, d = net.read(xin, s).astype(np.float64), net.read(out, s, grad=True).astype(np.float64)
            w, wa = w + ou.conv3d_wgrad(x, d), wa + ou.conv3d_wgrad(np.abs(x), np.abs(d))
            b, ba = b + d.sum((0, 1, 2)), ba + np.abs(d).sum((0, 1, 2))
        assert np.all(np.abs(grads[name + ".w"] - w) <= (4 * 17 * 17 + 2) * 2.0**-24 * wa + 1e-30), name
        assert np.all(np.abs(grads[name + ".b"] - b) <= (2 * 17 + 96 + 1) * 2.0**-24 * ba + 1e-30), name
