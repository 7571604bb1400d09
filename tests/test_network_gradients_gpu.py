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
