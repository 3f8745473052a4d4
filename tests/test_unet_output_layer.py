"""Backward pass of the network's output layer (k_head_grad) in closed form, at
voxel counts around its blocks of 256. All weights but the output layer's are zero and its biases
constant, so its output is the bias where positive and 0 elsewhere; the output
layer's weights are powers of two, so each voxel's gradient product is exact in
BF16. Layer 11's bias gradient is then the output layer's bias gradient times
that weight where the bias is positive, and 0 where it is not. All voxels'
gradients have one sign (targets far below the output), so the two FP32 sums
agree within 2 V roundings of 2^-24."""
import numpy as np
import pytest

import unet_oracle as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 4, 4, 4), (1, 4, 8, 8), (3, 8, 4, 4), (1, 12, 20, 28), (2, 16, 16, 20)])
def test_output_layer_input_gradient(shape):
    from mac_b200.unet import UNet
    rng = np.random.default_rng(sum(shape))
    m = np.where(rng.random(shape) < 0.8, 1, -1).astype(np.int8)
    r = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    e = np.where(m == 1, -1e3, 0.0).astype(np.float32)
    offs, _ = U.offsets()
    b11, (w12, b12) = offs[11][1], offs[12]
    bias = np.array([0.5, -0.5] * 8, np.float32)
    weight = np.array([2.0 ** (c % 5 - 2) * (1 if c % 3 else -1) for c in range(16)], np.float32)
    with UNet(0, seed=4) as net:
        p = np.zeros(net.nparams, np.float32)
        p[b11:b11 + 16] = bias
        p[w12:w12 + 16] = weight
        net.set_params(p, 1.0)
        _, g = net.loss_grad(r, m, e)
    total = g[b12]
    assert total != 0
    want = np.where(bias > 0, weight * total, 0.0)
    tol = 2 * np.prod(shape) * 2.0 ** -24
    assert np.all(np.abs(g[b11:b11 + 16] - want) <= tol * np.abs(want)), (g[b11:b11 + 16], want)
