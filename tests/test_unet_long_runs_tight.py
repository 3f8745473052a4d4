"""The marching convolutions' long runs (as test_unet_long_runs) at the bound that
equal sums have: at a width of 16 the staged weight gradient adds what the per-tap
kernel adds, in its order, so the gradients differ by the FP32 atomics between at
most 74 ranges alone (74 * 2^-24 = 4e-6). An edge column of a few samples off in an
input gradient would show here.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_long_runs_agree_to_the_atomics():
    from mac_b200.unet import UNet
    from test_unet import _layer_slices
    shape = (450, 20, 16, 16)
    rng = np.random.default_rng(78)
    m = (rng.random(shape) < 0.7).astype(np.int8)
    m[:, :, :, -1] = -1
    r = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    e = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    got = []
    with UNet(0, seed=6) as net:
        for staged in (True, False):
            net.set_conv(staged)
            got.append(net.loss_grad(r, m, e)[1])
    for k, (a, b) in enumerate(_layer_slices()):
        x, y = got[0][a:b], got[1][a:b]
        assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(y) + 1e-30, k
