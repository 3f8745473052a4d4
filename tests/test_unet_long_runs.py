"""Marching 3x3x3 convolutions over runs longer than the ring of accumulators
(four or eight output planes) at full, half and quarter resolution, against the
kernels that gather every tap (set_conv(False)). With 450 samples of 20 planes a
run is a whole column of planes, so the window of three crosses the ring's end
several times in every position.

The sums visit the same products in the same order, so activations agree bit for
bit; weight gradients agree within V / 16 FP32 roundings of 2^-24.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_long_runs_match_the_per_tap_kernels():
    from mac_b200.unet import UNet
    from test_unet import _layer_slices
    shape = (450, 20, 16, 16)
    rng = np.random.default_rng(77)
    m = (rng.random(shape) < 0.7).astype(np.int8)
    m[:, :, :, -1] = -1
    r = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    e = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    got = []
    with UNet(0, seed=5) as net:
        for staged in (True, False):
            net.set_conv(staged)
            got.append(net.loss_grad(r, m, e) + (net.forward(r, m),))
    (la, ga, fa), (lb, gb, fb) = got
    assert np.array_equal(fa, fb)
    assert abs(la - lb) <= 1e-12 * abs(lb)
    tol = np.prod(shape) / 16 * 2.0 ** -24
    for k, (a, b) in enumerate(_layer_slices()):
        assert np.linalg.norm(ga[a:b] - gb[a:b]) <= tol * np.linalg.norm(gb[a:b]) + 1e-30, k
