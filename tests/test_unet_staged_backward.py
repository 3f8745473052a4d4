"""The network's backward pass from staged planes and lines against the kernels
that gather every tap (set_conv(False)), on grids whose tiles and lines end at
and off their edges: widths below, at and above a multiple of 16, a single
tile, several samples, depth runs that end early, and a line too wide to stage.

Activations and their gradients are rounded to BF16 after the same FP32 sums in
the same order, so they agree bit for bit; weight gradients add the same
products in FP32, in the same order within a CTA's range where the width is a
multiple of 16 (only the atomics between at most 74 ranges then differ: 74 *
2^-24 = 4e-6), and else in ranges of at most V / 16 roundings of 2^-24 each.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("loss", ["mse", "energy"])
@pytest.mark.parametrize("shape", [(1, 4, 4, 4), (2, 16, 16, 16), (1, 12, 20, 28), (3, 8, 36, 44), (1, 20, 12, 64),
                                   (2, 64, 64, 64), (1, 8, 20, 128), (1, 4, 8, 132), (1, 40, 16, 72)])
def test_gradients_match_the_per_tap_kernels(shape, loss):
    from mac_b200.unet import UNet
    from test_unet import _layer_slices
    rng = np.random.default_rng(sum(shape))
    n, d, h, w = shape
    m = (rng.random(shape) < 0.7).astype(np.int8)
    m[:, :, :, -1] = -1
    r = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    e = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    got = []
    with UNet(0, seed=3) as net:
        net.set_loss(loss)
        for staged in (True, False):
            net.set_conv(staged)
            got.append(net.loss_grad(r, m, e) + (net.forward(r, m),))
    (la, ga, fa), (lb, gb, fb) = got
    assert np.array_equal(fa, fb)
    assert abs(la - lb) <= 1e-12 * abs(lb)
    tol = 1e-5 if w % 64 == 0 else max(1e-5, n * d * h * w / 16 * 2.0 ** -24)
    for k, (a, b) in enumerate(_layer_slices()):
        x, y = ga[a:b], gb[a:b]
        assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y) + 1e-30, k
