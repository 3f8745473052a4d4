"""The staged weight gradient where a CTA's range of voxels is shorter than a plane:
between the lines of the range, of the plane before and of the plane after lie gaps
that it must skip. Grids of few large planes, several samples (a range that crosses
a sample's end), odd widths and plane heights, a range that ends inside a line.

Both kernels add the same BF16 products in FP32. At a width that is a multiple of 64
(16 on every level) in the same order too, so they differ by the atomics between at
most 74 ranges (74 * 2^-24 = 4e-6); else by V / 16 roundings of 2^-24 at most.
The time is that of the whole call with either kernel; with the gaps walked the
staged one took 1.4 and 2.1 times the other's, without them it takes 0.8.
"""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(shape):
    rng = np.random.default_rng(sum(shape))
    m = (rng.random(shape) < 0.7).astype(np.int8)
    m[:, :, :, -1] = -1
    r = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    e = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    return r, m, e


@pytest.mark.parametrize("shape", [(1, 4, 128, 64), (3, 4, 132, 64), (1, 8, 100, 128), (5, 4, 60, 20), (2, 4, 200, 36),
                                   (1, 36, 36, 36), (1, 4, 256, 12), (7, 4, 20, 44)])
def test_gradients_of_flat_grids(shape):
    from mac_b200.unet import UNet
    from test_unet import _layer_slices
    r, m, e = _case(shape)
    got = []
    with UNet(0, seed=4) as net:
        for staged in (True, False):
            net.set_conv(staged)
            got.append(net.loss_grad(r, m, e)[1])
    tol = 1e-5 if shape[3] % 64 == 0 else max(1e-5, np.prod(shape) / 16 * 2.0 ** -24)
    for k, (a, b) in enumerate(_layer_slices()):
        x, y = got[0][a:b], got[1][a:b]
        assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y) + 1e-30, k


@pytest.mark.parametrize("shape", [(1, 4, 256, 128), (1, 8, 128, 128)])
def test_flat_grids_are_no_slower_than_the_per_tap_kernels(shape):
    from mac_b200.unet import UNet
    r, m, e = _case(shape)
    best = {}
    with UNet(0, seed=4) as net:
        for staged in (True, False, True, False):
            net.set_conv(staged)
            for _ in range(12):
                t = time.perf_counter()
                net.loss_grad(r, m, e)
                best[staged] = min(best.get(staged, 1e9), time.perf_counter() - t)
    print(best)
    assert best[True] <= 1.05 * best[False]
