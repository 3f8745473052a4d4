"""The marching convolutions on grids too small to fill the device with runs of four
planes, where a run has one to three: forward values have the per-tap kernel's bits
(BF16 after equal FP32 sums), and the pass is not held up by a run's planes.

Device time against the per-tap kernels': 0.49-0.51 with short runs, 0.64-0.66 with
runs of four planes throughout.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 4, 4, 4), (1, 8, 8, 8), (2, 12, 20, 8), (1, 128, 8, 8), (7, 20, 12, 16),
                                   (1, 36, 36, 36), (16, 16, 16, 16), (1, 4, 64, 128), (27, 8, 16, 8), (1, 44, 28, 52)])
def test_short_runs_keep_the_bits(shape):
    from mac_b200.unet import UNet
    rng = np.random.default_rng(sum(shape))
    m = rng.integers(-1, 2, shape).astype(np.int8)
    r = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    with UNet(0, seed=5) as net:
        a = net.forward(r, m)
        net.set_conv(False)
        b = net.forward(r, m)
    assert np.array_equal(a, b) and np.abs(a).max() > 0


@pytest.mark.parametrize("shape", [(1, 8, 8, 8), (1, 128, 8, 8)])
def test_small_grids_are_not_held_up_by_long_runs(shape):
    from mac_b200.unet import UNet
    best = {}
    with UNet(0, seed=5) as net:
        for staged in (True, False, True, False):
            net.set_conv(staged)
            best[staged] = min([best.get(staged, 1e9)] + [net.time_forward(*shape, reps=30)[0] for _ in range(3)])
    print(best)
    assert best[True] <= 0.57 * best[False]
