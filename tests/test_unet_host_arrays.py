"""The network's calls with pageable host arrays (staged in chunks by several
threads above 2 MB) against the same calls with pinned ones (plain copies), at
sizes below and above the line, whole and ragged chunks, fewer chunks than
lanes and many a lane. The same bytes must arrive: results are equal."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(a):
    import torch
    return torch.from_numpy(a).pin_memory().numpy()


@pytest.mark.parametrize("shape", [(1, 72, 76, 76), (1, 76, 80, 84), (2, 64, 64, 64), (1, 100, 124, 132), (3, 128, 96, 100)])
def test_pageable_and_pinned_arrays_agree(shape):
    from mac_b200.unet import UNet
    rng = np.random.default_rng(sum(shape))
    m = (rng.random(shape) < 0.7).astype(np.int8)
    m[:, :, :, -1] = -1
    r = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    e = np.where(m == 1, rng.standard_normal(shape), 0.0).astype(np.float32)
    pr, pm, pe, want = _pinned(r), _pinned(m), _pinned(e), _pinned(np.full(shape, np.nan, np.float32))
    f32, i8 = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int8)
    with UNet(0, seed=9) as net:
        net._check(net.lib.mac_unet_forward(net.h, *shape, pr.ctypes.data_as(f32), pm.ctypes.data_as(i8),
                                            want.ctypes.data_as(f32)), "forward")
        for _ in range(2):
            assert np.array_equal(net.forward(r, m), want)
        la, _ = net.loss_grad(pr, pm, pe)
        lb, _ = net.loss_grad(r, m, e)
        assert abs(la - lb) <= 1e-12 * abs(la)
