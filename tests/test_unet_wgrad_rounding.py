"""Rounding of the 3x3x3 weight gradients at widths that are no multiple of 16,
where staged lines are padded: tensor memory truncates each sum it adds to, so
what counts is how many additions a sum takes.

All activations of the test network are 1 and its output error is a power of two
constant on blocks of 4^3 voxels, which the centre taps carry to every level
unchanged in its bits (times 8 and 64). The gradient of a tap's weight is then a
sum of BF16 numbers that FP64 adds exactly, and what a device sum is off is its
own rounding. The exponents spread over 14 bits, so a sum needs more than FP32 has.

The staged sums take at most three quarters of the additions of the per-tap kernels'
(set_conv(False)), so their error is no larger but for the FP32 atomics that join
the ranges: up to 300, each rounding to nearest, 2^-24 sqrt(300) together.
"""
import numpy as np
import pytest

import unet_oracle as U

pytestmark = pytest.mark.gpu

#: 3x3x3 layers off the network's input, their level, and the channel whose centre tap carries the error on
CARRIED = {4: (2, None), 5: (2, 0), 7: (1, 32), 8: (1, 0), 10: (0, 16), 11: (0, 0)}


def _params():
    offs, n = U.offsets()
    p = np.zeros(n, np.float32)
    for k, ((wo, bo), (cin, cout, taps, *_r)) in enumerate(zip(offs, U.LAYERS)):
        w = p[wo:wo + taps * cout * cin].reshape(taps, cout, cin)
        if k < 12:
            p[bo:bo + cout] = 1.0
        ci = CARRIED[k][1] if k in CARRIED else (0 if k in (6, 9, 12) else None)
        if ci is not None:
            w[taps // 2, 0, ci] = 1.0
            p[bo] = 0.0  # channel 0 is carried forward too
    return p


def _errors(net, staged, r, m, e, g16, shape):
    net.set_conv(staged)
    _, grad = net.loss_grad(r, m, e)
    offs, _ = U.offsets()
    out = {}
    for k, (lvl, _c) in CARRIED.items():
        (wo, _b), (cin, cout, taps, *_r) = offs[k], U.LAYERS[k]
        got = grad[wo:wo + 27 * cout * cin].reshape(3, 3, 3, cout, cin)[:, :, :, 0].astype(np.float64)
        g = g16[:, ::2 ** lvl, ::2 ** lvl, ::2 ** lvl] * 8.0 ** lvl
        want = np.empty((3, 3, 3))
        for t in np.ndindex(3, 3, 3):  # the voxels whose neighbour at the tap is in the grid
            want[t] = g[(slice(None),) + tuple(slice(max(0, 1 - a), s + min(0, 1 - a))
                                               for a, s in zip(t, g.shape[1:]))].sum()
        out[k] = np.linalg.norm(got - want[..., None]) / (np.linalg.norm(want) * np.sqrt(cin))
    return out


@pytest.mark.parametrize("w", [4, 8, 12, 16, 20, 24, 28, 36, 40, 44, 60, 72, 100, 124])
def test_padded_lines_round_no_worse(w):
    import torch
    from mac_b200.unet import UNet
    shape = (8, 64, 64, w)
    rng = np.random.default_rng(w)
    k = rng.integers(0, 15, (8, 16, 16, (w + 3) // 4))
    d = np.ldexp(1.0, -k).repeat(4, 1).repeat(4, 2).repeat(4, 3)
    r, m = np.ones(shape, np.float32), np.ones(shape, np.int8)
    e = (1.0 - d).astype(np.float32)
    s16 = float(torch.tensor(2.0 / np.prod(shape), dtype=torch.float64).float().bfloat16())
    with UNet(0) as net:
        net.set_params(_params(), 1.0)
        tap = _errors(net, False, r, m, e, d * s16, shape)
        staged = _errors(net, True, r, m, e, d * s16, shape)
    print(w, {q: "%.2e %.2e" % (tap[q], staged[q]) for q in tap})
    for q in tap:
        assert tap[q] < 1e-3, q  # the error carried is the one meant
        assert staged[q] <= tap[q] + 2.0 ** -24 * 300 ** 0.5, (q, staged[q], tap[q])
