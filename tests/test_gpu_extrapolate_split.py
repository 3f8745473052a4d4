"""Layer extrapolation on both sides of the line (1,024 live bricks) between a
block per axis and a block per brick, bit for bit against its rule written out
over a dense grid. The layers are drawn at random over all existing cells, so
every combination of a face's layers and its neighbours' occurs, cut bricks
included. (The oracle grows its front from the layer-1 cells, so it stands for
the rule only where layers are distances; test_gpu_parity compares those.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rule(s):
    """Level by level: a face (between cell c and c - e_i) whose lower layer is L
    becomes the mean of the neighbouring faces of its axis that touch a layer
    below L, added in the order -x +x -y +y -z +z."""
    keys = s.cell_keys().reshape(-1, 3)
    ex = s.exists.astype(bool).reshape(-1)
    lo = keys.min(0) - 3
    dim = keys.max(0) - lo + 4
    at = tuple((keys - lo).T)
    lay = np.full(dim, -1, np.int32)
    lay[at] = np.where(ex, s.layer.reshape(-1), -1)
    const = np.zeros(dim, np.uint8)
    const[at] = s.flags.reshape(-1)
    sh = lambda a, d: np.roll(a, [-v for v in d], (0, 1, 2))  # value of cell c + d
    unit = np.eye(3, dtype=int)
    out = {}
    for i, f in enumerate(("u0x", "u0y", "u0z")):
        u = np.zeros(dim)
        u[at] = s.f64[f].reshape(-1)
        e = unit[i]
        la = sh(lay, -e)
        for L in range(1, s.params.layer_max + 2):
            write = ((la == L) & (lay >= L)) | ((lay == L) & ((la < 0) | (la >= L)))
            write &= (lay >= 0) & ((const >> i) & 1 == 0)
            n, val = np.zeros(dim), np.zeros(dim)
            for j in range(3):
                for d in (-unit[j], unit[j]):
                    l1 = sh(lay, d)
                    if j != i:
                        l0 = sh(lay, d - e)
                        take = (l0 >= 0) & (l1 >= 0) & ((l0 < L) | (l1 < L))
                    elif d[i] < 0:
                        l0 = sh(lay, -2 * e)
                        take = (la >= 0) & (l0 >= 0) & (l0 < L)
                    else:
                        take = (l1 >= 0) & (l1 < L)
                    n += take
                    val = np.where(take, val + sh(u, d), val)
            with np.errstate(invalid="ignore", divide="ignore"):
                u = np.where(write, val / n, u)
        out[f] = u[at].reshape(s.exists.shape)
    return out


@pytest.mark.parametrize("n,split", [(17, True), (62, True), (70, False)])
def test_both_forms_follow_the_rule(n, split):
    from mac_b200.gpu import Context
    from mac_b200.state import pool_spheres_world
    from mac_b200.world import setup_passes
    s = setup_passes(pool_spheres_world(n, nspheres=4, r_range=(0.05 * n, 0.15 * n), pool_frac=0.5)).sorted()
    assert (s.nbricks <= 1024) == split, s.nbricks
    layer = np.random.default_rng(n).integers(0, 7, s.layer.shape, dtype=s.layer.dtype)
    s.layer[:] = np.where(s.exists.astype(bool), layer, -1)
    with Context(s.params, max_bricks=s.nbricks + 64, max_particles=1024) as ctx:
        ctx.upload(s)
        ctx.extrapolate()
        got = ctx.download().sorted()
    want = _rule(s)
    ex = s.exists.astype(bool)
    for f in ("u0x", "u0y", "u0z"):
        assert np.array_equal(got.f64[f][ex], want[f][ex], equal_nan=True), f
