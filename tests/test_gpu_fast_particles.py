"""The particle move where a particle crosses several cells in one step: stencils of
the later Runge-Kutta stages lie partly or wholly outside the region staged around
the particle's brick, one cell below it included, and are then read through the brick
table. Against the oracle, bit for bit: uneven speeds around a mean that carries the
particles 1.2 to 3.6 cells along one, two or three axes, either way.

The runs of a falling, splashing or unstable flow reach such steps: dt follows the
speeds before the projection.
"""
import numpy as np
import pytest

from mac_b200.state import FLUID, Params, from_cells

N, H, DT = 28, 0.02, 0.01


def _world(direction, cells, sym):
    rng = np.random.default_rng(int(cells * 10) + sum(direction))
    g = np.arange(-4, N + 4)
    keys = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    u = np.asarray(direction) * cells * H / DT + rng.uniform(-0.4, 0.4, (len(keys), 3)) * H / DT
    # particles of the middle, every position inside a brick among them
    mid = keys[((keys >= 8) & (keys < N - 8)).all(1)]
    pos = (mid[:, None, :] + rng.uniform(-0.5, 0.5, (len(mid), 8, 3))).reshape(-1, 3) * H
    pr = Params(h=(H, H, H), dt_max=DT, dt=DT, layer_max=4, interp_symmetric=sym)
    s = from_cells(pr, keys, np.full(len(keys), FLUID, np.uint8), np.zeros(len(keys), np.uint8), u, pos)
    s.layer[s.exists != 0] = 0
    return s


CASES = [((0, 0, -1), 1.2), ((0, 0, -1), 2.4), ((0, 0, -1), 3.6), ((-1, 0, 0), 2.4), ((0, -1, 0), 2.4), ((-1, -1, -1), 2.4),
         ((-1, 0, -1), 3.0), ((0, -1, -1), 2.0), ((1, 1, 1), 2.4), ((0, 0, 1), 3.6), ((-1, 1, -1), 2.6)]


def _rows(p):
    return p[np.lexsort(p.T)]


def test_the_stencils_meant_are_among_them():
    """On CPU: in the second half of a downward move some particles' stencil corners lie exactly one cell below
    the twelve staged along an axis (local coordinate -3), the others inside."""
    s = _world((-1, -1, -1), 2.4, 1)
    cell = np.round(s.pos / H).astype(int)
    local = np.round(s.pos / H - 2.4).astype(int) - cell // 8 * 8
    assert ((local == -3).any(1) & (local >= -3).all(1)).sum() > 50


@pytest.mark.gpu
@pytest.mark.parametrize("sym", [1, 0])
@pytest.mark.parametrize("direction,cells", CASES)
def test_fast_particles_match_the_oracle(run_oracle, direction, cells, sym):
    from mac_b200.gpu import Context
    s = _world(direction, cells, sym)
    want, st = run_oracle("move" if sym else "movelin", s)
    assert st["invalid_reads"] == 0
    moved = np.abs(want.pos - s.pos).max() / H
    assert cells < moved < cells + 0.6
    with Context(s.params, max_bricks=s.nbricks + 64, max_particles=s.nparticles + 64) as ctx:
        ctx.upload(s)
        ctx.move()
        got = ctx.download()
    assert np.array_equal(_rows(got.pos), _rows(want.pos))
