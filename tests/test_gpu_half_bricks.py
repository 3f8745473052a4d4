"""The launch-by-launch MG-PCG's level-0 passes (a warp per half brick) against
the one-launch form of the solve, which stages bricks in shared memory. A coarse
block of 64 cells keeps the launches for every box of more than 64 bricks, with
the first kernel that the prefetching form (test_gpu_resident_solve) replaces.
Odd box sizes: bricks cut at every offset, absent neighbours, partial last
blocks of four bricks.

Both solve to a relative residual of 1e-12 with the same preconditioner, so each
is within 1e-10 of the exact pressure and they agree to 1e-9.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(s, solver, block):
    from mac_b200.gpu import Context
    with Context(s.params, max_bricks=int(s.nbricks * 1.2) + 64, max_particles=1024, solver=solver, rtol=1e-12,
                 max_iters=500) as ctx:
        if block:
            ctx.set_coarse_block(block)
        ctx.upload(s)
        before = ctx.launches()
        ctx.project(0)
        launched = ctx.launches() - before
        st, got = ctx.stats(), ctx.download()
    return got, st, launched


@pytest.mark.parametrize("solver", ["mgpcg64", "mixed"])
@pytest.mark.parametrize("n,frac", [(33, 0.4), (39, 0.8), (41, 0.6), (55, 0.45), (66, 0.7)])
def test_launches_match_one_launch(n, frac, solver):
    from mac_b200.state import pool_spheres_world
    from mac_b200.world import setup_passes
    s = setup_passes(pool_spheres_world(n, nspheres=4, r_range=(0.05 * n, 0.15 * n), pool_frac=frac))
    a, sa, la = _solve(s, solver, 64)
    b, sb, lb = _solve(s, solver, 0)
    assert la > lb + 20 * sa["iterations"] // 2, (la, lb)
    assert abs(sa["iterations"] - sb["iterations"]) <= 1
    ex = a.exists.astype(bool)
    for f in ("p", "u0x", "u0y", "u0z"):
        x, y = a.f64[f][ex], b.f64[f][ex]
        assert np.linalg.norm(x - y) <= 1e-9 * np.linalg.norm(y), f
