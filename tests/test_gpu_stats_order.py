"""Which solve the stats of an RK2-TVD pass are: the second projection's, also when
the first one's outcome is read after it.

The first solve starts from a pressure far off, stalls with a network that does
nothing, and falls back to the one-launch multigrid solve, whose outcome is read
late; the second starts within the (loose) tolerance and takes no iteration.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_stats_are_the_last_solves():
    from mac_b200.gpu import Context
    from mac_b200.state import pool_spheres_world
    from mac_b200.unet import UNet
    from mac_b200.world import setup_passes
    s = setup_passes(pool_spheres_world(24, nspheres=4, r_range=(1.2, 3.6)))
    s.f64["p"][:] = 3e3 * np.random.default_rng(1).standard_normal(s.f64["p"].shape)
    with UNet(0) as net:
        net.set_params(np.zeros(net.nparams, np.float32), 1.0)
        with Context(s.params, max_bricks=512, max_particles=1024, solver="learned", rtol=1.5, max_iters=200,
                     warm_start=1) as ctx:
            ctx.set_preconditioner(net)
            ctx.set_learned_smoothing(0.0)
            ctx.upload(s)
            ctx.rk2tvd()
            st = ctx.stats()
    assert st["solves"] == 2 and st["fallbacks"] == 1  # the first fell back, the second did not
    assert st["total_iterations"] > 8
    assert st["iterations"] == 0 and st["learned_iterations"] == 0
    assert 1.0 < st["relres"] <= 1.5  # what the second started from
