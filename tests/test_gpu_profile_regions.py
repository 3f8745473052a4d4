"""Timed regions of a profiled projection: a V-cycle region for every V-cycle that
was launched and none for a form that did not take the system.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 97])
def test_vcycle_regions(n):
    """n = 33 is one launch for the whole solve. n = 97 takes separate launches: a
    region per iteration, and one for the head of the V-cycle that finishes the
    last iteration and meets the tolerance."""
    from mac_b200.gpu import Context
    from test_gpu_resident_solve import _world
    s = _world(n, 0.5)
    with Context(s.params, max_bricks=int(s.nbricks * 1.2) + 64, max_particles=1024, solver="mixed", rtol=1e-10,
                 max_iters=500) as ctx:
        ctx.set_profiling(True)
        ctx.upload(s)
        ctx.profile()
        ctx.project(0)
        p, its = ctx.profile(), ctx.stats()["iterations"]
    ms, count = p["vcycle"]
    assert ms > 0
    if n == 33:
        assert count == 1 and p["spmv"][1] == 0
    else:
        assert p["spmv"][1] == its and count == its + 1
