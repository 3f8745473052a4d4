"""Lines between two forms of one pass: past a line a smaller world must not take
longer than a larger one that has the other form. Device times of the profile,
medians of 15; the margins are a tenth of the differences of 15-60% that a line in
the wrong place makes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _median(n, what):
    from mac_b200.gpu import Context
    from test_gpu_resident_solve import _world
    s = _world(n, 0.5)
    with Context(s.params, max_bricks=int(s.nbricks * 1.2) + 64, max_particles=1024, solver="mgpcg64", rtol=1e-10,
                 max_iters=500) as ctx:
        ctx.set_profiling(True)
        t = []
        for _ in range(15):
            ctx.upload(s)
            ctx.profile()
            if what == "vcycle":
                ctx.project(0)
                t.append(ctx.profile()["vcycle"][0] / ctx.stats()["iterations"])
            else:
                ctx.extrapolate()
                t.append(ctx.profile()["extrapolate"][0])
        return float(np.median(t)), s.nbricks


def test_extrapolation_split():
    (a, na), (b, nb) = _median(62, "extrapolate"), _median(70, "extrapolate")
    assert 700 < na <= 1024 < nb
    assert a <= 1.05 * b, (a, b)


@pytest.mark.parametrize("n", [48, 56])  # 512 and 729 live bricks
def test_extrapolation_follows_its_rule_on_both_sides(n):
    from test_gpu_extrapolate_split import test_both_forms_follow_the_rule as follows
    follows(n, True)
