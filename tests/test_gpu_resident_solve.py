"""The MG-PCG solve run as one resident kernel (small systems) against the
launch-by-launch loop on the same worlds. set_multigrid(2, prefetch=True) keeps
the launches (its first kernel prefetches bricks), so it serves as the general
path. Sizes sit at the edges of the resident form's layouts: one brick, part of
a cluster, a full cluster and one brick list beyond it, level 2 inside and
outside block 0's levels, several bricks a group, and the last and first box
sizes on either side of the line between the two forms; odd sizes throughout.

Both solve to a relative residual of 1e-12 with the same preconditioner; each
is within 1e-10 of the exact pressure there, so they agree to 1e-9 relative.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _world(n, frac):
    from mac_b200.state import pool_spheres_world
    from mac_b200.world import setup_passes
    return setup_passes(pool_spheres_world(n, nspheres=4, r_range=(0.05 * n, 0.15 * n), pool_frac=frac))


def _solve(s, solver, prefetch, rtol=1e-12, max_iters=500, **kw):
    from mac_b200.gpu import Context
    with Context(s.params, max_bricks=int(s.nbricks * 1.2) + 64, max_particles=1024, solver=solver, rtol=rtol,
                 max_iters=max_iters, **kw) as ctx:
        ctx.set_multigrid(2, prefetch)
        ctx.upload(s)
        before = ctx.launches()
        ctx.project(0)
        launched = ctx.launches() - before
        st, got = ctx.stats(), ctx.download()
    return got, st, launched


@pytest.mark.parametrize("solver", ["mgpcg64", "mixed"])
@pytest.mark.parametrize("n,frac", [(5, 0.7), (9, 0.4), (17, 0.6), (33, 0.4), (43, 0.6), (49, 0.4), (63, 0.45),
                                    (77, 0.55), (80, 0.6), (97, 0.5)])
def test_resident_matches_launches(n, frac, solver):
    s = _world(n, frac)
    a, sa, la = _solve(s, solver, False)
    b, sb, lb = _solve(s, solver, True)
    assert la < lb or n > 80, (la, lb)  # below the line the loop is one launch
    assert abs(sa["iterations"] - sb["iterations"]) <= 1
    ex = a.exists.astype(bool)
    for f in ("p", "u0x", "u0y", "u0z"):
        x, y = a.f64[f][ex], b.f64[f][ex]
        assert np.linalg.norm(x - y) <= 1e-9 * np.linalg.norm(y), f


@pytest.mark.parametrize("solver", ["mgpcg64", "mixed"])
def test_closed_box_has_no_exact_coarse_solve(solver):
    """A full box without a free surface: the operator is singular, the coarsest
    level keeps its sweeps, the speeds still become divergence-free."""
    s = _world(21, 1.1)
    a, sa, _ = _solve(s, solver, False, rtol=1e-10)
    b, sb, _ = _solve(s, solver, True, rtol=1e-10)
    ex = a.exists.astype(bool)
    for f in ("u0x", "u0y", "u0z"):
        x, y = a.f64[f][ex], b.f64[f][ex]
        assert np.linalg.norm(x - y) <= 1e-7 * np.linalg.norm(y), f


def test_solves_follow_one_another():
    """Several contexts and sizes in turn on one device, and a repeat on one
    context, give what each gives alone, bit for bit."""
    from mac_b200.gpu import Context
    worlds = [_world(9, 0.4), _world(49, 0.4), _world(33, 0.4)]
    alone = [_solve(s, "mixed", False)[0].f64["p"] for s in worlds]
    ctxs = [Context(s.params, max_bricks=int(s.nbricks * 1.2) + 64, max_particles=1024, solver="mixed", rtol=1e-12)
            for s in worlds]
    try:
        for _ in range(3):
            for s, c, want in zip(worlds, ctxs, alone):
                c.upload(s)
                c.project(0)
                assert np.array_equal(c.download().f64["p"], want)
    finally:
        for c in ctxs:
            c.close()


@pytest.mark.parametrize("warm", [False, True])
def test_cap_and_warm_start(warm):
    s = _world(33, 0.4)
    from mac_b200.gpu import MacError
    with pytest.raises(MacError) as e:
        _solve(s, "mixed", False, rtol=1e-14, max_iters=3, warm_start=warm)
    assert e.value.code == -4
    a, sa, _ = _solve(s, "mixed", False, warm_start=warm)
    b, sb, _ = _solve(s, "mixed", True, warm_start=warm)
    assert np.linalg.norm(a.f64["p"] - b.f64["p"]) <= 1e-9 * np.linalg.norm(b.f64["p"])
