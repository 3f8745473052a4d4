"""Waits of the one-launch solves that run out: the call returns the timeout
status and the context goes on to solve as a fresh one does. The limit is set to
so few polls that a wait gives up at once; every block then leaves on its own.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = -7


def test_csc_wait_that_runs_out_is_a_timeout():
    """The wait for a neighbour's value: its NaN ends the solve as a breakdown
    does, but the status tells the two apart."""
    from mac_b200.gpu import MacError
    from test_gpu_csc_resident import _ctx, _laplacian
    A = _laplacian((15, 16, 16), 0.05)
    b = np.random.default_rng(3).uniform(-1, 1, A.shape[0])
    with _ctx() as ctx:
        want = ctx.csc_solve(A.indptr, A.indices, A.data, b)
        ctx.set_wait_limit(0)
        with pytest.raises(MacError) as e:
            ctx.csc_solve(A.indptr, A.indices, A.data, b)
        assert e.value.code == TIMEOUT
        ctx.set_wait_limit()
        assert np.array_equal(ctx.csc_solve(A.indptr, A.indices, A.data, b), want)


def test_pressure_wait_that_runs_out_leaves_nothing_behind():
    """The grid barrier of the resident solve: blocks give up in different phases,
    so its count of arrivals is anywhere. The status stays until an upload, and
    the solve after that has the bits of a fresh context's."""
    from mac_b200.gpu import Context, MacError
    from test_gpu_resident_solve import _world
    s = _world(63, 0.45)
    make = lambda: Context(s.params, max_bricks=int(s.nbricks * 1.2) + 64, max_particles=1024, solver="mixed",
                           rtol=1e-10, max_iters=500)

    def project(ctx):
        try:
            ctx.project(0)
            return 0
        except MacError as e:
            return e.code
    with make() as ctx:
        ctx.upload(s)
        assert project(ctx) == 0
        want = ctx.download()
        its = ctx.stats()["iterations"]
    with make() as ctx:
        for polls in (0, 1, 4, 16, 0):
            ctx.upload(s)
            ctx.set_wait_limit(polls)
            code = project(ctx)
            assert code == TIMEOUT if polls == 0 else code in (0, TIMEOUT)
            ctx.set_wait_limit()
            assert code == 0 or project(ctx) == TIMEOUT
            ctx.upload(s)
            assert project(ctx) == 0 and ctx.stats()["iterations"] == its
            got = ctx.download()
            for f in ("p", "u0x", "u0y", "u0z"):
                assert np.array_equal(got.f64[f], want.f64[f]), (polls, f)
