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
