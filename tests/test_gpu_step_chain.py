"""Parts of a step that take another form by the size of the world: the particle
move's slices of a brick (sixteen for few particles, one for many), and the
RK2-TVD whose first projection's outcome is read with the second's when each
solve is one launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ctx(state, **kw):
    from mac_b200.gpu import Context
    kw.setdefault("rtol", 1e-13)
    return Context(state.params, max_bricks=4096, max_particles=1 << 22, **kw)


@pytest.mark.parametrize("copies", [1, 4, 16, 46])  # 16, 12, 3 and 1 slices of 67,000 particles
def test_move_slices(golden, copies):
    """Particles move independently of one another: every copy of a particle
    ends where the recorded run put it, to the last bit."""
    t30 = golden("c1_ref_t30")
    t30.params.interp_symmetric = 1
    want = golden("c1_ref_t30_move").pos
    t30.pos = np.tile(t30.pos, (copies, 1))
    with _ctx(t30) as ctx:
        ctx.upload(t30)
        ctx.move()
        got = ctx.download().pos
    rows, counts = np.unique(got, axis=0, return_counts=True)
    ref, each = np.unique(want, axis=0, return_counts=True)
    assert np.array_equal(rows, ref) and np.array_equal(counts, each * copies)


@pytest.mark.parametrize("prefetch", [False, True])  # one launch a solve; launch by launch
def test_rk2tvd_books_both_solves(golden, prefetch):
    from mac_b200.gpu import MacError
    t30 = golden("c1_ref_t30")
    with _ctx(t30, max_iters=3) as ctx:
        ctx.set_multigrid(2, prefetch)
        ctx.upload(t30)
        with pytest.raises(MacError) as e:
            ctx.rk2tvd()
        assert e.value.code == -4
        st = ctx.stats()
    assert (st["solves"], st["iterations"], st["total_iterations"]) == (2, 3, 6)
    with _ctx(t30, max_iters=2000) as ctx:
        ctx.set_multigrid(2, prefetch)
        ctx.upload(t30)
        ctx.rk2tvd()
        st = ctx.stats()
    assert st["solves"] == 2 and st["relres"] <= 1e-13
    assert st["iterations"] < st["total_iterations"] < 4 * st["iterations"]
