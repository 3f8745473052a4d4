"""Contexts solving at the same time from several threads, with resident kernels of
both forms (one cluster, the whole grid) and the drop-in solver between them: each
gets the bits it gets alone.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_contexts_in_threads_do_not_disturb_each_other():
    from mac_b200.gpu import Context
    from test_gpu_csc_resident import _ctx, _laplacian
    from test_gpu_resident_solve import _world
    worlds = [_world(n, 0.5) for n in (17, 49, 63)]
    A = _laplacian((15, 16, 16), 0.05)
    b = np.random.default_rng(9).uniform(-1, 1, A.shape[0])

    def projections(k, solver, reps, out):
        s = worlds[k]
        with Context(s.params, max_bricks=int(s.nbricks * 1.2) + 64, max_particles=1024, solver=solver, rtol=1e-10,
                     max_iters=500) as ctx:
            for _ in range(reps):
                ctx.upload(s)
                ctx.project(0)
                out.append(ctx.download().f64["p"])

    def systems(reps, out):
        with _ctx() as ctx:
            for _ in range(reps):
                out.append(ctx.csc_solve(A.indptr, A.indices, A.data, b))
    jobs = [(projections, 0, "mgpcg64"), (projections, 1, "mixed"), (projections, 2, "mgpcg64"), (projections, 2, "mixed"),
            (systems,)]
    alone = []
    for f, *a in jobs:
        out = []
        f(*a, 1, out)
        alone.append(out[0])
    outs = [[] for _ in jobs]
    threads = [threading.Thread(target=f, args=(*a, 8, o)) for (f, *a), o in zip(jobs, outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
        assert not t.is_alive()
    for want, got in zip(alone, outs):
        assert len(got) == 8 and all(np.array_equal(g, want) for g in got)
