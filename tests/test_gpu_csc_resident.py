"""The resident CSC solve and the rule that picks it, against a sparse direct
solve: sizes at the edges of its blocks (512 rows each), rows of exactly seven
and of more entries, a system of more rows than fit on the device at once,
unsorted columns, a column that repeats a row, a zero right-hand side and an
iteration cap. The solves run to a relative residual of 1e-12 on matrices of
condition number below 1e4, so solutions agree to 1e-8 relative.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _laplacian(shape, extra=0.0, far=()):
    """-(7-point operator + extra), Dirichlet outside the box; far: offsets along
    the flat index that add a symmetric coupling (rows of more entries)."""
    import scipy.sparse as sp
    one = [sp.diags([np.ones(n - 1), np.ones(n - 1)], [-1, 1], shape=(n, n)) for n in shape]
    eye = [sp.identity(n) for n in shape]
    k = sp.kron
    A = k(k(eye[0], eye[1]), one[2]) + k(k(eye[0], one[1]), eye[2]) + k(k(one[0], eye[1]), eye[2])
    N = A.shape[0]
    for d in far:
        A = A + sp.diags([np.full(N - d, 0.25), np.full(N - d, 0.25)], [-d, d], shape=(N, N))
    A = (A - sp.diags([np.full(N, 6.0 + 0.5 * len(far) + extra)], [0])).tocsc()
    A.sort_indices()
    return A


def _ctx(**kw):
    from mac_b200.gpu import Context
    from mac_b200.state import Params
    return Context(Params(h=(0.05, 0.05, 0.05)), max_bricks=64, max_particles=1024, rtol=1e-12,
                   max_iters=kw.get("max_iters", 5000))


def _direct(A, b):
    import scipy.sparse.linalg as spl
    return spl.spsolve(A, b)


def _check(A, b):
    with _ctx() as ctx:
        got = ctx.csc_solve(A.indptr, A.indices, A.data, b)
        it = ctx.stats()["iterations"]
    if A.shape[0] <= 4000:
        want = _direct(A, b)
        assert np.linalg.norm(got - want) <= 1e-8 * np.linalg.norm(want)
    assert np.linalg.norm(A @ got - b) <= 1e-11 * np.linalg.norm(b)
    return got, it


@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 7, 73), (8, 8, 8), (1, 19, 27), (3, 11, 31), (15, 16, 16)])
def test_sizes_at_block_edges(shape):
    A = _laplacian(shape, 0.05)
    _check(A, np.random.default_rng(1).uniform(-1, 1, A.shape[0]))


def test_longer_rows_take_the_launches():
    A = _laplacian((10, 10, 10), 0.05, far=(37,))
    assert np.diff(A.indptr).max() > 7
    _check(A, np.random.default_rng(2).uniform(-1, 1, A.shape[0]))


def test_more_rows_than_fit():
    A = _laplacian((60, 60, 60), 1.0)
    _check(A, np.random.default_rng(3).uniform(-1, 1, A.shape[0]))


def test_unsorted_columns_and_repeated_entries():
    A = _laplacian((6, 7, 8), 0.05)
    b = np.random.default_rng(4).uniform(-1, 1, A.shape[0])
    want, _ = _check(A, b)
    rng = np.random.default_rng(5)
    off, ind, val = [0], [], []
    for j in range(A.shape[0]):
        lo, hi = A.indptr[j], A.indptr[j + 1]
        for k in rng.permutation(np.arange(lo, hi)):
            i, v = A.indices[k], A.data[k]
            if {int(i), j} == {0, 1}:  # one coupling as two equal halves, both ways
                ind += [i, i]
                val += [v / 2, v / 2]
            else:
                ind.append(i)
                val.append(v)
        off.append(len(ind))
    with _ctx() as ctx:
        got = ctx.csc_solve(np.array(off), np.array(ind), np.array(val), b)
    assert np.linalg.norm(got - want) <= 1e-8 * np.linalg.norm(want)


def test_zero_right_hand_side_and_cap():
    from mac_b200.gpu import MacError
    A = _laplacian((9, 9, 9), 0.0)
    with _ctx() as ctx:
        assert not ctx.csc_solve(A.indptr, A.indices, A.data, np.zeros(A.shape[0])).any()
        assert ctx.stats()["iterations"] == 0
    with _ctx(max_iters=3) as ctx:
        with pytest.raises(MacError) as e:
            ctx.csc_solve(A.indptr, A.indices, A.data, np.random.default_rng(6).uniform(-1, 1, A.shape[0]))
        assert e.value.code == -4 and ctx.stats()["iterations"] == 3


def test_device_form_agrees_and_refuses():
    import torch
    from mac_b200.gpu import load
    lib = load()

    def solve(A, b):
        d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
             (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, b)]
        x = torch.full((len(b),), 7.0, dtype=torch.float64, device="cuda")
        its = ctypes.c_int(-1)
        rc = lib.mac_csc_solve_noalloc(torch.cuda.current_stream().cuda_stream, len(b), *[t.data_ptr() for t in d],
                                       x.data_ptr(), 1e-12, 5000, ctypes.byref(its), None)
        return rc, x.cpu().numpy(), its.value
    b = np.random.default_rng(7).uniform(-1, 1, 1000)
    for far in ((), (37,)):
        A = _laplacian((10, 10, 10), 0.05, far=far)
        rc, x, its = solve(A, b)
        want, it = _check(A, b)
        assert rc == 0 and abs(its - it) <= 1
        assert np.linalg.norm(x - want) <= 1e-9 * np.linalg.norm(want)
    A = _laplacian((10, 10, 10), 0.05)
    A.data[A.indptr[500]] *= 1.5  # not symmetric any more
    rc, x, _ = solve(A, b)
    assert rc == -8 and (x == 7.0).all()
