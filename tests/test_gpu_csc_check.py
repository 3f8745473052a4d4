"""The check that decides a CSC matrix's solver, on columns outside the
reference's seven entries: what it costs on a long column, and what it says of
a column that repeats a row.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_long_column_costs_its_length():
    """An arrowhead matrix through the allocation-free solve: one column and one
    row of n entries, each compared with its mirror (n^2 / 2 reads spread over n
    threads). A search of the column for repeats would be n^2 / 2 reads by one
    thread, seconds at this n; the solve takes a few iterations, each with one
    thread's pass over the column, well under a millisecond."""
    import torch
    from mac_b200.gpu import load
    lib = load()
    n = 40000
    off = np.concatenate([[0], n + 2 * np.arange(n)]).astype(np.int32)
    ind = np.empty(off[-1], np.int32)
    val = np.empty(off[-1])
    ind[:n], val[:n] = np.arange(n), 1e-3
    val[0] = -4.0
    ind[n::2], ind[n + 1::2] = 0, np.arange(1, n)
    val[n::2], val[n + 1::2] = 1e-3, -4.0
    b = np.random.default_rng(1).uniform(-1, 1, n)
    dev = [torch.from_numpy(a).cuda() for a in (off, ind, val, b)]
    x = torch.empty(n, dtype=torch.float64, device="cuda")
    t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    for _ in range(2):  # the first call loads the kernels
        t[0].record()
        rc = lib.mac_csc_solve_noalloc(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), n,
                                       *[a.data_ptr() for a in dev], x.data_ptr(), 1e-12, 200, None, None)
        t[1].record()
        t[1].synchronize()
        assert rc == 0
    got = x.cpu().numpy()
    res = -4.0 * got
    res[0] += 1e-3 * got[1:].sum()
    res[1:] += 1e-3 * got[0]
    assert np.linalg.norm(res - b) <= 1e-11 * np.linalg.norm(b)
    assert t[0].elapsed_time(t[1]) < 500.0


@pytest.mark.parametrize("split", ["one coupling", "all couplings"])
def test_unequal_parts_of_a_coupling_stay_with_cg(split):
    """Couplings stored as v / 4 and 3 v / 4 in one column and the other way round
    in its mirror: the same entries, so the matrix is symmetric and CG solves it,
    in the iterations of the matrix with whole entries (the parts add up exactly,
    up to the order of a row's sum)."""
    from test_gpu_csc_resident import _ctx, _laplacian
    A = _laplacian((9, 10, 11), 0.05)
    n = A.shape[0]
    off, ind, val = [0], [], []
    for j in range(n):
        for k in range(A.indptr[j], A.indptr[j + 1]):
            i, v = int(A.indices[k]), A.data[k]
            if i != j and (split == "all couplings" or {i, j} == {0, 1}):
                parts = [0.25 * v, 0.75 * v]
                ind += [i, i]
                val += parts if i < j else parts[::-1]
            else:
                ind.append(i)
                val.append(v)
        off.append(len(ind))
    b = np.random.default_rng(2).uniform(-1, 1, n)
    with _ctx() as ctx:
        want = ctx.csc_solve(A.indptr, A.indices, A.data, b)
        its = ctx.stats()["iterations"]
        got = ctx.csc_solve(np.array(off), np.array(ind), np.array(val), b)
        assert abs(ctx.stats()["iterations"] - its) <= 1
    assert np.linalg.norm(got - want) <= 1e-8 * np.linalg.norm(want)
