"""The resident CSC solve at the edges of its layouts: the polls of one warp (32 x 4
blocks of 512 rows), one block an SM, two blocks an SM with half the registers, and
one row more than the device holds. The launch count tells the forms apart.

Solved to a relative residual of 1e-12, recomputed here in FP64: 1e-11.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 512


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("blocks,extra", [("128", 0), ("128", 1), ("sms", 0), ("sms", 1), ("mid", -7), ("2 sms", 0),
                                          ("2 sms", 1)])
def test_rows_at_block_edges(blocks, extra):
    from test_gpu_csc_resident import _ctx, _laplacian
    sms = _sms()
    n = {"128": 128, "sms": sms, "mid": sms + sms // 2, "2 sms": 2 * sms}[blocks] * ROWS + extra
    # lines of 77 cells, then a chain for the rest: rows of every length up to seven
    A = _laplacian((n // (77 * 11), 11, 77), 0.05)
    if A.shape[0] < n:
        import scipy.sparse as sp
        A = sp.block_diag([A, _laplacian((1, 1, n - A.shape[0]), 0.05)]).tocsc()
        A.sort_indices()
    assert A.shape[0] == n
    b = np.random.default_rng(n).uniform(-1, 1, n)
    with _ctx() as ctx:
        before = ctx.launches()
        got = ctx.csc_solve(A.indptr, A.indices, A.data, b)
        launched, its = ctx.launches() - before, ctx.stats()["iterations"]
    assert np.linalg.norm(A @ got - b) <= 1e-11 * np.linalg.norm(b)
    if n <= 2 * sms * ROWS:
        assert launched == 2  # the check of the matrix and the solve
    else:
        assert launched > 3 * its


def test_device_form_at_its_largest():
    import torch
    from mac_b200.gpu import load
    from test_gpu_csc_resident import _laplacian
    lib = load()
    A = _laplacian((32, 32, 64), 0.05)
    b = np.random.default_rng(8).uniform(-1, 1, A.shape[0])
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
         (A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, b)]
    x = torch.empty(len(b), dtype=torch.float64, device="cuda")
    assert len(b) == 65536
    assert lib.mac_csc_solve_noalloc(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), len(b),
                                     *[t.data_ptr() for t in d], x.data_ptr(), 1e-12, 5000, None, None) == 0
    got = x.cpu().numpy()
    assert np.linalg.norm(A @ got - b) <= 1e-11 * np.linalg.norm(b)
