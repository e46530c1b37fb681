"""Jacobi-PCG on one thread-block cluster (pcg_cluster.cuh) at the edges of its range: one row, one
block, sizes that leave the last block short, one to five rows per thread, the largest
system it takes and the first it does not, rows wider and narrower than seven, operators that stay in
shared memory and ones that do not fit, a non-zero guess, and the iteration cap.

Against a dense or sparse FP64 solve on the host.  The solve stops at ||r|| <= 1e-12 ||b||; the
operators' condition number is below 1e5, so the solution is within 1e-7 relative."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from dopamine_b200.solver import lib

pytestmark = pytest.mark.gpu


def _operator(n, width, seed):
    """Symmetric positive definite band operator: `width` entries per row at most, offsets spread so
    that rows reach into neighbouring blocks."""
    rng = np.random.default_rng(seed)
    half = (width - 1) // 2
    offs = sorted({1, 3, 17, 129, 1111, 2500, 7}, key=lambda o: (o != 1, o))[:half]
    rows, cols, vals = [], [], []
    for o in offs:
        if o >= n:
            continue
        c = rng.uniform(0.5, 2.0, n - o)
        i = np.arange(n - o)
        rows += [i, i + o]
        cols += [i + o, i]
        vals += [-c, -c]
    if rows:
        A = sp.coo_matrix((np.concatenate(vals), (np.concatenate(rows), np.concatenate(cols))), shape=(n, n)).tocsr()
    else:
        A = sp.csr_matrix((n, n))
    d = -np.asarray(A.sum(axis=1)).ravel() + rng.uniform(0.05, 0.2, n)
    A = (A + sp.diags(d)).tocsr()
    A.sort_indices()
    return A


def _ell(A, width):
    n = A.shape[0]
    col = np.tile(np.arange(n, dtype=np.int32), (width, 1))
    val = np.zeros((width, n))
    row = np.repeat(np.arange(n), np.diff(A.indptr))
    slot = np.arange(A.nnz) - A.indptr[row]
    col[slot, row] = A.indices
    val[slot, row] = A.data
    return col, val


@pytest.mark.parametrize("n,width", [(1, 1), (2, 3), (31, 5), (513, 7), (1025, 7), (8191, 7), (8209, 9), (16385, 7),
                                     (16400, 15), (35937, 7), (36001, 16), (40959, 7),
                                     (40960, 7), (40961, 7)])
def test_cluster_solve_matches_sparse_direct(n, width):
    import torch
    A = _operator(n, width, n)
    col, val = _ell(A, width)
    rng = np.random.default_rng(1)
    x_ref, x0 = rng.standard_normal(n), rng.standard_normal(n)
    b = A @ x_ref
    dev = [torch.from_numpy(np.ascontiguousarray(q)).cuda() for q in (col, val, 1.0 / A.diagonal(), b, x0)]
    torch.cuda.synchronize()
    its, res = C.c_int(), C.c_double()
    p = [C.c_void_p(t.data_ptr()) for t in dev]
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    rc = lib().dpm_pcg_solve_noalloc(n, width, *p[:4], p[4], 1e-12, 0.0, 5000, 0, st, C.byref(its), C.byref(res))
    assert rc == 0, (rc, its.value)
    x = dev[4].cpu().numpy()
    assert np.linalg.norm(x - x_ref) <= 1e-7 * np.linalg.norm(x_ref)
    assert abs(res.value - np.linalg.norm(b - A @ x)) <= 1e-11 * np.linalg.norm(b)
    if its.value > 3:  # the cap: KSP_DIVERGED_ITS
        dev[4].copy_(torch.from_numpy(x0))
        rc = lib().dpm_pcg_solve_noalloc(n, width, *p[:4], p[4], 1e-12, 0.0, 3, 0, st, C.byref(its), C.byref(res))
        assert rc == -997 and its.value == 3
