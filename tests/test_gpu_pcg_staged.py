"""The staged grid form of Jacobi-PCG (k_pcg_staged) and the limits to the register and grid-stride forms:
row counts just above what the cluster form takes, a short last block, one and two rows per thread, rows
narrower and wider than seven (the widest, 16, at 131 072 rows: 177 of 223 KB are staged), 1024 and 4096
rows per SM and one row more.

Against the solution the right-hand side was formed from.  The solve stops at ||r|| <= 1e-12 ||b||; the
operators' condition number is below 1e5, so the solution is within 1e-7 relative."""
import ctypes as C

import numpy as np
import pytest

from dopamine_b200.solver import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,width", [(40961, 7), (41003, 9), (75777, 7), (75777, 16), (131072, 16), (131072, 7), (131072, 3)])
def test_noalloc_staged_solve(n, width):
    import torch
    from test_gpu_pcg_cluster import _ell, _operator
    A = _operator(n, width, n)
    col, val = _ell(A, width)
    rng = np.random.default_rng(1)
    x_ref, x0 = rng.standard_normal(n), rng.standard_normal(n)
    b = A @ x_ref
    dev = [torch.from_numpy(np.ascontiguousarray(q)).cuda() for q in (col, val, 1.0 / A.diagonal(), b, x0)]
    torch.cuda.synchronize()
    its, res = C.c_int(), C.c_double()
    p = [C.c_void_p(t.data_ptr()) for t in dev]
    rc = lib().dpm_pcg_solve_noalloc(n, width, *p, 1e-12, 0.0, 5000, 0,
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(its), C.byref(res))
    assert rc == 0, (rc, its.value)
    x = dev[4].cpu().numpy()
    assert np.linalg.norm(x - x_ref) <= 1e-7 * np.linalg.norm(x_ref)
    assert abs(res.value - np.linalg.norm(b - A @ x)) <= 1e-11 * np.linalg.norm(b)


@pytest.mark.parametrize("per_sm", [1024, 1025, 2700, 4096, 4097])
def test_drop_in_jacobi_by_rows_per_sm(per_sm):
    """The drop-in Jacobi solve of a path graph plus chords with per_sm rows on every SM."""
    import torch
    from test_zz_no_alloc import reference_solve
    L = lib()
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(per_sm)
    fo = np.concatenate([np.arange(n - 1), np.arange(n - 97), np.arange(n - 6145)]).astype(np.int64)
    fn = np.concatenate([np.arange(1, n), np.arange(97, n), np.arange(6145, n)]).astype(np.int64)
    coeff = rng.uniform(0.5, 2.0, fo.size)
    diag = np.bincount(fo, coeff, n) + np.bincount(fn, coeff, n)
    x_ref = rng.standard_normal(n)
    x_ref -= x_ref.mean()

    def apply(x):
        y = diag * x
        y -= np.bincount(fo, coeff * x[fn], n) + np.bincount(fn, coeff * x[fo], n)
        return y

    b = apply(x_ref)
    try:
        L.fvm_petsc_set_pressure_solver(b"jacobi")
        x, its, res = reference_solve(L, n, fo, fn, coeff, diag, b, np.zeros(n), 1e-10, 1e-50, 4000)
    finally:
        L.fvm_petsc_backend_finalize()
    assert np.linalg.norm(apply(x) - b) <= 1e-9 * np.linalg.norm(b), (its, res)
