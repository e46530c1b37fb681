"""The standalone-kernel form of the multilevel solve (mlkern.cuh, smoothed aggregation) where its
dispatch can go wrong: row counts around the 32-row slices, the size from which rows are taken in
slices on the finest, the restriction's and the first coarse level, wide rows, Chebyshev degrees 1 to
3, binary16 values, fewer aggregation passes (unsmoothed transfers), and a Dirichlet operator.

Against the plain Jacobi-PCG path on the same operator.  Both stop at ||r|| <= 1e-12 ||b||; with the
operators' condition number below 1e5 the solutions then differ by less than 1e-7 relative."""
import ctypes as C

import numpy as np
import pytest

from dopamine_b200 import abi, cases
from dopamine_b200.solver import Solver, lib

pytestmark = pytest.mark.gpu


def _box_faces(nx, ny, nz, seed):
    from test_zz_no_alloc import neumann_system
    return neumann_system(nx, ny, nz, seed)


@pytest.mark.parametrize("dims", [(13, 11, 9), (31, 33, 33), (41, 43, 43), (42, 41, 44), (96, 90, 73)])
def test_drop_in_amg_matches_jacobi(dims):
    from test_zz_no_alloc import reference_solve
    L = lib()
    n, fo, fn, coeff, diag = _box_faces(*dims, seed=3)
    rhs = np.random.default_rng(4).standard_normal(n) + 0.2
    x = {}
    try:
        for name in (b"jacobi", b"boomeramg"):
            L.fvm_petsc_set_pressure_solver(name)
            x[name], its, _ = reference_solve(L, n, fo, fn, coeff, diag, rhs, np.zeros(n), 1e-12, 1e-50, 4000)
            x[name] -= x[name].mean()
    finally:
        L.fvm_petsc_set_pressure_solver(b"jacobi")
        L.fvm_petsc_backend_finalize()
    assert 0 < its <= 40, its
    assert np.linalg.norm(x[b"boomeramg"] - x[b"jacobi"]) <= 1e-7 * np.linalg.norm(x[b"jacobi"])


def _step(case, **kw):
    p = abi.default_params(**dict(case.params, p_tol=1e-12, **kw))
    s = Solver(case, params=p)
    s.initialise()
    s.advance()
    s.advance()
    U, st = s.sync_host()["U"], s.stats()
    s.close()
    return U, st


@pytest.mark.parametrize("kw", [dict(p_ml_degree=1), dict(p_ml_degree=3), dict(p_ml_passes=2),
                                dict(p_ml_value_bits=16), dict(n_nonortho_corr=0)])
def test_step_options_match_plain_pcg(kw):
    case = cases.channel_config(nx=60, ny=37, nz=33, n_steps=2)  # 73 260 cells
    ref, _ = _step(case)
    U, st = _step(case, p_solver=abi.PSOLVER_MULTILEVEL_FCG, **kw)
    assert st["p_solver_used"] == abi.PSOLVER_MULTILEVEL_FCG and st["p_fallbacks"] == 0, st
    assert np.linalg.norm(U - ref) <= 1e-8 * np.linalg.norm(ref)


@pytest.mark.parametrize("name", ["outlet", "mixed"])
def test_step_operators_match_plain_pcg(name):
    if name == "outlet":  # Dirichlet pressure rows at the outlets
        ref = cases.regression_case("pdrop")
        case = cases.Case("pdrop", cases.skewed_unit_box(41, 0.04), ref.patches, dict(ref.params, dt=5e-4), ref.ic,
                          ref.ic_uref)
    else:
        case = cases.hybrid_config(n=31, kind="mixed", n_steps=2)
    U0, _ = _step(case)
    U, st = _step(case, p_solver=abi.PSOLVER_MULTILEVEL_FCG)
    assert st["p_fallbacks"] == 0 and st["p_iters"] <= 30 * st["p_solves"], st
    assert np.linalg.norm(U - U0) <= 1e-8 * np.linalg.norm(U0)
