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


def _fields(case, steps=2, **kw):
    s = Solver(case, params=abi.default_params(**dict(case.params, **kw)))
    s.initialise()
    for _ in range(steps):
        s.advance()
    h, st = s.sync_host(), s.stats()
    out = {"U": h["U"], "p": h["p"] - h["p"].mean()}
    if s.params.sgs_model != abi.SGS_NONE:
        out["nu_sgs"] = h["nu_sgs"]
    if s.params.boussinesq:
        out["T"] = h["T"]
    if s.params.n_scalars:
        out["C"] = s.scalars()[1]
    s.close()
    return out, st


@pytest.mark.parametrize("flow", ["channel", "rb"])
def test_every_field_matches_plain_pcg(flow):
    """U, p, nu_sgs, T and the scalars after two steps.  Both forms stop at ||r|| <= 1e-12 ||b||: with a
    condition number below 1e5 the pressures differ by less than 1e-7 and what they correct by less."""
    case = (cases.channel_config(nx=60, ny=37, nz=33, n_steps=2) if flow == "channel" else
            cases.rb_config(nx=48, ny=48, nz=33))
    ref, _ = _fields(case, p_tol=1e-12)
    out, st = _fields(case, p_tol=1e-12, p_solver=abi.PSOLVER_MULTILEVEL_FCG)
    assert st["p_fallbacks"] == 0
    err = {k: np.linalg.norm(out[k] - ref[k]) / np.linalg.norm(ref[k]) for k in ref}
    print(flow, {k: f"{v:.1e}" for k, v in err.items()})
    assert err.pop("p") <= 1e-7, err
    assert max(err.values()) <= 1e-8, err


def test_every_field_of_the_urban_flow():
    """At single near-ground cells the surface flux amplifies the last bits of the solve, whatever solves: plain
    PCG at p_tol 1e-10 against itself at 1e-13 moves U by 3.1e-6 (8.9e-6 on 60x60x19), p by 1.1e-4 (6.9e-4),
    nu_sgs by 2.5e-5 and the scalar by 1.1e-5 relative.  About four times that is allowed."""
    case = cases.urban_config(100, 100, 32)
    ref, _ = _fields(case, p_tol=1e-13)
    out, st = _fields(case, p_tol=1e-13, p_solver=abi.PSOLVER_MULTILEVEL_FCG)
    assert st["p_fallbacks"] == 0
    err = {k: np.linalg.norm(out[k] - ref[k]) / np.linalg.norm(ref[k]) for k in ref}
    print("urban", {k: f"{v:.1e}" for k, v in err.items()})
    for k, tol in {"U": 3.6e-5, "p": 2.8e-3, "nu_sgs": 1e-4, "C": 4.4e-5, "T": 1e-5}.items():
        assert err[k] <= tol, (k, err)


def test_solve_repeats_bit_for_bit():
    case = cases.urban_config(100, 100, 32)
    a, _ = _fields(case, steps=1, p_solver=abi.PSOLVER_MULTILEVEL_FCG)
    b, _ = _fields(case, steps=1, p_solver=abi.PSOLVER_MULTILEVEL_FCG)
    assert all(np.array_equal(a[k], b[k]) for k in a)
