"""What DPM_PSOLVER_AUTO chooses: on either side of its 131 072-cell limit, where the multilevel set-up
refuses, and for fluid regions that do not touch one another, which the multilevel form solves at its
usual iteration count."""
import numpy as np
import pytest

from dopamine_b200 import abi, cases
from dopamine_b200.solver import DopamineError, Solver

pytestmark = pytest.mark.gpu


def _step(case, **kw):
    s = Solver(case, params=abi.default_params(**dict(case.params, **kw)))
    s.initialise()
    s.advance()
    U, st = s.sync_host()["U"], s.stats()
    s.close()
    return U, st


@pytest.mark.parametrize("nx,form", [(64, abi.PSOLVER_TWOLEVEL_FCG), (65, abi.PSOLVER_MULTILEVEL_FCG)])
def test_choice_on_either_side_of_the_limit(nx, form):
    case = cases.channel_config(nx=nx, ny=64, nz=32, n_steps=1)
    _, st = _step(case, p_solver=abi.PSOLVER_AUTO)
    assert st["p_solver_used"] == form and st["p_fallbacks"] == 0


def test_two_level_where_the_multilevel_set_up_refuses():
    case = cases.channel_config(nx=65, ny=64, nz=32, n_steps=1)
    with pytest.raises(DopamineError):
        _step(case, p_solver=abi.PSOLVER_MULTILEVEL_FCG, p_ml_passes=4)
    _, st = _step(case, p_solver=abi.PSOLVER_AUTO, p_ml_passes=4)
    assert st["p_solver_used"] == abi.PSOLVER_TWOLEVEL_FCG and st["p_fallbacks"] == 0


@pytest.mark.parametrize("nx", [64, 65])
def test_bounds_of_the_smoother_are_checked_on_either_side(nx):
    with pytest.raises(DopamineError) as e:
        _step(cases.channel_config(nx=nx, ny=64, nz=32, n_steps=1), p_solver=abi.PSOLVER_AUTO, p_smooth_lmin=2.0,
              p_smooth_lmax=1.0)
    assert e.value.status == abi.ERR_ARG


def _beside(a, b, shift, patch=None):
    """Mesh a and, moved by shift in y, mesh b (all its faces on one patch when given)."""
    n = a.xyz.shape[0]
    return cases.RawMesh(
        xyz=np.concatenate([a.xyz, b.xyz + [0.0, shift, 0.0]]),
        cell_type=np.concatenate([a.cell_type, b.cell_type]),
        cell_off=np.concatenate([a.cell_off, b.cell_off[1:] + a.cell_off[-1]]),
        cell_nodes=np.concatenate([a.cell_nodes, b.cell_nodes + np.int32(n)]),
        bface_off=np.concatenate([a.bface_off, b.bface_off[1:] + a.bface_off[-1]]),
        bface_nodes=np.concatenate([a.bface_nodes, b.bface_nodes + np.int32(n)]),
        bface_patch=np.concatenate([a.bface_patch, b.bface_patch if patch is None else
                                    np.full_like(b.bface_patch, patch)]),
        patch_names=a.patch_names)


@pytest.mark.parametrize("kind", ["halves", "room", "pocket"])
def test_regions_that_do_not_touch(kind):
    half = kind == "halves"
    case = cases.channel_config(nx=60, ny=37 if half else 74, nz=33, n_steps=1)
    _, alone = _step(case, p_tol=1e-12, p_solver=abi.PSOLVER_MULTILEVEL_FCG)
    n = {"halves": 0, "room": 20, "pocket": 4}[kind]
    other = case.mesh if half else cases.uniform_box(n, n, n, 0.05 * n, 0.05 * n, 0.05 * n)
    case.mesh = _beside(case.mesh, other, 4.0, None if half else 2)  # closed boxes: wall faces only
    assert case.mesh.n_cells > 131072
    U0, _ = _step(case, p_tol=1e-12)
    U, st = _step(case, p_tol=1e-12, p_solver=abi.PSOLVER_AUTO)
    assert st["p_solver_used"] == abi.PSOLVER_MULTILEVEL_FCG and st["p_fallbacks"] == 0, st
    # the second region widens the preconditioned spectrum a little: 92 iterations in three solves by itself,
    # 96 with either box, where one null vector left alone costs hundreds
    assert st["p_iters"] <= alone["p_iters"] + 3 * st["p_solves"], (st, alone)
    # both stop at ||r|| <= 1e-12 ||b||, condition number below 1e5
    assert np.linalg.norm(U - U0) <= 1e-7 * np.linalg.norm(U0)
