"""Performance cases of the framework: what its users have it do, through its public entry points.

Three kinds of work are measured, over the sizes that the run configurations, the regression cases
and the drop-in interface are used at:

* ``step``: a host program that keeps the fields and has one RK3 time step done on the GPU
  (``dpm_upload_state``, ``dpm_advance``, ``dpm_download_state``: the drop-in sequence to_device,
  advance, sync_host, with the host's buffers pinned as ``bench.py`` has them).  The host's fields
  evolve from pass to pass, as in a run.
* ``solve`` / ``noalloc``: one pressure solve of a host that keeps its own step
  (``fvm_petsc_solve_pressure`` on host or device arrays; ``dpm_pcg_solve_noalloc`` on the caller's
  device operator).
* ``operators``: single operators swapped into a host's step (``Solver.ls_gradient_vector``,
  ``Solver.viscous_rhs_vector``), host arrays in and out.

``exact`` gives 64-bit references for the solves (fast diagonalisation of the tensor-product
operator) and the operators (numpy on the periodic box).  A whole step has none: it would be a
second solver; its outputs are compared between implementations.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from dopamine_b200 import abi, cases
from dopamine_b200.solver import Solver, lib

# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------


def listed():
    return [
        # Taylor-Green vortex 32^3, periodic, CDS, plain FP64 Jacobi-PCG: the smallest configuration,
        # and the size of the regression runs, where latency and launches count
        {"name": "step_tgv32", "kind": "step", "flow": "tgv", "nx": 32, "ny": 32, "nz": 32, "form": "plain"},
        # turbulent channel 96x64x64 on the plain FP64 path: walls, Vreman, log-law wall model
        {"name": "step_channel_plain", "kind": "step", "flow": "channel", "nx": 96, "ny": 64, "nz": 64,
         "form": "plain"},
        # the same channel in the form a production run chooses: precision form, automatic flexible
        # CG, the learned term trained at the start of the run
        {"name": "step_channel_chosen", "kind": "step", "flow": "channel", "nx": 96, "ny": 64, "nz": 64,
         "form": "learned"},
        # unstructured jittered hexes, prisms and pyramids: Koren TVD, AMD, three non-orthogonal
        # correctors, precision form
        {"name": "step_mixed_box", "kind": "step", "flow": "box", "nx": 40, "ny": 40, "nz": 40, "form": "chosen"},
        # the reference's default numerics (EXACT cell projection, dual Rhie-Chow, correctors) on the
        # 45-degree skewed box, an odd size, FP64
        {"name": "step_exact_skew", "kind": "step", "flow": "skew", "nx": 33, "ny": 33, "nz": 33, "form": "plain"},
        # Rayleigh-Benard with temperature and two passive scalars, van Leer
        {"name": "step_rb_1m", "kind": "step", "flow": "rb", "nx": 128, "ny": 128, "nz": 65, "form": "chosen"},
        # urban canopy at the half resolution: obstacles, MOST, AMD, temperature and a scalar
        {"name": "step_urban_2m", "kind": "step", "flow": "urban", "nx": 200, "ny": 200, "nz": 63, "form": "chosen"},
        # the largest: the urban canopy at three quarters of the full resolution (8.2M cells)
        {"name": "step_urban_8m", "kind": "step", "flow": "urban", "nx": 300, "ny": 300, "nz": 94, "form": "chosen"},
        # the pressure solve a Fortran host links: boomeramg, host arrays, odd sizes
        {"name": "solve_amg_host", "kind": "solve", "nx": 127, "ny": 101, "nz": 83, "walls": True, "amg": True,
         "device": False},
        # the same interface at a regression size with device arrays and Jacobi
        {"name": "solve_jacobi_device", "kind": "solve", "nx": 24, "ny": 24, "nz": 16, "walls": True, "amg": False,
         "device": True},
        # allocation-free solve on the caller's device operator
        {"name": "noalloc_solve", "kind": "noalloc", "nx": 45, "ny": 40, "nz": 37, "walls": False},
        # single operators swapped into a host's own step
        {"name": "operators", "kind": "operators", "nx": 64, "ny": 64, "nz": 63},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["solve"] * 2 + ["noalloc", "operators"])
    if kind == "operators":
        return {"kind": kind, "nx": rng.randint(17, 72), "ny": rng.randint(17, 72), "nz": rng.randint(17, 72)}
    if kind == "noalloc":
        return {"kind": kind, "nx": _log_int(rng, 9, 50), "ny": _log_int(rng, 9, 50), "nz": _log_int(rng, 9, 50),
                "walls": rng.random() < 0.5}
    if kind == "solve":
        amg = rng.random() < 0.5
        hi = 128 if amg else 72
        return {"kind": kind, "nx": _log_int(rng, 16, hi), "ny": _log_int(rng, 16, hi), "nz": _log_int(rng, 16, hi),
                "walls": rng.random() < 0.7, "amg": amg, "device": rng.random() < 0.5}
    flow = rng.choice(["tgv", "channel", "channel", "box", "skew", "rb", "urban", "urban"])
    case = {"kind": kind, "flow": flow}
    if flow in ("box", "skew"):
        n = _log_int(rng, 10, 44 if flow == "box" else 34)
        case.update(nx=n, ny=n, nz=n)
    elif flow == "tgv":
        n = _log_int(rng, 12, 56)
        case.update(nx=n, ny=n, nz=n)
    elif flow == "channel":
        case.update(nx=_log_int(rng, 24, 128), ny=_log_int(rng, 16, 96), nz=_log_int(rng, 16, 96))
    elif flow == "rb":
        case.update(nx=_log_int(rng, 32, 160), ny=_log_int(rng, 32, 160), nz=_log_int(rng, 16, 80))
    else:
        n = _log_int(rng, 60, 240)
        case.update(nx=n, ny=n + rng.randint(-9, 9), nz=max(19, int(n * 0.31) + rng.randint(-3, 3)))
    if flow in ("tgv", "skew"):
        case["form"] = "plain"
    elif flow == "channel":
        case["form"] = rng.choice(["plain", "chosen", "learned"])
    else:
        case["form"] = "chosen"
    return case


# ------------------------------------------------------------------------------------------
# time steps
# ------------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=2)
def _flow_case(flow, nx, ny, nz):
    """The run configuration of one flow and size (its mesh file, in a user's program)."""
    if flow == "tgv":
        return cases.tgv_config(nx)
    if flow == "channel":
        return cases.channel_config(nx, ny, nz)
    if flow == "box":
        return cases.hybrid_config(nx, "mixed")
    if flow == "skew":
        ref = cases.regression_case("tgv_skew_exact")
        params = dict(ref.params, dt=ref.params["dt"] * 16.0 / nx)
        return cases.Case(f"skew{nx}", cases.skewed_unit_box(nx, 0.08), ref.patches, params, ref.ic, ref.ic_uref)
    if flow == "rb":
        return cases.rb_config(nx, ny, nz)
    # obstacle sizes stay those of the configuration; only the resolution changes
    return cases.urban_config(nx, ny, nz)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True).numpy()
    t[...] = a
    return t


def _initial_state(case, base, s, seed):
    """U, p, T and the scalars of a run's start: the configuration's profile with seeded +-10 %
    noise (one part in a hundred for the smooth vortices), temperature and scalars perturbed."""
    rng = np.random.default_rng(seed)
    noise = base.noise
    base.noise = 0.0
    U = base.initial_velocity(s.centroid)
    base.noise = noise
    amp = 0.10 if case["flow"] in ("channel", "rb", "urban") else 0.01
    U *= 1.0 + amp * (2.0 * rng.random(U.shape) - 1.0)
    T = C0 = None
    if s.params.boussinesq:
        T = np.full(s.nc, s.params.T_ref)
        if case["flow"] == "rb":
            T = 1.0 - s.centroid[:, 2]
        T += (1.0e-3 if case["flow"] == "rb" else 0.1) * (2.0 * rng.random(s.nc) - 1.0)
    ns = int(s.params.n_scalars)
    if ns:
        C0 = 0.1 * rng.random((ns, s.nc))
    return U, T, C0


def _prepare_step(case, seed):
    base = _flow_case(case["flow"], case["nx"], case["ny"], case["nz"])
    more = {}
    if case["form"] != "plain":
        more = dict(form=abi.FORM_MIXED, p_solver=abi.PSOLVER_AUTO)
    s = Solver(base, params=abi.default_params(**dict(base.params, **more)))
    U, T, Cs = _initial_state(case, base, s, seed)
    s.to_device(U, np.zeros(s.nc), T)
    if Cs is not None:
        s.set_scalars(Cs)
    for _ in range(2):  # as Solver.initialise: the noise is projected out
        s.project_once(8.0 / 15.0 * s.params.dt)
    if case["form"] == "learned":
        s.learn_collect(3)
        s.learn_train(epochs=80, lr=1.0e-2)
    s.advance()
    host = s.sync_host()
    out = {"U": _pinned(host["U"]), "p": _pinned(host["p"])}
    if T is not None:
        out["T"] = _pinned(host["T"])
    if Cs is not None:
        out["C"] = _pinned(np.ascontiguousarray(s.scalars()[1].T))
    if s.params.sgs_model != abi.SGS_NONE:
        out["nu_sgs"] = _pinned(host["nu_sgs"])
    return {"kind": "step", "s": s, "dt": s.params.dt, "out": out}


def _dp(a):
    return None if a is None else a.ctypes.data_as(C.POINTER(C.c_double))


def _run_step(st):
    L, h, o = lib(), st["s"].h, st["out"]
    rc = L.dpm_upload_state(h, _dp(o["U"]), _dp(o["p"]), _dp(o.get("T")))
    if "C" in o:
        rc = rc or L.dpm_upload_scalars(h, _dp(o["C"]))
    rc = rc or L.dpm_advance(h, st["dt"])
    rc = rc or L.dpm_download_state(h, _dp(o["U"]), _dp(o["p"]), _dp(o.get("T")), _dp(o.get("nu_sgs")))
    if "C" in o:
        rc = rc or L.dpm_download_scalars(h, _dp(o["C"]))
    if rc:
        raise RuntimeError(f"time step failed with status {rc}")
    return o


# ------------------------------------------------------------------------------------------
# pressure solves: the two-point operator of a box of nx x ny x nz hexes, periodic in x and y (and
# in z without walls), Bump-graded in z with walls
# ------------------------------------------------------------------------------------------


def _spacings(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    hx, hy = np.full(nx, 2.0 / nx), np.full(ny, 2.0 / ny)
    hz = np.diff(cases.bump_nodes(nz, 0.25)) if case["walls"] else np.full(nz, 1.0 / nz)
    return hx, hy, hz


def _axis_coeffs(h, periodic):
    """1 / centre distance across the faces i | i+1 (the last entry closes a periodic axis)."""
    c = 2.0 / (h + np.roll(h, -1))
    if not periodic:
        c[-1] = 0.0
    return c


@functools.lru_cache(maxsize=2)
def _operator(nx, ny, nz, walls):
    """Face lists (1-based), coefficients and diagonal as the Fortran caller holds them; cells i fastest."""
    hx, hy, hz = _spacings({"nx": nx, "ny": ny, "nz": nz, "walls": walls})
    ids = np.arange(nx * ny * nz, dtype=np.int32).reshape(nz, ny, nx)
    own, nei, co = [], [], []
    A = (hz[:, None, None] * hy[None, :, None], hz[:, None, None] * hx[None, None, :],
         hy[None, :, None] * hx[None, None, :])
    cx, cy, cz = _axis_coeffs(hx, True), _axis_coeffs(hy, True), _axis_coeffs(hz, not walls)
    for ax, cf, area in ((2, cx[None, None, :], A[0]), (1, cy[None, :, None], A[1]), (0, cz[:, None, None], A[2])):
        full = np.broadcast_to(cf * area, ids.shape)
        keep = full != 0.0
        own.append(ids[keep])
        nei.append(np.roll(ids, -1, axis=ax)[keep])
        co.append(full[keep])
    own, nei, co = np.concatenate(own), np.concatenate(nei), np.ascontiguousarray(np.concatenate(co))
    n = ids.size
    diag = np.bincount(own, weights=co, minlength=n) + np.bincount(nei, weights=co, minlength=n)
    return dict(n=n, nf=own.size, l2g=np.arange(1, n + 1, dtype=np.int32), own=own + np.int32(1),
                nei=nei + np.int32(1), skip=np.zeros(own.size, np.int32), co=co, diag=diag)


def _rhs(case, seed):
    """A Poisson right-hand side as a step forms it: the divergence of a noisy face flux (zero sum),
    with both smooth and cell-scale content."""
    hx, hy, hz = _spacings(case)
    rng = np.random.default_rng(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    b = np.zeros(shape)
    x, y, z = (np.cumsum(h) - 0.5 * h for h in (hx, hy, hz))
    areas = (np.broadcast_to(hy[None, :, None] * hx[None, None, :], shape),
             np.broadcast_to(hz[:, None, None] * hx[None, None, :], shape),
             np.broadcast_to(hz[:, None, None] * hy[None, :, None], shape))
    for ax in range(3):
        ph = 2.0 * np.pi * rng.random(3)
        wave = (np.sin(np.pi * x + ph[0])[None, None, :] * np.sin(np.pi * y + ph[1])[None, :, None]
                * np.sin(2.0 * np.pi * z + ph[2])[:, None, None])
        F = areas[ax] * (wave + 0.1 * (2.0 * rng.random(shape) - 1.0))
        if ax == 0 and case["walls"]:
            F[-1] = 0.0
        b += F - np.roll(F, 1, axis=ax)
    return np.ascontiguousarray(b.ravel())


RTOL = 1.0e-10  # the configurations' Poisson tolerance
_assembled = {"key": None}


def _ip(a):
    return a.ctypes.data_as(C.POINTER(C.c_int))


def _call_solve(st):
    A, L = st["A"], lib()
    its, res = C.c_int(), C.c_double()
    L.fvm_petsc_set_pressure_solver(b"boomeramg" if st["amg"] else b"jacobi")
    L.fvm_petsc_set_io_on_device(1 if st["device"] else 0)
    p = (lambda t: C.cast(t.data_ptr(), C.POINTER(C.c_double))) if st["device"] else _dp
    rc = L.fvm_petsc_solve_pressure(A["n"], A["n"], A["nf"], _ip(A["l2g"]), _ip(A["own"]), _ip(A["nei"]), _ip(A["nei"]),
                                    _ip(A["skip"]), _dp(A["diag"]), p(st["b"]), _dp(A["co"]), 1, 1000, RTOL, 0.0, None,
                                    None, 0, p(st["x"]), C.byref(its), C.byref(res))
    L.fvm_petsc_set_io_on_device(0)
    if rc:
        raise RuntimeError(f"pressure solve failed with status {rc}")


def _prepare_solve(case, seed):
    A = _operator(case["nx"], case["ny"], case["nz"], case["walls"])
    b = _rhs(case, seed)
    st = {"kind": "solve", "A": A, "amg": case["amg"], "device": case["device"]}
    if case["device"]:
        st["b"], st["x"] = torch.from_numpy(b).cuda(), torch.zeros(A["n"], dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
    else:
        st["b"], st["x"] = b, np.zeros(A["n"])
    key = (case["nx"], case["ny"], case["nz"], case["walls"])
    if _assembled["key"] != key:  # the operator is assembled once per mesh and kept by the library
        lib().fvm_petsc_backend_finalize()
        _assembled["key"] = key
    _call_solve(st)  # a program's first solve assembles the operator and the hierarchy
    return st


def _run_solve(st):
    if st["device"]:
        st["x"].zero_()  # p' starts from zero each stage
        torch.cuda.current_stream().synchronize()  # device arrays are the caller's to order
    else:
        st["x"].fill(0.0)
    _call_solve(st)
    return st["x"]


@functools.lru_cache(maxsize=2)
def _ell(nx, ny, nz, walls):
    """The same operator in padded ELL [7][n], columns ascending, padding (own row, 0)."""
    A = _operator(nx, ny, nz, walls)
    n = A["n"]
    o, m = A["own"].astype(np.int64) - 1, A["nei"].astype(np.int64) - 1
    row = np.concatenate([np.arange(n), o, m])
    col = np.concatenate([np.arange(n), m, o])
    val = np.concatenate([A["diag"], -A["co"], -A["co"]])
    order = np.lexsort((col, row))
    row, col, val = row[order], col[order], val[order]
    first = np.searchsorted(row, np.arange(n))
    slot = np.arange(row.size) - first[row]
    ec = np.tile(np.arange(n, dtype=np.int32), (7, 1))
    ev = np.zeros((7, n))
    ec[slot, row] = col
    ev[slot, row] = val
    return ec, ev, 1.0 / A["diag"]


def _prepare_noalloc(case, seed):
    ec, ev, dinv = _ell(case["nx"], case["ny"], case["nz"], case["walls"])
    cuda = lambda a: torch.from_numpy(a).cuda()
    st = {"kind": "noalloc", "n": ec.shape[1], "col": cuda(ec), "val": cuda(ev), "dinv": cuda(dinv),
          "b": cuda(_rhs(case, seed)), "x": torch.zeros(ec.shape[1], dtype=torch.float64, device="cuda")}
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    lib().dpm_pcg_solve_noalloc(st["n"], 7, None, None, None, None, None, RTOL, 0.0, 0, 1, stream, None, None)
    torch.cuda.synchronize()
    return st


def _run_noalloc(st):
    st["x"].zero_()
    its, res = C.c_int(), C.c_double()
    ptr = lambda t: C.c_void_p(t.data_ptr())
    rc = lib().dpm_pcg_solve_noalloc(st["n"], 7, ptr(st["col"]), ptr(st["val"]), ptr(st["dinv"]), ptr(st["b"]),
                                     ptr(st["x"]), RTOL, 0.0, 5000, 1,
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(its), C.byref(res))
    if rc:
        raise RuntimeError(f"pressure solve failed with status {rc}")
    return st["x"]


def _exact_solve(case, seed):
    """A^-1 b by fast diagonalisation: A = Kx My Mz + Mx Ky Mz + Mx My Kz, each axis's pencil (K, M)
    diagonalised with M the cell sizes.  Zero-sum b; the mean is that of the zero initial guess, as
    Jacobi-PCG and flexible CG remove the constant from every direction."""
    hx, hy, hz = _spacings(case)
    V, lam = [], []
    for h, per in ((hz, not case["walls"]), (hy, True), (hx, True)):
        n = h.size
        c = _axis_coeffs(h, per)
        K = np.zeros((n, n))
        for i in range(n):
            j = (i + 1) % n
            K[i, i] += c[i]
            K[j, j] += c[i]
            K[i, j] -= c[i]
            K[j, i] -= c[i]
        sh = 1.0 / np.sqrt(h)
        w, Q = np.linalg.eigh(sh[:, None] * K * sh[None, :])
        V.append(sh[:, None] * Q)
        lam.append(w)
    b = _rhs(case, seed).reshape(case["nz"], case["ny"], case["nx"])
    b = b - b.mean()
    t = np.einsum("zyx,zk->kyx", b, V[0], optimize=True)
    t = np.einsum("kyx,yj->kjx", t, V[1], optimize=True)
    t = np.einsum("kjx,xi->kji", t, V[2], optimize=True)
    L = lam[0][:, None, None] + lam[1][None, :, None] + lam[2][None, None, :]
    L.flat[0] = 1.0
    t /= L
    t.flat[0] = 0.0
    t = np.einsum("kji,xi->kjx", t, V[2], optimize=True)
    t = np.einsum("kjx,yj->kyx", t, V[1], optimize=True)
    t = np.einsum("kyx,zk->zyx", t, V[0], optimize=True).ravel()
    return t - t.mean()


# ------------------------------------------------------------------------------------------
# single operators on the periodic box
# ------------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=2)
def _periodic_case(nx, ny, nz):
    return cases.Case("box", cases.uniform_box(nx, ny, nz, 1.0, 1.0, 1.0), [{"bc": "periodic"} for _ in range(6)],
                      dict(scheme=abi.SCHEME_CDS, nu=1.0e-3, dt=1.0e-3), "uniform")


NU = 1.0e-3


def _operator_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = case["nx"] * case["ny"] * case["nz"]
    return rng.standard_normal((n, 3)), 1.0e-3 * rng.random(n), rng.standard_normal((n, 3, 3))


def _prepare_operators(case, seed):
    s = Solver(_periodic_case(case["nx"], case["ny"], case["nz"]))
    U, nus, g = _operator_inputs(case, seed)
    return {"kind": "operators", "s": s, "U": U, "Ub": np.zeros((s.nb, 3)), "nus": nus, "g": g}


def _run_operators(st):
    s = st["s"]
    grad = s.ls_gradient_vector(st["U"], st["Ub"])
    visc = s.viscous_rhs_vector(st["U"], NU, st["nus"], st["g"], st["Ub"])
    return {"grad": grad, "visc": visc}


def _exact_operators(case, seed):
    U, nus, g = _operator_inputs(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    shape, h = (nz, ny, nx), np.array([1.0 / nx, 1.0 / ny, 1.0 / nz])
    U, nus, g = U.reshape(shape + (3,)), nus.reshape(shape), g.reshape(shape + (3, 3))
    kk, jj, ii = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    # least squares over the face neighbours (across the seams too) and the cells sharing a vertex
    # (within the box), weights 1 / distance squared
    A, r = np.zeros(shape + (3, 3)), np.zeros(shape + (3, 3))
    for dk in (-1, 0, 1):
        for dj in (-1, 0, 1):
            for di in (-1, 0, 1):
                if not (di or dj or dk):
                    continue
                on = np.ones(shape, bool)
                if abs(di) + abs(dj) + abs(dk) > 1:
                    for q, dq, m in ((ii, di, nx), (jj, dj, ny), (kk, dk, nz)):
                        on &= (q + dq >= 0) & (q + dq < m)
                d = np.array([di, dj, dk]) * h
                w = on / (d @ d)
                A += w[..., None, None] * np.outer(d, d)
                du = np.roll(U, (-dk, -dj, -di), axis=(0, 1, 2)) - U
                r += w[..., None, None] * d[:, None] * du[..., None, :]
    grad = np.linalg.solve(A, r).swapaxes(-1, -2)  # [j, i] = dU_j / dx_i
    visc = np.zeros(shape + (3,))
    for a, ax in ((0, 2), (1, 1), (2, 0)):  # the flux through each cell's upper face along axis a
        up = lambda q: np.roll(q, -1, axis=ax)
        nu = NU + 0.5 * (nus + up(nus))
        f = nu[..., None] * ((up(U) - U) / h[a] + 0.5 * (g + up(g))[..., a, :]) / h[a]
        visc += f - np.roll(f, 1, axis=ax)
    n = nx * ny * nz
    return {"grad": grad.reshape(n, 3, 3), "visc": visc.reshape(n, 3)}


# ------------------------------------------------------------------------------------------
# the interface
# ------------------------------------------------------------------------------------------
_PREPARE = {"step": _prepare_step, "solve": _prepare_solve, "noalloc": _prepare_noalloc, "operators": _prepare_operators}
_RUN = {"step": _run_step, "solve": _run_solve, "noalloc": _run_noalloc, "operators": _run_operators}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    if case["kind"] in ("solve", "noalloc"):
        return _exact_solve(case, seed)
    if case["kind"] == "operators":
        return _exact_operators(case, seed)
    return None


def work(case):
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] in ("solve", "noalloc"):
        # operator (three faces per cell: coefficient and neighbour), right-hand side, guess, solution
        return {"bytes": n * (3 * 12 + 8 + 3 * 8.0), "flops": n * 13.0 * 10}
    if case["kind"] == "operators":
        # U and the gradient twice (in and out), nu_sgs and the right-hand side
        return {"bytes": n * 8.0 * (3 + 9 + 3 + 1 + 9 + 3), "flops": n * (26 * 18.0 + 3 * 60.0)}
    if case["flow"] == "box":
        n = int(n * 2.35)  # cells after the split into prisms and pyramids
    fields = {"tgv": 4, "channel": 4, "box": 4, "skew": 4, "rb": 7, "urban": 6}[case["flow"]]
    # the state in and out, and the mesh once: three faces per cell (area vector, two cells,
    # coefficient), volume, centroid
    return {"bytes": n * (2.0 * 8 * fields + 3 * (24 + 8 + 8) + 32), "flops": n * 3 * 2500.0}


def tolerance(case):
    """About four times the largest difference measured between two correct implementations of the
    case: for the steps, between the Krylov forms (Jacobi-PCG, two-level, multilevel, other smoother
    degrees) at the configurations' Poisson tolerance of 1e-10, which bounds what a step can say of
    the pressure, and between the FP64 and the FP32 explicit half for the precision form; for the
    solves, between the solution and its 64-bit value."""
    if case["kind"] == "operators":
        return {"rel": 5e-14}
    if case["kind"] != "step":
        return {"rel": 4e-10, "max": 2e-9}
    if case["flow"] == "tgv":
        return {"rel": 8e-10, "max": 4e-9}
    if case["flow"] == "skew":  # the projection stops on the velocity energy of its last step (1e-2)
        return {"rel": 2e-5, "max": 2e-4}
    if case["flow"] == "channel" and case["form"] == "plain":
        return {"rel": 1.6e-7, "max": 1.2e-6}
    if case["flow"] == "channel":
        return {"rel": 1.6e-5, "max": 2.5e-4}
    if case["flow"] == "box":
        return {"rel": 1.5e-6, "max": 2e-5}
    if case["flow"] == "rb":
        return {"rel": 6e-6, "max": 8e-4}
    # urban: single near-ground cells, where a surface flux amplifies the tolerance's footprint
    return {"rel": 2e-3, "max": 0.2}
