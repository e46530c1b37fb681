"""The smoothed-aggregation hierarchy of the multilevel pressure solve on the CPU (compiled here from
its source): one hierarchy on any number of threads, and flexible CG with its V-cycle, restated in
numpy, on operators with one fluid region, with several, and with small sealed ones.

Every region without a Dirichlet row has its own constant in the null space.  The dense inverse of
the coarsest level lifts each of them and has no row for a region that has shrunk to one unknown;
otherwise the factorisation passes on rounding and the inverse holds entries of 1e9 and more."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import scipy.sparse as sp

HERE = os.path.dirname(os.path.abspath(__file__))
ENTRY = np.dtype([("col", np.int32), ("val", np.float32)])
DTYPES = [np.float32, np.int32, np.float32, np.uint16, np.int32, ENTRY, np.float32, np.float32, np.float32, np.int32,
          ENTRY, np.int32, ENTRY]


@pytest.fixture(scope="module")
def builder(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("sa") / "sa.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-fopenmp", "-shared",
                    os.path.join(HERE, "smoothed_multilevel.cpp"),
                    os.path.join(HERE, "..", "dopamine_b200", "csrc", "host", "multilevel.cpp"), "-o", so], check=True)
    L = C.CDLL(so)
    L.sa_array.restype = C.c_void_p

    def build(A, nullsp, passes=3, half=False):
        A = A.tocsr()
        n, W = A.shape[0], int(np.diff(A.indptr).max())
        col = np.tile(np.arange(n, dtype=np.int32), (W, 1))
        val = np.zeros((W, n))
        row = np.repeat(np.arange(n), np.diff(A.indptr))
        slot = np.arange(A.nnz) - A.indptr[row]
        col[slot, row], val[slot, row] = A.indices, A.data
        nl, nc = C.c_int(), C.c_int()
        rc = L.sa_build(n, W, col.ctypes.data_as(C.c_void_p), val.ctypes.data_as(C.c_void_p), int(nullsp), passes,
                        int(half), C.byref(nl), C.byref(nc))

        def array(l, which):
            m = C.c_longlong()
            p = L.sa_array(l, which, C.byref(m))
            nbytes = m.value * np.dtype(DTYPES[which]).itemsize
            return np.frombuffer((C.c_char * nbytes).from_address(p) if nbytes else b"", dtype=DTYPES[which]).copy()

        levels = []
        for l in range(nl.value if rc == 0 else 0):
            sizes, sc = (C.c_int * 3)(), (C.c_double * 2)()
            L.sa_level(l, sizes, sc)
            levels.append({"n": sizes[0], "next": sizes[1], "W": sizes[2], "oc": sc[0], "lmax": sc[1],
                           **{k: array(l, k) for k in range(1, 13)}})
        return rc, levels, (array(0, 0).reshape(nc.value, nc.value) if rc == 0 else None)

    return build


def _box(nx, ny, nz, region, dirichlet, seed=1):
    """Seven-point operator of a box with random coefficients; faces between regions are closed.
    dirichlet: the cells of the bottom layer have a boundary value."""
    rng = np.random.default_rng(seed)
    ids = np.arange(nx * ny * nz).reshape(nz, ny, nx)
    lab = np.zeros(ids.shape, int)
    for r, box in enumerate(region):
        lab[box] = r + 1
    a, b = [], []
    for ax in range(3):
        lo = tuple(slice(None, -1) if k == ax else slice(None) for k in range(3))
        hi = tuple(slice(1, None) if k == ax else slice(None) for k in range(3))
        same = lab[lo] == lab[hi]
        a.append(ids[lo][same])
        b.append(ids[hi][same])
    a, b = np.concatenate(a), np.concatenate(b)
    c = rng.uniform(0.5, 2.0, a.size)
    n = ids.size
    A = sp.coo_matrix((np.concatenate([-c, -c]), (np.concatenate([a, b]), np.concatenate([b, a]))), (n, n)).tocsr()
    d = np.bincount(a, c, n) + np.bincount(b, c, n)
    if dirichlet:
        d[ids[0].ravel()] += 2.0
    A = (A + sp.diags(d)).tocsr()
    A.sort_indices()
    return A


def _vcycle(levels, cinv, degree=2):
    """The V-cycle of csrc/cuda/mlkern.cuh as a function of the FP32 residual."""
    f = np.float32
    ops = []
    for L in levels:
        if L["W"]:
            col, row = L[1].reshape(L["W"], -1), np.tile(np.arange(L["n"]), L["W"])
            S = sp.csr_matrix((L[2], (row, col.ravel())), (L["n"], L["n"]))
        else:
            S = sp.csr_matrix((L[5]["val"], L[5]["col"], L[4]), (L["n"], L["n"]))
        lmax = 1.1 * L["lmax"]
        th, de = 0.55 * lmax, 0.45 * lmax
        ops.append((S + sp.diags(L[6]), sp.csr_matrix((L[10]["val"], L[10]["col"], L[9]), (L["n"], L["next"])),
                    sp.csr_matrix((L[12]["val"], L[12]["col"], L[11]), (L["next"], L["n"])), th, de))

    def smooth(l, b, x):
        S, _, _, th, de = ops[l]
        sig = th / de
        rho = 1.0 / sig
        d = f(1.0 / th) * (b if x is None else b - S @ x)
        x = d if x is None else x + d
        for _ in range(1, degree):
            rn = 1.0 / (2.0 * sig - rho)
            d = f(rn * rho) * d + f(2.0 * rn / de) * (b - S @ x)
            x, rho = x + d, rn
        return x

    def cycle(l, r):
        if l == len(levels):
            return cinv @ r
        L = levels[l]
        S, P, R = ops[l][:3]
        b = r * L[8]
        x = smooth(l, b, None)
        x = x + f(L["oc"]) * (P @ cycle(l + 1, R @ (L[7] * (b - S @ x))))
        return smooth(l, b, x)

    return lambda r: cycle(0, r.astype(f)).astype(float)


def _fcg(A, b, precond, nullsp, rtol=1e-10, maxit=60):
    n = b.size
    x, r = np.zeros(n), b - (b.mean() if nullsp else 0.0)
    p, q, pq, r0 = np.zeros(n), np.zeros(n), 1.0, np.linalg.norm(r)
    for it in range(maxit):
        if np.linalg.norm(r) <= rtol * r0:
            return x, it
        z = precond(r)
        if nullsp:
            z -= z.mean()
        w = A @ z
        beta = -(z @ q) / pq if it else 0.0
        p, q = z + beta * p, w + beta * q
        pq = p @ q
        if not pq > 0:
            return x, -1
        al = (z @ r) / pq
        x, r = x + al * p, r - al * q
    return x, maxit


HALVES = [np.s_[:, :, 15:]]
POCKET = [np.s_[10:14, 10:14, 10:14]]
ROOM = [np.s_[4:16, 8:20, 9:21]]
MANY = [np.s_[0:3, 5 * j:5 * j + 3, 5 * i:5 * i + 3] for j in range(6) for i in range(6)]


@pytest.mark.parametrize("dirichlet", [False, True])
@pytest.mark.parametrize("name", ["one", "halves", "pocket", "room", "many"])
def test_solve_on_several_regions(builder, name, dirichlet):
    region = {"one": [], "halves": HALVES, "pocket": POCKET, "room": ROOM, "many": MANY}[name]
    A = _box(30, 30, 24, region, dirichlet)
    rc, levels, cinv = builder(A, not dirichlet)
    assert rc == 0 and len(levels) == 2
    # The largest entry is at most 1 / (least eigenvalue of the lifted P^T A P): A's least non-zero one is
    # above 0.5 (2 - 2 cos(pi / 30)) = 1 / 182, and P^T P's above 0.1.
    # A factorisation that passes on rounding gives 1e9 and more.
    assert np.abs(cinv).max() < 182 / 0.1, np.abs(cinv).max()
    rng = np.random.default_rng(2)
    x_ref = rng.standard_normal(A.shape[0]) + np.sin(0.01 * np.arange(A.shape[0]))
    b = A @ x_ref
    x, its = _fcg(A, b, _vcycle(levels, cinv), not dirichlet)
    assert 0 < its <= 18, its  # one region: 12
    assert np.linalg.norm(b - A @ x) <= 2e-10 * np.linalg.norm(b)
    # the constants that the solve leaves in closed regions stay of the solution's size
    assert np.abs(x).max() <= 10 * np.abs(x_ref).max()


def test_more_regions_than_the_dense_level_holds_are_refused(builder):
    region = [np.s_[3 * k:3 * k + 2, 3 * j:3 * j + 2, 3 * i:3 * i + 2]
              for k in range(11) for j in range(11) for i in range(11)]
    rc, _, _ = builder(_box(33, 33, 33, region, False), True)
    assert rc < 0


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("region", [[], POCKET])
def test_same_hierarchy_on_any_thread_count(builder, region, half):
    from tests.test_host_setup import _Threads
    A = _box(30, 30, 24, region, False)
    threads = _Threads()
    out = []
    try:
        for t in (1, 3, max(8, threads.default)):
            threads(t)
            rc, levels, cinv = builder(A, True, half=half)
            assert rc == 0
            out.append([cinv.tobytes()] + [L[k].tobytes() for L in levels for k in range(1, 13)] +
                       [np.float64(L["lmax"]).tobytes() for L in levels])
    finally:
        threads(threads.default)
    assert out[0] == out[1] == out[2]
