"""The one-cluster Krylov run of the smallest systems: from less than one slice of rows to both
sides of the line where the chip-wide run takes over, on systems whose rows couple to far ends
(halo rows from every block), against the two-kernel iteration (host_loop=True)."""
import ctypes as C

import numpy as np
import pytest

import mhdarcy
from mhdarcy import _lib


def spread_system(n, seed):
    """Symmetric, diagonally dominant (condition below 4): off-diagonals at distances that reach
    from one end to the other."""
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    r, c, v = [], [], []
    for d in {1, 37, n // 3, n - 1} - {0}:
        if d < n:
            w = -0.12 * rng.random(n - d)
            r += [i[:-d], i[d:]]
            c += [i[d:], i[:-d]]
            v += [w, w]
    r, c, v = (np.concatenate(a + [b]) for a, b in ((r, i), (c, i), (v, 2.0 + rng.random(n))))
    o = np.lexsort((c, r))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    return rp, c[o].astype(np.int32), v[o], rng.normal(size=n)


def solve(n, rp, col, val, rhs, **kw):
    p = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
    h, o, st, x = C.c_void_p(), mhdarcy.solve_opts(**kw), _lib.SolveStats(), np.zeros(n)
    assert mhdarcy.lib.mh_csr_create(n, p(rp, C.c_int32), p(col, C.c_int32), C.byref(h)) == 0
    try:
        assert mhdarcy.lib.mh_csr_set_values(h, p(val, C.c_double), p(rhs, C.c_double)) == 0
        rc = mhdarcy.lib.mh_solve(h, C.byref(o), C.byref(st))
        mhdarcy.lib.mh_csr_get_solution(h, p(x, C.c_double), n)
    finally:
        mhdarcy.lib.mh_destroy(h)
    return rc, st.as_dict(), x


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 32, 65, 511, 513, 4097, 14335, 14336, 14337])
def test_iterates_match_two_kernel(gpu, n):
    """Sums in another order only: after k steps of a well conditioned system the iterates agree to
    1e-12 (FP64 rounding of at most 12 steps, with three decimals to spare)."""
    sysm = spread_system(n, n)
    for k in (1, 5, 12):
        _, s2, x2 = solve(n, *sysm, r_tol=1e-300, max_it=k, host_loop=True)
        _, s1, x1 = solve(n, *sysm, r_tol=1e-300, max_it=k)
        assert s1["iterations"] == s2["iterations"] and s1["status"] == s2["status"]
        assert np.abs(x1 - x2).max() <= 1e-12 * np.abs(x2).max()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [65, 14336])
def test_ir32_meets_tolerance(gpu, n):
    rp, col, val, rhs = spread_system(n, n + 1)
    rc, _, x = solve(n, rp, col, val, rhs, method=_lib.MH_SOLVER_IR32, r_tol=1e-12)
    rows = np.repeat(np.arange(n), np.diff(rp))
    r = rhs - np.bincount(rows, weights=val * x[col], minlength=n)
    assert rc == 0 and np.linalg.norm(r) <= 4e-12 * np.linalg.norm(rhs)
