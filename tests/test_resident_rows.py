"""The resident Krylov runs with two to four rows a thread: chip-wide at the sizes between those of
the other tests, and in one cluster on systems whose rows are so uneven (a band of 30 entries, then
one of three) that blocks of equal bytes hold more than 1024, 2048 and 3072 rows."""
import ctypes as C
import glob
import os
import re

import numpy as np
import pytest

import mhdarcy
from mhdarcy import _lib
from mhdarcy.cases import dirichlet_x_bc, make_case

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "svn-export_b200", "csrc")


def test_vectors_in_shared_memory_are_declared_so():
    """An access of 8 or 16 bytes needs an array of that type or alignment: no cast of another block's
    shared memory to a vector type."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = re.sub(r"\s+", " ", open(path).read())
        assert not re.search(r"reinterpret_cast<(const )?(double2|float2|float4|int4|uint4) \*>\(\w+\.map_shared_rank", text), path


def uneven_system(heavy, n=14336):
    """Diagonally dominant (condition below 4): 29 neighbours in the first `heavy` rows, two in the others."""
    rng = np.random.default_rng(heavy)
    i = np.arange(n)
    r, c, v = [i], [i], [2.0 + rng.random(n)]
    for d in range(1, 16):
        k = i[:-d] if d == 1 else i[:max(heavy - d, 0)]
        w = -0.03 * rng.random(len(k))
        r += [k, k + d]
        c += [k + d, k]
        v += [w, w]
    far = np.arange(32)  # the first rows and the last
    w = -0.03 * rng.random(32)
    r += [far, n - 1 - far]
    c += [n - 1 - far, far]
    v += [w, w]
    r, c, v = np.concatenate(r), np.concatenate(c), np.concatenate(v)
    o = np.lexsort((c, r))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    return rp, c[o].astype(np.int32), v[o], rng.normal(size=n)


def solve(rp, col, val, rhs, **kw):
    n = len(rhs)
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
@pytest.mark.parametrize("heavy", [700, 2900, 5200])
def test_uneven_rows_in_one_cluster(gpu, heavy):
    """Sums in another order than the two-kernel iteration's only: the iterates of a well conditioned
    system agree to 1e-12 (FP64 rounding of 12 steps at most, with three decimals to spare)."""
    sysm = uneven_system(heavy)
    for k in (1, 5, 12):
        _, s2, x2 = solve(*sysm, r_tol=1e-300, max_it=k, host_loop=True)
        _, s1, x1 = solve(*sysm, r_tol=1e-300, max_it=k)
        assert s1["iterations"] == s2["iterations"] == k
        assert np.abs(x1 - x2).max() <= 1e-12 * np.abs(x2).max()
    rp, col, val, rhs = sysm
    rows = np.repeat(np.arange(len(rhs)), np.diff(rp))
    for method in (_lib.MH_SOLVER_PCG64, _lib.MH_SOLVER_IR32):
        rc, st, x = solve(*sysm, method=method, r_tol=1e-12)
        r = rhs - np.bincount(rows, weights=val * x[col], minlength=len(rhs))
        assert rc == 0
        assert np.linalg.norm(r) <= 4e-12 * np.linalg.norm(rhs)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [24, 27, 29])
def test_two_rows_a_thread(gpu, n):
    mesh, coeffs = make_case(2, seed=3, n=n)
    with mhdarcy.MHSystem(mesh) as s:
        bc, _ = dirichlet_x_bc(s.topology(), mesh)
        s.set_coeffs(**coeffs)
        s.set_bc(bc["bc_type"], bc["pressure"])
        s.assemble()
        for k in (1, 10, 50):  # as the other sizes: 1e-10, the bound against the CPU's iterates
            two = s.solve(r_tol=1e-300, max_it=k, host_loop=True)
            x2 = s.solution()
            one = s.solve(r_tol=1e-300, max_it=k)
            assert one["iterations"] == two["iterations"] == k
            assert one["kernel_launches"] < two["kernel_launches"] - k
            for a, b in zip(s.split(s.solution()), s.split(x2)):
                assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()
        for method in (_lib.MH_SOLVER_PCG64, _lib.MH_SOLVER_IR32):
            st = s.solve(method=method, r_tol=1e-11)
            assert st["status"] == 0 and st["kernel_launches"] < st["iterations"]
            assert max(st["rel_residual"], st["rel_residual_unscaled"]) <= 1e-11
