"""The shared-memory-resident Krylov run (one cooperative launch per run, the default for one
system that fits on the chip) against the two-kernel iteration (host_loop=True, which keeps it):
the same recurrences with sums in another order.  Sizes from one block of one slice to the last
that fits; a general system whose columns reach from one end to the other; the iteration cap,
a zero right-hand side and an indefinite system."""
import ctypes as C

import numpy as np
import pytest

import mhdarcy
from mhdarcy import _lib
from mhdarcy.cases import dirichlet_x_bc, make_case


def system(cfg, n, seed=3):
    mesh, coeffs = make_case(cfg, seed=seed, n=n)
    s = mhdarcy.MHSystem(mesh)
    bc, _ = dirichlet_x_bc(s.topology(), mesh)
    s.set_coeffs(**coeffs)
    s.set_bc(bc["bc_type"], bc["pressure"])
    s.assemble()
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("cfg,n", [(1, 2), (1, 4), (1, 9), (2, 16), (5, 18), (2, 23), (1, 30)])
def test_pcg64_iterates_match_two_kernel(gpu, cfg, n):
    """After k iterations the FP64 iterates agree to 1e-10, the bound the two-kernel iteration
    itself is held to against the CPU's iterates."""
    with system(cfg, n) as s:
        for k in (1, 2, 10, 50):
            two = s.solve(r_tol=1e-300, max_it=k, host_loop=True)
            x2 = s.solution()
            one = s.solve(r_tol=1e-300, max_it=k)
            x1 = s.solution()
            assert one["status"] == two["status"] == mhdarcy.MH_NOT_CONVERGED
            assert one["iterations"] == two["iterations"] == k
            for a, b in zip(s.split(x1), s.split(x2)):
                assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()
        assert one["kernel_launches"] < two["kernel_launches"] - k  # the resident run was taken


@pytest.mark.gpu
@pytest.mark.parametrize("method", [_lib.MH_SOLVER_PCG64, _lib.MH_SOLVER_IR32])
@pytest.mark.parametrize("cfg,n", [(1, 2), (1, 9), (5, 18), (2, 30), (2, 35)])
def test_converged_residual(gpu, cfg, n, method):
    """Both norms of the residual, recomputed here on the exported system, meet r_tol."""
    with system(cfg, n) as s:
        st = s.solve(method=method, r_tol=1e-11)
        assert st["status"] == 0
        if method == _lib.MH_SOLVER_IR32 or n <= 30:  # (FP64 at n = 35 does not fit)
            assert st["kernel_launches"] < st["iterations"]
        rp, col, val, rhs = s.schur_system()
        x = s.split(s.solution())[2]
        rows = np.repeat(np.arange(len(rhs)), np.diff(rp))
        r = rhs - np.bincount(rows, weights=val * x[col], minlength=len(rhs))
        dg = np.zeros(len(rhs))
        on = rows == col
        dg[rows[on]] = val[on]
        sd = 1.0 / np.sqrt(dg)
        assert np.linalg.norm(r) <= 1.01e-11 * np.linalg.norm(rhs)
        assert np.linalg.norm(sd * r) <= 1.01e-11 * np.linalg.norm(sd * rhs)


class Csr:
    def __init__(self, A):
        n = len(A)
        nz = [np.nonzero(r)[0] for r in A]
        rp = np.concatenate([[0], np.cumsum([len(z) for z in nz])]).astype(np.int32)
        col = np.concatenate(nz).astype(np.int32)
        self.val, self.n, self.h = np.concatenate([A[i, z] for i, z in enumerate(nz)]), n, C.c_void_p()
        p = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
        self.p = p
        assert mhdarcy.lib.mh_csr_create(n, p(rp, C.c_int32), p(col, C.c_int32), C.byref(self.h)) == 0

    def solve(self, rhs, **kw):
        o, st, x = mhdarcy.solve_opts(**kw), _lib.SolveStats(), np.zeros(self.n)
        assert mhdarcy.lib.mh_csr_set_values(self.h, self.p(self.val, C.c_double), self.p(rhs, C.c_double)) == 0
        rc = mhdarcy.lib.mh_solve(self.h, C.byref(o), C.byref(st))
        mhdarcy.lib.mh_csr_get_solution(self.h, self.p(x, C.c_double), self.n)
        mhdarcy.lib.mh_destroy(self.h)
        return rc, st.as_dict(), x


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 700, 2049])
def test_arrow_system(gpu, n):
    """Every row couples to the first and the last: halo rows in every block.  CG on a diagonally
    dominant system of condition < 4 reaches 1e-12, so the error is below 4e-12 of the solution."""
    rng = np.random.default_rng(n)
    A = np.zeros((n, n))
    A[0, :], A[-1, :] = 0.5 / n, 0.25 / n
    A = A + A.T
    A[np.arange(n), np.arange(n)] = 2.0 + rng.random(n)
    rhs = rng.normal(size=n)
    rc, st, x = Csr(A).solve(rhs, r_tol=1e-12)
    ref = np.linalg.solve(A, rhs)
    assert rc == 0 and np.linalg.norm(x - ref) <= 4e-12 * np.linalg.norm(ref)


@pytest.mark.gpu
@pytest.mark.parametrize("host_loop", [False, True])
def test_ends_without_convergence(gpu, host_loop):
    A = np.array([[1.0, 3.0], [3.0, 1.0]])
    rc, st, _ = Csr(A).solve(np.array([1.0, -1.0]), host_loop=host_loop)
    assert rc == -8  # p'Sp <= 0
    rc, st, x = Csr(np.eye(40)).solve(np.zeros(40), host_loop=host_loop)
    assert rc == 0 and st["iterations"] == 0 and not x.any()
