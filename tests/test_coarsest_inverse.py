"""The dense inverse of the multigrid's coarsest level against the level's own matrix, and what
happens where that matrix is not positive definite to FP32 rounding."""
import ctypes as C

import numpy as np
import pytest

import mhdarcy
from mhdarcy import _lib
from mhdarcy.cases import dirichlet_x_bc, make_case

p = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731


class Csr:
    """A CSR system in a handle, solved by the multigrid."""

    def __init__(self, r, c, v, rhs):
        n = len(rhs)
        o = np.lexsort((c, r))
        self.rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
        self.col, self.val, self.rhs, self.h = c[o].astype(np.int32), v[o].copy(), rhs, C.c_void_p()
        assert mhdarcy.lib.mh_csr_create(n, p(self.rp, C.c_int32), p(self.col, C.c_int32), C.byref(self.h)) == 0

    def __enter__(self):
        return self

    def __exit__(self, *a):
        mhdarcy.lib.mh_destroy(self.h)

    def solve(self, **kw):
        o, st, x = mhdarcy.solve_opts(method=_lib.MH_SOLVER_AMG, **kw), _lib.SolveStats(), np.zeros(len(self.rhs))
        assert mhdarcy.lib.mh_csr_set_values(self.h, p(self.val, C.c_double), p(self.rhs, C.c_double)) == 0
        rc = mhdarcy.lib.mh_solve(self.h, C.byref(o), C.byref(st))
        assert mhdarcy.lib.mh_csr_get_solution(self.h, p(x, C.c_double), len(x)) == 0
        r = self.rhs - np.bincount(np.repeat(np.arange(len(x)), np.diff(self.rp)), weights=self.val * x[self.col],
                                   minlength=len(x))
        return rc, st.as_dict(), np.linalg.norm(r) / np.linalg.norm(self.rhs)


def coarsest(h):
    """(the coarsest level's matrix, its inverse or None)"""
    nl, rows, slots = np.zeros(1, np.int32), np.zeros(32, np.int64), np.zeros(32, np.int64)
    assert mhdarcy.lib.mh_amg_info(h, p(nl, C.c_int32), p(rows, C.c_int64), p(slots, C.c_int64), 32) == 0
    last, n, nnz, m = int(nl[0]) - 1, C.c_int64(), C.c_int64(), C.c_int64()
    null = [None] * 5
    assert mhdarcy.lib.mh_amg_level(h, last, C.byref(n), C.byref(nnz), *null) == 0
    rp, col, val = np.zeros(n.value + 1, np.int32), np.zeros(nnz.value, np.int32), np.zeros(nnz.value, np.float32)
    assert mhdarcy.lib.mh_amg_level(h, last, C.byref(n), C.byref(nnz), None, None, p(rp, C.c_int32), p(col, C.c_int32),
                                    p(val, C.c_float)) == 0
    A = np.zeros((n.value, n.value))
    A[np.repeat(np.arange(n.value), np.diff(rp)), col] = val
    assert mhdarcy.lib.mh_amg_coarsest(h, C.byref(m), None) == 0
    if m.value == 0:
        return A, None
    assert m.value == n.value == rows[last]
    inv = np.zeros((m.value, m.value), np.float32)
    assert mhdarcy.lib.mh_amg_coarsest(h, None, p(inv, C.c_float)) == 0
    return A, inv.astype(float)


def check_inverse(A, inv):
    """inv is the FP64 inverse rounded to FP32: |inv A - I| is at most 2^-24 m, m the largest row sum of
    |inv| |A|, and the elimination's own error, of the order of n eps m^2 (an SPD matrix: no growth)."""
    m = (np.abs(inv) @ np.abs(A)).sum(axis=1).max()
    assert np.abs(inv @ A - np.eye(len(A))).max() <= 2.0 ** -24 * m + len(A) * 2.0 ** -52 * m ** 2


@pytest.mark.gpu
@pytest.mark.parametrize("n", [170, 700, 1111, 2048, 2500, 3300, 3900, 4200])
def test_inverse_of_a_chain_level(gpu, monkeypatch, n):
    """One coarsening of a chain, so that the rows of the dense level follow n (about 0.32 n) over its
    32-row blocks and 64-row tiles to both sides of the limit."""
    monkeypatch.setenv("MH_AMG_LEVELS", "2")
    i = np.arange(n)
    rng = np.random.default_rng(n)
    w = 0.2 + rng.random(n - 1)
    d = 0.5 + rng.random(n)
    d[:-1] += w
    d[1:] += w
    r, c = np.concatenate([i, i[1:], i[:-1]]), np.concatenate([i, i[:-1], i[1:]])
    with Csr(r, c, np.concatenate([d, -w, -w]), rng.normal(size=n)) as s:
        rc, st, res = s.solve(r_tol=1e-12)
        assert rc == 0 and res <= 1e-12
        A, inv = coarsest(s.h)
        print("rows", len(A), "iterations", st["iterations"])
        assert (inv is not None) == (len(A) <= 1280)
        if inv is not None:
            check_inverse(A, inv)


@pytest.mark.gpu
@pytest.mark.parametrize("cfg,n", [(1, 16), (2, 21), (5, 32), (2, 47)])
def test_inverse_of_a_mesh_level(gpu, cfg, n):
    mesh, coeffs = make_case(cfg, seed=3, n=n)
    with mhdarcy.MHSystem(mesh) as s:
        bc, _ = dirichlet_x_bc(s.topology(), mesh)
        s.set_coeffs(**coeffs)
        s.set_bc(bc["bc_type"], bc["pressure"])
        s.assemble()
        with pytest.raises(mhdarcy.MHError):
            s.amg_coarsest()
        assert s.solve(method=_lib.MH_SOLVER_AMG, r_tol=1e-12)["status"] == 0
        A, inv = coarsest(s.h)
        assert inv is not None and np.array_equal(s.amg_coarsest(), inv.astype(np.float32))
        piv = np.linalg.cholesky(A).diagonal() ** 2 / A.diagonal()
        print("rows", len(A), "smallest pivot over its diagonal", piv.min())
        check_inverse(A, inv)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(12, 13, 14), (21, 22, 20), (40, 41, 43)])
@pytest.mark.parametrize("shift", [0.0, 1e-11])
def test_level_that_is_not_definite_in_fp32(gpu, shape, shift):
    """A diffusion operator without a Dirichlet boundary, alone or with a shift far below FP32 rounding
    (consistent: the right-hand side sums to zero).  The last pivot of its coarsest matrix is
    rounding; at these sizes it comes out negative or below the rounding of the diagonal: the level gets a
    polynomial and the solve converges without a fallback of the method."""
    nx, ny, nz = shape
    n = nx * ny * nz
    rng = np.random.default_rng(n)
    idx = np.arange(n).reshape(shape)
    r, c, v, d = [], [], [], np.zeros(n)
    for ax in range(3):
        a, b = np.take(idx, range(shape[ax] - 1), ax).ravel(), np.take(idx, range(1, shape[ax]), ax).ravel()
        w = 10.0 ** rng.uniform(-0.5, 0.5, len(a))
        r += [a, b]
        c += [b, a]
        v += [-w, -w]
        d += np.bincount(a, weights=w, minlength=n) + np.bincount(b, weights=w, minlength=n)
    i = np.arange(n)
    rhs = rng.normal(size=n)
    rhs -= rhs.mean()
    with Csr(np.concatenate(r + [i]), np.concatenate(c + [i]), np.concatenate(v + [d * (1 + shift)]), rhs) as s:
        rc, st, res = s.solve(r_tol=1e-9)
        A, inv = coarsest(s.h)
        print("rows", len(A), "iterations", st["iterations"], "residual", res)
        assert 160 < len(A) <= 1280 and inv is None
        assert rc == 0 and st["fell_back"] == 0 and res <= 1.01e-9
