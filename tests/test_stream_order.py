"""A handle's stream does not wait for the legacy stream: whatever a new handle lays down on the device
(zeroed vectors, the CSR pattern's padding, the exchange buffers of the resident Krylov run) goes
through the handle's own stream, and what is launched next finds it there."""
import ctypes as C
import glob
import os
import re

import numpy as np
import pytest

import mhdarcy
from mhdarcy import _lib

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "svn-export_b200", "csrc")


def test_no_call_on_the_legacy_stream():
    bad = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.c*"))):
        for no, line in enumerate(open(path), 1):
            if re.search(r"\bcudaMem(set|cpy)(2D|3D)?\(", line.split("//")[0]):
                bad.append("%s:%d" % (os.path.basename(path), no))
    assert not bad


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 131072, 1048576])
def test_first_values_of_a_new_csr_handle(gpu, n):
    """Sizes with and without padding rows (multiples of 1024 have none).  A chain with diagonal 4 and
    off-diagonals -1: condition below 3, so CG to 1e-13 leaves an error below 3e-13."""
    rng = np.random.default_rng(n)
    i = np.arange(n)
    r = np.concatenate([i, i[1:], i[:-1]])
    c = np.concatenate([i, i[:-1], i[1:]])
    v = np.concatenate([np.full(n, 4.0), np.full(2 * (n - 1), -1.0)])
    o = np.lexsort((c, r))
    rp = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32)
    col, val = c[o].astype(np.int32), v[o].copy()
    x = rng.normal(size=n)
    rhs = np.bincount(r[o], weights=val * x[col], minlength=n)
    p = lambda a, t: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
    for method in (_lib.MH_SOLVER_PCG64, _lib.MH_SOLVER_IR32) + ((_lib.MH_SOLVER_AMG,) if n > 1 else ()):
        h, st, got = C.c_void_p(), _lib.SolveStats(), np.zeros(n)
        opts = mhdarcy.solve_opts(method=method, r_tol=1e-13)
        assert mhdarcy.lib.mh_csr_create(n, p(rp, C.c_int32), p(col, C.c_int32), C.byref(h)) == 0
        try:
            assert mhdarcy.lib.mh_csr_set_values(h, p(val, C.c_double), p(rhs, C.c_double)) == 0
            rp2, col2, val2, rhs2 = np.zeros_like(rp), np.zeros_like(col), np.zeros_like(val), np.zeros_like(rhs)
            assert mhdarcy.lib.mh_get_schur_system(h, p(rp2, C.c_int32), p(col2, C.c_int32), p(val2, C.c_double),
                                                   p(rhs2, C.c_double)) == 0
            assert np.array_equal(rp2, rp) and np.array_equal(col2, col)
            assert np.array_equal(val2, val) and np.array_equal(rhs2, rhs)
            assert mhdarcy.lib.mh_solve(h, C.byref(opts), C.byref(st)) == 0
            assert mhdarcy.lib.mh_csr_get_solution(h, p(got, C.c_double), n) == 0
        finally:
            mhdarcy.lib.mh_destroy(h)
        assert np.linalg.norm(got - x) <= 3e-13 * np.linalg.norm(x)
