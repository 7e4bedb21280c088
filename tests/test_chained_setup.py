"""Launches that overlap, elsewhere than in the multigrid iteration: the multigrid setup against the same
setup with every launch waited for (a child process under CUDA_LAUNCH_BLOCKING), bit for bit, and
the Chebyshev steps (always inside a graph) against a numpy restatement of a few iterations."""
import os
import subprocess
import sys

import numpy as np
import pytest
import scipy.sparse as sp

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "svn-export_b200"))  # (run by itself)

import mhdarcy  # noqa: E402
from mhdarcy import _lib  # noqa: E402
from mhdarcy.cases import dirichlet_x_bc, make_case  # noqa: E402

CASES = [(1, 3), (1, 9), (5, 18), (2, 33), (5, 44)]


def system(cfg, n):
    mesh, coeffs = make_case(cfg, seed=5, n=n)
    s = mhdarcy.MHSystem(mesh)
    bc, _ = dirichlet_x_bc(s.topology(), mesh)
    s.set_coeffs(**coeffs)
    s.set_bc(bc["bc_type"], bc["pressure"])
    s.assemble()
    return s


def hierarchy(cfg, n):
    """Every array of the hierarchy, its coarsest inverse and the solution after two iterations."""
    out = {}
    with system(cfg, n) as s:
        s.solve(method=_lib.MH_SOLVER_AMG, r_tol=1e-300, max_it=2)
        for level in range(s.amg_info()["levels"]):
            (rp, col, val), agg, weight = s.amg_level(level)
            for k, a in dict(rp=rp, col=col, val=val, agg=agg, weight=weight).items():
                if a is not None:
                    out["%s%d" % (k, level)] = a
        inv = s.amg_coarsest()
        if inv is not None:
            out["inv"] = inv
        out["x"] = s.solution()
    return out


@pytest.mark.gpu
def test_setup_gives_the_same_bits(gpu, tmp_path):
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1")
    subprocess.run([sys.executable, os.path.abspath(__file__), str(tmp_path)], env=env, check=True, timeout=300)
    for cfg, n in CASES:
        apart = np.load(os.path.join(str(tmp_path), "%d_%d.npz" % (cfg, n)))
        for _ in range(3):
            got = hierarchy(cfg, n)
            assert sorted(got) == sorted(apart.files)
            for k in got:
                assert np.array_equal(got[k], apart[k]), (cfg, n, k)


@pytest.mark.gpu
@pytest.mark.parametrize("degree", [1, 2, 5])
@pytest.mark.parametrize("cfg,n", [(1, 3), (1, 9), (2, 23)])
def test_chebyshev_steps(gpu, cfg, n, degree):
    """x after 4 iterations from zero: FP32 vectors, so 1e-5 of the largest entry (rounding of some 20
    products and updates with a spectrum of at most 2, with a decimal to spare); a step that read
    what the one before had not written yet would be off in the first decimal."""
    its, f = 4, np.float32
    with system(cfg, n) as s:
        rp, col, val, rhs = s.schur_system()
        st = s.solve(method=_lib.MH_SOLVER_CHEB, cheb_degree=degree, r_tol=1e-300, max_it=its, inner_max_it=its,
                     inner_rtol=1e-30)
        got = s.split(s.solution())[2]
        for _ in range(4):
            s.solve(method=_lib.MH_SOLVER_CHEB, cheb_degree=degree, r_tol=1e-300, max_it=its, inner_max_it=its,
                    inner_rtol=1e-30)
            assert np.array_equal(s.split(s.solution())[2], got)
    assert st["iterations"] == its
    m = len(rhs)
    S = sp.csr_matrix((val, col, rp), shape=(m, m))
    sc = 1.0 / np.sqrt(S.diagonal())
    A, b = sp.diags(sc) @ S @ sp.diags(sc), rhs * sc
    hi = float(abs(A.astype(f)).sum(axis=1).max())
    theta, delta = 0.5 * (hi + hi / 30.0), 0.5 * (hi - hi / 30.0)

    def precondition(r):
        rho, sigma = delta / theta, theta / delta
        z = d = r / theta
        for _ in range(degree - 1):
            new = 1.0 / (2.0 * sigma - rho)
            d = new * rho * d + 2.0 * new / delta * (r - A @ z)
            z, rho = z + d, new
        return z

    r, x, p, q, pq = b.copy(), np.zeros(m), None, None, 0.0
    for k in range(its):
        z = precondition(r)
        p = z if p is None else z - (z @ q) / pq * p
        q = A @ p
        pq = p @ q
        alpha = (p @ r) / pq
        x, r = x + alpha * p, r - alpha * q
    assert np.abs(got - x * sc).max() <= 1e-5 * np.abs(x * sc).max()


if __name__ == "__main__":
    for c, m in CASES:
        np.savez(os.path.join(sys.argv[1], "%d_%d.npz" % (c, m)), **hierarchy(c, m))
