"""The resident Krylov run gives up when an exchange does not complete within its bounded wait.  The
solve then goes back to the start of the run and on with the two-kernel iteration, which the handle
keeps.  MH_RESIDENT_POLLS shortens the wait to no or one poll of a value, so that it runs out."""
import numpy as np
import pytest

import mhdarcy
from mhdarcy import _lib
from mhdarcy.cases import dirichlet_x_bc, make_case


def system(n):
    mesh, coeffs = make_case(2, seed=3, n=n)
    s = mhdarcy.MHSystem(mesh)
    bc, _ = dirichlet_x_bc(s.topology(), mesh)
    s.set_coeffs(**coeffs)
    s.set_bc(bc["bc_type"], bc["pressure"])
    s.assemble()
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("method", [_lib.MH_SOLVER_PCG64, _lib.MH_SOLVER_IR32])
@pytest.mark.parametrize("n,polls", [(14, "0"), (14, "1"), (23, "0")])
def test_wait_that_runs_out(gpu, monkeypatch, n, polls, method):
    with system(n) as s:
        monkeypatch.setenv("MH_RESIDENT_POLLS", polls)
        st = s.solve(method=method, r_tol=1e-12)
        x = s.solution()
        assert st["status"] == 0 and max(st["rel_residual"], st["rel_residual_unscaled"]) <= 1e-12
        assert st["kernel_launches"] > 2 * st["iterations"]  # the two-kernel iteration
        monkeypatch.delenv("MH_RESIDENT_POLLS")
        kept = s.solve(method=method, r_tol=1e-12)
        assert kept["status"] == 0 and kept["kernel_launches"] > 2 * kept["iterations"]
        host = s.solve(method=method, r_tol=1e-12, host_loop=True)
        xh = s.solution()
        assert host["status"] == 0
        if method == _lib.MH_SOLVER_PCG64:  # from the same start, the same bits
            assert st["iterations"] == host["iterations"] and np.array_equal(x, xh)
        warm = s.solve(method=method, r_tol=1e-12, use_initial_guess=True)
        assert warm["status"] == 0
    with system(n) as s:
        assert s.solve(method=method, r_tol=1e-12)["kernel_launches"] < host["iterations"]


@pytest.mark.gpu
def test_wait_that_runs_out_from_a_guess(gpu, monkeypatch):
    """The run works on the solution vector in place: what it started from is there again."""
    with system(14) as s:
        s.solve(r_tol=1e-6, host_loop=True)
        host = s.solve(r_tol=1e-12, use_initial_guess=True, host_loop=True)
        xh = s.solution()
    with system(14) as s:
        s.solve(r_tol=1e-6, host_loop=True)
        monkeypatch.setenv("MH_RESIDENT_POLLS", "0")
        st = s.solve(r_tol=1e-12, use_initial_guess=True)
        assert st["iterations"] == host["iterations"] and np.array_equal(s.solution(), xh)


@pytest.mark.gpu
@pytest.mark.parametrize("polls", ["", "many", "-1", "99999999999"])
def test_only_a_smaller_number_shortens_the_wait(gpu, monkeypatch, polls):
    monkeypatch.setenv("MH_RESIDENT_POLLS", polls)
    with system(14) as s:
        st = s.solve(r_tol=1e-10)
        assert st["status"] == 0 and st["kernel_launches"] < st["iterations"]
