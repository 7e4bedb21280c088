"""A multigrid solve to a tolerance of the order of FP64 rounding (r_tol 1e-15): flux vectors, which
are differences of the pressures, agree with those of a solve two decimals further to 4e-8 of the
larger of the value and the RMS, what the output stage's FP64 results are held to.  The seeds
are ones whose last segment ends just under r_tol.  Looser solves end where they did."""
import numpy as np
import pytest

import mhdarcy
from mhdarcy import _lib
from mhdarcy.cases import dirichlet_x_bc, make_case


def system(cfg, n, seed):
    mesh, coeffs = make_case(cfg, seed=seed, n=n)
    s = mhdarcy.MHSystem(mesh)
    bc, _ = dirichlet_x_bc(s.topology(), mesh)
    s.set_coeffs(**coeffs)
    s.set_bc(bc["bc_type"], bc["pressure"])
    s.assemble()
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("seed", [15, 22])
def test_flux_of_a_solve_to_rounding(gpu, seed):
    with system(2, 64, seed) as s:
        st = s.solve(method=_lib.MH_SOLVER_AMG, r_tol=1e-15)
        assert st["status"] == 0 and max(st["rel_residual"], st["rel_residual_unscaled"]) <= 1e-15
        flux = s.element_flux()
        s.solve(method=_lib.MH_SOLVER_AMG, r_tol=1e-17)
        ref = s.element_flux()
    scale = np.maximum(np.sqrt(np.mean(ref ** 2)), np.abs(ref))
    assert (np.abs(flux - ref) / scale).max() <= 4e-8


@pytest.mark.gpu
@pytest.mark.parametrize("method", [_lib.MH_SOLVER_AMG, _lib.MH_SOLVER_FCG_LEARNED])
@pytest.mark.parametrize("cfg,n", [(1, 3), (2, 13), (5, 18)])
def test_never_worse_than_the_tolerance(gpu, cfg, n, method):
    """At and below the line the solve still succeeds, within max_it, whatever the last segment did."""
    with system(cfg, n, 7) as s:
        for r_tol in (1.7e-15, 1e-15, 3e-16):
            st = s.solve(method=method, r_tol=r_tol)
            assert st["status"] == 0 and max(st["rel_residual"], st["rel_residual_unscaled"]) <= r_tol
            again = s.solve(method=method, r_tol=r_tol, max_it=st["iterations"])
            assert again["iterations"] <= st["iterations"] and again["status"] == 0
            warm = s.solve(method=method, r_tol=r_tol, use_initial_guess=True)
            assert warm["status"] == 0 and warm["iterations"] <= st["iterations"]
