"""The multigrid iteration's kernels overlap their launches (each waits for the one before by
itself).  With profile_kernels the same kernels are launched one after the other: both runs have to
give the same bits.  Sizes from one block per level to levels of more than one wave of blocks."""
import numpy as np
import pytest

import mhdarcy
from mhdarcy import _lib
from mhdarcy.cases import dirichlet_x_bc, make_case


@pytest.mark.gpu
@pytest.mark.parametrize("method", [_lib.MH_SOLVER_AMG, _lib.MH_SOLVER_FCG_LEARNED])
@pytest.mark.parametrize("cfg,n", [(1, 3), (1, 9), (5, 18), (2, 33), (5, 44)])
def test_overlap_gives_the_same_bits(gpu, cfg, n, method):
    mesh, coeffs = make_case(cfg, seed=5, n=n)
    with mhdarcy.MHSystem(mesh) as s:
        bc, _ = dirichlet_x_bc(s.topology(), mesh)
        s.set_coeffs(**coeffs)
        s.set_bc(bc["bc_type"], bc["pressure"])
        s.assemble()
        apart = s.solve(method=method, r_tol=1e-12, profile_kernels=True)
        xa = s.solution().copy()
        for host_loop in (False, True):
            st = s.solve(method=method, r_tol=1e-12, host_loop=host_loop)
            assert st["status"] == apart["status"] == 0
            assert st["iterations"] == apart["iterations"]
            assert np.array_equal(s.solution(), xa)
