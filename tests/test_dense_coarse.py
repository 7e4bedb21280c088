"""The dense inverse of the multigrid's coarsest level (block Gauss-Jordan, up to 1280 rows) at
sizes on and off its 32-row blocks and 64-row tiles.  The coarse solve is exact, so the cycle is at
least as good a preconditioner as with the next levels' cycles in its place (MH_AMG_COARSE=160);
a wrong entry of the inverse would make it a poor or an indefinite one.  Iterations are compared
with a quarter to spare, since a segment of the solve ends at a fixed reduction."""
import numpy as np
import pytest

import mhdarcy
from mhdarcy import _lib
from mhdarcy.cases import dirichlet_x_bc, make_case


@pytest.mark.gpu
@pytest.mark.parametrize("cfg,n,seed", [(1, 5, 3), (1, 6, 3), (1, 7, 3), (1, 8, 3), (2, 11, 3), (1, 16, 3), (2, 19, 3),
                                        (2, 21, 3), (5, 32, 5), (2, 47, 3)])
def test_dense_coarsest_level(gpu, monkeypatch, cfg, n, seed):
    mesh, coeffs = make_case(cfg, seed=seed, n=n)
    with mhdarcy.MHSystem(mesh) as s:
        bc, _ = dirichlet_x_bc(s.topology(), mesh)
        s.set_coeffs(**coeffs)
        s.set_bc(bc["bc_type"], bc["pressure"])
        out = {}
        for coarse in (160, 1280):
            monkeypatch.setenv("MH_AMG_COARSE", str(coarse))
            s.assemble()
            st = s.solve(method=_lib.MH_SOLVER_AMG, r_tol=1e-12)
            assert st["status"] == 0 and st["fell_back"] == 0
            out[coarse] = (st["iterations"], s.amg_info(), s.solution())
        assert out[1280][1]["rows"][-1] <= 1280
        assert out[1280][0] <= 1.25 * out[160][0], out
        print("coarsest", out[160][1]["rows"][-1], "->", out[1280][1]["rows"][-1], "iterations", out[160][0], "->",
              out[1280][0])
