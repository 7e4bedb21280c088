"""Node pressures against the oracle bit for bit where the blocks of 16 nodes can go wrong: ragged
last blocks, nodes of many elements (the serial path of a block whose terms do not fit), and lines,
triangles and tetrahedra side by side."""
import numpy as np
import pytest

import mhdarcy
import oracle as O
from helpers import oracle_problem
from mhdarcy.cases import dirichlet_x_bc, make_case
from mhdarcy.mesh import Mesh


def check(mesh, coeffs, bc_of):
    with mhdarcy.MHSystem(mesh) as s:
        topo = s.topology()
        bc = bc_of(topo)
        s.set_coeffs(**coeffs)
        s.set_bc(bc["bc_type"], bc["pressure"])
        s.assemble()
        s.solve(r_tol=1e-10)
        ref = O.node_pressure(oracle_problem(mesh, topo, s.n_edges, coeffs, bc), s.solution())
        assert np.array_equal(s.node_pressure(), ref)


@pytest.mark.gpu
@pytest.mark.parametrize("cfg,n", [(1, 2), (1, 3), (2, 7), (5, 16)])
def test_cubes(gpu, cfg, n):
    mesh, coeffs = make_case(cfg, seed=5, n=n)
    mesh.nodes[:] = mesh.nodes + 0.3 / n * np.random.default_rng(1).normal(size=mesh.nodes.shape) * (
        (mesh.nodes > 1e-9) & (mesh.nodes < 1.0 - 1e-9))  # no two distances alike
    check(mesh, coeffs, lambda t: dirichlet_x_bc(t, mesh)[0])


@pytest.mark.gpu
@pytest.mark.parametrize("rays", [30, 625, 626, 2500])
def test_star_of_lines(gpu, rays):
    """One node in `rays` elements: the centre and the first 15 outer nodes share a block of
    at most 640 pairs, so 625 rays are the last that fit."""
    a = np.linspace(0.0, 6.0, rays)
    nodes = np.concatenate([[[0.5, 0.5, 0.0]], np.stack([0.5 + 0.4 * np.cos(a), 0.5 + 0.4 * np.sin(a),
                                                          np.linspace(0.1, 0.9, rays)], 1)])
    el = np.stack([np.zeros(rays, int), np.arange(1, rays + 1), np.full(rays, -1), np.full(rays, -1)], 1)
    mesh = Mesh(nodes, np.ones(rays, np.int32), el)
    coeffs = dict(conductivity=np.random.default_rng(2).uniform(0.5, 2.0, rays), cross_section=np.full(rays, 0.1))

    def bc(topo):
        nb = len(topo["bdr_edge"])
        return dict(bc_type=np.ones(nb, np.int32), pressure=np.random.default_rng(3).normal(size=nb))

    check(mesh, coeffs, bc)
