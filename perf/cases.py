"""The work that a user of this framework has it do, as cases that can be timed and compared.

A case names a kind of call and its sizes; prepare() makes what a program holds before the call
(mesh handle, coefficient and boundary data, network weights), run() is one pass through the
public entry points, and exact() computes the same outputs in 64 bits with plain numpy and torch.

Kinds:
  steady    assembly, Krylov solve and back-substitution of one mesh (the reference's
            update_solution).  The meshes and fields are the repository's benchmark
            configurations 1, 2, 3 and 5 at the case's cube size n.
  batch     the same for independent instances of uneven size in one handle (configuration 3)
  unsteady  implicit Euler steps with a boundary pressure that changes every step (configuration 4)
  csr       an SPD system that the caller assembles (the LinSys seam: mh_csr_*)
  outputs   post-processing of a solution: element flux vectors, the transport's convection
            matrix, node pressures

Solves run to r_tol 1e-15, where the pressures are settled to about 1e-11: a looser solve may
stop anywhere within its tolerance, and on these systems that is orders of magnitude wider.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "svn-export_b200"))

import mhdarcy  # noqa: E402
from mhdarcy.cases import dirichlet_x_bc, make_case  # noqa: E402

METHODS = {"pcg64": mhdarcy.MH_SOLVER_PCG64, "ir32": mhdarcy.MH_SOLVER_IR32, "cheb": mhdarcy.MH_SOLVER_CHEB,
           "learned": mhdarcy.MH_SOLVER_FCG_LEARNED, "amg": mhdarcy.MH_SOLVER_AMG}
R_TOL = 1e-15
DT = 0.01  # configuration 4's time step


def listed():
    return [
        # a small model in a calibration loop: new coefficients up, the default solver, solution down
        dict(name="steady n8 pcg64 host", kind="steady", cfg=1, n=8, method="pcg64", host=True, options=False),
        # the same loop with the multigrid at an odd size, with every input a model can carry:
        # anisotropy, sources, transition coefficients, Robin and Neumann boundaries
        dict(name="steady n21 amg host opts", kind="steady", cfg=2, n=21, method="amg", host=True, options=True),
        # configuration 1 with the default solver: the plain FP64 baseline users start from
        dict(name="steady n16 pcg64", kind="steady", cfg=1, n=16, method="pcg64", host=False, options=False),
        # configuration 1 with the multigrid: launches and latency decide
        dict(name="steady n16 amg", kind="steady", cfg=1, n=16, method="amg", host=False, options=False),
        # mixed precision without a preconditioner setup, odd size, correlated field
        dict(name="steady n35 ir32", kind="steady", cfg=2, n=35, method="ir32", host=False, options=False),
        # the fractured family at middle size with the learned smoother (network forward pass)
        dict(name="steady n32 learned", kind="steady", cfg=5, n=32, method="learned", host=False, options=False),
        # configuration 2, the standard large model
        dict(name="steady n64 amg", kind="steady", cfg=2, n=64, method="amg", host=False, options=False),
        # configuration 5, the largest: 5.3M tetrahedra, six fractures, four channels
        dict(name="steady n96 amg", kind="steady", cfg=5, n=96, method="amg", host=False, options=False),
        # an ensemble of realisations on meshes of uneven size, solved together
        dict(name="batch 24 amg", kind="batch", instances=24, sizes=3, method="amg"),
        # configuration 4: four steps of a tidal boundary, matrix fixed, right-hand side moving
        dict(name="unsteady n48 amg", kind="unsteady", n=48, steps=4, method="amg", lumped=False),
        # a finite-volume pressure system handed over as CSR by a caller with its own assembly
        dict(name="csr 61x57x53 amg", kind="csr", nx=61, ny=57, nz=53, method="amg"),
        # output stage after a solve of configuration 2
        dict(name="outputs n64", kind="outputs", cfg=2, n=64),
    ]


def draw(rng):
    known = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    case = _draw(rng)
    while case in known:
        case = _draw(rng)
    return case


def _draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["steady"] * 5 + ["batch", "unsteady", "csr", "outputs"])
    if kind == "steady":
        method = rng.choice(["pcg64", "ir32", "cheb", "learned", "amg", "amg", "amg"])
        top = {"pcg64": 40, "ir32": 40, "cheb": 32, "learned": 56, "amg": 72}[method]
        cfg = rng.choice([1, 2, 5])
        return dict(kind="steady", cfg=cfg, n=size(16 if cfg == 5 else 6, top), method=method,
                    host=rng.random() < 0.3, options=rng.random() < 0.3)
    if kind == "batch":
        return dict(kind="batch", instances=size(2, 24), sizes=rng.randrange(1000),
                    method=rng.choice(["pcg64", "amg", "amg"]))
    if kind == "unsteady":
        return dict(kind="unsteady", n=size(8, 48), steps=rng.randrange(1, 5), method=rng.choice(["pcg64", "amg", "amg"]),
                    lumped=rng.random() < 0.5)
    if kind == "csr":
        return dict(kind="csr", nx=size(9, 70), ny=size(9, 70), nz=size(9, 70), method=rng.choice(["pcg64", "amg"]))
    return dict(kind="outputs", cfg=rng.choice([1, 2]), n=size(8, 64))


# ---- inputs -------------------------------------------------------------------------------
def _mesh_case(case, seed):
    """Mesh, coefficient fields and per-side boundary data (geometric) of a mesh case."""
    if case["kind"] == "batch":
        sizes = np.random.default_rng(case["sizes"]).choice([8, 12, 16, 24, 32], case["instances"])
        parts = [make_case(3, seed=1000 * seed + i, n=int(n)) for i, n in enumerate(sizes)]
        coeffs = {k: np.concatenate([c[k] for _, c in parts]) for k in parts[0][1]}
        return [m for m, _ in parts], coeffs
    cfg = 4 if case["kind"] == "unsteady" else case["cfg"]
    mesh, coeffs = make_case(cfg, seed=seed, n=case["n"])
    if case.get("options"):
        rng = np.random.default_rng(seed + 1)
        ne = mesh.n_elements
        q = np.linalg.qr(rng.normal(size=(ne, 3, 3)))[0]
        coeffs["anisotropy"] = np.einsum("eij,ej,ekj->eik", q, 10.0 ** rng.uniform(-0.5, 0.5, (ne, 3)), q).reshape(ne, 9)
        coeffs["water_source_density"] = 1e-7 * rng.normal(size=ne)
        coeffs["sigma"] = 10.0 ** rng.uniform(-1.0, 1.0, ne)
    return [mesh], coeffs


def _bc(case, topo, mesh, p_left=1.0):
    """Boundary data per boundary object: Dirichlet on x = 0 and x = 1, no flow elsewhere; with
    options x = 1 is a Robin boundary and the other sides carry a Neumann flux."""
    bc, left = dirichlet_x_bc(topo, mesh, p_left=p_left)
    out = dict(bc_type=bc["bc_type"], pressure=bc["pressure"])
    if case.get("options"):
        typ = bc["bc_type"].copy()
        right = (typ == mhdarcy.MH_BC_DIRICHLET) & (bc["pressure"] == 0.0)
        none = typ == mhdarcy.MH_BC_NONE
        typ[right], typ[none] = mhdarcy.MH_BC_ROBIN, mhdarcy.MH_BC_NEUMANN
        out = dict(bc_type=typ, pressure=np.where(right, 0.25, bc["pressure"]), flux=np.where(none, 1e-8, 0.0),
                   robin_sigma=np.where(right, 1e-5, 0.0))
    return out, left


def _csr_case(case, seed):
    """7-point finite volumes on an nx x ny x nz box with log-normal cell conductivities
    (harmonic means on the faces), Dirichlet on both x ends: (row_ptr, col, val, rhs)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    k = 10.0 ** rng.normal(-6.0, 1.0, (nz, ny, nx))
    n = nx * ny * nz
    idx = np.arange(n).reshape(nz, ny, nx)
    diag = np.zeros((nz, ny, nx))
    rows, cols, vals = [], [], []
    for ax in range(3):
        a = [slice(None)] * 3
        b = [slice(None)] * 3
        a[ax], b[ax] = slice(0, -1), slice(1, None)
        a, b = tuple(a), tuple(b)
        t = 2.0 * k[a] * k[b] / (k[a] + k[b])
        diag[a] += t
        diag[b] += t
        rows += [idx[a].ravel(), idx[b].ravel()]
        cols += [idx[b].ravel(), idx[a].ravel()]
        vals += [-t.ravel(), -t.ravel()]
    rhs = np.zeros((nz, ny, nx))
    rhs[:, :, 0] = 2.0 * k[:, :, 0]
    diag[:, :, 0] += 2.0 * k[:, :, 0]
    diag[:, :, -1] += 2.0 * k[:, :, -1]
    rows.append(idx.ravel())
    cols.append(idx.ravel())
    vals.append(diag.ravel())
    r, c, v = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    o = np.lexsort((c, r))
    r, c, v = r[o], c[o], v[o]
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(r, minlength=n))
    return rp, c.astype(np.int32), np.ascontiguousarray(v), rhs.ravel().copy()


# ---- prepare and run ----------------------------------------------------------------------
def _f64p(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_double)) if isinstance(t, torch.Tensor) else t.ctypes.data_as(
        C.POINTER(C.c_double))


def _i32p(a):
    return a.ctypes.data_as(C.POINTER(C.c_int32))


def _ok(rc):
    if rc < 0:
        raise RuntimeError(f"call returned {rc}: {mhdarcy.lib.mh_status_string(rc)}")


class _Csr:
    """A handle of mh_csr_create, destroyed with the state."""

    def __init__(self, n, rp, col):
        self.h = C.c_void_p()
        _ok(mhdarcy.lib.mh_csr_create(n, _i32p(rp), _i32p(col), C.byref(self.h)))

    def __del__(self):
        if self.h:
            mhdarcy.lib.mh_destroy(self.h)
            self.h = None


def prepare(case, seed):
    kind = case["kind"]
    if kind == "csr":
        rp, col, val, rhs = _csr_case(case, seed)
        return dict(kind=kind, sys=_Csr(len(rhs), rp, col), val=val, rhs=rhs, x=np.zeros(len(rhs)),
                    opts=mhdarcy.solve_opts(method=METHODS[case["method"]], r_tol=R_TOL))
    meshes, coeffs = _mesh_case(case, seed)
    s = mhdarcy.MHSystem.batch(meshes) if kind == "batch" else mhdarcy.MHSystem(meshes[0])
    bc, left = _bc(case, s.topology(), s.mesh)
    st = dict(kind=kind, sys=s, coeffs=coeffs, bc=bc, left=left, host=bool(case.get("host")),
              solve=dict(method=METHODS[case.get("method", "amg")], r_tol=R_TOL))
    if not st["host"]:
        s.set_coeffs(**coeffs)
        s.set_bc(**bc)
        st["out"] = torch.empty(s.sizes.mh_size, dtype=torch.float64, device="cuda")
    if case.get("method") == "learned":  # weights as training leaves them: a moderate output layer
        w = s.learned_weights()
        w[-33:] = np.random.default_rng(seed).normal(scale=0.2, size=33)
        s.set_learned_weights(w)
    if kind == "unsteady":
        st.update(steps=case["steps"], lumped=case["lumped"], init=np.zeros(s.n_elements))
    if kind == "outputs":
        s.assemble()
        s.solve(**st["solve"])
        nnz = C.c_int64()
        _ok(mhdarcy.lib.mh_transport_matrix(s.h, None, C.byref(nnz), None, None, None, None))
        st["flux"] = torch.empty((s.n_elements, 3), dtype=torch.float64, device="cuda")
        st["por"] = torch.full((s.n_elements,), 0.3, dtype=torch.float64, device="cuda")
        st["tr"] = torch.empty(nnz.value, dtype=torch.float64, device="cuda")
    return st


def run(st):
    lib, s = mhdarcy.lib, st["sys"]
    kind = st["kind"]
    if kind == "csr":
        stats = mhdarcy._lib.SolveStats()
        _ok(lib.mh_csr_set_values(s.h, _f64p(st["val"]), _f64p(st["rhs"])))
        _ok(lib.mh_solve(s.h, C.byref(st["opts"]), C.byref(stats)))
        _ok(lib.mh_csr_get_solution(s.h, _f64p(st["x"]), len(st["x"])))
        return st["x"]
    if kind == "outputs":
        cfl = C.c_double()
        _ok(lib.mh_get_element_flux_device(s.h, _f64p(st["flux"]), st["flux"].numel()))
        _ok(lib.mh_transport_matrix_device(s.h, _f64p(st["por"]), _f64p(st["tr"]), st["tr"].numel(), C.byref(cfl)))
        return dict(flux=st["flux"], transport=st["tr"], cfl=cfl.value, node=s.node_pressure())
    if kind == "unsteady":
        s.unsteady_init(DT, st["init"], lumped=st["lumped"])
        for k in range(st["steps"]):
            p = st["bc"]["pressure"].copy()
            p[st["left"]] = 1.0 + 0.5 * math.sin(2.0 * math.pi * DT * (k + 1))
            s.set_bc(st["bc"]["bc_type"], p)
            s.unsteady_step(DT, **st["solve"])
    else:
        if st["host"]:
            s.set_coeffs(**st["coeffs"])
            s.set_bc(**st["bc"])
        s.assemble()
        s.solve(**st["solve"])
        if st["host"]:
            return s.solution()
    _ok(lib.mh_get_solution_device(s.h, _f64p(st["out"]), st["out"].numel()))
    return st["out"]


def work(case):
    """Bytes that a pass cannot do without: element data and boundary data in, the outputs out,
    and for a solve the FP64 edge system (values and column indices) written and read once."""
    kind = case["kind"]
    if kind == "csr":
        n = case["nx"] * case["ny"] * case["nz"]
        return dict(bytes=7 * n * 12 + 16 * n, flops=2 * 7 * n)
    if kind == "batch":
        tets = int(sum(6 * int(n) ** 3 for n in np.random.default_rng(case["sizes"]).choice(
            [8, 12, 16, 24, 32], case["instances"])))
    else:
        tets = 6 * case["n"] ** 3
    edges = 2.06 * tets
    if kind == "outputs":
        # per tetrahedron: nodes, side fluxes, coefficients and 24 bytes of flux; 5 matrix entries
        return dict(bytes=int(tets * (16 + 32 + 16 + 24 + 5 * 8 + 32)), flops=int(tets * 120))
    steps = case.get("steps", 1)
    per = tets * (16 + 24 + 16 + 32 + 8) + edges * (7 * 12 * 2 + 8 * 3)
    return dict(bytes=int(per * steps), flops=int(steps * (tets * 900 + edges * 14)))


# ---- the same in 64 bits, with plain numpy and torch --------------------------------------
_SIDES = {1: [[0], [1]], 2: [[0, 1], [1, 2], [0, 2]], 3: [[1, 2, 3], [0, 2, 3], [0, 1, 3], [0, 1, 2]]}
_OPP = {1: [1, 0], 2: [2, 0, 1], 3: [0, 1, 2, 3]}


def _number_edges(dim, nodes, n_nodes):
    """Edges in the order in which a walk over the elements' sides meets them: the coincident
    sides of one dimension share an edge, except that the sides around an element of one
    dimension less get an edge each.  Returns side offsets, edge of each side, whether a side
    is on the boundary, and (lower element, higher side) pairs."""
    ne = len(dim)
    start = np.concatenate([[0], np.cumsum(dim + 1)])
    ns = int(start[-1])
    key = np.zeros(ns, np.int64)
    sdim = np.zeros(ns, np.int64)
    base = n_nodes + 1
    ekey = {}
    for d in (1, 2, 3):
        el = np.nonzero(dim == d)[0]
        if len(el):
            srt = np.sort(nodes[el, :d + 1], axis=1)
            k = np.zeros(len(el), np.int64)
            for j in range(min(d + 1, 3)):
                k = k * base + srt[:, j] + 1
            if d < 3:
                ekey[d] = (k, el)
        for i in range(d + 1):
            if len(el):
                sn = np.sort(nodes[el][:, _SIDES[d][i]], axis=1)
                k = np.zeros(len(el), np.int64)
                for j in range(d):
                    k = k * base + sn[:, j] + 1
                key[start[el] + i] = k
                sdim[start[el] + i] = d
    edge = np.zeros(ns, np.int64)
    first_of, cnt_of, inv_of, low_of = [], [], np.zeros(ns, np.int64), []
    shift = 0
    for d in (1, 2, 3):
        sd = np.nonzero(sdim == d)[0]
        if not len(sd):
            continue
        u, fi, inv, cnt = np.unique(key[sd], return_index=True, return_inverse=True, return_counts=True)
        low = np.full(len(u), -1, np.int64)
        if d >= 2 and (d - 1) in ekey:
            lk, le = ekey[d - 1]
            pos = np.searchsorted(u, lk)
            pos = np.minimum(pos, len(u) - 1)
            hit = u[pos] == lk
            low[pos[hit]] = le[hit]
        first_of.append(sd[fi])
        cnt_of.append(cnt)
        low_of.append(low)
        inv_of[sd] = inv + shift
        shift += len(u)
    first, cnt, low = np.concatenate(first_of), np.concatenate(cnt_of), np.concatenate(low_of)
    order = np.argsort(first, kind="stable")
    n_of = np.where(low >= 0, cnt, 1)
    e0 = np.zeros(len(first), np.int64)
    e0[order] = np.concatenate([[0], np.cumsum(n_of[order])[:-1]])
    # rank of a side within its group, in side order
    so = np.argsort(inv_of, kind="stable")
    gstart = np.concatenate([[0], np.cumsum(cnt)])[:-1]
    rank = np.zeros(ns, np.int64)
    rank[so] = np.arange(ns) - gstart[inv_of[so]]
    split = low[inv_of] >= 0
    edge = e0[inv_of] + np.where(split, rank, 0)
    bdr = (cnt[inv_of] == 1) & ~split
    ngh_side = np.nonzero(split)[0]
    return start, edge, bdr, low[inv_of[ngh_side]], ngh_side, int(n_of.sum())


class _Plain:
    """The mixed-hybrid system of one mesh (or union) in 64 bits on the GPU."""

    def __init__(self, case, mesh, coeffs):
        dev = "cuda"
        self.case = case
        dim, nodes, xyz = np.asarray(mesh.el_dim), np.asarray(mesh.el_nodes), np.asarray(mesh.nodes)
        start, edge, bdr, ngh_el, ngh_side, self.n_edges = _number_edges(dim, nodes, len(xyz))
        self.ne, self.ns, self.start = len(dim), int(start[-1]), start
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        self.edge, X = t(edge), t(xyz)
        get = lambda k, v: t(coeffs[k]) if coeffs.get(k) is not None else torch.full((self.ne,), v, dtype=torch.float64, device=dev)  # noqa: E731
        K, self.delta = get("conductivity", 1.0), get("cross_section", 1.0)
        src, self.sto, sigma = get("water_source_density", 0.0), get("storativity", 1.0), get("sigma", 1.0)
        self.meas = torch.zeros(self.ne, dtype=torch.float64, device=dev)
        side_meas = torch.ones(self.ns, dtype=torch.float64, device=dev)
        self.g = torch.zeros(self.ns, dtype=torch.float64, device=dev)
        self.c = torch.ones(self.ns, dtype=torch.float64, device=dev)
        self.fdiag = torch.zeros(self.ns, dtype=torch.float64, device=dev)
        self.bedge = torch.zeros(self.ns, dtype=torch.float64, device=dev)
        left = torch.zeros(self.ns, dtype=torch.bool, device=dev)
        right = torch.zeros(self.ns, dtype=torch.bool, device=dev)
        self.parts = []
        for d in (1, 2, 3):
            el = np.nonzero(dim == d)[0]
            if not len(el):
                continue
            e, P = t(el), X[t(nodes[el, :d + 1].astype(np.int64))]
            v = P[:, 1:] - P[:, :1]
            m = torch.sqrt(torch.linalg.det(v @ v.transpose(1, 2))) / math.factorial(d)
            self.meas[e] = m
            cen = P.mean(1)
            q = P - cen[:, None]
            cov = torch.einsum("eki,ekj->eij", q, q) / ((d + 1) * (d + 2))
            R = torch.linalg.inv(get("anisotropy", 0.0)[e].reshape(-1, 3, 3)) if coeffs.get("anisotropy") is not None \
                else torch.eye(3, dtype=torch.float64, device=dev).expand(len(el), 3, 3)
            y = cen[:, None] - P[:, _OPP[d]]  # centre minus the node opposite each side
            A = torch.einsum("eia,eab,ejb->eij", y, R, y) + (R * cov).sum((1, 2))[:, None, None]
            A = A * (m / (d * m) ** 2 / K[e] / self.delta[e])[:, None, None]
            s = t(start[el])[:, None] + torch.arange(d + 1, device=dev)
            self.parts.append((d, e, s, torch.linalg.inv(0.5 * (A + A.transpose(1, 2))), y))
            for i in range(d + 1):
                S = P[:, _SIDES[d][i]]
                self.g[s[:, i]] = cen[:, 2] - S[:, :, 2].mean(1)
                if d == 2:
                    side_meas[s[:, i]] = (S[:, 1] - S[:, 0]).norm(dim=1)
                elif d == 3:
                    side_meas[s[:, i]] = 0.5 * torch.linalg.cross(S[:, 1] - S[:, 0], S[:, 2] - S[:, 0]).norm(dim=1)
                left[s[:, i]] = S[:, :, 0].max(1).values < 1e-12
                right[s[:, i]] = S[:, :, 0].min(1).values > 1.0 - 1e-12
        self.bdr, el_of_side = t(bdr), t(np.repeat(np.arange(self.ne), dim + 1))
        self.left, self.right = left & self.bdr, right & self.bdr
        self.sd = side_meas * self.delta[el_of_side]
        self.src = self.meas * self.delta * src
        self.n_el, self.n_side = t(ngh_el), t(ngh_side)
        self.n_v = sigma[self.n_el] * side_meas[self.n_side] * self.delta[el_of_side[self.n_side]]
        self.el_of_side = el_of_side
        self.bc(1.0)

    def bc(self, p_left):
        self.c.fill_(1.0)
        self.fdiag.zero_()
        self.bedge.zero_()
        self.gd = self.g.clone()
        dirichlet = self.left if self.case.get("options") else self.left | self.right
        p = torch.full_like(self.g, p_left).masked_fill_(~self.left, 0.0)
        self.c[dirichlet] = 0.0
        self.gd[dirichlet] -= p[dirichlet]
        self.bedge[dirichlet] -= p[dirichlet]
        self.fdiag[dirichlet] -= 1.0
        if self.case.get("options"):
            none = self.bdr & ~self.left & ~self.right
            self.bedge[none] += 1e-8 * self.sd[none]
            self.bedge[self.right] -= self.sd[self.right] * 1e-5 * 0.25
            self.fdiag[self.right] -= self.sd[self.right] * 1e-5

    def assemble(self, mode=0, prev_p=None, prev_l=None):
        """Both eliminations: the edge system (CSR) and its right-hand side."""
        self.mode = mode
        dEE, bE = torch.zeros_like(self.meas), -self.src.clone()
        fd, be = self.fdiag.clone(), self.bedge.clone()
        if mode == 1:
            tt = -self.sto * self.meas / DT
            dEE, bE = dEE + tt, bE + tt * prev_p
        if mode == 2:
            nsd = torch.as_tensor(np.diff(self.start), device="cuda").to(torch.float64)
            self.lmh = (self.meas * self.sto * self.delta / DT / nsd)[self.el_of_side]
            self.src_side = (-self.src / nsd)[self.el_of_side]
            fd, be = fd - self.lmh, be - self.lmh * prev_l[self.edge]
        dEE = dEE.index_add(0, self.n_el, -self.n_v)
        s1, r1e = -dEE, -bE
        u = torch.zeros_like(self.g)
        bo = -be
        rows, cols, vals = [], [], []
        for d, e, s, Ai, _ in self.parts:
            a1 = Ai.sum(2)
            ag = (Ai @ self.gd[s][:, :, None])[:, :, 0]
            s1[e] += a1.sum(1)
            r1e[e] -= ag.sum(1)
            u[s] = -self.c[s] * a1
            bo[s] += self.c[s] * ag
        for d, e, s, Ai, _ in self.parts:
            cs = self.c[s]
            B = cs[:, :, None] * Ai * cs[:, None, :] - u[s][:, :, None] * u[s][:, None, :] / s1[e][:, None, None]
            B = B + torch.diag_embed(-fd[s])
            ed = self.edge[s]
            rows.append(ed[:, :, None].expand_as(B).reshape(-1))
            cols.append(ed[:, None, :].expand_as(B).reshape(-1))
            vals.append(B.reshape(-1))
        rhs = torch.zeros(self.n_edges, dtype=torch.float64, device="cuda")
        rhs.index_add_(0, self.edge, bo - u * (r1e / s1)[self.el_of_side])
        if len(self.n_el):
            ne_, nv, nd = self.n_el, self.n_v, self.edge[self.n_side]
            rhs.index_add_(0, nd, nv * (r1e / s1)[ne_])
            # neighbour-neighbour and neighbour-own couplings of each lower element
            o = torch.argsort(ne_, stable=True)
            le, lv, ld = ne_[o], nv[o], nd[o]
            cnt = torch.bincount(le, minlength=self.ne)
            first = torch.cumsum(cnt, 0) - cnt
            for k in range(int(cnt.max())):
                ok = k < cnt[le]
                j = first[le[ok]] + k
                w = -lv[ok] * lv[j] / s1[le[ok]]
                w = w + torch.where(torch.nonzero(ok)[:, 0] == j, lv[ok], torch.zeros_like(w))
                rows.append(ld[ok]), cols.append(ld[j]), vals.append(w)
            st = torch.as_tensor(self.start, device="cuda")
            nsd = st[1:] - st[:-1]
            for i in range(3):
                ok = i < nsd[le]
                sd = st[le[ok]] + i
                w = lv[ok] * u[sd] / s1[le[ok]]
                rows += [ld[ok], self.edge[sd]]
                cols += [self.edge[sd], ld[ok]]
                vals += [w, w]
        n = self.n_edges
        i = torch.stack([torch.cat(rows), torch.cat(cols)])
        S = torch.sparse_coo_tensor(i, torch.cat(vals), (n, n)).coalesce()
        self.u, self.s1, self.r1e = u, s1, r1e
        return S, rhs

    def back(self, lam, prev_l=None):
        acc = self.r1e.index_add(0, self.el_of_side, -self.u * lam[self.edge])
        if len(self.n_el):
            acc = acc.index_add(0, self.n_el, self.n_v * lam[self.edge[self.n_side]])
        p = acc / self.s1
        q = torch.zeros(self.ns, dtype=torch.float64, device="cuda")
        for d, e, s, Ai, _ in self.parts:
            rhs = self.gd[s] + p[e][:, None] - self.c[s] * lam[self.edge[s]]
            q[s] = (Ai @ rhs[:, :, None])[:, :, 0]
        if self.mode == 2:
            q = q - self.lmh * (lam - prev_l)[self.edge] + self.src_side
        return torch.cat([q, p, lam])

    def flux(self, sol):
        out = torch.zeros((self.ne, 3), dtype=torch.float64, device="cuda")
        for d, e, s, _, y in self.parts:
            out[e] = (sol[s][:, :, None] * y).sum(1) / (d * self.meas[e] * self.delta[e])[:, None]
        return out


def _solve_spd(S, b):
    """Jacobi-preconditioned CG in 64 bits, restarted from the recomputed residual until that
    does not fall any more."""
    i, v = S.indices(), S.values()
    diag = torch.zeros_like(b)
    on = i[0] == i[1]
    diag[i[0][on]] = v[on]
    sc = diag.rsqrt()
    A = torch.sparse_coo_tensor(i, v * sc[i[0]] * sc[i[1]], S.shape, is_coalesced=True).to_sparse_csr()
    bh = b * sc
    x = torch.zeros_like(b)
    best = math.inf
    for _ in range(8):
        r = bh - A @ x
        rr = torch.dot(r, r)
        now = math.sqrt(float(rr)) / float(bh.norm())
        if now < 1e-17 or now > 0.5 * best:
            break
        best = now
        p, d, stop = r.clone(), torch.zeros_like(b), float(rr) * 1e-18
        for it in range(40000):
            q = A @ p
            a = rr / torch.dot(p, q)
            d += a * p
            r -= a * q
            new = torch.dot(r, r)
            p.mul_(new / rr).add_(r)
            rr = new
            if it % 64 == 63 and float(rr) <= stop:
                break
        x += d
    return x * sc


def exact(case, seed):
    kind = case["kind"]
    if kind == "csr":
        rp, col, val, rhs = _csr_case(case, seed)
        rows = np.repeat(np.arange(len(rhs)), np.diff(rp))
        S = torch.sparse_coo_tensor(torch.as_tensor(np.stack([rows, col.astype(np.int64)])), torch.as_tensor(val),
                                    (len(rhs), len(rhs))).cuda().coalesce()
        return _solve_spd(S, torch.as_tensor(rhs).cuda())
    if kind != "batch" and case["n"] > 72:
        return None  # over 20 seconds
    meshes, coeffs = _mesh_case(case, seed)
    P = _Plain(case, mhdarcy.concat_meshes(meshes) if len(meshes) > 1 else meshes[0], coeffs)
    if kind == "unsteady":
        mode = 2 if case["lumped"] else 1
        sol = torch.zeros(P.ns + P.ne + P.n_edges, dtype=torch.float64, device="cuda")
        for k in range(case["steps"]):
            prev_p, prev_l = sol[P.ns:P.ns + P.ne], sol[P.ns + P.ne:]
            P.bc(1.0 + 0.5 * math.sin(2.0 * math.pi * DT * (k + 1)))
            sol = P.back(_solve_spd(*P.assemble(mode, prev_p, prev_l)), prev_l)
        return sol
    sol = P.back(_solve_spd(*P.assemble()))
    if kind == "outputs":
        return dict(flux=P.flux(sol), transport=None, cfl=None, node=None)
    return sol
