"""Timed cases of the accelerated path: operator assembly, matrix products, CG
solves, batched solves and the Total Lagrangian operators, each through the
public API (`stiffnessMatrix`, `massMatrix`, `heatConductionMatrix`,
`SystemMatrix * x`, `solveDisplacement`, `solveTemperature`,
`solveFieldBatched`, `deformationGradient`, `internalForceVector`,
`tangentMatrix`).

A case is a dict of plain values.  `kind` says what one pass does:

  csc       assemble K and take the SparseMatrixCSC arrays to the host (what a
            caller of the reference's stiffnessMatrix receives)
  product   assemble an operator on a kept mesh and pattern and apply it to a
            vector (the residual K u, M a or K_T T of a time or Newton step)
  analysis  a whole linear analysis from the mesh arrays: upload, pattern, K,
            load vector, the default solve (relative residual 1e-13)
  heat      steady heat conduction on a kept mesh: K_T, load, Jacobi-CG to
            1e-10 with random temperatures on two faces
  batched   many independent clamped bodies: one assembly and one IC(0)-CG to
            1e-10 over all of them
  tl        one Newton iteration of a hyperelastic body without its linear
            solve: F = I + grad u, internal force, consistent tangent and the
            tangent times an increment

`nx, ny, nz` are the cells per edge (a simplex mesh splits a cell into 2
triangles or 6 tetrahedra); `shape` is "box" (edges on the axes), "turned"
(the box rotated) or "curved" (every node moved smoothly, so that no element
is an affine image of the reference element).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from __graft_entry__ import load_package

DIM = {"quad": 2, "tri": 2, "hex": 3, "tet": 3}


def listed():
    return [
        # the smallest call: a test-sized model, matrix to the host; launches,
        # allocations and synchronisations count, not the work
        dict(name="csc_hex8_small", kind="csc", family="hex", order=1, nx=6, ny=6, nz=5, op="stiffness",
             shape="curved", precision="fp64"),
        # the headline workload: 3D Hooke K, hex27, 40^3 elements, 1.59 M DoFs
        dict(name="K_hex27_40", kind="product", family="hex", order=2, nx=40, ny=40, nz=40, op="stiffness",
             shape="box", precision="fp64"),
        # a body with curved elements (what a gmsh mesh of a real part has):
        # per-point quadrature instead of the affine form; ragged cell counts
        dict(name="K_hex27_curved", kind="product", family="hex", order=2, nx=19, ny=14, nz=17, op="stiffness",
             shape="curved", precision="fp64"),
        # tetrahedra of order 2, straight-sided, off the axes: the usual
        # automatic mesh (the batched workload's largest body, 2e5 elements)
        dict(name="K_tet10_turned", kind="product", family="tet", order=2, nx=33, ny=31, nz=29, op="stiffness",
             shape="turned", precision="fp64"),
        # scalar operator on first-order hexahedra: the reference's heat
        # benchmark shape (hex8), one entry per node pair
        dict(name="heat_hex8_64", kind="product", family="hex", order=1, nx=64, ny=64, nz=61, op="heat",
             shape="box", precision="fp64"),
        # the precision form (FP32 quadrature, FP64 sums) on a mid-size box
        dict(name="K_hex27_fp32", kind="product", family="hex", order=2, nx=25, ny=24, nz=23, op="stiffness",
             shape="box", precision="fp32"),
        # the 2D cantilever: 200x100 quad4, plane stress, whole analysis
        dict(name="analysis_quad4_200", kind="analysis", family="quad", order=1, nx=200, ny=100, nz=1),
        # the reference's published comparison: hex8 n=30 unit-cube-like body,
        # clamped left, traction right, pattern + K + solve
        dict(name="analysis_hex8_30", kind="analysis", family="hex", order=1, nx=30, ny=30, nz=30),
        # one request of the heat-serving stream, second-order tetrahedra
        dict(name="heat_solve_tet10", kind="heat", family="tet", order=2, nx=22, ny=23, nz=21),
        # a batch of uneven tet10 bodies (element counts log-uniform)
        dict(name="batched_tet10_8", kind="batched", family="tet", order=2, count=8, ne_min=1000, ne_max=60000),
        # the hyperelastic configuration's Newton iteration, first-order hex
        dict(name="tl_hex8_32", kind="tl", family="hex", order=1, nx=32, ny=31, nz=30, precision="fp64"),
        # its order-4 variant with the tangent on the tensor cores
        dict(name="tl_hex125_tc", kind="tl", family="hex", order=4, nx=9, ny=8, nz=8, precision="tf32x3"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _cells(rng, family, order, dofs_lo, dofs_hi, pdim):
    """Ragged cell counts for a log-uniform number of DoFs."""
    d = DIM[family]
    nodes = _log(rng, dofs_lo, dofs_hi) / pdim
    n = max(1.0, (nodes ** (1.0 / d) - 1.0) / order)
    c = [max(1, round(n * rng.uniform(0.75, 1.2))) for _ in range(d)]
    return dict(nx=c[0], ny=c[1], nz=c[2] if d == 3 else 1)


def draw(rng):
    kind = rng.choice(["csc", "product", "product", "product", "analysis", "heat", "batched", "tl"])
    if kind == "csc":
        family = rng.choice(["hex", "hex", "quad"])
        order = rng.choice([1, 2])
        return dict(kind=kind, family=family, order=order, op="stiffness", shape="curved", precision="fp64",
                    **_cells(rng, family, order, 300, 8000, DIM[family]))
    if kind == "product":
        family = rng.choice(["hex", "hex", "tet", "quad", "tri"])
        order = rng.choice([1, 2, 2, 3])
        op = rng.choice(["stiffness", "stiffness", "stiffness", "mass", "heat", "capacity"])
        pdim = DIM[family] if op in ("stiffness", "mass") else 1
        shape = rng.choice(["box", "turned", "curved"] if family in ("hex", "quad") else ["box", "turned"])
        top = 1.3e6 if shape != "curved" else 2.5e5
        case = dict(kind=kind, family=family, order=order, op=op, shape=shape,
                    precision=rng.choice(["fp64", "fp64", "fp64", "fp32"]))
        while True:
            case.update(_cells(rng, family, order, 1000, top, pdim))
            if _structural(case) * pdim ** 2 < 2.2e8:
                return case
    if kind == "analysis":
        family = rng.choice(["quad", "hex", "hex", "tet"])
        order = rng.choice([1, 1, 2])
        return dict(kind=kind, family=family, order=order,
                    **_cells(rng, family, order, 1000, 1e5, DIM[family]))
    if kind == "heat":
        family = rng.choice(["tri", "tet"])
        order = rng.choice([1, 2, 3, 4])
        return dict(kind=kind, family=family, order=order, **_cells(rng, family, order, 1000, 3e5, 1))
    if kind == "batched":
        return dict(kind=kind, family="tet", order=2, count=rng.randint(3, 12), ne_min=1000,
                    ne_max=int(_log(rng, 4000, 40000)))
    if rng.random() < 0.7:
        order = rng.choice([1, 1, 2])
        return dict(kind="tl", family="hex", order=order, precision="fp64",
                    **_cells(rng, "hex", order, 3000, 1.2e5 / order, 3))
    order = rng.choice([3, 4])
    return dict(kind="tl", family="hex", order=order, precision="tf32x3",
                **_cells(rng, "hex", order, 2000, 1.2e5, 3))


# ------------------------------------------------------------------ work
def _entities(case):
    """(mesh entity counts by dimension, ordered node pairs whose smallest
    common entity has that dimension) of one simplex mesh."""
    nx, ny, nz, p = case["nx"], case["ny"], case["nz"], case["order"]
    if case["family"] == "tri":
        count = [(nx + 1) * (ny + 1), nx * (ny + 1) + (nx + 1) * ny + nx * ny, 2 * nx * ny]
    else:
        v = (nx + 1) * (ny + 1) * (nz + 1)
        e = (nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
             + nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz)
        t = 6 * nx * ny * nz
        count = [v, e, 1 - v + e + t, t]
    pairs = []
    for d in range(len(count)):
        inside = math.comb(p + d, d) ** 2
        for k in range(d):
            inside -= math.comb(d + 1, k + 1) * pairs[k]
        pairs.append(inside)
    return count, pairs


def _structural(case):
    """Ordered node pairs that share an element."""
    p = case["order"]
    if case["family"] in ("hex", "quad"):
        n = [case["nx"], case["ny"]] + ([case["nz"]] if case["family"] == "hex" else [])
        return math.prod(c * (p + 1) ** 2 - (c - 1) for c in n)
    count, pairs = _entities(case)
    return sum(a * b for a, b in zip(count, pairs))


def _sizes(case):
    """(nodes, elements, nodes per element)."""
    p, d = case["order"], DIM[case["family"]]
    n = [case["nx"], case["ny"], case["nz"]][:d]
    nodes, cells = math.prod(p * c + 1 for c in n), math.prod(n)
    if case["family"] in ("hex", "quad"):
        return nodes, cells, (p + 1) ** d
    return nodes, cells * math.factorial(d), math.comb(p + d, d)


def _pdim(case):
    return 1 if case["kind"] == "heat" or case.get("op") in ("heat", "capacity") else DIM[case["family"]]


def work(case):
    """Each input read once, each output written once, the operator's values
    among them; the flops are the product's (one multiply-add per entry)."""
    if case["kind"] == "batched":
        bytes_ = flops = 0
        for m in _batch_sizes(case, np.random.default_rng(0)):
            w = work(dict(kind="analysis", family="tet", order=2, nx=m[0], ny=m[1], nz=m[2]))
            bytes_, flops = bytes_ + w["bytes"], flops + w["flops"]
        return {"bytes": bytes_, "flops": flops}
    pdim = _pdim(case)
    nodes, nel, npe = _sizes(case)
    nnz = _structural(case) * pdim * pdim
    bytes_ = 8 * nnz + 24 * nodes + 4 * npe * nel + 16 * pdim * nodes
    if case["kind"] == "csc":
        bytes_ += 8 * nnz + 8 * pdim * nodes     # the row indices and column pointers
    if case["kind"] == "tl":
        bytes_ += 8 * 3 * nodes                  # the force beside the product
    return {"bytes": bytes_, "flops": 2 * nnz}


# --------------------------------------------------------------- inputs
def _shape(case, rng, lattice):
    """Node coordinates from lattice coordinates (cells as the unit)."""
    d = DIM[case["family"]]
    size = np.ones(3)
    size[:d] = rng.uniform(0.5, 2.0, size=d)
    n = np.array([case["nx"], case["ny"], case["nz"]], dtype=float)
    x = lattice / n * size
    shape = case.get("shape", "box")
    if shape == "curved":
        y = x.copy()
        ph = rng.uniform(0.0, 2.0 * np.pi, size=(3, 3))
        for i in range(d):
            s = np.ones(len(x))
            for j in range(d):
                s = s * np.sin(2.0 * np.pi * lattice[:, j] / 5.3 + ph[i, j])
            y[:, i] += 0.08 * size[i] / n[i] * s
        x = y
    if shape in ("turned", "curved"):
        a = rng.uniform(0.2, 0.5, size=3)
        c, s = np.cos(a), np.sin(a)
        rot = np.array([[c[0], -s[0], 0.0], [s[0], c[0], 0.0], [0.0, 0.0, 1.0]])
        if d == 3:
            rot = rot @ np.array([[c[1], 0.0, s[1]], [0.0, 1.0, 0.0], [-s[1], 0.0, c[1]]])
            rot = rot @ np.array([[1.0, 0.0, 0.0], [0.0, c[2], -s[2]], [0.0, s[2], c[2]]])
        x = x @ rot.T
    return np.ascontiguousarray(x)


def _mesh(llf, case, rng):
    """(mesh, lattice coordinates of its nodes)."""
    simplex = case["family"] in ("tri", "tet")
    if DIM[case["family"]] == 2:
        m = llf.structured_rect_mesh(lx=float(case["nx"]), ly=float(case["ny"]), dx=1.0, dy=1.0,
                                     order=case["order"], simplex=simplex)
    else:
        m = llf.structured_box_mesh(lx=float(case["nx"]), ly=float(case["ny"]), lz=float(case["nz"]), dx=1.0,
                                    dy=1.0, order=case["order"], simplex=simplex)
    lattice = m.xyz
    m.xyz = _shape(case, rng, lattice)
    return m, lattice


def _type(case):
    if case["kind"] == "heat" or case.get("op") in ("heat", "capacity"):
        return "HeatConduction" if DIM[case["family"]] == 3 else "PlaneHeatConduction"
    return "Solid" if DIM[case["family"]] == 3 else "PlaneStress"


def _material(rng):
    """E, nu, conductivity, density and heat capacity of one body."""
    return dict(E=float(rng.uniform(1e4, 3e5)), nu=float(rng.uniform(0.2, 0.45)), k=float(np.exp(rng.normal())),
                rho=float(rng.uniform(1e-9, 1e-8)), c=float(rng.uniform(1e8, 1e9)))


def _batch_sizes(case, rng):
    """Cells per edge of every body; the counts are the same for every seed,
    so that the cost is the case's."""
    fixed = np.random.default_rng([case["count"], case["ne_max"]])
    out = []
    for _ in range(case["count"]):
        ne = math.exp(fixed.uniform(math.log(case["ne_min"]), math.log(case["ne_max"])))
        r = fixed.uniform(0.7, 1.4, size=3)
        n = (ne / 6.0 / np.prod(r)) ** (1.0 / 3.0)
        out.append(tuple(max(1, int(round(n * v))) for v in r))
    return out


def _inputs(case, seed):
    """Everything that the seed decides, as plain arrays beside the mesh."""
    llf = load_package()
    rng = np.random.default_rng(seed)
    if case["kind"] == "batched":
        parts, mats = [], []
        for nx, ny, nz in _batch_sizes(case, rng):
            parts.append(_mesh(llf, dict(kind="batched", family="tet", order=case["order"], nx=nx, ny=ny, nz=nz),
                               rng))
            mats.append(_material(rng))
        mesh, off = llf.concat_meshes([m for m, _ in parts])
        return dict(llf=llf, mesh=mesh, off=off, parts=parts, mats=mats, rng=rng)
    mesh, lattice = _mesh(llf, case, rng)
    return dict(llf=llf, mesh=mesh, lattice=lattice, mats=[_material(rng)], rng=rng)


def _smooth(rng, lattice, n, comps):
    """A smooth field with a little noise (displacements, temperatures)."""
    out = np.zeros((len(lattice), comps))
    for c in range(comps):
        k = rng.uniform(0.5, 3.0, size=3)
        ph = rng.uniform(0.0, 2.0 * np.pi, size=3)
        out[:, c] = np.prod(np.sin(k * lattice / n + ph), axis=1)
    return out + 0.02 * rng.standard_normal(out.shape)


def _vector(case, inp):
    n = np.array([case["nx"], case["ny"], case["nz"]], dtype=float)
    return _smooth(inp["rng"], inp["lattice"], n, _pdim(case)).reshape(-1)


def _tl_fields(case, inp):
    """Displacement (strains up to a few per cent) and a Newton increment."""
    n = np.array([case["nx"], case["ny"], case["nz"]], dtype=float)
    rng, X = inp["rng"], inp["mesh"].xyz
    A = 0.06 * rng.standard_normal((3, 3))
    h = float(np.min((X.max(axis=0) - X.min(axis=0)) / n)) / case["order"]
    u = X @ A.T + 0.01 * h * rng.standard_normal(X.shape)
    return u.reshape(-1), _smooth(rng, inp["lattice"], n, 3).reshape(-1)


TL = {"mu": 1.0, "lambda": 10.0}


def prepare(case, seed):
    inp = _inputs(case, seed)
    llf, mesh, rng, kind = inp["llf"], inp["mesh"], inp["rng"], case["kind"]
    st = dict(case=case, llf=llf, mesh=mesh)
    if kind == "batched":
        mats = [llf.Material(f"body#{i}", E=m["E"], nu=m["nu"]) for i, m in enumerate(inp["mats"])]
        P = llf.Problem(mats, type="Solid", mesh=mesh)
        P.pattern()
        st.update(P=P, off=inp["off"],
                  f=llf.loadVector(P, [llf.load(f"right#{i}", fx=1.0) for i in range(case["count"])]),
                  sup=[llf.displacementConstraint(f"left#{i}", ux=0, uy=0, uz=0) for i in range(case["count"])])
        return st
    mats = [llf.Material("body", **inp["mats"][0])]
    if kind == "analysis":
        d = DIM[case["family"]]
        st.update(mats=mats, type=_type(case), load=[llf.load("right", fx=float(rng.uniform(0.5, 2.0)))],
                  sup=[llf.displacementConstraint("left", ux=0, uy=0, uz=0 if d == 3 else None)])
        return st
    P = llf.Problem(mats, type=_type(case), mesh=mesh)
    P.pattern()
    st.update(P=P)
    if kind == "product":
        st.update(x=_vector(case, inp))
    elif kind == "heat":
        T = rng.uniform(0.0, 100.0, size=(mesh.non, 1))
        st.update(T=[llf.temperatureConstraint(g, T=llf.ScalarField(T, P)) for g in ("left", "right")])
    elif kind == "tl":
        u, du = _tl_fields(case, inp)
        st.update(u=llf.VectorField(u.reshape(-1, 1), P), du=du)
    return st


# ------------------------------------------------------------------ run
def _operator(st):
    llf, case, P = st["llf"], st["case"], st["P"]
    if case["op"] == "stiffness":
        return llf.stiffnessMatrix(P, precision=case["precision"])
    if case["op"] == "mass":
        return llf.massMatrix(P, lumped=False, precision=case["precision"])
    if case["op"] == "heat":
        return llf.heatConductionMatrix(P, precision=case["precision"])
    return llf.heatCapacityMatrix(P, precision=case["precision"])


def run(st):
    llf, case = st["llf"], st["case"]
    kind = case["kind"]
    if kind == "csc":
        colptr, rowval, nzval = _operator(st).csc()
        return {"colptr": colptr, "rowval": rowval, "nzval": nzval}
    if kind == "product":
        return _operator(st) * st["x"]
    if kind == "analysis":
        P = llf.Problem(st["mats"], type=st["type"], mesh=st["mesh"])
        return llf.solveDisplacement(P, load=st["load"], support=st["sup"]).a
    if kind == "heat":
        return llf.solveTemperature(st["P"], temperatureConstraint=st["T"], iterative=True, reltol=1e-10,
                                    preconditioner="jacobi").a
    if kind == "batched":
        K = llf.stiffnessMatrix(st["P"])
        return llf.solveFieldBatched(K, st["f"], support=st["sup"], node_offsets=st["off"], preconditioner="ic0",
                                     reltol=1e-10).a
    P = st["P"]
    F = llf.deformationGradient(st["u"])
    f = llf.internalForceVector(P, F=F, energy="NeoHookeCompressible", params=TL)
    K = llf.tangentMatrix(P, F, params=TL, precision=case["precision"])
    return {"force": f.a, "tangent_du": K * st["du"]}


# ---------------------------------------------------- the same in plain torch
def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda" if torch.cuda.is_available() else "cpu")


def _monomials(x, p, tensor, deriv=None):
    """Monomials of 2 x - 1 that span the element's polynomial space at points
    x (n, d) of [0,1]^d, or their derivative along one axis."""
    d = x.shape[1]
    exps = [e for e in np.ndindex(*([p + 1] * d)) if tensor or sum(e) <= p]
    y = 2.0 * x - 1.0
    cols = []
    for e in exps:
        c = np.ones(len(x))
        for j in range(d):
            if j == deriv:
                c = c * (2.0 * e[j] * y[:, j] ** (e[j] - 1) if e[j] else 0.0)
            else:
                c = c * y[:, j] ** e[j]
        cols.append(c)
    return np.stack(cols, axis=1)


def _gauss(n, d, verts=None):
    """Points and weights: tensor Gauss on [0,1]^d, or (vertices given) the
    collapsed rule of that simplex."""
    g, w = np.polynomial.legendre.leggauss(n)
    g, w = (g + 1.0) / 2.0, w / 2.0
    pts = np.stack([a.ravel() for a in np.meshgrid(*([g] * d), indexing="ij")], axis=1)
    wts = np.prod(np.stack([a.ravel() for a in np.meshgrid(*([w] * d), indexing="ij")], axis=1), axis=1)
    if verts is None:
        return pts, wts
    bary, left = [], np.ones(len(pts))
    for j in range(d):
        bary.append(left * pts[:, j])
        if j < d - 1:
            wts = wts * left * (1.0 - pts[:, j])
        left = left * (1.0 - pts[:, j])
    lam = np.stack(bary, axis=1)
    e = verts[1:] - verts[0]
    vol = abs(np.linalg.det(e)) if d > 1 else abs(e[0, 0])
    return verts[0] + lam @ e, wts * vol


class _Elements:
    """Shape functions, Jacobians and weights at the quadrature points of the
    elements of one kind (one congruent class of lattice elements)."""

    def __init__(self, xyz, lattice, conn, p, tensor, nq, dim):
        ref = lattice[conn[0]][:, :dim]
        ref = ref - np.floor(ref.min(axis=0) + 1e-9)
        V = np.linalg.inv(_monomials(ref, p, tensor))
        pts, w = _gauss(nq, dim, None if tensor else ref[: dim + 1])
        self.dim, self.conn = dim, _t(conn, torch.int64)
        self.N = _t(_monomials(pts, p, tensor) @ V)
        self.dN = _t(np.stack([_monomials(pts, p, tensor, j) @ V for j in range(dim)], axis=2))
        self.dNn = _t(np.stack([_monomials(ref, p, tensor, j) @ V for j in range(dim)], axis=2))
        self.X = _t(xyz[:, :dim])[self.conn]
        J = torch.einsum("eai,qaj->eqij", self.X, self.dN)
        self.inv = torch.linalg.inv(J)                         # d ref_i / d x_j
        self.w = torch.linalg.det(J).abs() * _t(w)

    def grad(self, u):
        """Physical gradients (e, q, comp, dim) of nodal values (n, comp)."""
        return torch.einsum("eac,qak->eqck", u[self.conn], self.dN) @ self.inv

    def scatter(self, out, s):
        """out += sum over points of s (e, q, comp, dim) : grad N."""
        r = s @ self.inv.transpose(-1, -2)
        out.index_add_(0, self.conn.reshape(-1), torch.einsum("eqck,qak->eac", r, self.dN).reshape(-1, s.shape[2]))


def _kinds(family):
    return {"hex": 1, "quad": 1, "tri": 2, "tet": 6}[family]


def _elements(case, mesh, lattice, nq=None):
    conn, T, p = mesh.conn - 1, _kinds(case["family"]), case["order"]
    return [_Elements(mesh.xyz, lattice, conn[t::T], p, case["family"] in ("hex", "quad"), nq or p + 1,
                      DIM[case["family"]]) for t in range(T)]


def _lame(case, m, dim):
    E, nu = m["E"], m["nu"]
    lam = E * nu / ((1 - nu) * (1 + nu)) if dim == 2 else E * nu / ((1 + nu) * (1 - 2 * nu))
    return lam, E / (2 * (1 + nu))


def _apply(blocks, op, u, coef):
    """The operator times u (n, comp): coef is (lam, mu) or one number, per
    block."""
    out = torch.zeros_like(u)
    for el, c in zip(blocks, coef):
        if op in ("mass", "capacity"):
            v = torch.einsum("eac,qa->eqc", u[el.conn], el.N) * (c * el.w)[..., None]
            out.index_add_(0, el.conn.reshape(-1), torch.einsum("eqc,qa->eac", v, el.N).reshape(-1, u.shape[1]))
            continue
        G = el.grad(u)
        if op == "heat":
            s = c * G
        else:
            tr = torch.einsum("eqii->eq", G)
            s = c[1] * (G + G.transpose(-1, -2))
            s = s + (c[0] * tr)[..., None, None] * torch.eye(el.dim, dtype=u.dtype, device=u.device)
        el.scatter(out, s * el.w[..., None, None])
    return out


def _stored(blocks, op, coef, shape):
    """The operator's stored matrix: sorted keys column * n + row and the
    values there."""
    n = shape[0] * shape[1]
    dev = blocks[0].w.device
    keys, vals = torch.zeros(0, dtype=torch.int64, device=dev), torch.zeros(0, dtype=torch.float64, device=dev)
    for el, c in zip(blocks, coef):
        e, k, d = len(el.conn), el.conn.shape[1], el.dim
        g = torch.einsum("qak,eqkj->eqaj", el.dN, el.inv)
        if op == "heat":
            g = g.transpose(2, 3).reshape(e, -1, k)
            K = g.transpose(1, 2) @ (g * (c * el.w).repeat_interleave(d, dim=1)[..., None])
        else:
            f = g.reshape(e, -1, k * d)
            O = (f.transpose(1, 2) @ (f * el.w[..., None])).reshape(e, k, d, k, d)
            tr = torch.einsum("eaibi->eab", O)
            K = c[0] * O + c[1] * O.transpose(2, 4) + c[1] * tr[:, :, None, :, None] * torch.eye(
                d, dtype=O.dtype, device=dev)[None, None, :, None, :]
        dof = (el.conn[:, :, None] * shape[1] + torch.arange(shape[1], device=dev)).reshape(e, -1)
        key = torch.cat([keys, (dof[:, None, :] * n + dof[:, :, None]).reshape(-1)])
        val = torch.cat([vals, K.reshape(-1)])
        keys, at = torch.unique(key, return_inverse=True)
        vals = torch.zeros(len(keys), dtype=torch.float64, device=dev).index_add_(0, at, val)
    return keys, vals


def _solve(blocks, op, coef, f, x0, free):
    """K u = f on the free entries (Jacobi-CG in 64 bits, restarted from the
    true residual until it stops falling)."""
    n = f.numel()
    keys, vals = _stored(blocks, op, coef, f.shape)
    rows = torch.bincount(keys // n, minlength=n)     # symmetric: columns as rows
    ptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=keys.device), rows.cumsum(0)])
    K = torch.sparse_csr_tensor(ptr, keys % n, vals, size=(n, n))
    d = vals[keys // n == keys % n]
    free, b, x = free.reshape(-1).to(f.dtype), f.reshape(-1), x0.reshape(-1).clone()
    d = free / d
    first = None
    for _ in range(4):
        r = free * (b - K @ x)
        start = float(r.norm())
        first = start if first is None else first
        if start <= 3e-16 * first:
            break
        z = d * r
        p, rho, step = z.clone(), torch.dot(r, z), torch.zeros_like(x)
        goal = 1e-14 * first if start > 1e-12 * first else 1e-2 * start
        for it in range(12000):
            q = free * (K @ p)
            a = rho / torch.dot(p, q)
            step += a * p
            r -= a * q
            if it % 25 == 24 and float(r.norm()) <= goal:
                break
            z = d * r
            new = torch.dot(r, z)
            p = z + (new / rho) * p
            rho = new
        x = x + step
    return x.reshape(f.shape)


def _traction(case, mesh, lattice, scale):
    """Consistent nodal loads of a traction along x on the face "right"."""
    d, T = DIM[case["family"]], _kinds(case["family"])
    conn = mesh.group("right").conn - 1
    tensor = case["family"] in ("hex", "quad")
    f = torch.zeros((mesh.non, d), dtype=torch.float64, device=_t([0.0]).device)
    T = 1 if tensor or d == 2 else 2
    for t in range(T):
        c = conn[t::T]
        ref = lattice[c[0]][:, 1:d]
        ref = ref - np.floor(ref.min(axis=0) + 1e-9)
        V = np.linalg.inv(_monomials(ref, case["order"], tensor or d == 2))
        pts, w = _gauss(case["order"] + 1, d - 1, None if tensor or d == 2 else ref[:d])
        dN = _t(np.stack([_monomials(pts, case["order"], tensor or d == 2, j) @ V for j in range(d - 1)], axis=2))
        J = torch.einsum("eai,qaj->eqij", _t(mesh.xyz[:, :d])[_t(c, torch.int64)], dN)
        area = torch.linalg.det(J.transpose(-1, -2) @ J).sqrt() * _t(w)
        v = torch.einsum("eq,qa->ea", area, _t(_monomials(pts, case["order"], tensor or d == 2) @ V)) * scale
        f[:, 0].index_add_(0, _t(c, torch.int64).reshape(-1), v.reshape(-1))
    return f


def _csc(case, inp):
    """The stored matrix: on these meshes no entry is zero, so every pair of
    DoFs that share an element is stored."""
    blocks = _elements(case, inp["mesh"], inp["lattice"])
    d = blocks[0].dim
    n = inp["mesh"].non * d
    keys, vals = _stored(blocks, "stiffness", [_lame(case, inp["mats"][0], d)], (inp["mesh"].non, d))
    cols = torch.bincount(keys // n, minlength=n)
    colptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=keys.device), cols.cumsum(0)]) + 1
    return {"colptr": colptr, "rowval": keys % n + 1, "nzval": vals}


def _tl(case, inp):
    mesh = inp["mesh"]
    u, du = (_t(v).reshape(-1, 3) for v in _tl_fields(case, inp))
    el = _elements(case, mesh, inp["lattice"])[0]
    eye = torch.eye(3, dtype=torch.float64, device=u.device)
    # nodal deformation gradients of every element, interpolated to the points
    Jn = torch.einsum("eai,baj->ebij", el.X, el.dNn)
    Fn = eye + torch.einsum("eac,bak->ebck", u[el.conn], el.dNn) @ torch.linalg.inv(Jn)
    F = torch.einsum("eaij,qa->eqij", Fn, el.N)
    Ft = F.transpose(-1, -2)
    Ci = torch.linalg.inv(Ft @ F)
    lnJ = torch.log(torch.linalg.det(F))[..., None, None]
    mu, lam = TL["mu"], TL["lambda"]
    S = mu * (eye - Ci) + lam * lnJ * Ci
    w = el.w[..., None, None]
    force, Kdu = torch.zeros_like(u), torch.zeros_like(u)
    el.scatter(force, F @ S * w)
    G = el.grad(du)
    dE = 0.5 * (Ft @ G + G.transpose(-1, -2) @ F)
    dS = lam * Ci * torch.einsum("eqij,eqij->eq", Ci, dE)[..., None, None] + 2.0 * (mu - lam * lnJ) * (Ci @ dE @ Ci)
    el.scatter(Kdu, (G @ S + F @ dS) * w)
    return {"force": force.reshape(-1, 1), "tangent_du": Kdu.reshape(-1)}


def exact(case, seed):
    inp = _inputs(case, seed)
    mesh, rng, kind = inp["mesh"], inp["rng"], case["kind"]
    d = DIM[case["family"]]
    if kind == "csc":
        return _csc(case, inp)
    if kind == "tl":
        return _tl(case, inp)
    if kind == "batched":
        blocks, coef, f, free = [], [], [], []
        for (m, lattice), mat, o in zip(inp["parts"], inp["mats"], inp["off"]):
            sub = dict(family="tet", order=case["order"])
            part = _elements(sub, m, lattice)
            for el in part:
                el.conn = el.conn + int(o)
            blocks += part
            coef += [_lame(sub, mat, 3)] * len(part)
            f.append(_traction(sub, m, lattice, 1.0))
            free.append(np.repeat(lattice[:, :1] > 0, 3, axis=1))
        f, free = torch.cat(f), _t(np.concatenate(free), torch.bool)
        return _solve(blocks, "stiffness", coef, f, torch.zeros_like(f), free).reshape(-1, 1)
    lattice, mat = inp["lattice"], inp["mats"][0]
    if kind == "analysis":
        blocks = _elements(case, mesh, lattice)
        f = _traction(case, mesh, lattice, float(rng.uniform(0.5, 2.0)))
        free = _t(np.repeat(lattice[:, :1] > 0, d, axis=1), torch.bool)
        return _solve(blocks, "stiffness", [_lame(case, mat, d)] * len(blocks), f, torch.zeros_like(f),
                      free).reshape(-1, 1)
    if kind == "heat":
        T = _t(rng.uniform(0.0, 100.0, size=(mesh.non, 1)))
        free = _t((lattice[:, :1] > 0) & (lattice[:, :1] < case["nx"]), torch.bool)
        blocks = _elements(case, mesh, lattice)
        x0 = torch.where(free, torch.zeros_like(T), T)
        return _solve(blocks, "heat", [mat["k"]] * len(blocks), torch.zeros_like(T), x0, free)
    op = case["op"]
    x = _t(_vector(case, inp)).reshape(mesh.non, -1)
    c = {"stiffness": _lame(case, mat, d), "mass": mat["rho"], "heat": mat["k"], "capacity": mat["c"] * mat["rho"]}[op]
    nq = case["order"] + (2 if op in ("mass", "capacity") and case["family"] in ("tri", "tet") else 1)
    blocks = _elements(case, mesh, lattice, nq)
    return _apply(blocks, op, x, [c] * len(blocks)).reshape(-1)
