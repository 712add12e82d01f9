"""Kernels that take several small elements per CTA, at element counts that
leave a partly filled CTA, against the oracle bit for bit."""
import numpy as np
import pytest

from helpers import assert_csc_identical

pytestmark = pytest.mark.gpu

PRM = {"mu": 1.0, "lambda": 10.0}
# nx, ny, nz, order, simplex
TL_CASES = {"hex8-1": (1, 1, 1, 1, False), "hex8-27": (3, 3, 3, 1, False), "hex8-35": (5, 7, 1, 1, False),
            "tet4-18": (3, 1, 1, 1, True), "tet10-30": (5, 1, 1, 2, True), "hex27-3": (3, 1, 1, 2, False)}


def _box(llf, nx, ny, nz, order, simplex):
    m = llf.structured_box_mesh(lx=float(nx), ly=float(ny), lz=float(nz), dx=1.0, dy=1.0, order=order, simplex=simplex)
    m.xyz = m.xyz + 0.02 * np.random.default_rng(7).standard_normal(m.xyz.shape)
    return m


@pytest.mark.parametrize("masked", [False, True], ids=["all", "part"])
@pytest.mark.parametrize("case", TL_CASES.values(), ids=TL_CASES.keys())
def test_tl_operators_bit_identical(llf, orc, case, masked):
    m = _box(llf, *case)
    sel = np.arange(m.nel)
    if masked:   # every third element outside the problem's material
        sel = sel[sel % 3 != 1]
        m.groups["part"] = llf.Group("part", 3, np.unique(m.conn[sel]), m.family, m.order, m.conn[sel], sel)
    p = llf.Problem([llf.Material("part" if masked else "body")], type="Solid", mesh=m)
    u = llf.VectorField(0.02 * np.random.default_rng(11).standard_normal((3 * m.non, 1)), p)
    F = llf.grad(u, add_identity=True)
    rule = llf._lib.builtin_rule(m.family, m.order)
    conn, T = m.conn[sel], F.A[sel]
    law = dict(energy="NeoHookeCompressible", params=PRM)
    got = {0: llf.materialTangentMatrix(p, F=F, **law), 1: llf.initialStressMatrix(p, S=F),
           2: llf.initialStressMatrix(p, C=llf.TensorField(_cauchy_green(F.A, m), p), **law),
           3: llf.tangentMatrix(p, F, **law)}
    for mode, K in got.items():
        Tm = _cauchy_green(F.A, m)[sel] if mode == 2 else T
        ref = orc.tl_matrix(mode, m.xyz, conn, rule, Tm, orc.LAW_NEOHOOKE, [1.0, 10.0])
        assert_csc_identical(K.csc(), ref.julia(), f"mode {mode}")
    if not masked:
        f = llf.internalForceVector(p, F=F, **law)
        assert np.array_equal(f.a[:, 0], orc.tl_internal_force(0, m.xyz, conn, rule, T, orc.LAW_NEOHOOKE, [1.0, 10.0]))
        fp = llf.internalForceVector(p, P=F)
        assert np.array_equal(fp.a[:, 0], orc.tl_internal_force(1, m.xyz, conn, rule, T))


def _cauchy_green(A, m):
    Fm = np.swapaxes(A.reshape(m.nel, m.npe, 3, 3), -1, -2)
    C = np.einsum("eaki,eakj->eaij", Fm, Fm)
    return np.ascontiguousarray(np.swapaxes(C, -1, -2).reshape(m.nel, 9 * m.npe))


# cells, order, simplex: element counts that give every CTA its full number of
# elements on the GPU's SMs and leave the last one partly filled
ASM_CASES = {"hex8": ((11, 10, 11), 1, False), "tet4": ((8, 7, 7), 1, True), "tet10": ((5, 4, 5), 2, True),
             "quad4": ((49, 47), 1, False), "tri3": ((61, 59), 1, True), "tri6": ((29, 29), 2, True),
             "quad9": ((28, 28), 2, False), "hex27": ((7, 7, 7), 2, False), "tet20": ((4, 4, 5), 3, True),
             "quad25": ((18, 18), 4, False),
             # beyond the packed kernel, with a CTA per column node in the gather
             "hex64": ((3, 2, 2), 3, False), "hex125": ((2, 1, 2), 4, False), "tet35": ((2, 2, 1), 4, True)}


def _shaped(llf, cells, order, simplex, shape):
    if len(cells) == 3:
        m = llf.structured_box_mesh(lx=float(cells[0]), ly=float(cells[1]), lz=float(cells[2]), dx=1.0, dy=1.0,
                                    order=order, simplex=simplex)
    else:
        m = llf.structured_rect_mesh(lx=float(cells[0]), ly=float(cells[1]), dx=1.0, dy=1.0, order=order,
                                     simplex=simplex)
    x = m.xyz.copy()
    if "curved" in shape:   # the nodes beyond the middle move: axis-aligned or turned elements beside curved ones
        far = x[:, 0] > 0.5 * cells[0]
        x[far, : m.dim] += 0.05 * np.sin(x[far][:, [1, 0, 2]][:, : m.dim] * 2.1 + 0.3)
    if "turned" in shape:
        c, s = np.cos(0.3), np.sin(0.3)
        x = x @ np.array([[c, -s, 0.0], [s, c, 0.0], [0.0, 0.0, 1.0]]).T
    m.xyz = np.ascontiguousarray(x)
    return m


@pytest.mark.parametrize("shape", ["box", "turned", "curved", "turned-curved", "curved-part"])
@pytest.mark.parametrize("case", ASM_CASES.values(), ids=ASM_CASES.keys())
def test_small_element_operators_bit_identical(llf, orc, case, shape):
    m = _shaped(llf, *case, shape)
    sel = np.arange(m.nel)
    if shape.endswith("part"):   # every third element outside the problem's material
        sel = sel[sel % 3 != 1]
        m.groups["part"] = llf.Group("part", m.dim, np.unique(m.conn[sel]), m.family, m.order, m.conn[sel], sel)
    mat = llf.Material("part" if len(sel) < m.nel else "body", E=2.1e5, nu=0.3, rho=7.85e-9, k=45.0)
    rule = llf._lib.builtin_rule(m.family, m.order)
    d, conn = m.dim, m.conn[sel]
    P = llf.Problem([mat], type="Solid" if d == 3 else "PlaneStress", mesh=m)
    H = llf.Problem([mat], type="HeatConduction" if d == 3 else "PlaneHeatConduction", mesh=m)
    pt = 0 if d == 3 else 1
    for K, ref in ((llf.stiffnessMatrix(P), (orc.ELASTIC, pt, d, d, [mat.E, mat.nu])),
                   (llf.massMatrix(P, lumped=False), (orc.MASS, pt, d, d, [mat.rho])),
                   (llf.heatConductionMatrix(H), (orc.HEAT, 3 if d == 3 else 4, d, 1, [mat.k]))):
        r = orc.assemble(*ref[:4], m.xyz, conn, rule, ref[4])
        assert_csc_identical(K.csc(), r.julia(), f"kind {ref[0]}")
