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
