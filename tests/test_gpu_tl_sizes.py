"""Total Lagrangian operators at the sizes where the choice of kernel or of
the elements per CTA turns, against the oracle bit for bit."""
import numpy as np
import pytest

from helpers import assert_csc_identical

pytestmark = pytest.mark.gpu
PRM = {"mu": 1.0, "lambda": 10.0}


def _problem(llf, cells, order, simplex, seed):
    m = llf.structured_box_mesh(lx=float(cells[0]), ly=float(cells[1]), lz=float(cells[2]), dx=1.0, dy=1.0, order=order,
                                simplex=simplex)
    p = llf.Problem([llf.Material("body")], type="Solid", mesh=m)
    u = llf.VectorField(0.03 * np.random.default_rng(seed).standard_normal((3 * m.non, 1)), p)
    return m, p, llf.grad(u, add_identity=True)


def _rule(llf, m, nip):
    """The built-in rule with points of weight zero after its own, nip in all."""
    r = llf._lib.builtin_rule(m.family, m.order)
    q = np.arange(nip) % r["nip"]
    w = np.where(np.arange(nip) < r["nip"], r["w"][q], 0.0)
    return {"nip": nip, "npe": r["npe"], "w": w, "N": np.ascontiguousarray(r["N"][q]),
            "dN": np.ascontiguousarray(r["dN"][q]), "node_ref": None}


def test_largest_rules(llf, orc):
    """Caller-supplied rules up to the shared-memory limit of an element:
    hex125 takes 300 points (376 in the tensor-core form) and no more."""
    m, p, F = _problem(llf, (1, 1, 1), 4, False, 1)
    r = _rule(llf, m, 300)
    p.device_mesh().set_tables(r["w"], r["N"], r["dN"])
    K = llf.materialTangentMatrix(p, F=F, energy="NeoHookeCompressible", params=PRM)
    ref = orc.tl_matrix(orc.TL_KMAT, m.xyz, m.conn, r, F.A, orc.LAW_NEOHOOKE, [1.0, 10.0])
    assert_csc_identical(K.csc(), ref.julia(), "Kmat hex125, 300 points")
    r = _rule(llf, m, 376)
    p.device_mesh().set_tables(r["w"], r["N"], r["dN"])
    Kt = llf.tangentMatrix(p, F, params=PRM, precision="tf32x3")
    with pytest.raises(llf.LLFError, match="too large"):
        llf.tangentMatrix(p, F, params=PRM)
    r = _rule(llf, m, 377)
    p.device_mesh().set_tables(r["w"], r["N"], r["dN"])
    with pytest.raises(llf.LLFError, match="too large"):
        llf.tangentMatrix(p, F, params=PRM, precision="tf32x3")
    r = _rule(llf, m, 125)   # the points that have weight
    p.device_mesh().set_tables(r["w"], r["N"], r["dN"])
    want = llf.tangentMatrix(p, F, params=PRM, precision="tf32x3")
    for a, b in zip(Kt.csc(), want.csc()):
        assert np.array_equal(a, b)


# meshes of one element per CTA, of fewer than a full CTA holds and of full
# CTAs; internal force with a thread per component (at most two CTAs per SM)
# and per node
@pytest.mark.parametrize("cells,order,simplex", [((1, 1, 1), 1, False), ((8, 7, 6), 1, False), ((13, 12, 11), 1, False),
                                                 ((14, 13, 13), 1, False), ((1, 1, 1), 1, True), ((8, 7, 7), 1, True),
                                                 ((4, 3, 2), 2, True), ((5, 6, 7), 2, True), ((3, 3, 2), 2, False),
                                                 ((7, 7, 7), 2, False), ((2, 1, 1), 4, True), ((5, 4, 3), 3, True)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_elements_per_cta(llf, orc, cells, order, simplex):
    m, p, F = _problem(llf, cells, order, simplex, 2)
    rule = llf._lib.builtin_rule(m.family, m.order)
    f = llf.internalForceVector(p, F=F, energy="NeoHookeCompressible", params=PRM)
    assert np.array_equal(f.a[:, 0], orc.tl_internal_force(0, m.xyz, m.conn, rule, F.A, orc.LAW_NEOHOOKE, [1.0, 10.0]))
    P = llf.TensorField(np.random.default_rng(5).standard_normal((m.nel, 9 * m.npe)), p)
    f = llf.internalForceVector(p, P=P)
    assert np.array_equal(f.a[:, 0], orc.tl_internal_force(1, m.xyz, m.conn, rule, P.A))
    K = llf.tangentMatrix(p, F, params=PRM)
    ref = orc.tl_matrix(3, m.xyz, m.conn, rule, F.A, orc.LAW_NEOHOOKE, [1.0, 10.0])
    assert_csc_identical(K.csc(), ref.julia(), f"tangent {cells} p{order}")
