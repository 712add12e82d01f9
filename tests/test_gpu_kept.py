"""Matrices assembled into a kept stored layout: the product from the stored
values and keep bits, and the structural values expanded from them, against
the first assembly of the same operator, which holds the structural values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# kind, (nx, ny, nz), order, simplex, operator: 1 to 3 components, columns of
# 4 to 1029 entries, axis-aligned boxes (most columns drop entries) and turned
# ones (nearly none do)
CASES = {
    "hex8": ("box", (5, 4, 3), 1, False, "K"), "hex27": ("box", (4, 3, 3), 2, False, "K"),
    "hex64": ("box", (2, 2, 1), 3, False, "K"), "tet4": ("box", (1, 1, 1), 1, True, "K"),
    "tet10": ("box", (3, 2, 3), 2, True, "K"), "quad4": ("rect", (7, 5), 1, False, "K"),
    "tri6": ("rect", (3, 4), 2, True, "K"), "hex8-heat": ("box", (5, 4, 3), 1, False, "heat"),
    "hex125-heat": ("box", (2, 1, 2), 4, False, "heat"), "hex27-mass": ("box", (3, 2, 2), 2, False, "mass"),
}


def _problem(llf, kind, cells, order, simplex, op, turned):
    if kind == "box":
        m = llf.structured_box_mesh(lx=float(cells[0]), ly=float(cells[1]), lz=float(cells[2]), dx=1.0, dy=1.0,
                                    order=order, simplex=simplex)
    else:
        m = llf.structured_rect_mesh(lx=float(cells[0]), ly=float(cells[1]), dx=1.0, dy=1.0, order=order,
                                     simplex=simplex)
    if turned:
        c, s = np.cos(0.3), np.sin(0.3)
        R = np.array([[c, -s, 0.0], [s, c, 0.0], [0.0, 0.0, 1.0]])
        m.xyz = np.ascontiguousarray(m.xyz @ R.T)
    t = {"K": ("PlaneStrain", "Solid"), "mass": ("PlaneStrain", "Solid"),
         "heat": ("PlaneHeatConduction", "HeatConduction")}[op][m.dim - 2]
    return llf.Problem([llf.Material("body", E=2.1e5, nu=0.3)], type=t, mesh=m)


def _assemble(llf, P, op, **kw):
    if op == "K":
        return llf.stiffnessMatrix(P, **kw)
    return llf.massMatrix(P, lumped=False, **kw) if op == "mass" else llf.heatConductionMatrix(P, **kw)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("turned", [False, True], ids=["box", "turned"])
@pytest.mark.parametrize("case", CASES.values(), ids=CASES.keys())
def test_kept_product_and_expansion_equal_structural(llf, case, turned, precision):
    if precision == "fp32" and case[2] == 4:
        pytest.skip("the precision form refuses order-4 hexahedra (their tables exceed shared memory)")
    P = _problem(llf, *case, turned)
    op = case[-1]
    first = _assemble(llf, P, op, precision=precision)     # structural values
    x = np.random.default_rng(3).standard_normal(P.pdim * P.non)
    want, nz = first * x, first.dm.copy_structural()
    kept = _assemble(llf, P, op, precision=precision)      # into the kept layout
    assert np.array_equal(kept * x, want)                  # from the stored values
    assert np.array_equal(kept.dm.copy_structural(), np.where(nz == 0.0, 0.0, nz))
    assert np.array_equal(kept * x, want)                  # from the expanded values
    # a value that is not finite reaches the same entries either way
    x[1], x[-1] = np.nan, np.inf
    again = _assemble(llf, P, op, precision=precision)
    assert np.array_equal(again * x, kept * x, equal_nan=True)
