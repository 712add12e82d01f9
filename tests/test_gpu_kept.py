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
    "hex125": ("box", (2, 1, 1), 4, False, "K"), "tet35": ("box", (2, 1, 1), 4, True, "K"),
    "hex125-mass": ("box", (1, 2, 1), 4, False, "mass"), "hex125-heat": ("box", (2, 1, 2), 4, False, "heat"), "hex27-mass": ("box", (3, 2, 2), 2, False, "mass"),
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


@pytest.mark.parametrize("case", [("Solid", (5, 4, 6), 2, 3), ("PlaneStress", (9, 7), 2, 2), ("HeatConduction", (6, 5, 4), 1, 1)],
                         ids=["hex27", "quad9", "heat"])
@pytest.mark.parametrize("precond", [0, 1, 2])
def test_noalloc_from_the_stored_values(llf, case, precond):
    """A product lets llf_pcg_noalloc take a matrix that holds its stored CSC
    only; it allocates nothing and gives the bits of the expanded matrix."""
    typ, cells, order, P = case
    L = [float(c) for c in cells]
    m = (llf.structured_box_mesh(lx=L[0], ly=L[1], lz=L[2], dx=1.0, dy=1.0, order=order) if len(cells) == 3 else
         llf.structured_rect_mesh(lx=L[0], ly=L[1], dx=1.0, dy=1.0, order=order))
    prob = llf.Problem([llf.Material("body", E=2.1e5, nu=0.3, k=45.0)], type=typ, mesh=m)
    make = llf.heatConductionMatrix if typ == "HeatConduction" else llf.stiffnessMatrix
    K1 = make(prob)
    K2, K3 = make(prob), make(prob)   # assembled into the kept layout
    fixed = np.repeat(m.xyz[:, 0] < 1e-9, P)
    b = np.random.default_rng(5).standard_normal(P * m.non)
    with pytest.raises(llf.LLFError, match="not expanded"):
        _noalloc(llf, K2, b, fixed, precond)
    assert np.array_equal(K2.dm.spmv(b), K1.dm.spmv(b))
    K3.dm.prepare()
    got, want = _noalloc(llf, K2, b, fixed, precond), _noalloc(llf, K3, b, fixed, precond)
    assert got[1] == want[1] and np.array_equal(got[0], want[0])


def _noalloc(llf, K, b, fixed, precond):
    import ctypes as C

    torch = pytest.importorskip("torch")
    db = torch.from_numpy(b).cuda()
    dx = torch.zeros_like(db)
    df = torch.from_numpy(fixed.astype(np.uint8)).cuda()
    torch.cuda.synchronize()
    it, rr, allocs0 = C.c_int64(0), C.c_double(0.0), K.dm.ctx.allocs()
    rc = llf._lib.lib().llf_pcg_noalloc(K.dm.ctx.h, K.dm.h, C.c_void_p(db.data_ptr()), C.c_void_p(dx.data_ptr()),
                                        C.c_void_p(df.data_ptr()), precond, 1e-8, 20 * len(b), C.byref(it), C.byref(rr))
    K.dm.ctx.check(rc, "llf_pcg_noalloc")
    assert K.dm.ctx.allocs() == allocs0
    return dx.cpu().numpy(), it.value


@pytest.mark.parametrize("case", [("box", (3, 3, 2), 4, False, "K"), ("box", (44, 43, 42), 1, True, "K"),
                                  ("rect", (190, 210), 2, False, "K")], ids=["long-rows", "by-degree", "by-degree-2d"])
def test_product_against_the_stored_matrix(llf, case):
    """Long rows in node order and the product by degree (77,824 nodes and
    more), from structural and stored values, against scipy on the CSC."""
    P = _problem(llf, *case, turned=True)
    first = _assemble(llf, P, case[-1])
    x = np.random.default_rng(9).standard_normal(P.pdim * P.non)
    y = first * x
    A = first.A
    bound = abs(A) @ abs(x)   # of a row's sum: 2,187 terms at most, each rounded twice
    assert np.all(np.abs(y - A @ x) <= 2 * 2187 * 2.0**-53 * bound)
    assert np.array_equal(_assemble(llf, P, case[-1]) * x, y)
