"""Repeated products of a matrix assembled into a kept stored layout: the
stored values serve the first three, the fourth expands the structural ones,
and every product has the same bits."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kept(llf, typ, n, order):
    m = llf.structured_box_mesh(n=n, order=order)
    P = llf.Problem([llf.Material("body", E=2.1e5, nu=0.3, k=45.0)], type=typ, mesh=m)
    make = llf.heatConductionMatrix if typ == "HeatConduction" else llf.stiffnessMatrix
    return make(P), make(P), np.random.default_rng(n).standard_normal(P.pdim * P.non)


def _product(ctx, K, x):
    ctx.profile_reset()
    ctx.profile(True)
    y = K.dm.spmv(x)
    ctx.sync()
    ctx.profile(False)
    return y, set(ctx.profile_report())


@pytest.mark.parametrize("typ,n,order", [("Solid", 4, 1), ("HeatConduction", 2, 4)])
def test_fourth_product_expands(llf, typ, n, order):
    first, K, x = _kept(llf, typ, n, order)
    ctx, want = K.dm.ctx, first.dm.spmv(x)
    kernels = []
    for _ in range(6):
        y, k = _product(ctx, K, x)
        assert np.array_equal(y, want)
        kernels.append(k)
    assert kernels == [{"k_spmv_kept"}] * 3 + [{"k_expand_nz", "k_spmv"}] + [{"k_spmv"}] * 2
    nz = first.dm.copy_structural()
    assert np.array_equal(K.dm.copy_structural(), np.where(nz == 0.0, 0.0, nz))


def test_products_from_two_contexts(llf):
    """Threads with a context each multiply by one matrix while it expands."""
    first, K, x = _kept(llf, "Solid", 12, 2)
    want = first.dm.spmv(x)
    bad = []

    def work():
        ctx = llf._lib.Context(0)
        y = np.empty(len(x))
        for _ in range(8):
            ctx.check(llf._lib.lib().llf_matrix_spmv(ctx.h, K.dm.h, llf._lib.ptr(x, llf._lib.C.c_double),
                                                     llf._lib.ptr(y, llf._lib.C.c_double)))
            if not np.array_equal(y, want):
                bad.append(1)

    ts = [threading.Thread(target=work) for _ in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
