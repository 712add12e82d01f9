"""The CG whose whole loop runs in one kernel, one CTA per chunk, against the
launches (the allocation-free path, a batch with too many chunks for it, and
the fallback when its waits run out): the same bits."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(llf, kind, n, order=1):
    if kind == "rect":
        m = llf.structured_rect_mesh(n=n, order=order)
        P = llf.Problem([llf.Material("body")], type="PlaneStress", mesh=m)
        K = llf.stiffnessMatrix(P)
    else:
        m = llf.structured_box_mesh(n=n, order=order)
        P = llf.Problem([llf.Material("body")], type="Solid" if kind == "box" else "HeatConduction", mesh=m)
        K = llf.stiffnessMatrix(P) if kind == "box" else llf.heatConductionMatrix(P)
    nd = P.pdim * P.non
    fixed = np.zeros(nd, dtype=np.uint8)
    for c in range(P.pdim):
        fixed[P.pdim * (m.group("left").nodes - 1) + c] = 1
    rng = np.random.default_rng(n)
    x0 = np.where(fixed, rng.standard_normal(nd), 0.0)
    return P, K, rng.standard_normal(nd), x0, fixed


def _noalloc(llf, K, b, x0, fixed, precond, reltol, maxiter):
    torch = pytest.importorskip("torch")
    t = lambda a: torch.tensor(a, device="cuda")
    db, dx, df = t(b), t(x0), t(fixed)
    torch.cuda.synchronize()
    it, rr = C.c_int64(0), C.c_double(0.0)
    rc = llf._lib.lib().llf_pcg_noalloc(K.dm.ctx.h, K.dm.h, C.c_void_p(db.data_ptr()), C.c_void_p(dx.data_ptr()),
                                        C.c_void_p(df.data_ptr()), precond, reltol, maxiter, C.byref(it), C.byref(rr))
    assert rc in (0, -4), llf._lib.lib().llf_last_error(K.dm.ctx.h).decode()
    torch.cuda.synchronize()
    return dx.cpu().numpy(), it.value, rr.value


# one chunk, a ragged last chunk, chunks of 192 to 768 DoFs (one CTA per SM),
# and more chunks than SMs (two CTAs per SM)
CASES = [("box", 1, 1), ("box", 9, 1), ("box", 6, 2), ("box", 30, 1), ("box", 33, 1), ("rect", 3, 1),
         ("rect", 101, 1), ("heat", 2, 1), ("heat", 40, 1), ("heat", 48, 1)]


@pytest.mark.parametrize("precond", [0, 1, 2])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-{c[1]}-p{c[2]}")
def test_resident_equals_launches(llf, case, precond):
    P, K, b, x0, fixed = _problem(llf, *case)
    maxiter = 60
    got = K.dm.pcg(b, x0, fixed, precond=precond, reltol=1e-9, maxiter=maxiter, raise_on_fail=False)
    want = _noalloc(llf, K, b, x0, fixed, precond, 1e-9, maxiter)
    assert np.array_equal(got[0], want[0]) and got[1:] == want[1:]


@pytest.mark.parametrize("n,order", [(12, 1), (22, 2)], ids=["fits", "no-room"])
def test_resident_with_nodes_in_random_order(llf, n, order):
    """A chunk whose columns meet nodes all over the system: its halo is most
    of it, or does not fit beside the chunk."""
    m = llf.structured_box_mesh(n=n, order=order)
    new = np.random.default_rng(n).permutation(m.non)
    xyz = np.empty_like(m.xyz)
    xyz[new] = m.xyz
    conn = new[m.conn - 1] + 1
    body = llf.Group("body", 3, np.arange(1, m.non + 1), m.family, m.order, conn, np.arange(m.nel))
    sh = llf.Mesh(3, m.family, m.order, xyz, conn, {"body": body})
    P = llf.Problem([llf.Material("body", k=2.0)], type="Solid" if order == 1 else "HeatConduction", mesh=sh)
    K = llf.stiffnessMatrix(P) if order == 1 else llf.heatConductionMatrix(P)
    nd = P.pdim * m.non
    fixed = np.repeat(xyz[:, 0] < 1e-9, P.pdim).astype(np.uint8)
    b, x0 = np.random.default_rng(2).standard_normal(nd), np.zeros(nd)
    got = K.dm.pcg(b, x0, fixed, precond=1, reltol=1e-9, maxiter=50, raise_on_fail=False)
    want = _noalloc(llf, K, b, x0, fixed, 1, 1e-9, 50)
    assert np.array_equal(got[0], want[0]) and got[1:] == want[1:]


def test_resident_batches(llf):
    """A system with more than two chunks per SM alone (the launches), a
    batch of uneven systems in one launch, and a batch with more chunks than
    CTAs (the launches): every system as it is alone."""
    ms = [llf.structured_box_mesh(n=n, order=1) for n in (62, 62, 62)]
    small = [llf.structured_box_mesh(n=n, order=1) for n in (3, 17, 8, 1)]
    for group in (ms, small):
        m, off = llf.concat_meshes(group)
        mats = [llf.Material(f"body#{i}", k=1.0 + i) for i in range(len(group))]
        P = llf.Problem(mats, type="HeatConduction", mesh=m)
        K = llf.heatConductionMatrix(P)
        b = np.random.default_rng(1).standard_normal(P.non)
        fixed = np.zeros(P.non, dtype=np.uint8)
        for i in range(len(group)):
            fixed[m.group(f"left#{i}").nodes - 1] = 1
        x, its, rr = K.dm.pcg_batched(b, np.zeros(P.non), fixed, off, precond=1, reltol=1e-9, maxiter=80,
                                      raise_on_fail=False)
        for i, g in enumerate(group):
            Pi = llf.Problem([llf.Material("body", k=1.0 + i)], type="HeatConduction", mesh=g)
            s = slice(off[i], off[i + 1])
            xi, ii, ri = llf.heatConductionMatrix(Pi).dm.pcg(b[s], np.zeros(g.non), fixed[s], precond=1, reltol=1e-9,
                                                             maxiter=80, raise_on_fail=False)
            assert np.array_equal(x[s], xi) and its[i] == ii and rr[i] == ri, i


def test_waits_that_run_out_fall_back_to_launches(llf, monkeypatch):
    P, K, b, x0, fixed = _problem(llf, "box", 20, 1)
    want = K.dm.pcg(b, x0, fixed, precond=2, reltol=1e-10, maxiter=500)
    monkeypatch.setenv("LLF_RESIDENT_WAIT_NS", "0")
    got = K.dm.pcg(b, x0, fixed, precond=2, reltol=1e-10, maxiter=500)
    assert np.array_equal(got[0], want[0]) and got[1:] == want[1:]
    monkeypatch.delenv("LLF_RESIDENT_WAIT_NS")
    again = K.dm.pcg(b, x0, fixed, precond=2, reltol=1e-10, maxiter=500)
    assert np.array_equal(again[0], want[0])


def test_breakdown_is_reported(llf):
    P, K, b, x0, fixed = _problem(llf, "box", 6, 1)
    with pytest.raises(llf.LLFError, match="breakdown"):
        (-1.0 * K).dm.pcg(b, x0, fixed, precond=0, reltol=1e-9, maxiter=50)
