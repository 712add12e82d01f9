"""Which form of the CG a solve takes: the resident loop with its halo, the
one that exchanges directions (a halo that does not fit), or the launches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HALO, DIRECTIONS, LAUNCHES = "k_cg_resident", "k_cg_resident_directions", "k_seg_spmv"


def _forms(ctx, f):
    ctx.profile_reset()
    ctx.profile(True)
    f()
    ctx.sync()
    ctx.profile(False)
    return {HALO, DIRECTIONS, LAUNCHES} & set(ctx.profile_report())


def _solve(llf, m, typ, precond=1):
    P = llf.Problem([llf.Material("body")], type=typ, mesh=m)
    K = llf.heatConductionMatrix(P) if typ == "HeatConduction" else llf.stiffnessMatrix(P)
    nd = P.pdim * P.non
    fixed = np.repeat(m.xyz[:, 0] < 1e-9, P.pdim).astype(np.uint8)
    b = np.random.default_rng(1).standard_normal(nd)
    return K.dm.ctx, lambda: K.dm.pcg(b, np.zeros(nd), fixed, precond=precond, reltol=1e-9, maxiter=40,
                                      raise_on_fail=False)


def _shuffled(llf, n, order):
    m = llf.structured_box_mesh(n=n, order=order)
    new = np.random.default_rng(n).permutation(m.non)
    xyz = np.empty_like(m.xyz)
    xyz[new] = m.xyz
    conn = new[m.conn - 1] + 1
    body = llf.Group("body", 3, np.arange(1, m.non + 1), m.family, m.order, conn, np.arange(m.nel))
    return llf.Mesh(3, m.family, m.order, xyz, conn, {"body": body})


# one chunk; a CTA per SM; two per SM; a halo of most of the system; halos that
# do not fit, found by the kernel and seen from the row lengths alone;
# more chunks than two per SM; IC(0), whose sweeps need the launches
@pytest.mark.parametrize("mesh,typ,precond,want", [
    (lambda l: l.structured_box_mesh(n=1, order=1), "Solid", 1, {HALO}),
    (lambda l: l.structured_box_mesh(n=30, order=1), "Solid", 2, {HALO}),
    (lambda l: l.structured_rect_mesh(n=101, order=1), "PlaneStress", 0, {HALO}),
    (lambda l: l.structured_box_mesh(n=33, order=1), "Solid", 1, {HALO}),
    (lambda l: _shuffled(l, 12, 1), "Solid", 1, {HALO}),
    (lambda l: _shuffled(l, 22, 2), "HeatConduction", 1, {HALO, DIRECTIONS}),
    (lambda l: l.structured_box_mesh(n=6, order=4), "HeatConduction", 1, {HALO, DIRECTIONS}),
    (lambda l: l.structured_box_mesh(n=24, order=2), "HeatConduction", 1, {DIRECTIONS}),
    (lambda l: l.structured_box_mesh(n=62, order=1), "HeatConduction", 1, {LAUNCHES}),
    (lambda l: l.structured_box_mesh(n=4, order=1), "Solid", 3, {LAUNCHES}),
], ids=["one-chunk", "one-per-sm", "one-per-sm-2d", "two-per-sm", "wide-halo", "no-room", "long-rows", "longer-rows", "too-many", "ic0"])
def test_form(llf, mesh, typ, precond, want):
    ctx, solve = _solve(llf, mesh(llf), typ, precond)
    assert _forms(ctx, solve) == want


def test_fallback_runs_the_launches(llf, monkeypatch):
    ctx, solve = _solve(llf, llf.structured_box_mesh(n=20, order=1), "Solid")
    monkeypatch.setenv("LLF_RESIDENT_WAIT_NS", "0")
    assert _forms(ctx, solve) == {HALO, LAUNCHES}
    monkeypatch.delenv("LLF_RESIDENT_WAIT_NS")
    monkeypatch.setenv("LLF_RESIDENT_GIVE_UP", "1,2")
    assert _forms(ctx, solve) == {HALO, LAUNCHES}
    monkeypatch.delenv("LLF_RESIDENT_GIVE_UP")
    assert _forms(ctx, solve) == {HALO}


def test_meeting_points_only_where_the_loop_may_run(llf):
    """A solve with more chunks than the resident CG takes allocates nothing
    for it: one allocation fewer than a solve that it takes."""
    count = []
    for n in (20, 62):
        ctx, solve = _solve(llf, llf.structured_box_mesh(n=n, order=1), "HeatConduction")
        a = ctx.allocs()
        solve()
        count.append(ctx.allocs() - a)
    assert count[0] == count[1] + 1


def test_contexts_that_share_the_gpu_take_the_launches(llf):
    ctx, solve = _solve(llf, llf.structured_box_mesh(n=12, order=1), "Solid")
    want = solve()
    ctx.share_gpu()
    try:
        assert _forms(ctx, solve) == {LAUNCHES}
        got = solve()
    finally:
        ctx.share_gpu(False)
    assert _forms(ctx, solve) == {HALO}
    assert np.array_equal(got[0], want[0]) and got[1:] == want[1:]
