"""A resident CG in which one CTA gives up while the others of its system
finish: nothing that the kernel wrote is kept, and the solution, iteration
counts and residuals are those of an undisturbed solve, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _heat(llf, meshes):
    """Conduction on independent bodies: matrix, DoF offsets, load, fixed DoFs."""
    m, off = llf.concat_meshes(meshes)
    P = llf.Problem([llf.Material(f"body#{i}", k=1.0 + i) for i in range(len(meshes))], type="HeatConduction", mesh=m)
    fixed = np.zeros(P.non, dtype=np.uint8)
    for i in range(len(meshes)):
        fixed[np.flatnonzero(m.xyz[off[i]:off[i + 1], 0] < 1e-9) + off[i]] = 1
    return llf.heatConductionMatrix(P), np.asarray(off), np.random.default_rng(3).standard_normal(P.non), fixed


def _shuffled(llf, n, order):
    """A box with its nodes in random order: a chunk meets nodes all over it."""
    m = llf.structured_box_mesh(n=n, order=order)
    new = np.random.default_rng(n).permutation(m.non)
    xyz = np.empty_like(m.xyz)
    xyz[new] = m.xyz
    conn = new[m.conn - 1] + 1
    body = llf.Group("body", 3, np.arange(1, m.non + 1), m.family, m.order, conn, np.arange(m.nel))
    return llf.Mesh(3, m.family, m.order, xyz, conn, {"body": body})


def _same(monkeypatch, solve, chunk, it):
    want = solve()
    monkeypatch.setenv("LLF_RESIDENT_GIVE_UP", f"{chunk},{it}")
    got = solve()
    monkeypatch.delenv("LLF_RESIDENT_GIVE_UP")
    assert np.isfinite(want[0]).all() and np.abs(want[0]).max() > 0
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


# (chunk, iteration that gives up, iterations asked for): the first CTA, which
# publishes the system's state, another and the last one, where the system
# ends and before it
@pytest.mark.parametrize("chunk,it,maxiter", [(0, 1, 1), (1, 1, 1), (0, 4, 4), (1, 4, 4), (-1, 4, 4), (2, 2, 5)])
@pytest.mark.parametrize("kind", ["Solid", "HeatConduction"])
def test_one_system(llf, monkeypatch, kind, chunk, it, maxiter):
    m = llf.structured_box_mesh(n=16, order=1)
    P = llf.Problem([llf.Material("body")], type=kind, mesh=m)
    K = llf.stiffnessMatrix(P) if kind == "Solid" else llf.heatConductionMatrix(P)
    nd = P.pdim * P.non
    fixed = np.repeat(m.xyz[:, 0] < 1e-9, P.pdim).astype(np.uint8)
    b = np.random.default_rng(1).standard_normal(nd)
    nch = -(-nd // 192)   # nd / 148 is below the smallest chunk
    solve = lambda: K.dm.pcg(b, np.zeros(nd), fixed, precond=1, reltol=1e-9, maxiter=maxiter, raise_on_fail=False)
    _same(monkeypatch, solve, chunk % nch, it)


# a chunk of the second of two systems, which is the last to end
@pytest.mark.parametrize("chunk", [0, 3])
def test_batch(llf, monkeypatch, chunk):
    K, off, b, fixed = _heat(llf, [llf.structured_box_mesh(n=n, order=1) for n in (9, 14)])
    solve = lambda: K.dm.pcg_batched(b, np.zeros(len(b)), fixed, off, precond=1, reltol=1e-9, maxiter=6,
                                     raise_on_fail=False)
    _same(monkeypatch, solve, -(-off[1] // 192) + chunk, 6)


# the second system's halo does not fit, so it runs in a second launch, after
# which the first system's result counts no more either
@pytest.mark.parametrize("chunk", [0, 5])
def test_batch_with_a_halo_that_does_not_fit(llf, monkeypatch, chunk):
    K, off, b, fixed = _heat(llf, [llf.structured_box_mesh(n=3, order=2), _shuffled(llf, 22, 2)])
    solve = lambda: K.dm.pcg_batched(b, np.zeros(len(b)), fixed, off, precond=1, reltol=1e-9, maxiter=6,
                                     raise_on_fail=False)
    _same(monkeypatch, solve, -(-off[1] // 192) + chunk, 6)
