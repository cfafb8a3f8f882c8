"""GPU tests of the factorised solve (the default for a symmetric J on a tissue small enough for a
sparse factorisation): against SuperLU on the oracle's systems, at front sizes around the 64-pivot
panels, for every column height, indefinite systems, slave-master pairs and uneven batches."""
import numpy as np
import pytest
import scipy.sparse.linalg as sla

from oracle import oracle as O
from tissueorigami_b200 import capi, mesh
from tissueorigami_b200.newton import BatchSolver, NewtonRaphsonSolver

pytestmark = pytest.mark.gpu


def _system(t):
    fg, inv, _, _ = O.grow(t, t.x, t.fg)
    vs = O.viscosity_surfaces(t, t.x)
    rowptr, colidx = O.block_pattern(t)
    vals, g = O.assemble_bsr(t, t.x, t.x, vs, inv, rowptr, colidx)
    return vals, g, O.bsr_to_scipy(rowptr, colidx, vals, t.n_nodes).tocsc()


# Columns of 2, 3 and 4 nodes (6, 9 and 12 unknowns); one to many fronts; root separators of under
# one, one to two and several 64-pivot panels (60 / 66 pivots: 10 and 11 columns of two nodes).
TISSUES = {
    "one_front": lambda: mesh.small_rectangle(nx=3, ny=2),
    "two_levels": lambda: mesh.small_rectangle(nx=6, ny=4),
    "root_60": lambda: mesh.small_rectangle(nx=20, ny=10),
    "root_66": lambda: mesh.small_rectangle(nx=23, ny=11),
    "disc_odd": lambda: mesh.small_disc(7, 1311, 1200.0),
    "disc_large": lambda: mesh.small_disc(3, 9000, 800.0),
    "three_nodes": lambda: mesh.wing_disc(n_surface_points=1203),
    "four_nodes": lambda: mesh.large_slab(nx=31, ny=23),
}


@pytest.mark.parametrize("name", list(TISSUES))
@pytest.mark.parametrize("refine", [0, 1])
def test_factorised_solve_matches_direct(name, refine):
    """du within 1e-8 of SuperLU relative in the norm (a Krylov residual of 1e-13 and condition numbers
    up to ~1e5), in the one or two iterations an exact preconditioner takes, fixed unknowns zero."""
    t = TISSUES[name]()
    vals, g, J = _system(t)
    ref = sla.spsolve(J, g)
    with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-13, krylov_refine=refine) as s:
        du, rc, iters, rr = s.solveForDeltaU(vals, g)
        assert s.preconditioner()[0] == capi.TF_PRECOND_TWO_LEVEL and s.preconditioner()[1] > 0
        assert s.preconditioner()[2] == 1  # one factorisation, also with refinement
    assert rc == capi.TF_OK and iters <= 3 * (1 + refine)
    if refine == 0:
        assert rr <= 1e-13
    assert np.linalg.norm(du - ref) <= 1e-8 * np.linalg.norm(ref)
    assert np.all(du[t.fixed.reshape(-1) != 0] == 0.0)


def test_factorised_solve_of_an_indefinite_system():
    """Negative pivots (one node's diagonal block negated, and a whole negated system): the signs of the
    factorisation carry them."""
    t = mesh.small_disc(7, 1500, 1200.0)
    vals, g, J = _system(t)
    rowptr, colidx = O.block_pattern(t)
    free = np.nonzero(t.fixed.sum(axis=1) == 0)[0]
    node = int(free[len(free) // 2])
    k = int(np.nonzero(colidx[rowptr[node]:rowptr[node + 1]] == node)[0][0]) + rowptr[node]
    one = vals.copy()
    one[k] = -one[k]
    for v in (one, -vals):
        ref = sla.spsolve(O.bsr_to_scipy(rowptr, colidx, v, t.n_nodes).tocsc(), g)
        with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-13) as s:
            du, rc, iters, rr = s.solveForDeltaU(v, g)
        assert rc == capi.TF_OK and rr <= 1e-13 and iters <= 4
        assert np.linalg.norm(du - ref) <= 1e-8 * np.linalg.norm(ref)


@pytest.mark.parametrize("share", [0.02, 0.3])
def test_negative_pivots_in_some_panels_of_a_front(share):
    """Fronts of several 64-pivot panels (the root of 9,000 prisms has six), some of them with negative pivots and
    some without, beside fronts with none: every panel's update takes its own signs. Five solves of one
    system are equal to the last bit."""
    t = mesh.small_disc(3, 9000, 800.0)
    vals, g, _ = _system(t)
    rowptr, colidx = O.block_pattern(t)
    free = np.nonzero(t.fixed.sum(axis=1) == 0)[0]
    node = np.random.default_rng(5).choice(free, int(share * len(free)), replace=False)
    rows = np.repeat(np.arange(t.n_nodes), np.diff(rowptr))
    vals[(rows == colidx) & np.isin(rows, node)] *= -1.0
    ref = sla.spsolve(O.bsr_to_scipy(rowptr, colidx, vals, t.n_nodes).tocsc(), g)
    with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-13) as s:
        first, rc, iters, rr = s.solveForDeltaU(vals, g)
        assert rc == capi.TF_OK and rr <= 1e-13 and iters <= 4
        assert s.preconditioner()[2] == 1
        for _ in range(4):
            assert np.array_equal(s.solveForDeltaU(vals, g)[0], first)
    assert np.linalg.norm(first - ref) <= 1e-8 * np.linalg.norm(ref)


def test_singular_system_falls_back():
    """A free node cut off from everything (zero row and column): a zero pivot. The call returns what the
    iterative path makes of it, without a non-finite du on the other nodes."""
    t = mesh.small_disc(7, 700, 1200.0)
    vals, g, _ = _system(t)
    rowptr, colidx = O.block_pattern(t)
    node = int(np.nonzero(t.fixed.sum(axis=1) == 0)[0][3])
    rows = np.repeat(np.arange(t.n_nodes), np.diff(rowptr))
    vals = vals.copy()
    vals[(rows == node) | (colidx == node)] = 0.0
    with NewtonRaphsonSolver.from_tissue(t, krylov_max_iters=500) as s:
        _, rc, _, _ = s.solveForDeltaU(vals, g)
    assert rc in (capi.TF_OK, capi.TF_KRYLOV_MAX_ITERS, capi.TF_KRYLOV_BREAKDOWN, capi.TF_NONFINITE)


@pytest.mark.parametrize("name", ["one_front", "root_66", "three_nodes"])
def test_launches_outside_graphs(name):
    """use_graphs = 0 launches the same kernels one by one: equal to the last bit."""
    t = TISSUES[name]()
    vals, g, _ = _system(t)
    out = []
    for graphs in (0, 1):
        with NewtonRaphsonSolver.from_tissue(t, use_graphs=graphs) as s:
            out.append([s.solveForDeltaU(vals, g)[0] for _ in range(2)])
            assert s.krylov_method() == 2 and s.preconditioner()[2] == 2
    assert all(np.array_equal(a, out[0][0]) for r in out for a in r)


def test_slaves_and_boundary_changes_rebuild_the_plan():
    """Slave-master pairs couple distant columns (a new pattern, a new dissection); setting the boundary
    again returns to the first one. Positions against the iterative path (krylov_warm_start = 0)."""
    t = mesh.small_rectangle(nx=14, ny=9)
    pairs = np.array([[3 * 30 + 0, 3 * 200 + 0], [3 * 31 + 1, 3 * 120 + 1], [3 * 41 + 2, 3 * 33 + 2]], np.int32)
    out = {}
    for warm in (0, 1):
        with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-14, krylov_warm_start=warm) as s:
            res = []
            for sm in (None, pairs, None):
                s.set_boundary(t.fixed, t.ext_visc, sm)
                s.set_growth(fg=t.fg)
                x, rc, st = s.runOneStep(t.x, t.dt)
                assert rc == capi.TF_OK
                res.append((x, st["newton_iters"]))
        out[warm] = res
    for a, b in zip(out[0], out[1]):
        assert a[1] == b[1]
        assert np.abs(a[0] - b[0]).max() <= 1e-9 * t.size


@pytest.mark.parametrize("count", [1, 7])
def test_batch_matches_single_runs(count):
    """Uneven tissues factorised together (trees of different depth, tissues that converge in different
    rounds) against single-tissue runs: 1e-9 of the size, equal Newton counts."""
    sizes = [4000, 60, 700, 12, 2500, 333, 1201][:count]
    ts = [mesh.small_disc(50 + i, max(n, 40), 700.0 + 300 * i) if i % 2 == 0 else mesh.small_rect_sized(50 + i, n, 900.0)
          for i, n in enumerate(sizes)]
    with BatchSolver(ts, krylov_rtol=1e-14) as b:
        x = b.join([t.x for t in ts])
        its = []
        for _ in range(2):
            x, rc, _ = b.runOneStep(x, ts[0].dt)
            assert rc == capi.TF_OK
            its.append(b.tissue_stats()["newton_iters"].tolist())
        xs = b.split(x)
    for i, t in enumerate(ts):
        with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-14) as s:
            y = t.x
            for k in range(2):
                y, rc, st = s.runOneStep(y, t.dt)
                assert rc == capi.TF_OK and st["newton_iters"] == its[k][i]
        assert np.abs(xs[i] - y).max() <= 1e-9 * t.size


@pytest.mark.parametrize("eta", [4.0, 1e5])
def test_viscous_steps_match_bicgstab(eta):
    """Internal viscosity makes J unsymmetric: the factor of its symmetric part in a minimal residual
    iteration against BiCGStab, two steps, 1e-9 of the size and equal Newton counts; and back to a
    symmetric J on the same solver."""
    t = mesh.wing_disc(n_surface_points=700)
    t.eta[:] = eta
    out = {}
    for method in (capi.TF_KRYLOV_AUTO, capi.TF_KRYLOV_BICGSTAB):
        with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-13, krylov_method=method) as s:
            x, its = t.x, []
            for _ in range(2):
                x, rc, st = s.runOneStep(x, t.dt)
                assert rc == capi.TF_OK
                assert st["krylov_method"] == (5 if method == capi.TF_KRYLOV_AUTO else 1)
                its.append(st["newton_iters"])
            s.set_material(t.lam, t.mu, None)
            s.set_growth(fg=t.fg)
            y, rc, st = s.runOneStep(t.x, t.dt)
            assert rc == capi.TF_OK
        out[method] = (x, its, y)
    a, b = out.values()
    assert a[1] == b[1]
    assert np.abs(a[0] - b[0]).max() <= 1e-9 * t.size
    assert np.abs(a[2] - b[2]).max() <= 1e-9 * t.size


@pytest.mark.parametrize("bad", [0.0, np.nan])
def test_set_growth_rejects_singular_tensors_and_keeps_the_inverse(bad):
    """A singular or non-finite Fg is refused and leaves InvFg as it was; a valid one sets it."""
    t = mesh.small_disc(5, 301, 1000.0)
    rng = np.random.default_rng(3)
    fg = np.tile(np.eye(3), (t.n_elems, 1, 1)) + rng.uniform(-0.1, 0.1, (t.n_elems, 3, 3))
    with NewtonRaphsonSolver.from_tissue(t) as s:
        s.set_growth(fg=fg)
        inv = s.get_growth()[1].reshape(-1, 3, 3)
        assert np.abs(inv - np.linalg.inv(fg)).max() <= 1e-13
        wrong = fg.copy()
        wrong[-1] = bad
        with pytest.raises(capi.TFError):
            s.set_growth(fg=wrong)
        assert np.array_equal(s.get_growth()[1].reshape(-1, 3, 3), inv)


@pytest.mark.parametrize("rows", [(0, 1), (1, 2), (0, 2)])
def test_set_growth_rejects_a_tensor_with_two_equal_rows(rows):
    """Its determinant is zero where every product is rounded (the other minors cancel exactly), but not where the
    products are contracted into fused operations."""
    t = mesh.small_disc(5, 301, 1000.0)
    rng = np.random.default_rng(7)
    fg = np.tile(np.eye(3), (t.n_elems, 1, 1)) + rng.uniform(-0.1, 0.1, (t.n_elems, 3, 3))
    i, j = rows

    def det(m):
        m = m.reshape(9)
        return (m[0] * (m[4] * m[8] - m[5] * m[7]) - m[1] * (m[3] * m[8] - m[5] * m[6])) + m[2] * (m[3] * m[7] - m[4] * m[6])

    with NewtonRaphsonSolver.from_tissue(t) as s:
        refused = 0
        for _ in range(20):
            wrong = fg.copy()
            wrong[-1] = rng.uniform(0.5, 1.5, (3, 3))
            wrong[-1, j] = wrong[-1, i]
            if det(wrong[-1]) == 0.0:
                refused += 1
                with pytest.raises(capi.TFError):
                    s.set_growth(fg=wrong)
            else:
                s.set_growth(fg=wrong)
        assert refused > 0


@pytest.mark.parametrize("apart", [1e-2, 1e-13, 1e-15])
def test_set_growth_inverts_nearly_singular_tensors_by_the_determinant_it_tests(apart):
    """Tensors with two nearly equal rows: InvFg to the last bit what the adjugate over the determinant, every
    product rounded, gives in numpy; a determinant rounded differently is off by its whole size there, or zero."""
    t = mesh.small_disc(5, 301, 1000.0)
    rng = np.random.default_rng(11)
    fg = rng.uniform(0.5, 1.5, (t.n_elems, 3, 3))
    fg[:, 2] = fg[:, 0] * (1.0 + apart * rng.uniform(-1.0, 1.0, (t.n_elems, 3)))
    m = fg.reshape(-1, 9).T
    det = (m[0] * (m[4] * m[8] - m[5] * m[7]) - m[1] * (m[3] * m[8] - m[5] * m[6])) + m[2] * (m[3] * m[7] - m[4] * m[6])
    fg[det == 0.0] = np.eye(3)
    m = fg.reshape(-1, 9).T.copy()
    det = (m[0] * (m[4] * m[8] - m[5] * m[7]) - m[1] * (m[3] * m[8] - m[5] * m[6])) + m[2] * (m[3] * m[7] - m[4] * m[6])
    adj = np.stack([m[4] * m[8] - m[5] * m[7], m[2] * m[7] - m[1] * m[8], m[1] * m[5] - m[2] * m[4],
                    m[5] * m[6] - m[3] * m[8], m[0] * m[8] - m[2] * m[6], m[2] * m[3] - m[0] * m[5],
                    m[3] * m[7] - m[4] * m[6], m[1] * m[6] - m[0] * m[7], m[0] * m[4] - m[1] * m[3]])
    with NewtonRaphsonSolver.from_tissue(t) as s:
        s.set_growth(fg=fg)
        assert np.array_equal(s.get_growth()[1].reshape(-1, 9), (adj * (1.0 / det)).T)
