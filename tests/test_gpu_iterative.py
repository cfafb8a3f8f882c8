"""GPU tests of the iterative solve by name (krylov_method = TF_KRYLOV_CG, which takes no sparse factor): the
two-level preconditioner of single tissues and of batches, the warm-started history, and what else solves
through it. It serves every tissue too large for a factorisation and whatever the factor fails on.

Tolerances: positions within 1e-9 of the tissue size of the oracle's, with equal Newton counts; solutions within
1e-8 of SuperLU's (residual 1e-13, condition numbers up to ~1e5).
"""
import numpy as np
import pytest
import scipy.sparse.linalg as sla

from oracle import oracle as O
from tissueorigami_b200 import capi, mesh
from tissueorigami_b200.newton import BatchSolver, NewtonRaphsonSolver

pytestmark = pytest.mark.gpu

CG = dict(krylov_method=capi.TF_KRYLOV_CG)


def _steps(s, x, dt, n):
    """n steps from x: positions, Newton counts, Krylov iterations per step."""
    its, kry = [], []
    for _ in range(n):
        x, rc, st = s.runOneStep(x, dt)
        assert rc == capi.TF_OK and st["solve_launches"] >= st["newton_iters"]
        its.append(st["newton_iters"])
        kry.append(st["krylov_iters_total"])
    return x, its, kry


def test_warm_started_conjugate_gradients_match_cold_ones():
    """krylov_warm_start: from the second step on fewer iterations, the same steps."""
    t = mesh.wing_disc(n_surface_points=1500)
    x_ref, _, it_ref, _ = O.simulate_sparse(t, n_steps=4)
    res = {}
    for warm in (0, 1):
        with NewtonRaphsonSolver.from_tissue(t, krylov_warm_start=warm, **CG) as s:
            res[warm] = _steps(s, t.x, t.dt, 4)
        assert res[warm][1] == it_ref
        assert np.abs(res[warm][0] - x_ref).max() <= 1e-9 * t.size
    assert sum(res[1][2][1:]) < sum(res[0][2][1:])


def test_two_level_solve_matches_direct_with_fewer_iterations():
    t = mesh.wing_disc(n_surface_points=1500)
    _, inv, _, _ = O.grow(t, t.x, t.fg)
    rowptr, colidx = O.block_pattern(t)
    vals, g = O.assemble_bsr(t, t.x, t.x, O.viscosity_surfaces(t, t.x), inv, rowptr, colidx)
    ref = sla.spsolve(O.bsr_to_scipy(rowptr, colidx, vals, t.n_nodes).tocsc(), g)
    iters = {}
    for pc in (capi.TF_PRECOND_BLOCK_JACOBI, capi.TF_PRECOND_TWO_LEVEL):
        with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-13, precond=pc, **CG) as s:
            du, rc, iters[pc], rr = s.solveForDeltaU(vals, g)
            eff, n_coarse, refreshes = s.preconditioner()
        assert eff == pc and (n_coarse, refreshes) == (0, 0) if pc == capi.TF_PRECOND_BLOCK_JACOBI else n_coarse % 6 == 0 < n_coarse
        assert pc == capi.TF_PRECOND_BLOCK_JACOBI or refreshes == 1
        assert rc == capi.TF_OK and rr <= 1e-13
        assert np.linalg.norm(du - ref) <= 1e-8 * np.linalg.norm(ref)
        assert np.all(du[t.fixed.reshape(-1) != 0] == 0.0)
    assert iters[capi.TF_PRECOND_TWO_LEVEL] < iters[capi.TF_PRECOND_BLOCK_JACOBI]


@pytest.mark.parametrize("warm", [0, 1])
def test_two_level_steps_match_oracle(warm):
    t = mesh.small_disc(11, 3000, 2000.0, n_steps=3)
    x_ref, _, it_ref, _ = O.simulate_sparse(t, n_steps=3)
    with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-14, krylov_warm_start=warm, **CG) as s:
        x, its, _ = _steps(s, t.x, t.dt, 3)
    assert its == it_ref
    assert np.abs(x - x_ref).max() <= 1e-9 * t.size


def test_two_level_with_slaves_matches_block_jacobi():
    """Slave DoFs are left out of the coarse modes."""
    t = mesh.small_rectangle(nx=12, ny=8)
    t.slave_master = np.array([[3 * 30 + 0, 3 * 20 + 0], [3 * 30 + 1, 3 * 20 + 1], [3 * 41 + 2, 3 * 33 + 2]], np.int32)
    out = {}
    for pc in (capi.TF_PRECOND_BLOCK_JACOBI, capi.TF_PRECOND_TWO_LEVEL):
        with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-14, precond=pc, **CG) as s:
            out[pc] = _steps(s, t.x, t.dt, 2)[0]
            assert (s.preconditioner()[1] > 0) == (pc == capi.TF_PRECOND_TWO_LEVEL)
    assert np.abs(out[capi.TF_PRECOND_TWO_LEVEL] - out[capi.TF_PRECOND_BLOCK_JACOBI]).max() <= 1e-9 * t.size
    x = out[capi.TF_PRECOND_TWO_LEVEL].reshape(-1)
    for s_, m_ in t.slave_master:
        assert x[s_] - t.x.reshape(-1)[s_] == pytest.approx(x[m_] - t.x.reshape(-1)[m_], abs=1e-12 * t.size)


def test_batch_coarse_space_matches_oracle():
    """One coarse space per tissue (at least one aggregate of six modes each), tissues that converge in different
    rounds."""
    ts = [mesh.small_disc(100 + k, n, 600.0 + 400.0 * k) if k % 2 == 0 else mesh.small_rect_sized(100 + k, n, 600.0 + 400.0 * k)
          for k, n in enumerate([400, 1500, 700, 3000, 500, 2200])]
    with BatchSolver(ts, krylov_rtol=1e-14, **CG) as b:
        x, its = b.join([t.x for t in ts]), []
        for _ in range(2):
            x, rc, st = b.runOneStep(x, ts[0].dt)
            assert rc == capi.TF_OK and st["solve_launches"] >= st["newton_iters"]
            its.append(b.tissue_stats()["newton_iters"].tolist())
        pc, n_coarse, refreshes = b.preconditioner()
        assert pc == capi.TF_PRECOND_TWO_LEVEL and n_coarse % 6 == 0 and n_coarse >= 6 * len(ts) and refreshes >= 1
        xs = b.split(x)
    for i, t in enumerate(ts):
        x_ref, _, it_ref, _ = O.simulate_sparse(t, n_steps=2)
        assert [k[i] for k in its] == it_ref
        assert np.abs(xs[i] - x_ref).max() <= 1e-9 * t.size


def test_newton_step_matches_reference_run():
    """Run 07008's first step (tests/test_golden_newton.py has the tolerances)."""
    from tests.test_golden_newton import _check_trace, _tissue

    t, z = _tissue()
    with NewtonRaphsonSolver.from_tissue(t, **CG) as s:
        x, rc, st = s.runOneStep(t.x, t.dt)
    assert rc == capi.TF_OK and st["solve_launches"] > 0
    assert np.abs(x - z["x_step1"]).max() <= 1e-8
    assert st["newton_iters"] == len(z["du_trace"])
    _check_trace(st["du_norm"], list(z["du_trace"]))


def test_lumen_steps_match_oracle():
    t = mesh.small_rectangle(nx=8, ny=6)
    elems = np.nonzero(t.exposed & 1)[0].astype(np.int32)
    x_ref, _, it_ref, _ = O.simulate_sparse(t, n_steps=3, lumen=(elems, 1.0e5, 2.0))
    with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-14, **CG) as s:
        s.set_lumen(elems, 1.0e5, 2.0, t.x)
        x, its, _ = _steps(s, t.x, t.dt, 3)
    assert its == it_ref
    assert np.abs(x - x_ref).max() <= 1e-9 * t.size


def test_adjoint_gradient_matches_the_factorised_one():
    """Four steps, checkpoints every two: gradients of a misfit by the growth rates and the start, 1e-8 of the
    largest entry between the two solves (both residuals 1e-14, condition numbers up to ~1e5)."""
    t = mesh.small_disc(21, 900, 1500.0)
    t.newton_tol = 1e-12
    target = t.x * 1.01
    out = {}
    for method in (capi.TF_KRYLOV_AUTO, capi.TF_KRYLOV_CG):
        with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-14, krylov_method=method) as s:
            x, rc, _ = s.adjoint_forward(t.x, 4, t.dt, 2)
            assert rc == capi.TF_OK
            dr, dx, rc, st = s.adjoint_backward(2.0 * (x - target), want_dx0=True)
            assert rc == capi.TF_OK and (st["solve_launches"] > 0) == (method == capi.TF_KRYLOV_CG)
        out[method] = (dr, dx)
    for a, b in zip(*out.values()):
        assert np.abs(b).max() > 0 and np.abs(a - b).max() <= 1e-8 * np.abs(b).max()
