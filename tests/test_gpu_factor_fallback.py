"""GPU tests of what happens where a factorised solve does not get there: a kept factor that no longer fits the
Jacobian is replaced, a system it cannot solve goes to the iterative solve, the others stay with it."""
import numpy as np
import pytest
import scipy.sparse.linalg as sla

from oracle import oracle as O
from tissueorigami_b200 import capi, mesh
from tissueorigami_b200.newton import BatchSolver, NewtonRaphsonSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate", [1.0, 2.0])
def test_second_right_hand_side_of_a_lumen_replaces_a_kept_factor(rate):
    """Two steps of 2,000 s with a lumen: in the second the factor kept from an earlier Newton iteration serves
    the residual but not the lumen's gradient. It is replaced by one of the current J, so that the iterative
    solve (15,000 iterations a step here) never runs; equal Newton counts and positions (1e-9 of the size) to
    runs that keep no factor (krylov_max_iters = 2). The updates' norms end 3.5e-4, 3e-11: the Newton tolerance
    lies between."""
    out = {}
    for cap in (20000, 2):
        t = mesh.small_rectangle(nx=60, ny=40)
        t.rates *= rate
        with NewtonRaphsonSolver.from_tissue(t, krylov_max_iters=cap, newton_tol=1e-8) as s:
            s.set_lumen(np.nonzero(t.exposed & 1)[0].astype(np.int32), 1.0e5, 2.0, t.x)
            x, its, launches = t.x, [], []
            for _ in range(2):
                x, rc, st = s.runOneStep(x, 2000.0)
                assert rc == capi.TF_OK
                its.append(st["newton_iters"])
                launches.append(st["solve_launches"])
            out[cap] = (x, its, s.preconditioner()[2])
        assert launches == [0, 0]
    assert out[20000][1] == out[2][1] and out[20000][2] < out[2][2]
    assert np.abs(out[20000][0] - out[2][0]).max() <= 1e-9 * t.size


def test_kept_factor_is_replaced_where_newton_moves_far():
    """Steps of 600 s of fast growth: the factor kept from the second Newton iteration does not serve all of the
    later ones and is made anew (a third time and more), without the iterative solve. Positions within 1e-9 of
    the size of those of runs that keep no factor (krylov_max_iters = 2), equal Newton counts (the updates' norms
    end 1e-5, 1e-12, the tolerance lies between)."""
    out = {}
    for cap in (20000, 2):
        t = mesh.small_rectangle(nx=60, ny=40)
        t.rates *= 5.0
        with NewtonRaphsonSolver.from_tissue(t, krylov_max_iters=cap, krylov_rtol=1e-13, newton_tol=1e-8) as s:
            x, its = t.x, []
            for _ in range(2):
                x, rc, st = s.runOneStep(x, 600.0)
                assert rc == capi.TF_OK and st["solve_launches"] == 0
                its.append(st["newton_iters"])
            out[cap] = (x, its, s.preconditioner()[2])
    assert out[20000][1] == out[2][1] and 6 <= out[20000][2] < out[2][2]
    assert np.abs(out[20000][0] - out[2][0]).max() <= 1e-9 * t.size


@pytest.mark.parametrize("cap", [2, 3])
def test_kept_factor_is_replaced_at_a_low_iteration_cap(cap):
    """krylov_max_iters below what a kept factor needs (three to five iterations, where a factor of J itself needs
    one): the steps converge all the same, to the positions without a cap (1e-9 of the size)."""
    t = mesh.wing_disc(n_surface_points=1500)
    out = {}
    for most in (cap, 20000):
        with NewtonRaphsonSolver.from_tissue(t, krylov_max_iters=most) as s:
            x = t.x
            for _ in range(2):
                x, rc, st = s.runOneStep(x, t.dt)
                assert rc == capi.TF_OK and st["solve_launches"] == 0
            out[most] = (x, s.preconditioner()[2])
    assert out[20000][1] == 4 and out[cap][1] > 4  # two factorisations a step without a cap
    assert np.abs(out[cap][0] - out[20000][0]).max() <= 1e-9 * t.size


def test_packing_pairs_that_come_and_go_on_one_solver():
    """Two sheets apart, in contact and apart again, each step from given positions: the factor serves the first
    and the last, MINRES the one with pairs, and what the solver says of its preconditioner is what a solver
    with that step alone says. Positions to 1e-9 of the size, equal Newton counts."""
    t = mesh.stacked_sheets()
    apart = t.x.copy()
    apart[t.x[:, 2] > 0.5 * (t.x[:, 2].min() + t.x[:, 2].max()), 2] += 20.0
    starts = [apart, t.x, apart]

    def step(s, x):
        s.set_growth(fg=t.fg)
        y, rc, st = s.runOneStep(x, t.dt)
        assert rc == capi.TF_OK
        return y, st["newton_iters"], s.krylov_method(), s.preconditioner()[:2]

    with NewtonRaphsonSolver.from_tissue(t, packing=True, krylov_rtol=1e-13) as s:
        one = [step(s, x) for x in starts]
    alone = []
    for x in starts:
        with NewtonRaphsonSolver.from_tissue(t, packing=True, krylov_rtol=1e-13) as s:
            alone.append(step(s, x))
    assert [r[2] for r in one] == [2, 4, 2]
    for a, b in zip(one, alone):
        assert a[1:] == b[1:]
        assert np.abs(a[0] - b[0]).max() <= 1e-9 * t.size


def _system(t):
    """(values, right-hand side) of the oracle's first Newton iteration, and the block pattern."""
    _, inv, _, _ = O.grow(t, t.x, t.fg)
    rowptr, colidx = O.block_pattern(t)
    vals, g = O.assemble_bsr(t, t.x, t.x, O.viscosity_surfaces(t, t.x), inv, rowptr, colidx)
    return vals, g, rowptr, colidx


def _cut_off(t, vals, g, rowptr, colidx):
    """The system with one free node's rows, columns and forces zero (a zero pivot, and a solution all the same),
    and the solution on the other unknowns (the node's own are free): their indices and values."""
    node = int(np.nonzero(t.fixed.sum(axis=1) == 0)[0][3])
    rows = np.repeat(np.arange(t.n_nodes), np.diff(rowptr))
    vals, g = vals.copy(), g.copy()
    vals[(rows == node) | (colidx == node)] = 0.0
    g[3 * node:3 * node + 3] = 0.0
    keep = np.setdiff1d(np.arange(3 * t.n_nodes), 3 * node + np.arange(3))
    J = O.bsr_to_scipy(rowptr, colidx, vals, t.n_nodes).tocsc()
    return vals, g, keep, sla.spsolve(J[keep][:, keep], g[keep])


def test_singular_system_is_left_to_the_iterative_solve():
    """The factorisation meets a zero pivot; the conjugate gradients that follow do not: the solution of the rest
    within 1e-8 of SuperLU's (a residual of 1e-13 and condition numbers up to ~1e5). The next system of the same solver is a factorised one again."""
    t = mesh.small_disc(7, 700, 1200.0)
    vals, g, rowptr, colidx = _system(t)
    with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-13) as s:
        good, rc, it, _ = s.solveForDeltaU(vals, g)
        root = s.preconditioner()[1]
        assert rc == capi.TF_OK and it <= 3 and root > 0
        v, b, keep, ref = _cut_off(t, vals, g, rowptr, colidx)
        du, rc, it, rr = s.solveForDeltaU(v, b)
        assert rc == capi.TF_OK and rr <= 1e-13 and it > 3
        assert s.preconditioner()[1] != root
        assert np.all(np.isfinite(du)) and np.linalg.norm(du[keep] - ref) <= 1e-8 * np.linalg.norm(ref)
        again, rc, _, _ = s.solveForDeltaU(vals, g)
        assert rc == capi.TF_OK and s.preconditioner()[1] == root
        assert np.array_equal(again, good)


@pytest.mark.parametrize("bad", [[0], [1], [2, 3], [0, 1, 2, 3]])
def test_tissues_of_a_batch_whose_factor_fails_leave_the_others_alone(bad):
    """Some tissues of a batch with a zero pivot: the others' solutions equal, to the last bit, those of the batch
    without it; the bad ones' come from the iterative solve (1e-8 of SuperLU's as above)."""
    ts = [mesh.small_disc(50 + i, n, 900.0) for i, n in enumerate([700, 1500, 333, 1201])]
    sys = [_system(t) for t in ts]
    cut = [_cut_off(t, *s) for t, s in zip(ts, sys)]
    cat = np.concatenate
    with BatchSolver(ts, krylov_rtol=1e-13) as b:
        good, rc, _, _ = b.solveForDeltaU(cat([s[0] for s in sys]), cat([s[1] for s in sys]))
        assert rc == capi.TF_OK
        du, rc, _, _ = b.solveForDeltaU(cat([(cut if i in bad else sys)[i][0] for i in range(4)]),
                                        cat([(cut if i in bad else sys)[i][1] for i in range(4)]))
        assert rc == capi.TF_OK
        good, du = b.split(good), b.split(du)
    for i in range(4):
        if i in bad:
            keep, ref = cut[i][2:]
            assert np.linalg.norm(du[i].reshape(-1)[keep] - ref) <= 1e-8 * np.linalg.norm(ref)
        else:
            assert np.array_equal(du[i], good[i])


@pytest.mark.parametrize("batch", [False, True])
def test_a_factor_that_fails_is_not_tried_again_in_the_step(batch):
    """A node that nothing holds (no stiffness around it, no drag): every Newton iteration has a zero pivot. The
    step factorises that tissue once; the other Newton iterations go to the iterative solve at once. Equal
    Newton counts and positions (1e-9 of the size) to steps of that solve alone."""
    t = mesh.small_disc(7, 700, 1200.0)
    node = int(np.nonzero(t.fixed.sum(axis=1) == 0)[0][40])
    around = (t.conn == node).any(axis=1)
    t.lam[around] = t.mu[around] = 0.0
    t.ext_visc.reshape(-1, 3)[node] = 0.0
    other = mesh.small_disc(8, 900, 1000.0)
    out = {}
    for warm in (1, 0):  # 0: no factor
        make = (lambda **kw: BatchSolver([other, t], **kw)) if batch else (lambda **kw: NewtonRaphsonSolver.from_tissue(t, **kw))
        with make(krylov_rtol=1e-13, krylov_warm_start=warm) as s:
            x0 = s.join([other.x, t.x]) if batch else t.x
            x, rc, st = s.runOneStep(x0, t.dt)
            assert rc == capi.TF_OK and st["newton_iters"] >= 4
            out[warm] = (x, st["newton_iters"], st["solve_launches"], s.preconditioner()[2])
    a, b = out[1], out[0]
    assert a[1] == b[1] and a[2] == b[2]  # every Newton iteration has its iterative solve
    # refreshes: coarse operators as without a factor, and factorisations: one, or for a batch one per
    # Newton iteration (the other tissue's)
    assert a[3] <= b[3] + (a[1] if batch else 1)
    assert np.abs(a[0] - b[0]).max() <= 1e-9 * t.size


def test_without_memory_for_the_factor_the_steps_are_iterative():
    """Device memory held back until only so much is left, around every point at which one of the factor's buffers
    no longer fits: the step succeeds all the same, equal Newton counts and positions (1e-9 of the size)."""
    import torch

    t = mesh.wing_disc(n_surface_points=6000)
    mb = 1 << 20

    def step(left=None):
        with NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-13) as s:
            free = torch.cuda.mem_get_info()[0]
            hold = torch.empty(free - left, dtype=torch.uint8, device="cuda") if left else None
            free = torch.cuda.mem_get_info()[0]
            x, rc, st = s.runOneStep(t.x, t.dt)
            used = free - torch.cuda.mem_get_info()[0]
        del hold
        torch.cuda.empty_cache()
        assert rc == capi.TF_OK
        return x, st["newton_iters"], st["solve_launches"], used

    with NewtonRaphsonSolver.from_tissue(t, krylov_warm_start=0) as s:  # the iterative kernels' local memory is the process's
        s.runOneStep(t.x, t.dt)
    step()
    x, its, launches, used = step()
    assert launches == 0 and used > 100 * mb
    ways = []
    for left in [3 * used, 2 * used + 8 * mb, 2 * used - 8 * mb] + [used + k * mb for k in range(4, -13, -2)]:
        y, n, launches, _ = step(left)
        assert n == its and np.abs(y - x).max() <= 1e-9 * t.size
        ways.append(launches > 0)
    assert not ways[0] and all(ways[3:])
