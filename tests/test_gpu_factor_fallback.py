"""GPU tests of what happens where a factorised solve does not get there: a kept factor that no longer fits the
Jacobian is replaced, a system it cannot solve goes to the iterative solve, the others stay with it."""
import numpy as np
import pytest

from tissueorigami_b200 import capi, mesh
from tissueorigami_b200.newton import NewtonRaphsonSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate", [1.0, 2.0])
def test_second_right_hand_side_of_a_lumen_replaces_a_kept_factor(rate):
    """Two steps of 2,000 s with a lumen: in the second the factor kept from an earlier Newton iteration serves
    the residual but not the lumen's gradient. It is replaced by one of the current J, so that the iterative
    solve never runs; equal Newton counts and positions (1e-9 of the size) to runs of that solve alone, where
    it converges (not at twice the rate: 20,000 iterations)."""
    out = {}
    for warm in (1, 0) if rate == 1.0 else (1,):  # 0: no factor
        t = mesh.small_rectangle(nx=60, ny=40)
        t.rates *= rate
        with NewtonRaphsonSolver.from_tissue(t, krylov_warm_start=warm) as s:
            s.set_lumen(np.nonzero(t.exposed & 1)[0].astype(np.int32), 1.0e5, 2.0, t.x)
            x, its, launches = t.x, [], []
            for _ in range(2):
                x, rc, st = s.runOneStep(x, 2000.0)
                assert rc == capi.TF_OK
                its.append(st["newton_iters"])
                launches.append(st["solve_launches"])
        out[warm] = (x, its, launches)
    assert out[1][2] == [0, 0]
    if 0 not in out:
        return
    assert min(out[0][2]) > 0
    assert out[1][1] == out[0][1]
    assert np.abs(out[1][0] - out[0][0]).max() <= 1e-9 * t.size


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
