"""Errors that a stage finds on the device: every way of stepping reports the same one."""
import numpy as np
import pytest

from dacti_b200 import cases
from dacti_b200.solver import Batch, DgError, Solver

pytestmark = pytest.mark.gpu
MISSING_BC = -5
CAN_UNSPLIT = 1 << 4


def coarsens_into_missing_boundary(base, levels, **kw):
    """Uniform gas whose grid may coarsen below the base level: it does so at once, and the parents on the domain's
    boundary have no boundary condition, which the next substep's face sums find first."""
    c = cases.lax_liu3(base, levels, **kw)
    t = c.tree
    leaf = t.leaf_mask()
    t.p[1:] = (1.0, 0.0, 0.0, 1.0)
    t.flags[leaf] |= CAN_UNSPLIT
    t.bc[~leaf] = -1
    return c


def step_until_error(solver, hook=None, most=12):
    for k in range(most):
        try:
            solver.integrate(hook)
        except DgError as e:
            return k, e.code
    return None


@pytest.mark.parametrize("base,levels", [(3, 2), (4, 3), (6, 2), (7, 2)])
def test_face_sum_error_ends_a_run(base, levels):
    """One thread-block cluster (up to 2048 cells) and the whole GPU: every block leaves the run together, with the
    error of the stage launches, and the GPU goes on."""
    s = Solver(coarsens_into_missing_boundary(base, levels))
    want = step_until_error(s, hook=lambda *_: None)
    s.close()
    assert want is not None and want[1] == MISSING_BC
    for _ in range(5):
        s = Solver(coarsens_into_missing_boundary(base, levels))
        assert step_until_error(s) == want
        s.close()
    s = Solver(cases.lax_liu3(base, levels))
    assert not s.integrate()[1]
    assert np.isfinite(s.active_cells().u).all()
    s.close()


def test_failing_trees_of_a_batch_leave_the_others_alone():
    """Ten trees side by side, two of which fail: the batch reports the error, and every other tree is where
    Solver.integrate takes it, step after step, the failing ones readable."""
    trees = [cases.lax_liu3(3 + k % 3, 2, max_cfl=0.5 - 0.01 * k) for k in range(10)]
    bad = {3: coarsens_into_missing_boundary(4, 2), 8: coarsens_into_missing_boundary(5, 2)}
    trees = [bad.get(k, c) for k, c in enumerate(trees)]
    together, alone = [Solver(c) for c in trees], [Solver(c) for c in trees]
    b = Batch(together)
    failed = 0
    for _ in range(6):
        codes = set()
        for k, s in enumerate(alone):
            try:
                s.integrate()
            except DgError as e:
                assert k in bad
                codes.add(e.code)
        try:
            b.step()
            assert not codes
        except DgError as e:
            failed += 1
            assert {e.code} == codes
        for k, (x, y, c) in enumerate(zip(together, alone, trees)):
            n = x.n_active_cells()
            a = x.active_cells()
            assert a.n == n and np.isfinite(a.u).all()
            if k in bad:
                continue
            w = y.active_cells().sorted(c.params.side_length)
            a = a.sorted(c.params.side_length)
            assert a.n == w.n and a.u.tobytes() == w.u.tobytes() and np.array_equal(a.acti_level, w.acti_level)
            assert x.stats().cell_updates == y.stats().cell_updates
    assert failed > 1
    b.close()
    for s in together + alone:
        s.close()
