"""Errors that a stage finds on the device: every way of stepping reports the same one."""
import numpy as np
import pytest

from dacti_b200 import cases
from dacti_b200.solver import DgError, Solver

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
