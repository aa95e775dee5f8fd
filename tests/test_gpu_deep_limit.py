"""A level limit far above what the flow refines to (deeper than a Morton key resolves) changes nothing: the re-sort after
a global step orders the same cells the same way."""
import dataclasses

import numpy as np
import pytest

from dacti_b200 import cases
from dacti_b200.solver import Solver

pytestmark = pytest.mark.gpu


def _blob3(thresholds):
    c = cases.blast3d(3, 2, thresholds)
    t = c.tree
    r2 = (t.center ** 2).sum(axis=1)
    t.p[1:] = 0.0
    t.p[1:, 0] = (1.0 + 0.3 * np.exp(-r2 / 0.04))[1:]
    t.p[1:, 4] = 1.0
    return c


@pytest.mark.parametrize("make,limits", [(lambda: cases.smooth_periodic(5, 2, (0.05, 0.3)), (12, 29, 30, 31)),
                                         (lambda: _blob3((0.05, 0.15)), (8, 19, 20, 31))])
def test_level_limit_beyond_the_sort_keys(make, limits):
    seen = []
    for limit in limits:
        case = make()
        s = Solver(dataclasses.replace(case, params=dataclasses.replace(case.params, max_level=limit)))
        for _ in range(4):
            assert not s.integrate()[1]
        a, st = s.active_cells(), s.stats()
        s.close()
        assert a.tree_level.max() < limits[0]
        seen.append([(st.cell_updates, st.n_splits, st.n_substeps, st.tree_size)] +
                    [getattr(a, f).tobytes() for f in ("tree_level", "acti_level", "center", "t", "u", "p", "error")])
    assert all(x == seen[0] for x in seen[1:])
