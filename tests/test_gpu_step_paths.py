"""Which way a step takes: device-resident runs, the host's stage launches and the lockstep batch, each seen in the launch
counts, and each with the bits of the others."""
import dataclasses

import numpy as np
import pytest

from dacti_b200 import cases
from dacti_b200.solver import KERNEL_KINDS, Batch, Solver

pytestmark = pytest.mark.gpu
FLUX, REGRID = KERNEL_KINDS.index("flux"), KERNEL_KINDS.index("regrid")


def _launches(case, steps, hook=None):
    """Of some steps: launches of runs, stage launches of the face sums and of the regrid, substeps, the largest cluster
    that a step left, and the cells."""
    s = Solver(case)
    a, largest = s.stats(), 0
    for _ in range(steps):
        s.integrate(hook)
        largest = max(largest, *s.stats().n_clusters)
    b, cells = s.stats(), s.active_cells().sorted(case.params.side_length)
    s.close()
    kinds = [y - x for x, y in zip(a.kernel_launches, b.kernel_launches)]
    return b.n_launches - a.n_launches - sum(kinds), kinds[FLUX], kinds[REGRID], b.n_substeps, largest, cells


# one thread-block cluster throughout; from one cluster to the whole GPU; the whole GPU
@pytest.mark.parametrize("base,levels,steps,low,high", [(3, 2, 4, 0, 2048), (5, 2, 18, 2048, 65536), (6, 2, 3, 2048, 65536)])
def test_steps_are_runs(base, levels, steps, low, high):
    case = cases.lax_liu3(base, levels)
    runs, flux, _, substeps, largest, cells = _launches(case, steps)
    assert runs >= steps and flux == 0 and low < largest <= high
    runs, flux, _, n, _, want = _launches(case, steps, hook=lambda *_: None)
    assert runs == 0 and flux == n == substeps
    assert cells.n == want.n and cells.u.tobytes() == want.u.tobytes()


def test_large_clusters_are_the_hosts():
    runs, flux, _, substeps, largest, _ = _launches(cases.shock_drop(3, 5, 3), 3)
    assert runs > 0 and 0 < flux < substeps and largest > 65536


def test_tight_pool_stops_runs():
    case = cases.lax_liu3(4, 3)
    small = dataclasses.replace(case.params, pool_capacity=case.tree.n_nodes + 1024)
    runs, flux, regrid, _, _, _ = _launches(dataclasses.replace(case, params=small), 8)
    assert runs > 8 and flux == 0 and regrid > 0


LOCKSTEP = {
    "euler2": lambda: cases.riemann_batch(12, seed=11, base_levels=(4, 6), extra_levels=(2, 3)),
    "nan_trees": lambda: cases.riemann_batch(24, seed=3, base_levels=(4, 5), extra_levels=(2, 3)),
    "drops3": lambda: [cases.shock_drop(3, 3, 2), cases.shock_drop(3, 4, 1)],
    "drops2": lambda: [cases.shock_drop(2, 4, 3), cases.shock_drop(2, 5, 2), cases.shock_drop(2, 4, 2)],
    "tension": lambda: [cases.osc_drop(4, 2, rho_gas=0.5), cases.osc_drop(4, 1, rho_gas=0.5)],
    "walls3": lambda: [cases.blast3d(3, 2), cases.blast3d(4, 1)],
}


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("name", sorted(LOCKSTEP))
def test_lockstep_and_runs_equal_single_steps(name, form):
    """The same trees in lockstep (asked for by the timing of its stages), as one run per tree or what else the batch
    chooses, and one by one."""
    trees = LOCKSTEP[name]()
    lock, free, alone = ([Solver(c) for c in trees] for _ in range(3))
    for s in lock + free + alone:
        s.set_form(form)
    bl, bf = Batch(lock), Batch(free)
    bl.set_profiling(True)
    breaks = 0
    for _ in range(3):
        want = [s.integrate()[1] for s in alone]
        assert bl.step() == bf.step() == want
        breaks += sum(want)
    assert bl.stage_times()["face_sum"][1] > 0 and bf.stage_times()["face_sum"][1] == 0
    assert breaks > 0 or name != "nan_trees"
    bl.close()
    bf.close()
    for a, b, w, c in zip(lock, free, alone, trees):
        sw, tw = w.active_cells().sorted(c.params.side_length), w.stats()
        for s in (a, b):
            x, t = s.active_cells().sorted(c.params.side_length), s.stats()
            assert x.n == sw.n and s.global_dt == w.global_dt
            for f in ("u", "p", "t", "error"):
                assert np.array_equal(getattr(x, f), getattr(sw, f), equal_nan=True)
            assert np.array_equal(x.acti_level, sw.acti_level) and np.array_equal(x.tree_level, sw.tree_level)
            assert (t.cell_updates, t.n_substeps, t.n_splits, t.n_unsplits, t.tree_size) == \
                (tw.cell_updates, tw.n_substeps, tw.n_splits, tw.n_unsplits, tw.tree_size)
    for s in lock + free + alone:
        s.close()
