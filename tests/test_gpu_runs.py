"""Device-resident runs (one launch for many substeps) give the bits of the stage-by-stage launches.

A substep callback makes the host issue every stage of every substep itself; without one the same step
runs on the device. Both use the same arithmetic, so cells, time levels, state and counters are equal bit
for bit. The cases cover a cluster of a few cells, the edges of the sizes that choose a run's shape (one
thread-block cluster up to 2048 cells, the whole GPU above, the launches above 65536), clusters that
outgrow the scratch, runs that stop for a pool without room, surface tension, both forms, and a NaN.
"""
import dataclasses

import numpy as np
import pytest

from dacti_b200 import cases
from dacti_b200.models import ModelId
from dacti_b200.parity import _keys
from dacti_b200.solver import Solver, step_many

pytestmark = pytest.mark.gpu

NS = dict(model=ModelId.NAVIER_STOKES, mu=2e-3, prandtl=0.72)
CASES = {
    "few_cells": (lambda: cases.lax_liu3(2, 1), 6, "fp64"),
    "tiny": (lambda: cases.lax_liu3(3, 2), 8, "fp64"),
    "cluster_edge": (lambda: cases.lax_liu3(5, 2), 10, "fp64"),  # its largest cluster grows through 2048
    "viscous2": (lambda: cases.lax_liu3(4, 3, **NS), 6, "fp64"),
    "periodic": (lambda: cases.periodic_blob(5, 2), 6, "fp64"),
    "limiter": (lambda: cases.smooth_periodic(5, 2, limiter=5), 5, "fp64"),
    "walls3": (lambda: cases.blast3d(3, 2), 3, "fp64"),
    "viscous3": (lambda: cases.blast3d(3, 2, model=ModelId.NAVIER_STOKES, mu=2e-3), 3, "fp64"),
    "drop2": (lambda: cases.shock_drop(2, 4, 3), 2, "fp64"),
    "drop2_terms": (lambda: cases.shock_drop(2, 4, 2, mu=(1e-3, 1.8e-5), conductivity=(0.6, 0.026)), 2, "mixed"),
    "drop3_mixed": (lambda: cases.shock_drop(3, 4, 2), 2, "mixed"),
    "above_runs": (lambda: cases.shock_drop(3, 5, 3), 3, "fp64"),  # clusters of up to 127 thousand cells
}


def _run(case, steps, form="fp64", hook=None):
    s = Solver(case)
    s.set_form(form)
    dts, breaks = [], []
    for _ in range(steps):
        dt, fb = s.integrate(hook)
        dts.append(dt)
        breaks.append(fb)
        if fb:
            break
    snap, st = s.active_cells(), s.stats()
    counters = (st.cell_updates, st.n_splits, st.n_unsplits, st.n_substeps, st.tree_size, st.n_gc, st.max_acti_level,
                list(st.acti_time), list(st.acti_counter), list(st.n_clusters), list(st.n_buffers))
    s.close()
    o = np.argsort(_keys(snap, case.params.side_length))
    fields = [getattr(snap, f)[o] for f in ("tree_level", "acti_level", "center", "t", "u", "p", "error", "max_dt", "cfl")]
    if snap.k is not None:
        fields.append(np.delete(snap.k, 1, axis=1)[o])  # column 1 is not used
    return dts, breaks, counters, fields


def _same(a, b):
    assert a[0] == b[0] and a[1] == b[1]
    assert a[2] == b[2]
    for x, y in zip(a[3], b[3]):
        assert x.tobytes() == y.tobytes()


@pytest.mark.parametrize("name", sorted(CASES))
def test_run_equals_stage_launches(name):
    make, steps, form = CASES[name]
    case = make()
    seen = []
    by_stage = _run(case, steps, form, hook=lambda s, level, *_: seen.append(level))
    _same(_run(case, steps, form), by_stage)
    assert len(seen) == by_stage[2][3]


def test_run_resumes_after_pool_growth():
    """A pool with room for hardly a split: the run stops before the regrid, the host grows the pool and
    finishes that substep, and the next run goes on."""
    case = cases.lax_liu3(4, 3)
    small = dataclasses.replace(case.params, pool_capacity=case.tree.n_nodes + 1024)
    roomy = dataclasses.replace(case.params, pool_capacity=200000)
    tight = _run(dataclasses.replace(case, params=small), 8)
    _same(tight, _run(dataclasses.replace(case, params=roomy), 8))
    _same(tight, _run(dataclasses.replace(case, params=small), 8, hook=lambda *_: None))


def test_run_with_surface_tension():
    case = cases.osc_drop(4, 2, rho_gas=0.5)
    _same(_run(case, 2), _run(case, 2, hook=lambda *_: None))


def test_run_stops_at_a_nan():
    case = cases.lax_liu3(4, 1)
    case.tree.p[np.nonzero(case.tree.leaf_mask())[0][37], 0] = -1.0
    a, b = _run(case, 1), _run(case, 1, hook=lambda *_: None)
    assert a[1] == b[1] == [True]
    assert a[2] == b[2]


def test_runs_side_by_side():
    """More solvers at once than the GPU holds thread-block clusters, of different sizes."""
    batch = [cases.lax_liu3(3 + k % 4, 2, max_cfl=0.5 - 0.01 * k) for k in range(11)]
    side = [Solver(c) for c in batch]
    for _ in range(3):
        step_many(side, threads=11)
    for c, s in zip(batch, side):
        got, st = s.active_cells(), s.stats()
        s.close()
        want = _run(c, 3)
        o = np.argsort(_keys(got, 1.0))
        assert got.u[o].tobytes() == want[3][4].tobytes() and st.cell_updates == want[2][0]


def test_large_runs_side_by_side():
    """Fewer solvers than make one-cluster runs: clusters that the host steps (262144 cells), grid-wide runs and a
    small tree at once, on a thread each."""
    batch = [cases.lax_liu3(9, 1), cases.lax_liu3(6, 3), cases.lax_liu3(9, 1, max_cfl=0.4), cases.lax_liu3(7, 2), cases.lax_liu3(3, 2)]
    side = [Solver(c) for c in batch]
    for _ in range(3):
        step_many(side, threads=5)
    for c, s in zip(batch, side):
        got, st = s.active_cells(), s.stats()
        s.close()
        want = _run(c, 3)
        o = np.argsort(_keys(got, 1.0))
        assert got.u[o].tobytes() == want[3][4].tobytes() and st.cell_updates == want[2][0]


@pytest.mark.parametrize("name", ["tiny", "walls3", "drop2", "drop3_mixed"])
def test_fields_equal_records(name):
    """active_cells (field arrays) and the record read-back give the same values, before and after steps."""
    make, _, form = CASES[name]
    s = Solver(make())
    s.set_form(form)
    for _ in range(2):
        a, b = s.active_cells(), s.active_cells_noalloc()
        for f in ("tree_level", "acti_level", "center", "t", "u", "p", "error", "max_dt", "cfl", "k"):
            x, y = getattr(a, f), getattr(b, f)
            assert (x is None and y is None) or (x.dtype == y.dtype and x.shape == y.shape and x.tobytes() == y.tobytes())
        s.integrate()
    s.close()
