"""What the framework is timed on: whole runs through its public entry points.

A solver case is a short simulation as a program of this framework runs it: the initial tree is in hand
(host arrays, from the scene builders), `run` constructs the solver on the GPU, advances a number of
global steps and reads every active cell back, as a driver does for a frame. The batched cases do the
same for many independent trees at once; the forecaster cases train and apply the regrid network on host
samples. All solver outputs are FP64 and follow the reference's arithmetic, so there is no second value
to hold them against short of another adaptive solver; the forecaster's are checked in 64 bits.

Families (`kind`), with the sizes of the repository's own tests, fixtures and benchmark:
- lax      2D Euler or Navier-Stokes quadrant problem on the unit square (`model`), zero-gradient sides;
- cylinder 2D Navier-Stokes flow past a no-slip cylinder, inflow, outflow and free-slip sides;
- drop     air-water shock-drop, five equations, 2D or 3D (`dims`), plain or mixed form (`form`), with
           viscous and heat terms or without (`viscous`);
- blast    3D Euler or Navier-Stokes blast with both wall types and a periodic side;
- trees    independent 2D Euler quadrant problems, stepped as a lockstep batch or concurrently (`via`);
- train, predict   the regrid forecaster's network.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from dacti_b200 import cases
from dacti_b200.casefile import Case, SolverParams, prune_inactive
from dacti_b200.forecast import Mlp
from dacti_b200.models import BcType, ModelId, ModelShape
from dacti_b200.scene import BoundarySpec, SceneSpec, build_tree
from dacti_b200.scene_gpu import build_tree_device
from dacti_b200.solver import Batch, Solver, step_many

N_IN = 15  # forecaster inputs of a 2D case (5 + 5 D)
HIDDEN = 64


def listed():
    return [
        # the smallest simulation: a few hundred to two thousand cells, where every launch and wait counts
        {"name": "lax_tiny", "kind": "lax", "model": "euler", "base": 4, "levels": 2, "steps": 12},
        # the 2D Euler configuration of the tests and documents (64^2 base, +3 levels)
        {"name": "lax_config", "kind": "lax", "model": "euler", "base": 6, "levels": 3, "steps": 16},
        # the Navier-Stokes cylinder at its stated size (128 x 64 base, +5 levels)
        {"name": "cylinder", "kind": "cylinder", "base": 7, "levels": 5, "steps": 5},
        # 2D five-equation shock-drop: deep time levels over few cells
        {"name": "drop2d", "kind": "drop", "dims": 2, "base": 6, "levels": 3, "steps": 3, "form": "fp64", "viscous": False},
        # 3D Euler blast: a refined shell that grows from a uniform grid, pools that grow with it
        {"name": "blast3d", "kind": "blast", "model": "euler", "base": 5, "levels": 2, "steps": 3},
        # 3D shock-drop at a quarter of the benchmark's resolution per axis less one level, plain form
        {"name": "drop3d", "kind": "drop", "dims": 3, "base": 5, "levels": 3, "steps": 2, "form": "fp64", "viscous": False},
        # the same in the mixed form
        {"name": "drop3d_mixed", "kind": "drop", "dims": 3, "base": 5, "levels": 3, "steps": 2, "form": "mixed", "viscous": False},
        # the largest: the benchmark's depth (64 base cells along x, +4 levels) in a box half as wide and high
        {"name": "drop3d_large", "kind": "drop", "dims": 3, "base": 6, "levels": 4, "steps": 1, "form": "fp64", "viscous": False},
        # a parameter study: independent small trees in lockstep
        {"name": "trees_batch", "kind": "trees", "via": "batch", "count": 24, "base": 5, "levels": 2, "steps": 3},
        # the same study with one stream per tree
        {"name": "trees_many", "kind": "trees", "via": "many", "count": 24, "base": 5, "levels": 2, "steps": 3},
        # one epoch of the forecaster's training on a modest sample set, the minibatch that training uses
        {"name": "forecast_train", "kind": "train", "samples": 12000, "batch": 512, "epochs": 1},
        # the forecast over the cells of a large 2D frame
        {"name": "forecast_predict", "kind": "predict", "samples": 300000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lax", "lax", "cylinder", "drop", "drop", "drop", "blast", "trees", "train", "predict"])
    if kind == "lax":
        return {"kind": kind, "model": rng.choice(["euler", "navier_stokes"]), "base": rng.randint(4, 7),
                "levels": rng.randint(1, 3), "steps": rng.randint(3, 13)}
    if kind == "cylinder":
        return {"kind": kind, "base": rng.randint(5, 7), "levels": rng.randint(3, 5), "steps": rng.randint(2, 7)}
    if kind == "drop":
        dims = rng.choice([2, 3])
        base, levels = (rng.randint(4, 6), rng.randint(2, 4)) if dims == 2 else (rng.randint(4, 5), rng.randint(2, 3))
        return {"kind": kind, "dims": dims, "base": base, "levels": levels, "steps": rng.randint(1, 3),
                "form": rng.choice(["fp64", "fp64", "mixed"]), "viscous": rng.random() < 0.35}
    if kind == "blast":
        return {"kind": kind, "model": rng.choice(["euler", "navier_stokes"]), "base": rng.randint(3, 5), "levels": rng.randint(1, 2),
                "steps": rng.randint(2, 3)}
    if kind == "trees":
        return {"kind": kind, "via": rng.choice(["batch", "many"]), "count": rng.randint(5, 40), "base": rng.randint(4, 5),
                "levels": 2, "steps": rng.randint(2, 3)}
    if kind == "train":
        return {"kind": kind, "samples": _log_int(rng, 3000, 15000), "batch": rng.choice([500, 512, 1000, 1024]), "epochs": 1}
    return {"kind": kind, "samples": _log_int(rng, 1000, 1000000)}


# ---- inputs -------------------------------------------------------------------------------------

def _quadrants(rng, base, levels):
    """A 2D Euler quadrant problem with moderate random states (no near-vacuum that breaks the run)."""
    q = np.empty((4, 4))
    q[:, 0] = rng.uniform(0.5, 2.0, 4)
    q[:, 1] = rng.uniform(-0.4, 0.4, 4)
    q[:, 2] = rng.uniform(-0.4, 0.4, 4)
    q[:, 3] = rng.uniform(0.5, 2.0, 4)

    def x2p(c):
        x, y = c[:, 0], c[:, 1]
        return q[np.where(x > 0, np.where(y > 0, 0, 3), np.where(y > 0, 1, 2))].copy()

    side = BoundarySpec(BcType.ZERO_GRADIENT)
    spec = SceneSpec(ModelShape(ModelId.EULER, 2), (1.0, 1.0), base, base + levels, x2p, [(side, side), (side, side)])
    prm = SolverParams(side_length=1.0, active_size=(1.0, 1.0), periodic=(False, False), max_cfl=0.5, max_dt=1.0,
                       error_threshold=(0.02, 0.05), max_level=base + levels, min_level=base, weights=(1.0, 0.0, 0.0, 0.0))
    return Case(build_tree(spec), prm)


def _net_params(rng):
    w = [rng.uniform(-1, 1, HIDDEN * N_IN) * math.sqrt(6.0 / N_IN), rng.uniform(-0.1, 0.1, HIDDEN),
         rng.uniform(-1, 1, HIDDEN * HIDDEN) * math.sqrt(6.0 / HIDDEN), rng.uniform(-0.1, 0.1, HIDDEN),
         rng.uniform(-1, 1, HIDDEN) * math.sqrt(6.0 / (HIDDEN + 1)), rng.uniform(-0.1, 0.1, 1)]
    return np.concatenate(w).astype(np.float32)


def _samples(rng, n):
    """Feature rows as the solver gives them: compressed variations >= 0, levels, velocities; labels that
    follow the steepest of them with some noise, a fifth positive."""
    x = np.log1p(100.0 * np.abs(rng.standard_normal((n, N_IN))) * 10.0 ** rng.uniform(-4, -0.5, (n, 1)))
    x[:, 3] = rng.integers(5, 13, n) / 16.0
    x[:, 5:7] = rng.uniform(-0.5, 0.5, (n, 2))
    score = x[:, 0] + 0.5 * x[:, 1] + 0.3 * rng.standard_normal(n)
    return x.astype(np.float32), (score > np.quantile(score, 0.8)).astype(np.float32)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "lax":
        model = ModelId.EULER if case["model"] == "euler" else ModelId.NAVIER_STOKES
        c = cases.lax_liu3(case["base"], case["levels"], model=model, **({"mu": 2e-3, "prandtl": 0.72} if case["model"] != "euler" else {}))
        c.tree.p[:, 0] *= rng.uniform(0.995, 1.005)
        c.tree.p[:, 3] *= rng.uniform(0.995, 1.005)
        return {"case": case, "tree": c}
    if kind == "cylinder":
        spec, prm = cases.cylinder_ns_spec(mach=rng.uniform(0.2, 0.4), base_level=case["base"], levels=case["levels"])
        return {"case": case, "tree": Case(build_tree_device(spec), prm)}
    if kind == "drop":
        more = {"mu": (1e-3, 1.8e-5), "conductivity": (0.6, 0.026)} if case["viscous"] else {}
        deep = case["dims"] == 3 and case["base"] + case["levels"] >= 10
        spec, prm = cases.shock_drop_spec(case["dims"], case["base"], case["levels"], aspect=4 if deep else 2,
                                          mach=rng.uniform(1.45, 1.55), **more)
        c = Case(build_tree_device(spec), prm)
        if deep:  # large trees go up without their inactive parts, into a pool with room for the run
            c = prune_inactive(c)
            c.params.pool_capacity = int(3.3 * c.tree.n_nodes)
        return {"case": case, "tree": c}
    if kind == "blast":
        model = ModelId.EULER if case["model"] == "euler" else ModelId.NAVIER_STOKES
        c = cases.blast3d(case["base"], case["levels"], model=model, **({"mu": 2e-3} if case["model"] != "euler" else {}))
        c.tree.p[:, 4] *= np.where(c.tree.p[:, 4] > 2.0, rng.uniform(0.9, 1.0), 1.0)
        return {"case": case, "tree": c}
    if kind == "trees":
        return {"case": case, "trees": [_quadrants(rng, case["base"] + k % 2, case["levels"]) for k in range(case["count"])]}
    state = {"case": case, "net": Mlp(N_IN), "params": _net_params(rng)}
    state["net"].params = state["params"]
    state["x"], state["y"] = _samples(rng, case["samples"])
    return state


# ---- one pass -----------------------------------------------------------------------------------

def _rows(case):
    """Rows of a pass's output arrays: room for the cells of any run of the case (how many there are
    depends on the flow), the rest zero."""
    kind, base, full = case["kind"], case["base"], case["base"] + case["levels"]
    if kind == "lax":  # fronts: a band of finest cells along lines
        return min(4 ** full, 4 ** base + 60 * 2 ** full)
    if kind == "trees":
        return 12 * 4 ** base * case["count"]
    if kind == "cylinder":
        return 4 ** base + 16 * 2 ** full
    if kind == "blast":  # shells: a layer of finest cells over areas
        return min(8 ** full, 44 * 4 ** full)
    if case["dims"] == 2:
        return 4 ** base + 20 * 2 ** full
    return (8 + 5 * case["steps"]) * 4 ** full // 4 if full < 10 else 5 * 4 ** full // 4


def _frame(case, snaps):
    """Every field of the frames' cells, one array per field over all trees."""
    out = {"cells": sum(s.n for s in snaps)}
    for name in ("tree_level", "acti_level", "center", "t", "u", "p", "error", "max_dt", "cfl", "k"):
        parts = [getattr(s, name) for s in snaps]
        if parts[0] is not None:
            a = parts[0] if len(parts) == 1 else np.concatenate(parts)
            a.resize((_rows(case),) + a.shape[1:], refcheck=False)
            out[name] = a
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "predict":
        return state["net"].predict(state["x"])
    if kind == "train":
        net = state["net"]
        net.params = state["params"]
        loss = net.train(state["x"], state["y"], epochs=case["epochs"], batch=case["batch"], lr=3e-3, pos_weight=4.0)
        return {"loss": loss, "params": net.params}
    if kind == "trees":
        solvers = [Solver(c) for c in state["trees"]]
        if case["via"] == "batch":
            batch = Batch(solvers)
            for _ in range(case["steps"]):
                batch.step()
            batch.close()
        else:
            for _ in range(case["steps"]):
                step_many(solvers)
        out = _frame(case, [s.active_cells() for s in solvers])
        for s in solvers:
            s.close()
        return out
    solver = Solver(state["tree"])
    if kind == "drop":
        solver.set_form(case["form"])
    for _ in range(case["steps"]):
        solver.integrate()
    out = _frame(case, [solver.active_cells()])
    solver.close()
    return out


# ---- what a pass cannot do without ---------------------------------------------------------------

def _updates(case):
    """Leaf cell-updates of a pass, estimated from the base grid and the depth: base cells x level
    substeps x a factor of the family (measured on the listed sizes)."""
    kind, base, levels = case["kind"], case["base"], case["levels"]
    if kind == "lax":
        return 2.0 * 4.0 ** base * 2.0 ** (levels + 3) * case["steps"]
    if kind == "cylinder":
        return 1.0 * 4.0 ** base * 2.0 ** (levels + 3) * case["steps"]
    if kind == "blast":
        return 4.0 * 8.0 ** base * 2.0 ** (levels + 2) * case["steps"]
    if kind == "trees":
        return 2.0 * case["count"] * 2.5 * 4.0 ** base * 2.0 ** (levels + 2) * case["steps"]
    if case["dims"] == 2:
        return 0.2 * 4.0 ** base * 2.0 ** (levels + 6) * case["steps"]
    return (0.3 * 8.0 ** base * 2.0 ** (levels + 6) if base + levels < 10 else 1.3e8) * case["steps"]


def work(case):
    """Solver: state in and out per leaf cell-update (16 E + 8 D + 12 bytes; about 60 operations per face
    and component). Forecaster: samples in, predictions or weights out; 2 operations per weight and
    sample forward, 4 more backward."""
    kind = case["kind"]
    weights = HIDDEN * (N_IN + 1) + HIDDEN * (HIDDEN + 1) + HIDDEN + 1
    if kind == "predict":
        return {"bytes": 4.0 * case["samples"] * (N_IN + 1), "flops": 2.0 * weights * case["samples"]}
    if kind == "train":
        n = case["samples"] * case["epochs"]
        return {"bytes": 4.0 * n * (N_IN + 1) + 28.0 * weights * math.ceil(case["samples"] / case["batch"]) * case["epochs"],
                "flops": 6.0 * weights * n}
    three = kind == "blast" or case.get("dims") == 3
    D = 3 if three else 2
    E = D + 4 if kind == "drop" else D + 2
    n = _updates(case)
    return {"bytes": (16.0 * E + 8.0 * D + 12.0) * n, "flops": 60.0 * D * E * n}


# ---- 64-bit values of the forecaster --------------------------------------------------------------

def _unpack(w):
    cut = np.cumsum([HIDDEN * N_IN, HIDDEN, HIDDEN * HIDDEN, HIDDEN, HIDDEN])
    w1, b1, w2, b2, w3, b3 = np.split(w, cut)
    return w1.reshape(HIDDEN, N_IN), b1, w2.reshape(HIDDEN, HIDDEN), b2, w3, b3


def _shuffle(perm, state):
    """The training order: Fisher-Yates with splitmix64 (Steele, Lea and Flood, 2014)."""
    mask = (1 << 64) - 1
    for k in range(len(perm) - 1, 0, -1):
        state = (state + 0x9E3779B97F4A7C15) & mask
        z = state
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (k + 1)
        perm[k], perm[j] = perm[j], perm[k]
    return state


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("train", "predict"):
        return None  # FP64 already, and adaptive: no plain 64-bit value within seconds
    rng = np.random.default_rng(seed)
    params = _net_params(rng)
    x, y = (a.astype(np.float64) for a in _samples(rng, case["samples"]))
    if kind == "predict":  # the network predicts with its weights rounded to bfloat16
        w = torch.from_numpy(params).bfloat16().double().numpy()
        w1, b1, w2, b2, w3, b3 = _unpack(w)
        a2 = np.maximum(np.maximum(x @ w1.T + b1, 0.0) @ w2.T + b2, 0.0)
        return 1.0 / (1.0 + np.exp(-(a2 @ w3 + b3)))
    w = params.astype(np.float64)
    m, v, t, state, loss, pw, lr = np.zeros_like(w), np.zeros_like(w), 0, 7, 0.0, 4.0, float(np.float32(3e-3))
    perm = list(range(case["samples"]))
    for _ in range(case["epochs"]):
        state = _shuffle(perm, state)
        order, loss = np.array(perm), 0.0
        for first in range(0, case["samples"], case["batch"]):
            idx = order[first:first + case["batch"]]
            w1, b1, w2, b2, w3, b3 = _unpack(w)
            a1 = np.maximum(x[idx] @ w1.T + b1, 0.0)
            a2 = np.maximum(a1 @ w2.T + b2, 0.0)
            z, yt = a2 @ w3 + b3[0], y[idx]
            loss += float((pw * yt * np.logaddexp(0.0, -z) + (1.0 - yt) * np.logaddexp(0.0, z)).sum())
            dz = (pw * yt + 1.0 - yt) / (1.0 + np.exp(-z)) - pw * yt
            d2 = np.where(a2 > 0.0, dz[:, None] * w3, 0.0)
            d1 = np.where(a1 > 0.0, d2 @ w2, 0.0)
            g = np.concatenate([(d1.T @ x[idx]).ravel(), d1.sum(0), (d2.T @ a1).ravel(), d2.sum(0), dz @ a2, [dz.sum()]]) / len(idx)
            t += 1
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            w = w - lr * (m / (1.0 - 0.9 ** t)) / (np.sqrt(v / (1.0 - 0.999 ** t)) + 1e-8)
    return {"loss": loss / case["samples"], "params": w}
