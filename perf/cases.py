"""Performance cases of the GB300 Implicit Monte Carlo engine.

Each case is work that a program built on ``mpimc`` has it do through its
public entry points: whole simulations (``Engine`` + ``run`` + the cell
fields), single timesteps of a running simulation, batched ensembles, and the
training of the thick-cell surrogate.  Decks are the repository's own
(tests/golden/decks), with the cell and particle counts of the case.

    listed()            the cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the caller holds before the call
    run(state)          one pass; returns every output of it
    work(case)          bytes and operations that a pass cannot do without
    exact(case, seed)   the pass's outputs in 64 bits, where they have a closed form
"""
import os
import sys

import numpy as np

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(REPO, "mixedprecisionimc.jl_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import mpimc  # noqa: E402
from mpimc import _lib, surrogate  # noqa: E402

DECKS = os.path.join(REPO, "tests", "golden", "decks")
PREC = {"fp64": 0, "fp32": 1, "fp16": 2}
STATE_BYTES = {"fp64": 8, "fp32": 4, "fp16": 2}

# deck file, timesteps of a full run, transport segments per history, and the
# share of a full particle list that a step moves (the channel's walls absorb
# most births in the step that made them)
FAMILY = {
    "slab": ("c2_slab_fine.txt", 602, 1.5),
    "coarse": ("c1_slab.txt", 101, 1.2),
    "suolson": ("suolson.txt", 5001, 1.2),
    "wave": ("c3_heatwave.txt", 150, 12.0),
    "thick": ("thick_heated.txt", 21, 60.0),
    "channel": ("c4_channel2d.txt", 1001, 2.4),
}


def listed():
    return [
        # one timestep of a simulation under way, then its temperature, as a
        # program that watches or couples the run takes it: the Su-Olson
        # benchmark deck as shipped (1000 cells, binary16 state).  Latency and
        # launches are all of it.
        {"name": "step_suolson_fp16", "kind": "step", "deck": "suolson", "prec": "fp16", "cells": 1000,
         "ninput": 1000, "nmax": 50000},
        # a whole small simulation, set-up included: the coarse linearized
        # slab deck as shipped (100 cells, 1e5 particles, double precision)
        {"name": "run_coarse_slab_fp64", "kind": "run", "deck": "coarse", "prec": "fp64", "cells": 100,
         "ninput": 10000, "nmax": 100000, "steps": 101, "learned": False},
        # the flagship deck at full particle count for a third of its clock:
        # short histories, two thousand cells
        {"name": "run_slab_fp32", "kind": "run", "deck": "slab", "prec": "fp32", "cells": 2000,
         "ninput": 2000000, "nmax": 20000000, "steps": 200, "learned": False},
        # the same deck in double precision, the reference's default type, at
        # a tenth of the particles
        {"name": "run_slab_fp64", "kind": "run", "deck": "slab", "prec": "fp64", "cells": 2000,
         "ninput": 200000, "nmax": 2000000, "steps": 60, "learned": False},
        # half-precision particle state (the reference's FLOAT16 decks), an odd mesh
        {"name": "run_slab_fp16", "kind": "run", "deck": "slab", "prec": "fp16", "cells": 1250,
         "ninput": 500000, "nmax": 5000000, "steps": 100, "learned": False},
        # nonlinear heat wave, whole clock at a fifth of the particles: long
        # histories of unequal length
        {"name": "run_wave_fp32", "kind": "run", "deck": "wave", "prec": "fp32", "cells": 500,
         "ninput": 400000, "nmax": 4000000, "steps": 150, "learned": False},
        # the same in double precision, small
        {"name": "run_wave_fp64", "kind": "run", "deck": "wave", "prec": "fp64", "cells": 250,
         "ninput": 20000, "nmax": 200000, "steps": 60, "learned": False},
        # the 2D channel through thick walls: births dominate, the list is
        # compacted every step
        {"name": "run_channel_fp32", "kind": "run", "deck": "channel", "prec": "fp32", "cells": 10,
         "ninput": 4000000, "nmax": 20000000, "steps": 100, "learned": False},
        # 2D in double precision on an odd mesh (98 x 28 cells)
        {"name": "run_channel_fp64", "kind": "run", "deck": "channel", "prec": "fp64", "cells": 7,
         "ninput": 100000, "nmax": 500000, "steps": 60, "learned": False},
        # thick heated cells with the learned surrogate (RANDOMWALK = TRUE)
        {"name": "run_thick_learned", "kind": "run", "deck": "thick", "prec": "fp32", "cells": 30,
         "ninput": 200000, "nmax": 2000000, "steps": 21, "learned": True},
        # a batched ensemble of unlike decks, one transport launch per step
        {"name": "ensemble_fused", "kind": "batch", "decks": 24, "scale": 0.05, "fused": True},
        # training of the surrogate, which every program that turns it on
        # waits for: walks, then Adam steps
        {"name": "train_surrogate", "kind": "train", "samples": 1 << 18, "batch": 8192, "iterations": 1000},
    ]


def _log(rng, a, b):
    return float(np.exp(rng.uniform(np.log(a), np.log(b))))


def _draw_run(rng):
    deck = rng.choice(["slab", "slab", "coarse", "suolson", "wave", "wave", "channel", "channel", "thick"])
    prec = rng.choice(["fp64", "fp32", "fp32", "fp16"])
    learned = deck == "thick"
    segs = FAMILY[deck][2] * (0.5 if learned else 1.0)
    cells = {"slab": lambda: round(_log(rng, 100, 5000)), "coarse": lambda: round(_log(rng, 20, 400)),
             "suolson": lambda: 1000, "wave": lambda: round(_log(rng, 50, 2000)),
             "channel": lambda: rng.randint(3, 13), "thick": lambda: rng.randint(12, 60)}[deck]()
    steps = min(FAMILY[deck][1], round(_log(rng, 10, 200)))
    if prec == "fp16" and deck in ("channel", "wave") or prec == "fp64" and deck == "thick":
        prec = "fp32"
    if prec == "fp64" and deck == "wave":  # its step waits for the longest history
        steps = min(steps, 60)
    # at most the histories of the largest listed case, whose segments and
    # type cost what they do
    most = 2.5e9 / (steps * segs) / {"fp64": 24.0, "fp32": 1.0, "fp16": 1.1}[prec]
    nmax = round(_log(rng, 2.0e4, min(2.0e7, max(4.0e4, most))))
    return {"kind": "run", "deck": deck, "prec": prec, "cells": cells, "ninput": max(1000, nmax // rng.choice([5, 10, 12])),
            "nmax": nmax, "steps": steps, "learned": learned}


def draw(rng):
    kind = rng.choice(["run"] * 7 + ["step", "batch", "train"])
    if kind == "step":
        nmax = round(_log(rng, 1.0e4, 1.0e6))
        deck = rng.choice(["suolson", "coarse"])
        return {"kind": "step", "deck": deck, "prec": rng.choice(["fp64", "fp32", "fp16"]),
                "cells": 1000 if deck == "suolson" else rng.randint(20, 400), "ninput": max(500, nmax // 20), "nmax": nmax}
    if kind == "batch":
        fused = rng.choice([True, True, False])
        return {"kind": "batch", "decks": rng.randint(4, 16 if fused else 8), "scale": round(_log(rng, 0.01, 0.05), 4),
                "fused": fused}
    if kind == "train":
        batch = 64 * rng.choice([32, 48, 64, 96, 128])
        return {"kind": "train", "samples": batch * rng.randint(8, 32), "batch": batch, "iterations": rng.randint(200, 1000)}
    return _draw_run(rng)


# ------------------------------------------------------------------ inputs
def _deck(case, seed):
    """(inputs, mesh, overrides) of a deck with the case's mesh, counts and state type."""
    deck, cells = case["deck"], case["cells"]
    inputs = mpimc.Input.readInputs(os.path.join(DECKS, FAMILY[deck][0]))
    if deck == "channel":  # square cells, `cells` per half unit of length: 14 c x 4 c
        inputs["DX"] = inputs["DY"] = repr(0.5 / cells)
    elif deck != "suolson":
        inputs["DX"] = repr(float(inputs["XSIZE"]) / cells)
    inputs["NINPUT"], inputs["NMAX"], inputs["SEED"] = str(case["ninput"]), str(case["nmax"]), str(1 + seed)
    p = PREC[case["prec"]]
    ov = {"precision": p, "scale_select_precision": p if deck == "suolson" else min(p, 1)}
    return inputs, mpimc.Mesh.mesh_generation(inputs), ov


def _ensemble(case, seed):
    """Decks drawn like the repository's batched ensemble: heat-wave physics
    with the mesh, opacity, heat capacity, surface and counts of each drawn."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["decks"]):
        inputs = mpimc.Input.readInputs(os.path.join(DECKS, FAMILY["wave"][0]))
        # the ensemble's sizes are the case's and not the seed's: another
        # seed is other physics on the same meshes and counts
        u = ((i * 0.6180339887) % 1.0, (i * 0.7548776662) % 1.0)
        nin = max(1000, int(10.0 ** (4.0 + 2.0 * u[1]) * case["scale"]))
        inputs.update({
            "DX": repr(1.0 / round(50.0 * 40.0 ** u[0])),
            "SIGMA_A_VALS": [repr(float(10.0 ** rng.uniform(0.5, 1.5)))],
            "SIGMA_A_POWERS": [repr(0.0 if i % 2 else -3.0)],
            "BEE_VALS": [repr(float(rng.uniform(0.05, 1.0)))],
            "T_SURFACE_VALS": [np.float32(rng.uniform(0.2, 1.0)), np.float32(0.0)],
            "NINPUT": str(nin), "NMAX": str(10 * nin), "SEED": str(1000 * seed + i),
        })
        out.append((inputs, mpimc.Mesh.mesh_generation(inputs)))
    return out


class _Step:
    """A simulation under way: its list filled, its clock open-ended."""

    def __init__(self, case, seed):
        inputs, mesh, ov = _deck(case, seed)
        self.engine = mpimc.Engine(inputs, mesh, dict(ov, t_end=1.0e9))
        self.engine.run(max(32, 2 * case["nmax"] // case["ninput"]))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return {"case": case, "sim": _Step(case, seed)}
    if kind == "run":
        if case["learned"]:
            surrogate.trained_params()  # once per process, as a program that turns it on does
        return {"case": case, "deck": _deck(case, seed)}
    if kind == "batch":
        return {"case": case, "decks": _ensemble(case, seed)}
    return {"case": case, "seed": 1 + seed}


# -------------------------------------------------------------------- pass
def _fields(engine):
    return {k: engine.field(k) for k in ("temp", "radenergydens", "matenergydens")}


def _step_numbers(steps):
    """A run's per-step records: whole numbers, and the energies of the balance."""
    return {"n_census": np.array([s["n_census_out"] for s in steps], np.int64),
            "n_sourced": np.array([s["n_sourced"] for s in steps], np.int64),
            "segments": np.array([s["segments"] for s in steps], np.int64),
            "queries": np.array([s["surrogate_calls"] for s in steps], np.int64),
            "total_energy": np.array([s["total_energy"] for s in steps]),
            "energy_dep": np.array([s["energy_dep"] for s in steps]),
            "rad_energy": np.array([s["rad_energy"] for s in steps])}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        engine = state["sim"].engine
        record, _ = engine.step()
        out = _step_numbers([record])
        out["temp"] = engine.field("temp")
        return out
    if kind == "run":
        inputs, mesh, ov = state["deck"]
        with mpimc.Engine(inputs, mesh, ov) as engine:
            if case["learned"]:
                surrogate.enable(engine)
            steps, _ = engine.run(case["steps"])
            return dict(_fields(engine), **_step_numbers(steps))
    if kind == "batch":
        engines = [mpimc.Engine(i, m) for i, m in state["decks"]]
        try:
            steps, _ = mpimc.run_batch(engines, threads=32, fused=case["fused"])
            return {"steps": np.array(steps, np.int64),
                    "totals": np.array([e.totals() for e in engines], np.int64),
                    "temp": np.concatenate([e.field("temp") for e in engines]),
                    "radenergydens": np.concatenate([e.field("radenergydens") for e in engines])}
        finally:
            for e in engines:
                e.close()
    params, loss = surrogate.train(seed=state["seed"], n_samples=case["samples"], batch=case["batch"],
                                   iterations=case["iterations"], return_loss=True)
    return {"params": params, "loss": loss}


# -------------------------------------------------------------------- work
def _histories(ninput, nmax, steps):
    """Histories moved in `steps` steps of a list that fills to nmax."""
    fill = max(1, min(steps, nmax // max(1, ninput)))
    return ninput * fill * (fill + 1) / 2 + (steps - fill) * nmax


def _run_work(deck, prec, ninput, nmax, steps, full=False):
    # a history's state read once and its census state written once: five
    # state-typed fields (seven in 2D, the starting energy never narrower than
    # 32 bits), cell and scale, and the alive byte; per segment the flight, the
    # attenuation and the two compensated sums
    s = STATE_BYTES[prec]
    dims = 2 if deck == "channel" else 0
    read, write = (4 + dims) * s + max(4, s) + 5, (4 + dims) * s
    if deck == "channel":  # most births die in the step that made them
        h = ninput * steps
        return {"bytes": h * (read + 0.2 * write), "flops": h * 2.4 * 60.0}
    h = steps * nmax if full else _histories(ninput, nmax, steps)
    return {"bytes": h * (read + write), "flops": h * FAMILY[deck][2] * 60.0}


def work(case):
    kind = case["kind"]
    if kind == "step":
        return _run_work(case["deck"], case["prec"], case["ninput"], case["nmax"], 1, full=True)
    if kind == "run":
        return _run_work(case["deck"], case["prec"], case["ninput"], case["nmax"], case["steps"])
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for i in range(case["decks"]):
            nin = max(1000, int(10.0 ** (4.0 + 2.0 * ((i * 0.7548776662) % 1.0)) * case["scale"]))
            w = _run_work("wave", "fp32", nin, 10 * nin, 150)
            total = {k: total[k] + w[k] for k in total}
        return total
    # forward and two backward products per Adam step; inputs, classes and targets read once
    per_walk = 2.0 * 3.0 * (4 * 64 + 3 * 64 * 64)
    return {"bytes": case["samples"] * 28.0 + 3 * 4 * 12800.0,
            "flops": case["iterations"] * case["batch"] * per_walk}


def exact(case, seed):
    # A simulation is a long chain of random histories and a training run a
    # long chain of Adam steps on simulated walks: neither has a closed form
    # that torch or numpy gives within seconds.
    return None
