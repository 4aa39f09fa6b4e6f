"""What imc_step reads back and keeps from one call for the next: the list's
length, the step's statistics in host memory, and the step graph."""
import time

import numpy as np
import pytest

from conftest import load_deck

pytestmark = pytest.mark.gpu


def _engine(precision=1):
    import mpimc
    inputs, mesh = load_deck("c1_slab", NINPUT="500", NMAX="6000")
    return mpimc.Engine(inputs, mesh, {"precision": precision, "t_end": 1e6})


def _longer_list(e):
    """Three times the list, the copies in the cells that the originals are in."""
    p = e.particles()
    e.set_particles({k: np.concatenate([v, v, v]) for k, v in p.items()})


def _batch(e, fused):
    import mpimc
    other = _engine(e.deck.precision)
    mpimc.run_batch([e, other], max_steps=5, threads=2, fused=fused)
    other.close()


CHANGES = {
    "set_particles": _longer_list,
    "empty_list": lambda e: e.set_particles({"E": [], "E0": [], "cell": []}),
    "clean": lambda e: e.clean(),
    "sourcing": lambda e: (e.update(), e.sourcing()),
    "run": lambda e: e.run(7),
    "batch": lambda e: _batch(e, False),
    "fused_batch": lambda e: _batch(e, True),
    "load_state": None,
}


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("change", sorted(CHANGES))
def test_step_after_the_list_changed(change, precision, gpu_lib):
    """Steps, another call that changes the list, steps: as a fresh handle that
    loads the state in between goes on, record by record and field by field."""
    e = _engine(precision)
    e.run(6)
    early = e.save_state()
    for _ in range(8):
        e.step()
    if change == "load_state":
        e.load_state(early)
    else:
        CHANGES[change](e)
    fresh = _engine(precision)
    fresh.load_state(e.save_state())
    for _ in range(4):
        a, da = e.step()
        b, db = fresh.step()
        assert a == b and da == db
        assert e.num_particles() == fresh.num_particles()
    for f in ("temp", "radenergydens", "matenergydens"):
        assert np.array_equal(e.field(f), fresh.field(f))
    e.close()
    fresh.close()


def test_records_of_steps_and_runs_agree(gpu_lib):
    """The records that steps read in host memory are those that a run copies."""
    a, b = _engine(), _engine()
    steps = [a.step()[0] for _ in range(20)]
    runs, _ = b.run(20)
    assert steps == runs
    a.close()
    b.close()


def test_first_step_after_a_run(gpu_lib):
    """It reuses the run's graph and allocates nothing: no slower than twice a
    later step (a capture, an instantiation and pinned memory made it four
    times as long).  Medians over engines."""
    first, later = [], []
    for _ in range(9):
        e = _engine()
        e.run(40)
        t = []
        for _ in range(20):
            t0 = time.perf_counter()
            e.step()
            t.append(time.perf_counter() - t0)
        first.append(t[0])
        later.append(np.median(t[4:]))
        e.close()
    assert np.median(first) <= 2.0 * np.median(later)
