"""A handle that has taken part in a batch of handles side by side, whose
transport launches are small, has the whole GPU again afterwards: its transport
takes as long as that of a handle that ran alone.  (The batch's launches are 13
blocks on this deck, the handle's own 152, three to five times as fast; the
bound is twice, which leaves room for clocks and noise.)"""
import pytest

from conftest import load_deck

pytestmark = pytest.mark.gpu


def _stages(e):
    for call in (e.update, e.sourcing, e.transport, e.clean, e.tally, e.energycheck, e.timestep):
        call()


def _transport_ms(e, how):
    e.set_timing(True)
    e.transport_timing()  # reading resets
    for _ in range(8):
        {"stages": lambda: _stages(e), "step": e.step, "run": lambda: e.run(1)}[how]()
    ms, launches = e.transport_timing()
    assert launches == 8
    e.set_timing(False)
    return ms


@pytest.mark.parametrize("how", ["stages", "step", "run"])
def test_whole_gpu_after_a_batch(how, gpu_lib):
    import mpimc
    inputs, mesh = load_deck("c1_slab")
    alone = mpimc.Engine(inputs, mesh)
    alone.run(40)
    pair = [mpimc.Engine(inputs, mesh) for _ in range(2)]
    steps, _ = mpimc.run_batch(pair, max_steps=40, threads=2)
    assert steps == [40, 40]
    want = _transport_ms(alone, how)
    for e in pair:
        assert _transport_ms(e, how) <= 2.0 * want
    for e in pair + [alone]:
        e.close()


def test_shapes_change_no_result(gpu_lib):
    """Batches and runs in turn: every field as that of the same steps alone."""
    import mpimc
    import numpy as np
    inputs, mesh = load_deck("c1_slab")
    alone = mpimc.Engine(inputs, mesh)
    alone.run(24)
    pair = [mpimc.Engine(inputs, mesh) for _ in range(2)]
    for _ in range(4):
        mpimc.run_batch(pair, max_steps=3, threads=2)
        for e in pair:
            e.run(2)
            e.step()
    for e in pair:
        assert e.time() == alone.time()
        for f in ("temp", "radenergydens", "matenergydens"):
            assert np.array_equal(e.field(f), alone.field(f))
        e.close()
    alone.close()
