"""The fused batch's blocks each start at the deck of their share of the work
and go through the others in turn: with any number of decks (one, a lane's
eight and one more, more than a warp, the most there can be) every list is
walked once, and each deck's fields equal its own run's bit for bit."""
import os
import sys

import numpy as np
import pytest

from conftest import REPO

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(REPO, "tests", "golden"))


@pytest.mark.parametrize("n", [1, 8, 9, 33, 256])
def test_every_deck_is_walked_once(gpu_lib, n):
    import mpimc
    from c5_decks import c5_decks
    decks = c5_decks(n, particle_scale=0.002)
    engines = [mpimc.Engine(i, m) for i, m in decks]
    steps, _ = mpimc.run_batch(engines, max_steps=4, fused=True)
    assert steps == [4] * n
    for (inputs, mesh), e in zip(decks, engines):
        alone = mpimc.Engine(inputs, mesh)
        alone.run(4)
        assert e.totals() == alone.totals()
        assert np.array_equal(e.field("temp"), alone.field("temp"))
        assert np.array_equal(e.field("radenergydens"), alone.field("radenergydens"))
        alone.close()
        e.close()
