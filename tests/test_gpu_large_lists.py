"""Sizes beyond one round of the kernels that stride or scan in rounds: more
source slots than the birth counts' last block scans at once (128 blocks of 128
slots), more list tiles than the compaction has blocks, and than its last block
scans at once."""
import numpy as np
import pytest

from conftest import load_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_births_of_a_large_mesh(precision, gpu_lib):
    """120 x 80 cells are 19,600 slots, 154 blocks: every birth where and with
    what energy the oracle has it.  1e-14: the same FP64 formulas; binary32
    births 1e-6."""
    import mpimc
    import oracle
    nodes = {"XMESHNODES": np.linspace(0.0, 1.0, 121), "YMESHNODES": np.linspace(0.0, 1.0, 81)}
    inputs, mesh = load_deck("tiny_2d", NINPUT="30000", NMAX="90000", **nodes)
    ov = {"precision": precision}
    g, o = mpimc.Engine(inputs, mesh, ov), oracle.Oracle(inputs, mesh, ov)
    assert g.ncells == 9600
    for e in (g, o):
        e.update()
        e.sourcing()
    pg, po = g.particles(), o.particles()
    assert len(pg["E"]) == len(po["E"]) > 9600
    assert np.array_equal(pg["cell"], po["cell"])
    rtol = 1e-14 if precision == 0 else 1e-6
    for k in ("E", "E0", "t", "x", "y"):
        np.testing.assert_allclose(pg[k], po[k], rtol=rtol, atol=rtol * 1e-3, err_msg=k)
    g.close()
    o.close()


@pytest.mark.parametrize("n", [4096 * 257 + 1, 4096 * 1216, 4096 * 1216 + 12345])
@pytest.mark.parametrize("alive", [0.03, 0.9])
def test_compaction_of_a_long_list(n, alive, gpu_lib):
    """The survivors, in order, as numpy's mask selects them."""
    import mpimc
    inputs, mesh = load_deck("tiny_1d")
    e = mpimc.Engine(inputs, mesh, {"precision": 1})
    rng = np.random.default_rng(n)
    live = rng.random(n) < alive
    live[[0, n - 1]] = True  # the ends of the list
    cols = {"t": np.zeros(n), "x": rng.random(n).astype(np.float32).astype(np.float64) * 0.04, "mu": rng.random(n),
            "E": np.arange(n, dtype=np.float64) + 1.0, "E0": np.where(live, 1.0, -1.0),
            "cell": rng.integers(0, e.ncells, n).astype(np.int32)}
    e.set_particles(cols)
    e.clean()
    p = e.particles()
    assert len(p["E"]) == live.sum()
    assert np.array_equal(p["E"], cols["E"][live])  # whole numbers below 2^24: exact in binary32
    assert np.array_equal(p["cell"], cols["cell"][live])
    assert np.array_equal(p["mu"], cols["mu"][live].astype(np.float32).astype(np.float64))
    assert (p["E0"] == 1.0).all()
    e.close()
