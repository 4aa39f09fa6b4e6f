"""Negative opacities, which a deck may state and a cell below zero temperature
has: histories gain energy, exp(-sigma_a f d) above 1, and FP64 state follows
the reference's arithmetic there as FP32 state does."""
import numpy as np
import pytest

from conftest import load_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deck", ["tiny_1d", "tiny_2d"])
@pytest.mark.parametrize("y", [-1e-6, -0.05, -0.4])
def test_a_history_gains_energy(deck, y, gpu_lib):
    """Flights to census through a medium of y mean free paths of negative
    absorption, no collision on the way: every weight is E exp(-y) to 3 units of
    2^-53 for exp and the product, and the deposits are what the list gained."""
    import mpimc
    inputs, mesh = load_deck(deck)
    e = mpimc.Engine(inputs, mesh)
    e.update()
    c, dt = float(inputs["PHYS_C"]), e.time()[1]
    nc = len(e.field("temp"))
    e.set_field("fleck", np.ones(nc))
    e.set_field("sigma_s", np.full(nc, 1e-12))
    e.set_field("sigma_a", np.full(nc, y / (c * dt)))
    n = 500
    rng = np.random.default_rng(5)
    E = rng.uniform(0.5, 1.5, n)
    cols = {"t": np.zeros(n), "E": E, "E0": E, "cell": np.zeros(n, np.int32)}
    if deck == "tiny_1d":
        # from the left (reflecting) end, on to the right
        cols.update(x=rng.uniform(0.0, 0.05, n), mu=rng.uniform(0.5, 1.0, n))
    else:
        # from the bottom left, on to the right (the bottom reflects)
        a = rng.uniform(0.0, 1.2, n)
        cols.update(x=rng.uniform(0.0, 0.1, n), y=rng.uniform(0.0, 0.25, n), ux=np.cos(a), uy=np.sin(a))
    e.set_particles(cols)
    before = e.particles()["E"].sum()
    e.transport()
    p = e.particles()
    assert (p["E0"] >= 0).all()
    np.testing.assert_allclose(p["E"], E * np.exp(-y), rtol=2.0 ** -50, atol=0)
    width = np.asarray(mesh.dx) if deck == "tiny_1d" else np.outer(mesh.dy, mesh.dx).ravel()
    dep = (e.field("energydep").reshape(-1, nc)[0] * width).sum()
    np.testing.assert_allclose(dep, before - p["E"].sum(), rtol=1e-9)
    e.close()


@pytest.mark.parametrize("deck", ["tiny_1d", "tiny_2d"])
@pytest.mark.parametrize("precision", [0, 1])
def test_births_of_negative_energy_end_at_the_cutoff(deck, precision, gpu_lib):
    """The cells of such a deck emit negative energy.  A negative weight is below
    its cut-off, 1 % of itself, from the first segment on: those histories end
    there, as the reference's comparison has it, and none reaches census."""
    import mpimc
    inputs, _ = load_deck(deck)
    n = len(inputs["SIGMA_A_VALS"])
    inputs, mesh = load_deck(deck, SIGMA_A_VALS=["-1e-3"] * n, SIGMA_A_POWERS=["0.0"] * n, SIGMA_S_VALS=["20.0"])
    e = mpimc.Engine(inputs, mesh, {"precision": precision})
    e.update()
    e.sourcing()
    born = e.particles()["E"]
    assert (born < 0).sum() >= 20 and (born > 0).sum() >= 100
    e.transport()
    e.clean()
    left = e.particles()["E"]
    assert 0 < len(left) < len(born) and (left > 0).all()
    e.close()
