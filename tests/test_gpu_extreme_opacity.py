"""Scattering opacities at the ends of their range: an infinite one collides at
once and for ever (the history stops at the segment cap, which the caller is
told), one of 0 never, FP64 state as FP32."""
import numpy as np
import pytest

from conftest import load_deck

pytestmark = pytest.mark.gpu


def _transport(deck, precision, sigma_s):
    import mpimc
    inputs, mesh = load_deck(deck, SEGMENTCAP="50")
    e = mpimc.Engine(inputs, mesh, {"precision": precision})
    e.update()
    nc = len(e.field("temp"))
    e.set_field("fleck", np.ones(nc))
    e.set_field("sigma_a", np.full(nc, 1e-3))
    e.set_field("sigma_s", np.full(nc, sigma_s))
    n = 96
    cols = {"t": np.zeros(n), "E": np.ones(n), "E0": np.ones(n), "cell": np.zeros(n, np.int32),
            "x": np.linspace(0.01, 0.04, n)}
    if deck == "tiny_1d":
        cols["mu"] = np.linspace(0.5, 1.0, n)
    else:
        a = np.linspace(0.1, 1.2, n)
        cols.update(y=np.linspace(0.02, 0.2, n), ux=np.cos(a), uy=np.sin(a))
    e.set_particles(cols)
    try:
        e.transport()
        return None, e.particles()
    except mpimc._lib.ImcError as err:
        return str(err), e.particles()
    finally:
        e.close()


@pytest.mark.parametrize("deck", ["tiny_1d", "tiny_2d"])
@pytest.mark.parametrize("precision", [0, 1])
def test_infinite_opacity_stops_at_the_cap(deck, precision, gpu_lib):
    err, p = _transport(deck, precision, np.inf)
    assert err is not None and "segment cap" in err
    assert (p["E0"] < 0).all()  # every history ended


@pytest.mark.parametrize("deck", ["tiny_1d", "tiny_2d"])
@pytest.mark.parametrize("precision", [0, 1])
def test_no_opacity_never_collides(deck, precision, gpu_lib):
    err, p = _transport(deck, precision, 0.0)
    assert err is None and (p["E0"] >= 0).all()
    if deck == "tiny_1d":
        np.testing.assert_allclose(p["mu"], np.linspace(0.5, 1.0, 96), rtol=1e-7)
    else:
        np.testing.assert_allclose(p["ux"], np.cos(np.linspace(0.1, 1.2, 96)), rtol=1e-6)
