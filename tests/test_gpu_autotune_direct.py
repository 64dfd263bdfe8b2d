"""The autotuner times the plane-resident and direct-load passes, which take no
geometry, among its candidates, and keeps them where they are the fastest: a step
of 32^3 complex64 is four launches that way and nine with the tile ring (measured
15 against 46 us)."""
import pytest

import qaxions_b200 as qx

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _fresh_tune_cache():
    qx.clear_tune_cache()
    yield
    qx.clear_tune_cache()


@pytest.mark.parametrize("nsteps", [1, 12])
def test_autotune_keeps_the_plane_passes(nsteps):
    with qx.Field(3, 32, dtype="c64", dt=0.2 / 32**2) as f:
        f.ic_config(qx.IC_GRF, 3, 2, 0.02, 0.05)
        ms, cached = f.autotune(nsteps)
        assert ms > 0 and not cached
        t = f.get_tune()
        assert t["tma"] == 1
        assert not any(t[k] for k in ("x_rows", "y_tx", "la_tx", "nbuf", "pw", "plan", "chain", "pencil_warp"))
        assert len(f.profile_step(1)) == 4


@pytest.mark.parametrize("cosmo", [0, 1])
def test_autotune_leaves_the_clock(cosmo):
    """The timed steps are not taken: step count, time, and in the MRE cosmology
    the scale factor and the time step that follows it, are those before."""
    with qx.Field(3, 16, dtype="c128", dt=1e-4) as f:
        f.ic_config(qx.IC_GRF, 3, 0)
        if cosmo:
            f.set_cosmology(1, 0.5)
        f.step(3)
        psi, clock, cosmology = f.psi, (f.curr(), f.time(), f.a()), f.cosmology()
        f.autotune(2)
        assert (f.curr(), f.time(), f.a()) == clock
        assert f.cosmology() == cosmology
        assert (f.psi == psi).all()
