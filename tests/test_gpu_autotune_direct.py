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
