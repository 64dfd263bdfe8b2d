"""A launch geometry that is asked for runs, also on the grids that have
plane-resident or direct-load passes, and gives the same step: the tile ring in
its forms (pencils per thread, ring depth, tile columns, radix plan, warp per
pencil) against the direct-load kernels of set_tune(tma=0), and settings that a
grid has no form for leave its default alone.

Tolerances: FP64 1e-12, FP32 2e-6 for one operation and 1e-5 for a run, as for
every other pass."""
import numpy as np
import pytest

import qaxions_b200 as qx
from oracle import sp_oracle as O

pytestmark = pytest.mark.gpu


def _names(f):
    return [n for n, _ in f.profile_step(1)]


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("N", [32, 64, 96])
def test_asked_geometry_replaces_the_plane_passes(N, dtype):
    with qx.Field(3, N, dtype=dtype, dt=0.2 / N**2) as f:
        f.psi = O.ic_config("grf", 3, N, seed=N)
        planes = _names(f)
        assert len(planes) == 4
        asked = [dict(pw=1), dict(nbuf=2), dict(y_tx=8), dict(la_tx=16), dict(x_rows=4), dict(tma=0)]
        for t in asked:
            f.set_tune(**{"tma": 1, **t})
            assert len(_names(f)) == 8, t
        f.set_tune(tma=1)
        assert _names(f) == planes
        # a radix plan or warp form that the grid does not have changes nothing
        f.set_pencil_warp(2)
        assert _names(f) == planes
        f.set_plan(1)
        assert len(_names(f)) == (8 if N == 96 else 4)  # (32 = 8 4 is not compiled, 64 = 8 8)


# drift, potential, three steps
TOL = {"c64": (2e-6, 2e-6, 1e-5), "c128": (1e-12, 1e-12, 1e-12)}
RING = [dict(pw=1), dict(nbuf=2), dict(y_tx=16, la_tx=16), dict(pw=1, nbuf=4, la_tx=16)]


def _ops(f, psi, dt):
    f.psi = psi
    f.drift(dt)
    d = f.psi
    f.psi = psi
    f.updatePotential()
    V = f.V
    f.step(3)
    return d, V, f.psi


@pytest.mark.parametrize("dtype", ["c64", "c128"])
@pytest.mark.parametrize("dim,N", [(3, 32), (3, 64), (3, 96), (3, 128), (2, 64), (2, 96), (2, 128), (2, 256),
                                   (2, 512)])
def test_ring_forms_match_direct_loads(dim, N, dtype):
    tol = TOL[dtype]
    dt = 0.37 / N**2
    rng = np.random.default_rng(N + dim)
    psi = 1.0 + 0.3 * (rng.normal(size=(N,) * dim) + 1j * rng.normal(size=(N,) * dim))
    with qx.Field(dim, N, pref=30.0, dtype=dtype, k0="zero", dt=0.2 / N**2) as f:
        f.set_tune(tma=0)
        want = _ops(f, psi, dt)
        for t in RING + [dict()]:
            f.set_tune(**{"tma": 1, **t})
            if N == 512 and t.get("nbuf") == 4 and (dtype == "c128" or t.get("la_tx") == 16):
                # four 64 KB tiles do not fit an SM's shared memory
                with pytest.raises(qx.QxError, match="smem attribute"):
                    f.drift(dt)
                continue
            for a, b, e in zip(_ops(f, psi, dt), want, tol):
                assert O.rel_l2(a, b) < e, t


@pytest.mark.parametrize("wp", [1, 2, 3, 4])
@pytest.mark.parametrize("N,dtype", [(256, "c64"), (512, "c64"), (512, "c128")])
def test_pencil_warp_forms_in_2d(N, dtype, wp):
    """The last-axis passes of a 2D grid in warp-per-pencil form (column 0 pairs
    with its mirror mode within the pencil) against the direct loads."""
    tol = TOL[dtype]
    dt = 0.37 / N**2
    rng = np.random.default_rng(N + wp)
    psi = 1.0 + 0.3 * (rng.normal(size=(N, N)) + 1j * rng.normal(size=(N, N)))
    with qx.Field(2, N, pref=30.0, dtype=dtype, k0="zero", dt=0.2 / N**2) as f:
        f.set_tune(tma=0)
        want = _ops(f, psi, dt)
        Vw, _ = O.update_potential(psi, 30.0, k0="zero")
        assert O.rel_l2(want[1], Vw) < tol[1]
        f.set_tune(tma=1)
        f.set_pencil_warp(wp)
        for a, b, e in zip(_ops(f, psi, dt), want, tol):
            assert O.rel_l2(a, b) < e
