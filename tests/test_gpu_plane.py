"""Plane-resident passes (3D N = 32, 64, 96 and, complex64, 128: the x and y
transforms of a z plane in one launch) and the direct-load last-axis passes
(3D N <= 128, 2D N = 64..512), against the NumPy oracle and against the
general row and strided passes (set_tune(tma=0)) on the same state: the drift,
the potential (column 0 with both k = 0 conventions), the merged loop, the
measured loop's kick + forward transform, and stacked boxes.

Tolerances: FP64 1e-12 (round-off of two orders of summation), FP32 2e-6 for
one operation and 1e-5 for a run, as for every other pass."""
import numpy as np
import pytest

import qaxions_b200 as qx
from oracle import sp_oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(3, 32), (3, 64), (3, 96), (3, 128), (2, 64), (2, 96), (2, 128), (2, 256), (2, 512)]


def _field(dim, N, dtype, general, k0="zero", dt=None):
    f = qx.Field(dim, N, pref=30.0, dtype=dtype, k0=k0, dt=dt or 0.2 / N**2)
    if general:
        f.set_tune(tma=0)
    return f


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("dim,N", GRIDS)
def test_operators_match_oracle_and_general_passes(dim, N, dtype):
    one = 1e-12 if dtype == "c128" else 2e-6
    rng = np.random.default_rng(N + dim)
    psi = 1.0 + 0.3 * (rng.normal(size=(N,) * dim) + 1j * rng.normal(size=(N,) * dim))
    dt = 0.37 / N**2  # not representable
    want = O.drift(psi, dt)
    Vw, _ = O.update_potential(psi, 30.0, k0="zero")
    got = []
    for general in (False, True):
        with _field(dim, N, dtype, general) as f:
            f.psi = psi
            f.drift(dt)
            d = f.psi
            f.psi = psi
            f.updatePotential()
            got.append((d, f.V, f.Vhat))
            assert O.rel_l2(d, want) < one
            assert O.rel_l2(f.V, Vw) < one
    for a, b in zip(*got):
        assert O.rel_l2(a, b) < one


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("dim,N", [g for g in GRIDS if g[1] <= 128])
def test_loops_match_general_passes(dim, N, dtype):
    """step() with graph replays, the measured loop (kick, x and y forward from
    real space; the last step measured too) and a call of another length."""
    tol = 1e-12 if dtype == "c128" else 1e-5
    psi = O.ic_config("grf+solitons", dim, N, seed=N, n_solitons=2, rc_lo=0.05, rc_hi=0.1)
    got = []
    for general in (False, True):
        with _field(dim, N, dtype, general, k0="reference") as f:
            f.psi = psi
            f.step(7)
            a = f.psi
            recs = f.run(5, 3, qx.MEAS_RHO_MAX | qx.MEAS_ENERGY)
            b = f.psi
            f.step(1)
            got.append((a, b, f.psi, np.array([[r["rhomax"], r["energy"]] for r in recs])))
    for x, y in zip(*got):
        assert O.rel_l2(x, y) < tol
    if N <= 64:
        ref, _ = O.run(psi, 0.2 / N**2, 7, 30.0)
        assert O.rel_l2(got[0][0], ref) < tol


@pytest.mark.parametrize("dtype", ["c128", "c64"])
def test_stacked_boxes(dtype):
    """Planes and columns of several boxes in one launch, the mirror rows of
    column 0 within their own box."""
    tol = 1e-13 if dtype == "c128" else 1e-6
    groups = [(32, 3), (64, 2), (128, 2)]
    dt = 0.2 / 128**2
    psi = [O.ic_config("grf", 3, n, seed=10 * n + i) for n, c in groups for i in range(c)]
    ens = qx.Ensemble(groups, dtype=dtype, dt=dt, pref=30.0)
    for b, p in enumerate(psi):
        ens.set_psi(b, p)
    ens.step(5)
    for b, p in enumerate(psi):
        with _field(3, p.shape[0], dtype, True, dt=dt) as f:
            f.psi = p
            f.step(5)
            assert O.rel_l2(ens.psi(b), f.psi) < tol, b
    ens.close()
