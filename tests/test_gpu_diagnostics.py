"""Mass and energy from one transform per axis, and the shell binning by sorted
runs, against the NumPy oracle at the edges of their ranges: rows shorter than a
warp (N = 4 .. 32), a row length that is no multiple of a warp (N = 96), 2D and
3D, one bin to many, few states that fill no block.

Tolerances: FP64 sums 1e-12 relative; FP32 1e-5 (FP32 transforms of an FP32
state, white round-off of 1e-7 per mode).  Mode counts are exact."""
import numpy as np
import pytest

import qaxions_b200 as qx
from oracle import sp_oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(2, 4), (2, 8), (2, 16), (2, 64), (2, 96), (2, 512), (3, 4), (3, 8), (3, 16), (3, 32), (3, 64), (3, 96),
         (3, 128)]


def _psi(dim, N):
    rng = np.random.default_rng(7 * N + dim)
    x = np.arange(N) / N
    p = 1.0 + 0.2 * rng.normal(size=(N,) * dim) + 0.3j * rng.normal(size=(N,) * dim)
    return p * np.exp(2j * np.pi * x)  # a carrier along x: the axes' shares differ


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("dim,N", GRIDS)
def test_mass_and_energy(dim, N, dtype):
    tol = 1e-12 if dtype == "c128" else 1e-5
    psi = _psi(dim, N)
    V = np.random.default_rng(N).normal(size=(N,) * dim)
    with qx.Field(dim, N, dtype=dtype, k0="zero") as f:
        f.psi = psi
        f.updatePotential()
        f.V = V
        M, E, K, W = f.mass_energy()
        Eo, Ko, Wo = O.energy(psi, V)
        scale = 0.5 * np.mean(np.abs(V) * np.abs(psi) ** 2)
        assert M == pytest.approx(O.mass(psi), rel=tol)
        assert K == pytest.approx(Ko, rel=tol)
        assert abs(W - Wo) < tol * scale
        assert abs(E - Eo) < tol * (Ko + scale)
        r = f.measure(qx.MEAS_RHO_MAX | qx.MEAS_ENERGY)
        rho = np.abs(psi) ** 2
        assert r["rhomax"] == pytest.approx(rho.max() / rho.mean(), rel=tol)
        assert r["vmax"] == pytest.approx(np.abs(V).max(), rel=tol)
        assert (r["mass"], r["kinetic"]) == (M, K)


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("dim,N", GRIDS)
def test_spectrum_bins(dim, N, dtype):
    psi = _psi(dim, N)
    with qx.Field(dim, N, dtype=dtype) as f:
        f.psi = psi
        for mode, nb in ((0, N // 2 + 1), (1, 1), (1, 5), (1, 300), (2, 1), (2, 7), (2, 257)):
            k, P, c = f.spectrum(0, mode, nb)
            ko, Po, co = O.density_spectrum(psi, mode, nb)
            np.testing.assert_array_equal(c, co)
            sel = c > 0
            rtol, atol = (1e-11, 1e-13) if dtype == "c128" else (1e-4, 1e-6)
            np.testing.assert_allclose(P[sel], Po[sel], rtol=rtol, atol=atol * max(Po.max(), 1e-300))


def test_nan_reaches_the_diagnostics():
    psi = _psi(3, 16)
    psi[3, 2, 1] = np.nan
    with qx.Field(3, 16, dtype="c128") as f:
        f.psi = psi
        f.V = np.ones((16,) * 3)
        assert all(np.isnan(v) for v in f.mass_energy())
