"""Mass and energy of 3D 256^3 and 512^3 against the sums of their definition with
torch's FP64 transforms, for every form of the strided passes that the grid has
(the kinetic sum's own passes run whatever set_tune(tma) says).

Tolerances: the sums are FP64 over the field's own values, so the mass and the
potential energy (relative to the sum of |V| |psi|^2, as V changes sign) agree to
round-off, 1e-12, and so does the kinetic energy of an FP64 field.  An FP32 field's
kinetic energy takes one FP32 transform per axis: at most 9 radix-2 levels of one
rounding, 2 * 9 * 6e-8 in |psi^|^2 = 1.1e-6; the bound is 3e-6."""
import numpy as np
import pytest

import qaxions_b200 as qx

pytestmark = pytest.mark.gpu

FORMS = {
    (256, "c64"): [dict(), dict(tune=dict(pw=1)), dict(wp=1), dict(wp=2), dict(tune=dict(tma=0))],
    (256, "c128"): [dict(), dict(tune=dict(nbuf=2)), dict(tune=dict(tma=0))],
    (512, "c64"): [dict(), dict(wp=0), dict(wp=2), dict(wp=4)],
    (512, "c128"): [dict(), dict(wp=0)],
}


def _energies(psi, V, L=1.0):
    """(M, K, W, sum |V| rho) of the definition (mass_energy's normalisation)."""
    import torch

    N = psi.shape[0]
    dV = (L / N) ** 3
    k2 = (2.0 * np.pi / L * torch.fft.fftfreq(N, 1.0 / N, dtype=torch.float64, device="cuda")) ** 2
    p = torch.as_tensor(psi, device="cuda")
    rho = p.real.square() + p.imag.square()
    v = torch.as_tensor(V, device="cuda")
    M, W, scale = rho.sum() * dV, 0.5 * dV * (v * rho).sum(), 0.5 * dV * (v.abs() * rho).sum()
    del v, rho
    p = torch.fft.fftn(p)
    h = p.real.square() + p.imag.square()
    del p
    K = sum((h.sum(dim=[b for b in range(3) if b != a]) * k2).sum() for a in range(3)) * 0.5 * dV / N**3
    return tuple(float(x) for x in (M, K, W, scale))


@pytest.mark.parametrize("N,dtype", list(FORMS))
def test_mass_energy_of_large_grids(N, dtype):
    rng = np.random.default_rng(N)
    psi = np.empty((N,) * 3, np.complex128)
    psi.real = 1.0 + 0.2 * rng.standard_normal((N,) * 3, dtype=np.float32)
    psi.imag = 0.2 * rng.standard_normal((N,) * 3, dtype=np.float32)
    with qx.Field(3, N, pref=20.0, dtype=dtype, k0="zero") as f:
        f.psi = psi
        f.updatePotential()
        want = _energies(f.psi, f.V)
        default_wp = f.get_tune()["pencil_warp"]
        for form in FORMS[N, dtype]:
            f.set_tune(**{"tma": 1, **form.get("tune", {})})
            f.set_pencil_warp(form.get("wp", default_wp))
            M, E, K, W = f.mass_energy()
            assert M == pytest.approx(want[0], rel=1e-12), form
            assert K == pytest.approx(want[1], rel=1e-12 if dtype == "c128" else 3e-6), form
            assert abs(W - want[2]) < 1e-12 * want[3], form
            assert E == K + W
