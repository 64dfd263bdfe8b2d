"""Field.propagate runs kick, drift, updateTime, updatePotential, kick with the
pointwise work inside the transform passes; it must leave psi, V, the clock and
Vmax as the five calls do, from a V that is not the potential of psi too (the
first kick takes V as it is).  Tolerances: the same operations on the same values,
up to fused multiply-adds: 1e-13 (FP64), 1e-6 (FP32)."""
import numpy as np
import pytest

import qaxions_b200 as qx
from oracle import sp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("cosmo", [0, 1])
@pytest.mark.parametrize("dim,N", [(3, 8), (3, 64), (3, 128), (3, 256), (2, 16), (2, 256)])
def test_propagate_is_its_five_operations(dim, N, cosmo, dtype):
    tol = 1e-13 if dtype == "c128" else 1e-6
    rng = np.random.default_rng(N)
    psi = 1.0 + 0.2 * (rng.normal(size=(N,) * dim) + 1j * rng.normal(size=(N,) * dim))
    V = 50.0 * rng.normal(size=(N,) * dim)
    out = []
    for fused in (True, False):
        with qx.Field(dim, N, pref=20.0, dtype=dtype, k0="zero", dt=0.2 / N**2) as f:
            f.psi, f.V = psi, V
            if cosmo:
                f.set_cosmology(1, 0.01)
            for _ in range(3):
                if fused:
                    f.propagate()
                else:
                    f.kick(0.5 * f.cosmology()[2])
                    f.drift(f.cosmology()[2])
                    f.updateTime()
                    f.updatePotential()
                    f.kick(0.5 * f.cosmology()[2])
            out.append((f.psi, f.V, f.Vmax(), f.time(), f.curr(), f.a()))
    a, b = out
    assert O.rel_l2(a[0], b[0]) < tol
    assert O.rel_l2(a[1], b[1]) < 10 * tol
    assert a[2] == pytest.approx(np.abs(a[1]).max(), rel=1e-15 if dtype == "c128" else 1e-7)
    assert a[3:] == b[3:]
