"""FP64 512-point strided passes in warp-per-pencil form (qx_set_pencil_warp, the
default at 3D 512^3): the same butterflies, phases and Poisson divide as the
plain tiles, so the state agrees to FP64 round-off (a few 1e-16 per pass; the
bound leaves two orders)."""
import numpy as np
import pytest

import qaxions_b200 as qx
from oracle import sp_oracle as O

pytestmark = pytest.mark.gpu


def test_warp_per_pencil_fp64_matches_plain_tiles():
    N = 512
    out = []
    with qx.Field(3, N, pref=50.0, dtype="c128", k0="reference", dt=0.2 / N**2) as f:
        assert f.get_tune()["pencil_warp"] == 1
        f.ic_config(qx.IC_GRF, 5, 2, 0.02, 0.05)
        psi0 = f.psi
        for wp in (1, 0):
            f.set_pencil_warp(wp)
            f.psi = psi0
            f.step(2)
            V, energy = f.V, f.mass_energy()
            f.drift(0.1 / N**2)
            out.append((f.psi, V, energy))
    a, b = out
    assert O.rel_l2(a[0], b[0]) < 1e-13
    assert O.rel_l2(a[1], b[1]) < 1e-12  # low modes dominate V; its round-off is that of the density
    assert np.allclose(a[2], b[2], rtol=1e-12)
