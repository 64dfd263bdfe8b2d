"""A launch that the runtime refuses (an x_rows whose blocks are larger than the
row kernels are built for, a histogram larger than an SM's shared memory) is
reported once, by the call that made it: the next call on valid settings is not
told of it again."""
import numpy as np
import pytest

import qaxions_b200 as qx
from oracle import sp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("after", ["kick", "computeEnergy", "step"])
def test_refused_launch_is_reported_once(after):
    N = 512  # 32 threads per row: 16 rows are 512 threads of a 256-thread kernel
    psi = O.ic_config("grf", 2, N, seed=3)
    with qx.Field(2, N, dtype="c64", dt=0.2 / N**2) as f:
        f.psi = psi
        f.set_tune(x_rows=16)
        with pytest.raises(qx.QxError, match="kernel launch"):
            f.drift(1e-6)
        f.set_tune()
        f.psi = psi
        getattr(f, after)(*{"kick": (1e-6,), "step": (2,)}.get(after, ()))
        assert np.isfinite(f.psi).all()


def test_refused_histogram_is_reported_once():
    N = 64
    psi = O.ic_config("grf", 2, N, seed=4)
    with qx.Field(2, N, dtype="c128", dt=0.2 / N**2) as f:
        f.psi = psi
        with pytest.raises(qx.QxError, match="smem attribute"):
            f.spectrum(0, qx.SPEC_LOG, 4000)  # 8 warps x 4000 bins x 16 bytes
        f.kick(1e-6)
        assert np.isfinite(f.psi).all()
