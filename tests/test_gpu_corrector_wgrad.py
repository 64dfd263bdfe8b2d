"""Weight and bias gradients of the tensor-core path (MN-major operands read in
place, GELU derivative in the convolution epilogue) against the CUDA-core sums,
per layer, at the edges: two bricks only (N = 8, where the convolutions run on
mma.sync and the weight gradients on tcgen05), fewer bricks than SMs, an odd
number of bricks per block.  The paths differ by the BF16 rounding of dZ in the
weight gradients (2^-9 per term, random in sign) and by FP32 summation order
elsewhere: 4e-3 for the weights as for the whole gradient, 1e-3 for the biases
(BF16 activations that flip between convolutions summed in another order)."""
import numpy as np
import pytest

import qaxions_b200 as qx
from qaxions_b200 import corrector as cr
from oracle import corrector_oracle as CO
from oracle import sp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 16, 32, 64, 96])
def test_layer_gradients(N):
    rng = np.random.default_rng(N)
    k = np.fft.fftfreq(N) * N
    kk = k[:, None, None] ** 2 + k[None, :, None] ** 2 + k[None, None, :] ** 2

    def smooth(a):
        f = np.fft.ifftn(np.fft.fftn(rng.normal(size=(N,) * 3)) * np.exp(-kk / 8.0)).real
        return a * f / f.std()

    with qx.Field(3, N, dtype="c64") as c, qx.Field(3, N, dtype="c64") as f:
        psi = 1.0 + smooth(0.3) + 1j * smooth(0.2)
        c.psi, c.V, f.psi = psi, smooth(1.0), psi + 1e-3 * (smooth(1.0) + 1j * smooth(1.0))
        g = {}
        for tensor in (True, False):
            corr = cr.Corrector(N, seed=2)
            corr.set_tensor_path(tensor)
            corr.set_scales(1.0, 1e-3)
            corr.gradients(c, f)
            g[tensor] = corr.gradients(c, f)[1].astype(np.float64)
            corr.close()
    at = 0
    for ci, co in CO.DIMS:
        for n, tol in ((27 * ci * co, 4e-3), (co, 1e-3)):
            assert np.linalg.norm(g[False][at:at + n]) > 0
            assert O.rel_l2(g[True][at:at + n], g[False][at:at + n]) <= tol, (ci, co, n)
            at += n
