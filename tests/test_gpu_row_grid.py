"""The grid of a row pass depends on the field alone, not on what ran before it in
the process: a 2D grid runs the row kernels in smaller blocks, more of which fit
an SM, than a 3D one of the same N.  The sums of mass_energy are formed block by
block, so another grid shows in their last bits."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import sys
import numpy as np
import qaxions_b200 as qx

N = 128
for dim in map(int, sys.argv[2:]):
    with qx.Field(dim, N, dtype=sys.argv[1], pref=3.0) as f:
        rng = np.random.default_rng(dim)
        f.psi = 1.0 + 0.3 * (rng.normal(size=(N,) * dim) + 1j * rng.normal(size=(N,) * dim))
        print(dim, *[x.hex() for x in f.mass_energy()])
"""


def _lines(dtype, *dims):
    r = subprocess.run([sys.executable, "-c", PROGRAM, dtype, *map(str, dims)], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    return dict(ln.split(" ", 1) for ln in r.stdout.splitlines())


@pytest.mark.parametrize("dtype", ["c64", "c128"])
def test_row_grid_is_the_fields_own(dtype):
    want = {**_lines(dtype, 3), **_lines(dtype, 2)}
    assert _lines(dtype, 2, 3) == want
    assert _lines(dtype, 3, 2) == want
