"""The measured time loop with more measurements than steps: meas_list then
repeats entries, and the loop of main() (src/main.cxx:71-81) measures where its
step index equals the next entry, so a repeated entry ends the measurements.
Whatever the list, run(n, m) takes n steps: the state and clock of step(n) and
one record per scheduled measurement beside the first.

Tolerances as for every other comparison of two forms of the loop: FP64 1e-12,
FP32 1e-5."""
import numpy as np
import pytest

import qaxions_b200 as qx
from oracle import sp_oracle as O

pytestmark = pytest.mark.gpu


def _records(nsteps, nmeas):
    """Steps after which the loop measures: idx == list[next]."""
    ml, out = qx.meas_list(nsteps, nmeas), [0]
    for idx in range(nsteps):
        if len(out) - 1 < len(ml) and ml[len(out) - 1] == idx:
            out.append(idx + 1)
    return out


# (40, 60): one entry repeats behind a measured one, then graph replays to the end
RUNS = [(1, 3), (2, 5), (3, 4), (5, 8), (5, 9), (10, 20), (40, 60), (7, 3), (4, 0)]


@pytest.mark.parametrize("nsteps,nmeas", RUNS)
@pytest.mark.parametrize("dim,N,dtype", [(3, 32, "c64"), (3, 16, "c128"), (2, 64, "c128")])
def test_run_takes_nsteps(dim, N, dtype, nsteps, nmeas):
    tol = 1e-12 if dtype == "c128" else 1e-5
    psi = O.ic_config("grf+solitons", dim, N, seed=N + nsteps, n_solitons=2, rc_lo=0.05, rc_hi=0.1)
    with qx.Field(dim, N, pref=20.0, dtype=dtype, dt=0.2 / N**2) as f:
        f.psi = psi
        f.step(nsteps)
        want, V, time, curr = f.psi, f.V, f.time(), f.curr()
        f.psi = psi
        recs = f.run(nsteps, nmeas)
        assert f.curr() - curr == nsteps
        assert f.time() == pytest.approx(2 * time, rel=1e-12)
        assert [r["number"] for r in recs] == list(range(len(recs)))
        assert [r["step"] - curr for r in recs] == _records(nsteps, nmeas)
        assert O.rel_l2(f.psi, want) < tol
        assert O.rel_l2(f.V, V) < 10 * tol  # (the low modes dominate V)
