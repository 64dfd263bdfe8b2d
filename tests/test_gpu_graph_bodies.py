"""The loop's bodies run in groups from a captured graph, the rest one by one: the
same state whatever the split -- calls shorter than a group, one group and a rest,
several groups, a field with and without a graph yet, a changed time step, and an
eager drift with another step in between (its factor tables are inputs of the
graph).  Bit for bit: the same kernels on the same operands."""
import numpy as np
import pytest

import qaxions_b200 as qx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["c128", "c64"])
@pytest.mark.parametrize("dim,N", [(2, 64), (2, 256), (3, 32), (3, 16), (3, 256)])
def test_split_of_the_loop_does_not_matter(dim, N, dtype):
    dt = 0.2 / N**2
    out = []
    for graph in (True, False):
        with qx.Field(dim, N, pref=20.0, dtype=dtype, k0="zero", dt=dt) as f:
            f.ic_config(qx.IC_GRF, 3, 1, 0.05, 0.1)
            for n in (3, 18, 9, 1, 26):  # eager; two groups and one; a group; none; three groups and one
                f.time_steps(n, graph)
            f.drift(0.3 * dt)
            f.time_steps(18, graph)
            f.set_dt(0.5 * dt)
            f.time_steps(18, graph)
            f.run(20, 2, qx.MEAS_RHO_MAX)
            out.append((f.psi, f.V))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("n", [2, 10, 17, 18, 19, 27])
def test_ensemble_groups_of_steps(n):
    groups = [(32, 2), (64, 1), (96, 1)]
    dt = 0.2 / 96**2
    a = qx.Ensemble(groups, dtype="c64", dt=dt)
    b = qx.Ensemble(groups, dtype="c64", dt=dt)
    for e in (a, b):
        e.ic_config(qx.IC_GRF, seed_base=3, n_sol=1)
    a.step(n)
    a.step(n)  # replays the captured groups
    for box in range(a.nboxes):
        with qx.Field(3, a.box_n(box), dtype="c64", k0="zero", dt=dt) as f:
            f.psi = b.psi(box)
            f.time_steps(n, False)
            f.time_steps(n, False)
            assert np.array_equal(a.psi(box), f.psi)
    a.close()
    b.close()
