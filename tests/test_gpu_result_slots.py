"""The pinned lines the reductions' results come back through: many fields alive
at once, closed out of order, and fields of several threads each read their own
results; opening a field does not make the driver pin a block of memory anew."""
import ctypes
import threading
import time

import numpy as np
import pytest

import qaxions_b200 as qx

pytestmark = pytest.mark.gpu

N = 8


def _field(c):
    f = qx.Field(2, N, dtype="c128")
    f.psi = np.full((N, N), np.sqrt(c), np.complex128)
    return f


def _check(f, c):
    # L = 1: the mass is the mean of |psi|^2; sqrt(c)^2 and the sum's round-off
    assert f.mass_energy()[0] == pytest.approx(c, rel=1e-14)
    assert f.rho_stats()[0] == pytest.approx(1.0, rel=1e-14)


def test_many_fields_at_once():
    live = {c: _field(c) for c in range(1, 81)}
    for c in list(live)[::3]:
        live.pop(c).close()
    for c in range(200, 230):
        live[c] = _field(c)
    for c, f in live.items():
        _check(f, c)
        f.close()


def test_fields_of_several_threads():
    errors = []

    def work(k):
        try:
            for i in range(20):
                fs = [_field(100 * k + j + 1) for j in range(4)]
                for j, f in enumerate(fs):
                    _check(f, 100 * k + j + 1)
                for f in fs:
                    f.close()
        except Exception as e:  # noqa: BLE001 (reported by the main thread)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


def test_pinning_stays_short_between_fields():
    """Pinning a few bytes takes the driver milliseconds when no block is pinned yet
    and microseconds otherwise; a field that opens and closes leaves one pinned."""
    rt = ctypes.CDLL("libcudart.so.12")
    qx.Field(2, N).close()
    times = []
    for _ in range(15):
        p = ctypes.c_void_p()
        t0 = time.perf_counter()
        assert rt.cudaHostAlloc(ctypes.byref(p), ctypes.c_size_t(64), ctypes.c_uint(2)) == 0
        assert rt.cudaFreeHost(p) == 0
        times.append(time.perf_counter() - t0)
    assert min(times) < 0.5e-3
