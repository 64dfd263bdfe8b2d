"""The FP64 Poisson multiplier of the passes (pois_mult: reciprocal, Newton-Raphson,
residual correction) is the quotient pois_c / |n|^2 bit for bit: every |n|^2 of a
512^3 grid, and a stretch up to the bound it is stated for, for numerators of all
binades that a box gives and random and extreme significands.  The kernel under
test is compiled from the library's header; the quotients are the division of the
device and, for a part, of the host."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "qaxions_b200", "csrc")

SOURCE = r"""
#include "qx_kernels.cuh"

__global__ void k_mult(const double* c, int nc, long m0, long nm, double* out, unsigned long long* differ) {
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= nm * nc) return;
    qx::SArgs<double> s{};
    s.pois_c = c[i / nm];
    const long m = m0 + i % nm;
    const double got = qx::pois_mult<double>(m, s), want = s.pois_c / (double)m;
    if (__double_as_longlong(got) != __double_as_longlong(want)) atomicAdd(differ, 1ull);
    if (out) out[i] = got;
}

extern "C" int run(const double* c, int nc, long m0, long nm, double* out, unsigned long long* differ) {
    const long n = nm * nc;
    k_mult<<<(unsigned)((n + 255) / 256), 256>>>(c, nc, m0, nm, out, differ);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def mult(tmp_path_factory):
    import torch

    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    d = tmp_path_factory.mktemp("mult")
    (d / "mult.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    "-Xcompiler", "-fPIC", "-shared", "-I", CSRC, str(d / "mult.cu"), "-o", str(d / "mult.so")], check=True)
    lib = C.CDLL(str(d / "mult.so"))
    lib.run.argtypes = [C.c_void_p, C.c_int, C.c_long, C.c_long, C.c_void_p, C.c_void_p]

    def call(c, m0, nm, values=False):
        cd = torch.tensor(c, dtype=torch.float64, device="cuda")
        out = torch.empty(len(c) * nm, dtype=torch.float64, device="cuda") if values else None
        differ = torch.zeros(1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        assert lib.run(cd.data_ptr(), len(c), m0, nm, out.data_ptr() if values else None, differ.data_ptr()) == 0
        return int(differ.item()), out.cpu().numpy().reshape(len(c), nm) if values else None

    return call


def _numerators():
    """-1 / (dk^2 S) of boxes L = 1e-3 ... 1e3, N = 4 ... 512, and significands at
    random, all ones and next to a power of two in the binades around them."""
    box = [-1.0 / ((2.0 * np.pi / L) * (2.0 * np.pi / L) * float(N) ** dim)
           for L in (1e-3, 0.37, 1.0, 20.0, 1e3) for N in (4, 32, 96, 128, 256, 512) for dim in (2, 3)]
    rng = np.random.default_rng(5)
    rand = [-np.ldexp(1.0 + rng.random(), int(e)) for e in rng.integers(-60, 20, 60)]
    edge = [-np.ldexp(s, e) for s in (1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), 1.5) for e in (-60, -31, 0, 9)]
    return box + rand + edge


def test_every_m_of_a_512_box(mult):
    c = _numerators()
    for part in range(0, len(c), 20):
        differ, _ = mult(c[part:part + 20], 1, 3 * 256**2)
        assert differ == 0
    differ, _ = mult(c[::10], 2**24 - 200000, 200000)
    assert differ == 0


def test_against_the_hosts_division(mult):
    c = _numerators()[::7]
    differ, got = mult(c, 1, 3 * 256**2, values=True)
    m = np.arange(1, 3 * 256**2 + 1, dtype=np.float64)
    assert differ == 0
    for k, ck in enumerate(c):
        assert np.array_equal(got[k], ck / m)
