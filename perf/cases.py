"""The calls whose time counts, with their inputs, outputs and 64-bit values.

A case is one call sequence of a user's program on one GPU: time steps of one
box, the measured time loop, the reference's unfused operators, the
diagnostics of a snapshot, an ensemble of small boxes, and the learned
corrector's training gradient and corrected coarse step.  The boxes hold a
Gaussian random field (P(k) ~ k^-2 exp(-(k/kc)^2), kc = N/8 modes, sigma 0.3,
clipped at -0.9) plus Schive-profile solitons, mean |psi|^2 = 1, made with
torch on the GPU from the seed and written into the field's own device
memory, as a program does that makes its states on the device.

exact() restates each call in complex128 with torch.fft.
"""
import math

import numpy as np
import torch

import qaxions_b200 as qx
from qaxions_b200 import corrector as cr

GRIDS_2D = (64, 96, 128, 256, 512)
GRIDS_3D = (32, 64, 96, 128, 256, 512)
ENSEMBLE_GRIDS = (32, 64, 96, 128)
TRAIN_GRIDS = (32, 64, 96, 128)
CHANNELS = ((4, 32), (32, 32), (32, 2))  # the corrector's layers


def _box(name, call, dim, N, dtype, steps=1, **more):
    return dict({"name": name, "call": call, "dim": dim, "N": N, "dtype": dtype, "steps": steps, "dt_dx2": 0.2,
                 "pref": 1.0, "solitons": 8}, **more)


def listed():
    return [
        # the smallest run: the smoke test's 32^3 box and step count; launches and latency
        _box("step-3d-32-c64", "step", 3, 32, "c64", 8, solitons=2),
        # 2D 256^2 plain FP64 run of 8 solitons: 50 steps between two 64-bin P(k)
        _box("step-spectrum-2d-256-c128", "step+spectrum", 2, 256, "c128", 50, mode=1, nbins=64),
        # the reference's own operator surface (kick, drift, updatePotential, kick), as its tests drive it
        _box("propagate-3d-64-c64", "propagate", 3, 64, "c64", 10),
        # a radix-3 grid in the plain FP64 form
        _box("step-3d-96-c128", "step", 3, 96, "c128", 10),
        # the 128^3 accuracy runs, both forms
        _box("step-3d-128-c64", "step", 3, 128, "c64", 20),
        _box("step-3d-128-c128", "step", 3, 128, "c128", 10),
        # the measured time loop of main(): 20 steps, 3 measurements of rhomax, Vmax, mass and energy
        _box("run-3d-256-c64", "run", 3, 256, "c64", 20, nmeas=3, solitons=16),
        # the headline box: 512^3, complex64 form and complex128 form
        _box("step-3d-512-c64", "step", 3, 512, "c64", 10, solitons=32),
        _box("step-3d-512-c128", "step", 3, 512, "c128", 5, solitons=32),
        # diagnostics of a 512^3 snapshot: mass and energy, 256-bin log P(k)
        _box("diagnose-3d-512-c64", "diagnose", 3, 512, "c64", mode=2, nbins=256, solitons=32),
        # boxes of three sizes advanced together, then fetched
        {"name": "ensemble-64-96-128-c64", "call": "ensemble", "groups": "64x4,96x2,128x2", "dtype": "c64",
         "mixed": "", "steps": 200, "solitons": 0},
        # one training gradient of the corrector at its training size
        {"name": "gradient-128", "call": "gradient", "N": 128, "dtype": "c64", "dt_dx2": 0.2, "pref": 1.0,
         "solitons": 16},
    ]


def draw(rng):
    call = rng.choice(["step", "step", "step", "step", "step+spectrum", "propagate", "run", "diagnose", "ensemble",
                       "gradient", "corrected"])
    dtype = rng.choice(["c64", "c64", "c128"])
    common = {"dt_dx2": round(math.exp(rng.uniform(math.log(0.02), math.log(0.37))), 4),
              "solitons": rng.randrange(0, 33)}
    if call == "ensemble":
        sizes = sorted(rng.sample(ENSEMBLE_GRIDS, rng.randrange(1, 4)))
        groups = ",".join("%dx%d" % (n, rng.randrange(1, 5)) for n in sizes)
        # dt follows the finest grid of the ensemble
        return {"call": call, "groups": groups, "dtype": dtype, "mixed": rng.choice(["", "", "step", "passes"]),
                "steps": rng.randrange(3, 120), "solitons": rng.randrange(0, 5)}
    if call in ("gradient", "corrected"):
        N = rng.choice(TRAIN_GRIDS if call == "gradient" else (32, 64, 128, 256))
        return dict(common, call=call, N=N, dtype="c64", pref=1.0)
    dim = rng.choice([2, 3, 3, 3])
    N = rng.choice(GRIDS_2D if dim == 2 else GRIDS_3D)
    # at most the work of the listed 512^3 runs, spread over its logarithm
    most = {512: 4, 256: 30}.get(N, 100) if dim == 3 else 200
    steps = max(1, int(round(math.exp(rng.uniform(0.0, math.log(most))))))
    c = dict(common, call=call, dim=dim, N=N, dtype=dtype, steps=steps,
             pref=round(math.exp(rng.uniform(math.log(0.3), math.log(300.0))), 4))
    if call in ("diagnose", "step+spectrum"):
        c["mode"] = rng.choice([0, 1, 2])
        c["nbins"] = N // 2 + 1 if c["mode"] == 0 else rng.choice([24, 64, 100, 256])
    if call == "run":
        c["nmeas"] = rng.randrange(1, 4)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _rng(seed, stream=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + stream)
    return g


def _modes(N, half=False):
    n = torch.fft.rfftfreq(N, 1.0 / N) if half else torch.fft.fftfreq(N, 1.0 / N)
    return n.to("cuda", torch.float64)


def _n2(dim, N, half=False):
    """Integer |n|^2 over the (half) spectrum, reference site order (x fastest)."""
    m = [_modes(N, half and a == dim - 1) ** 2 for a in range(dim)]
    out = m[0].reshape([-1] + [1] * (dim - 1))
    for a in range(1, dim):
        out = out + m[a].reshape([-1] + [1] * (dim - 1 - a))
    return out


def _initial(dim, N, n_sol, seed, stream=0):
    """psi of one box in complex128: sqrt(1 + GRF) plus solitons, mean |psi|^2 = 1."""
    g = _rng(seed, stream)
    axes = tuple(range(dim))
    h = torch.fft.rfftn(torch.randn((N,) * dim, generator=g, device="cuda", dtype=torch.float64), dim=axes)
    k2 = _n2(dim, N, half=True)
    P = torch.exp(-k2 / (N / 8.0) ** 2) / k2.clamp(min=1.0)
    P[(0,) * dim] = 0.0
    h *= P.sqrt_()
    del P, k2
    d = torch.fft.irfftn(h, s=(N,) * dim, dim=axes)
    del h
    d *= 0.3 / d.square().mean().sqrt()
    psi = torch.complex((1.0 + d.clamp_(min=-0.9)).sqrt_(), torch.zeros((), device="cuda", dtype=torch.float64))
    del d
    u = torch.rand((n_sol, 5), generator=g, device="cuda", dtype=torch.float64).tolist()
    x = torch.arange(N, device="cuda", dtype=torch.float64) / N
    lo, hi = (0.02, 0.05) if dim == 2 else (0.01, 0.03)
    for c in u:
        rc = lo + (hi - lo) * c[0]
        amp = math.sqrt(1e-6) / rc ** 2
        r2 = 0.0
        for a in range(dim):
            t = x - c[2 + a]
            t = (t - t.round()) ** 2
            r2 = r2 + t.reshape([-1] + [1] * (dim - 1 - a))
        f = amp / (1.0 + (0.091 / rc ** 2) * r2) ** 4
        psi += f * complex(math.cos(2 * math.pi * c[1]), math.sin(2 * math.pi * c[1]))
        del f, r2
    v = torch.view_as_real(psi)
    v *= 1.0 / math.sqrt(float(v.square().sum()) / N ** dim)
    return psi


class _DeviceArray:
    """A field's own device memory (Field.device_pointers) for torch; a tensor
    made of it keeps this object, and with it the field, alive."""

    def __init__(self, field, ptr, shape, typestr):
        self.field = field
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (int(ptr), False),
                                         "version": 2}


def _views(f, c128):
    p, v = f.device_pointers()
    return (torch.as_tensor(_DeviceArray(f, p, f.shape, "<c16" if c128 else "<c8"), device="cuda"),
            torch.as_tensor(_DeviceArray(f, v, f.shape, "<f8" if c128 else "<f4"), device="cuda"))


def _groups(case):
    return [tuple(int(x) for x in g.split("x")) for g in case["groups"].split(",")]


def _boxes(case):
    return [n for n, count in _groups(case) for _ in range(count)]


def _dt(case):
    return case["dt_dx2"] / case["N"] ** 2


def _cplx(case):
    return torch.complex128 if case["dtype"] == "c128" else torch.complex64


def _params(seed):
    """Network parameters: uniform in the fan-in range, the last layer small."""
    r = np.random.default_rng(int(seed))
    out = []
    for l, (ci, co) in enumerate(CHANNELS):
        a = math.sqrt(3.0 / (27 * ci)) * (0.1 if l == 2 else 1.0)
        out += [r.uniform(-a, a, 27 * ci * co), r.uniform(-0.05, 0.05, co)]
    return np.concatenate(out).astype(np.float32)


TAU = 1e-6       # scale of the corrector's output: the size of a coarse step's error
V_SCALE = 1e-3   # scale of its potential feature


def _pair(case, seed):
    """Coarse state, its potential and the fine state, as complex64 / float32."""
    N = case["N"]
    psi = _initial(3, N, case["solitons"], seed).to(torch.complex64)
    V = _potential(psi.to(torch.complex128), 1.0, "zero").to(torch.float32)
    e = _initial(3, N, 0, seed, 1)
    fine = (psi.to(torch.complex128) + TAU * (e.real - e.real.mean()) * complex(1.5, 2.5)).to(torch.complex64)
    return psi, V, fine


def _field(case, dt=None):
    c128 = case["dtype"] == "c128"
    # FP32 boxes set the k = 0 mode of V to zero, FP64 boxes keep the reference's convention
    return qx.Field(case.get("dim", 3), case["N"], pref=case["pref"], dtype=case["dtype"],
                    k0="reference" if c128 else "zero", dt=_dt(case) if dt is None else dt)


def _written(f, psi):
    """Put a device state into the field and say so."""
    p, v = _views(f, psi.dtype == torch.complex128)
    p.copy_(psi)
    torch.cuda.synchronize()
    cr.psi_changed(f)
    return p, v


def prepare(case, seed):
    call = case["call"]
    if call == "ensemble":
        e = qx.Ensemble(_groups(case), dtype=case["dtype"], mixed={"": False, "step": True}.get(case["mixed"], "passes"))
        for b, n in enumerate(_boxes(case)):
            e.set_psi(b, _initial(3, n, case["solitons"], seed, b).to(_cplx(case)).cpu().numpy())
        return {"case": case, "ens": e}
    if call == "gradient":
        psi, V, fine = _pair(case, seed)
        fc, ff = _field(case), _field(case)
        _, v = _written(fc, psi)
        v.copy_(V)
        _written(ff, fine)
        corr = cr.Corrector(case["N"])
        corr.params = _params(seed)
        corr.set_scales(V_SCALE, TAU)
        return {"case": case, "coarse": fc, "fine": ff, "corr": corr}
    f = _field(case)
    psi, V = _written(f, _initial(f.dim(), case["N"], case["solitons"], seed).to(_cplx(case)))
    st = {"case": case, "f": f, "psi": psi, "V": V}
    if call == "corrected":
        st["backup"] = _field(case)
        st["corr"] = cr.Corrector(case["N"])
        st["corr"].params = _params(seed)
        st["corr"].set_scales(V_SCALE, TAU)
    if call in ("diagnose", "corrected"):
        f.updatePotential()  # a snapshot within a run: its potential is there
    return st


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------


def _spectrum_out(case, k, P, count):
    # the powers of a complex64 box carry its precision
    return {"k": k, "P": P if case["dtype"] == "c128" else P.astype(np.float32), "count": count}


def run(st):
    case = st["case"]
    call = case["call"]
    if call == "ensemble":
        e = st["ens"]
        e.step(case["steps"])
        kind = np.complex128 if case["dtype"] == "c128" else np.complex64
        return [e.psi(b).astype(kind, copy=False) for b in range(e.nboxes)]
    if call == "gradient":
        loss, grad = st["corr"].gradients(st["coarse"], st["fine"])
        return {"loss": loss, "grad": grad}
    f = st["f"]
    if call == "corrected":
        n = cr.corrected_steps(f, st["corr"], 1, _dt(case), backup=st["backup"])
        return {"psi": st["psi"], "fallbacks": n}
    if call == "diagnose":
        M, E, K, W = f.mass_energy()
        return dict(_spectrum_out(case, *f.spectrum(0, case["mode"], case["nbins"])), M=M, E=E, K=K, W=W)
    if call == "propagate":
        for _ in range(case["steps"]):
            f.propagate()
        return {"psi": st["psi"], "V": st["V"]}
    if call == "run":
        recs = f.run(case["steps"], case["nmeas"], qx.MEAS_RHO_MAX | qx.MEAS_ENERGY)
        keep = ("number", "rhomax", "vmax", "mass", "energy", "kinetic", "potential")
        return {"psi": st["psi"], "V": st["V"], "records": [{k: r[k] for k in keep} for r in recs]}
    f.step(case["steps"])
    out = {"psi": st["psi"], "V": st["V"]}
    if call == "step+spectrum":
        out.update(_spectrum_out(case, *f.spectrum(0, case["mode"], case["nbins"])))
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------


def _fft_flops(S):
    return 5.0 * S * math.log2(S)


def _step_flops(S):
    # drift: two complex transforms; potential: one real pair; phases, density, Poisson
    return 3.0 * _fft_flops(S) + 40.0 * S


def _net_flops(S):
    return 2.0 * 27 * S * sum(ci * co for ci, co in CHANNELS)


def work(case):
    call = case["call"]
    w = 8 if case["dtype"] == "c128" else 4
    if call == "ensemble":
        S = [n ** 3 for n in _boxes(case)]
        return {"bytes": sum(4 * w * s for s in S), "flops": case["steps"] * sum(_step_flops(s) for s in S)}
    S = case["N"] ** case.get("dim", 3)
    if call == "gradient":
        # forward, weight gradients, data gradients of the last two layers
        back = 2.0 * 27 * S * (32 * 32 + 32 * 2)
        return {"bytes": 20 * S, "flops": 2 * _net_flops(S) + back}
    if call == "corrected":
        return {"bytes": 16 * S, "flops": _step_flops(S) + _net_flops(S) + 2 * _fft_flops(S)}
    if call == "diagnose":
        return {"bytes": 3 * w * S, "flops": 1.5 * _fft_flops(S) + 20.0 * S}
    flops = case["steps"] * _step_flops(S)
    if call == "run":
        flops += (case["nmeas"] + 1) * _fft_flops(S)
    if call == "step+spectrum":
        flops += 0.5 * _fft_flops(S)
    return {"bytes": 5 * w * S, "flops": flops}


# ---------------------------------------------------------------------------
# the same values in 64 bits
# ---------------------------------------------------------------------------


def _potential(psi, pref, k0):
    """pref (|psi|^2 - 1) through -1/k^2; the k = 0 mode divided by 1 (reference) or zero."""
    dim, N = psi.dim(), psi.shape[0]
    axes = tuple(range(dim))
    h = torch.fft.rfftn(pref * (torch.view_as_real(psi).square().sum(-1) - 1.0), dim=axes)
    k2 = _n2(dim, N, half=True) * (2 * math.pi) ** 2
    k2[(0,) * dim] = 1.0
    h /= -k2
    if k0 == "zero":
        h[(0,) * dim] = 0.0
    return torch.fft.irfftn(h, s=(N,) * dim, dim=axes)


def _kick(psi, V, dt):
    return psi.mul_(torch.polar(torch.ones_like(V), -dt * V))


def _drift(psi, dt):
    axes = tuple(range(psi.dim()))
    phase = _n2(psi.dim(), psi.shape[0]) * (-0.5 * dt * (2 * math.pi) ** 2)
    h = torch.fft.fftn(psi, dim=axes)
    h *= torch.polar(torch.ones_like(phase), phase)
    del phase
    return torch.fft.ifftn(h, dim=axes)


def _steps(psi, n, dt, pref, k0):
    """n merged kick-drift-kick steps: (psi, V)."""
    V = _potential(psi, pref, k0)
    psi = _kick(psi, V, 0.5 * dt)
    for i in range(n):
        psi = _drift(psi, dt)
        V = _potential(psi, pref, k0)
        psi = _kick(psi, V, dt if i < n - 1 else 0.5 * dt)
    return psi, V


def _mass_energy(psi, V):
    dim, N = psi.dim(), psi.shape[0]
    dV = 1.0 / N ** dim
    rho = torch.view_as_real(psi).square().sum(-1)
    h = torch.view_as_real(torch.fft.fftn(psi, dim=tuple(range(dim)))).square().sum(-1)
    K = 0.5 * dV * dV * (2 * math.pi) ** 2 * float((_n2(dim, N) * h).sum())
    W = 0.5 * dV * float((V * rho).sum())
    return {"mass": dV * float(rho.sum()), "energy": K + W, "kinetic": K, "potential": W}


def _spectrum(psi, mode, nbins):
    """Shell-binned power of |psi|^2 over the full spectrum (k, P, count)."""
    dim, N = psi.dim(), psi.shape[0]
    half = N // 2
    h = torch.fft.fftn(torch.view_as_real(psi).square().sum(-1), dim=tuple(range(dim)))
    p = torch.view_as_real(h).square().sum(-1).reshape(-1) / float(N ** dim) ** 2
    del h
    r = np.sqrt(np.arange(dim * half * half + 1, dtype=np.float64))
    if mode == 0:
        nbins = half + 1
        b = np.rint(r)
        k = np.arange(nbins) * 2 * math.pi
    else:
        with np.errstate(divide="ignore"):
            b = np.floor(nbins * r / half) if mode == 1 else np.floor(nbins * np.log(r) / math.log(half) + 1e-9)
        b[0] = nbins
        b[r >= half] = nbins
        e = (np.arange(nbins) + 0.5) / nbins
        k = 2 * math.pi * (half * e if mode == 1 else half ** e)
    b = torch.from_numpy(np.clip(b, 0, nbins).astype(np.int64)).cuda()
    bins = b[_n2(dim, N).reshape(-1).long()]
    count = torch.bincount(bins, minlength=nbins + 1)[:nbins]
    P = torch.bincount(bins, weights=p, minlength=nbins + 1)[:nbins]
    return {"k": k, "P": (P / count.clamp(min=1)).cpu().numpy(), "count": count.cpu().numpy()}


def _conv(x, w, b):
    """Periodic 3^3 convolution of x [N, N, N, ci] with w [27, ci, co]."""
    y = b.expand(x.shape[:3] + b.shape)
    for o in range(27):
        s = (1 - o // 9, 1 - (o // 3) % 3, 1 - o % 3)
        y = y + torch.roll(x, s, (0, 1, 2)) @ w[o]
    return y


def _net(psi, V, p):
    x = torch.stack([psi.real, psi.imag, V / V_SCALE, torch.view_as_real(psi).square().sum(-1) - 1.0], -1)
    at = 0
    for l, (ci, co) in enumerate(CHANNELS):
        w, b = p[at:at + 27 * ci * co].reshape(27, ci, co), p[at + 27 * ci * co:at + 27 * ci * co + co]
        at += 27 * ci * co + co
        x = _conv(x, w, b)
        if l < 2:
            x = torch.nn.functional.gelu(x)
    return x


def exact(case, seed):
    call = case["call"]
    if call == "ensemble":
        boxes = _boxes(case)
        dt = 0.2 / max(boxes) ** 2
        return [_steps(_initial(3, n, case["solitons"], seed, b).to(_cplx(case)).to(torch.complex128), case["steps"],
                       dt, 1.0, "reference")[0].cpu().numpy() for b, n in enumerate(boxes)]
    p = torch.from_numpy(_params(seed)).cuda().double() if call in ("gradient", "corrected") else None
    if call == "gradient":
        psi, V, fine = _pair(case, seed)
        psi, V, fine = psi.to(torch.complex128), V.double(), fine.to(torch.complex128)
        p.requires_grad_(True)
        target = torch.view_as_real((fine - psi) / TAU)
        loss = (_net(psi, V, p) - target).square().mean()
        loss.backward()
        return {"loss": float(loss), "grad": p.grad.cpu().numpy()}
    dim, N, dt, pref = case.get("dim", 3), case["N"], _dt(case), case["pref"]
    k0 = "reference" if case["dtype"] == "c128" else "zero"
    psi = _initial(dim, N, case["solitons"], seed).to(_cplx(case)).to(torch.complex128)
    if call == "corrected":
        mass = float(torch.view_as_real(psi).square().sum())
        psi, V = _steps(psi, 1, 4 * dt, pref, k0)
        with torch.no_grad():
            psi = psi + TAU * torch.view_as_complex(_net(psi, V, p).contiguous())
        psi = psi * math.sqrt(mass / float(torch.view_as_real(psi).square().sum()))
        return {"psi": psi, "fallbacks": 0}
    if call == "diagnose":
        e = _mass_energy(psi, _potential(psi, pref, k0))
        return dict(_spectrum(psi, case["mode"], case["nbins"]), M=e["mass"], E=e["energy"], K=e["kinetic"],
                    W=e["potential"])
    if call == "propagate":
        V = torch.zeros((N,) * dim, device="cuda", dtype=torch.float64)
        for _ in range(case["steps"]):
            psi = _drift(_kick(psi, V, 0.5 * dt), dt)
            V = _potential(psi, pref, k0)
            psi = _kick(psi, V, 0.5 * dt)
        return {"psi": psi, "V": V}
    if call == "run":
        n, m = case["steps"], case["nmeas"]
        at = [n - 1] if m == 1 else [k * (n - 1) // (m - 1) for k in range(m)]
        recs = []

        def measure(psi, V):
            rho = torch.view_as_real(psi).square().sum(-1)
            recs.append(dict(_mass_energy(psi, V), number=len(recs), rhomax=float(rho.max() / rho.mean()),
                             vmax=float(V.abs().max())))

        V = _potential(psi, pref, k0)
        measure(psi, V)
        psi = _kick(psi, V, 0.5 * dt)
        for i in range(n):
            psi = _drift(psi, dt)
            V = _potential(psi, pref, k0)
            if len(recs) - 1 < m and at[len(recs) - 1] == i:
                measure(psi, V)
            psi = _kick(psi, V, dt if i < n - 1 else 0.5 * dt)
        return {"psi": psi, "V": V, "records": recs}
    psi, V = _steps(psi, case["steps"], dt, pref, k0)
    out = {"psi": psi, "V": V}
    if call == "step+spectrum":
        out.update(_spectrum(psi, case["mode"], case["nbins"]))
    return out
