"""The work that users of mcstar_b200 have it do, as cases of a performance measurement.

Every case goes through the package's public entry points:

  step      Stepper.step: the fused conserved (or relaxing) steps of one resident field -- the
            simulation itself, 2D and 3D, FP32 and FP64, with and without thermal noise
  loop      the driver loop written against the mcstar-libs names (C2R, psi3_split, R2C,
            fill_kspace, update_eom), one call per kernel
  ensemble  Ensemble.run: many fields of mixed sizes stepped together
  analysis  the observables of an output interval: free energy, peaks, bond order
  adjoint   AdjointRun.sf_loss_and_grads: a run and its gradient
  lowpass   the local-amplitude low-pass of a 2D field

Fields are liquids (mean density plus uniform noise) or one-mode crystals with noise, made on
the GPU from the seed.  ``exact`` restates each case in plain FP64 torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mcstar-libs_b200"))

import mcstar_b200 as pfc  # noqa: E402

DX = math.pi / 4
PSI0, AMP = -0.2, 0.05
THS, RLIM = 0.0, 10.0  # peak threshold and neighbour radius of the analysis
DIVS = 2.0             # divisions per sigma of the low-pass


def listed():
    def case(name, kind, nx, ny, nz, dtype, **more):
        return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, dtype=dtype, **more)

    return [
        # the smallest call: a small noisy film advanced one step at a time by an interactive
        # driver that looks at the state after every step
        case("film-128-single", "step", 128, 128, 1, "f32", T=1e-3, dt=0.5, steps=1, prop="conserved"),
        # the 2D validation run of the repository's configurations: 256^2, FP64, no noise
        case("film-256-f64", "step", 256, 256, 1, "f64", T=0.0, dt=0.5, steps=100, prop="conserved"),
        # 2D grain growth in a large box commensurate with the crystal (a 2-3-5 size)
        case("grains-2400x2000", "step", 2400, 2000, 1, "f32", T=1e-3, dt=0.5, steps=20, prop="conserved"),
        # 3D nucleation, the repository's noisy 128^3 configuration between two outputs
        case("nucleation-128", "step", 128, 128, 128, "f32", T=1e-3, dt=0.5, steps=100, prop="conserved"),
        # a 3D box fitted to a crystal orientation: no power-of-two side
        case("slab-240x200x180", "step", 240, 200, 180, "f32", T=1e-3, dt=0.5, steps=20, prop="conserved"),
        # the FP64 side of a precision study
        case("cube-192-f64", "step", 192, 192, 192, "f64", T=0.0, dt=0.25, steps=10, prop="conserved"),
        # the headline workload of the benchmark: 512^3, FP32, no noise, 20 steps per call
        case("bulk-512", "step", 512, 512, 512, "f32", T=0.0, dt=0.25, steps=20, prop="conserved"),
        # a driver ported from mcstar-libs name by name, kernel call by kernel call
        case("driver-loop-256", "loop", 256, 256, 256, "f32", T=1e-3, dt=0.5, steps=4),
        # the batched workload of the benchmark: 48 films and 16 cubes of mixed sizes
        dict(name="ensemble-48-16", kind="ensemble", n2d=48, n3d=16, members=4, dtype="f32", steps=10),
        # the observables of one output interval on a bcc crystal
        case("analysis-256", "analysis", 256, 256, 256, "f32"),
        # the gradient of a structure-factor loss through a short 3D run
        case("gradient-128", "adjoint", 128, 128, 128, "f32", T=0.0, dt=0.25, steps=10, every=5),
        # post-processing of a large film: its local amplitude
        case("amplitude-2048", "lowpass", 2048, 2048, 1, "f32"),
    ]


# ---- drawn cases ----------------------------------------------------------------------------------
_SMOOTH = sorted(2 ** a * 3 ** b * 5 ** c for a in range(13) for b in range(8) for c in range(6)
                 if 2 ** a * 3 ** b * 5 ** c <= 4096)


def _side(rng, lo, hi):
    """A 2-3-5 length between lo and hi, spread over their logarithm (odd ones among them);
    a power of two now and then, as simulations prefer them."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if rng.random() < 0.25:
        return min(max(2 ** round(math.log2(v)), lo), hi)
    return min((s for s in _SMOOTH if lo <= s <= hi), key=lambda s: abs(math.log(s / v)))


def _steps(rng, cells, dtype, most):
    budget = 8e7 if dtype == "f32" else 4e7  # cell updates of a call
    return max(1, min(int(budget / cells), round(math.exp(rng.uniform(0.0, math.log(most))))))


def draw(rng):
    kind = rng.choices(("step2d", "step3d", "loop", "ensemble", "analysis", "adjoint", "lowpass"),
                       (6, 8, 3, 1, 2, 2, 1))[0]
    dtype = "f32" if rng.random() < 0.7 else "f64"
    T = rng.choice((0.0, 1e-3))
    dt = rng.choice((0.25, 0.5))
    if kind == "ensemble":
        return dict(kind="ensemble", n2d=rng.randint(4, 32), n3d=rng.randint(1, 8), members=rng.randint(1, 1 << 20),
                    dtype=dtype, steps=rng.randint(1, 10))
    if kind in ("step2d", "lowpass"):
        nx, ny, nz = _side(rng, 64, 3072), _side(rng, 64, 3072), 1
    elif kind == "analysis":  # (the bond order takes a cubic box)
        nx = ny = nz = _side(rng, 48, 288)
    elif kind == "adjoint":
        nx, ny, nz = (_side(rng, 32, 144) for _ in range(3))
    elif kind == "loop" and rng.random() < 0.4:
        nx, ny, nz = _side(rng, 64, 2048), _side(rng, 64, 2048), 1
    else:
        nx, ny, nz = (_side(rng, 32, 320) for _ in range(3))
    c = dict(kind="step" if kind.startswith("step") else kind, nx=nx, ny=ny, nz=nz, dtype=dtype)
    if kind in ("analysis", "lowpass"):
        return c
    c.update(T=T, dt=dt, steps=_steps(rng, nx * ny * nz, dtype, 100 if c["kind"] == "step" else 10))
    if c["kind"] == "step":
        c["prop"] = rng.choices(("conserved", "conserved_exp", "relax"), (8, 1, 1))[0]
        if c["prop"] == "relax":
            c["T"] = 0.0
    if kind == "adjoint":
        c.update(T=0.0, steps=min(c["steps"], 10), every=rng.randint(2, 10))
    return c


# ---- inputs -----------------------------------------------------------------------------------------
def _np(case):
    return np.float32 if case["dtype"] == "f32" else np.float64


def _eps(case):
    return 0.1 if case["kind"] == "adjoint" else 0.25


def _lens(case):
    return tuple(case[k] * DX for k in ("nx", "ny", "nz"))


def _namp(case):
    return pfc.namp_from_temperature(case["T"], case["dt"]) if case.get("T") else 0.0


def _liquid(case, seed):
    """psi0 + U(-amp, amp), FP64, (nz, ny, nx)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand((case["nz"], case["ny"], case["nx"]), dtype=torch.float64, device="cuda", generator=g)
    return PSI0 + AMP * (2.0 * u - 1.0)


def _crystal(case, seed, amp=0.1, noise=0.01):
    """A one-mode crystal (bcc; in 2D triangular) fitted to the box, at a random offset, with
    noise; FP64, (nz, ny, nx)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    h = 1.0 / math.sqrt(2.0)
    qs = [(h, h, 0), (h, -h, 0), (h, 0, h), (h, 0, -h), (0, h, h), (0, h, -h)]
    if case["nz"] == 1:
        qs = [(1.0, 0, 0), (0.5, math.sqrt(0.75), 0), (0.5, -math.sqrt(0.75), 0)]
    off = torch.rand(3, dtype=torch.float64, device="cuda", generator=g).tolist()
    z, y, x = (torch.arange(n, dtype=torch.float64, device="cuda") / n for n in shape)
    f = PSI0 + noise * (2.0 * torch.rand(shape, dtype=torch.float64, device="cuda", generator=g) - 1.0)
    for q in qs:
        m = [round(a * n * DX / (2 * math.pi)) for a, n in zip(q, (case["nx"], case["ny"], case["nz"]))]
        f += amp * torch.cos(2 * math.pi * (m[0] * (x + off[0])[None, None, :] + m[1] * (y + off[1])[None, :, None] +
                                            m[2] * (z + off[2])[:, None, None]))
    return f


def _cdtype(case):
    return torch.complex64 if case["dtype"] == "f32" else torch.complex128


def _fdtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.float64


def _spectrum(case, psi):
    """The half spectrum of a real field in the case's precision: what the run starts from."""
    return torch.fft.rfftn(psi).to(_cdtype(case))


def _members(case, seed):
    ms = pfc.ensemble_members(seed=case["members"], n2d=case["n2d"], n3d=case["n3d"])
    for i, m in enumerate(ms):  # other inputs for another seed, the same sizes
        m["seed"] = (m["seed"] + 7919 * seed + i) % (2 ** 31)
    return ms


def _target(case, seed):
    """The structure factor a gradient run is fitted to: that of another crystal."""
    n = case["nx"] * case["ny"] * case["nz"]
    t = torch.fft.rfftn(_crystal(case, seed + 1000003, amp=0.08) - 0.01)
    return (t.abs() ** 2 / n).to(_fdtype(case)).reshape(-1)


def prepare(case, seed):
    kind, dt = case["kind"], _np(case)
    if kind == "ensemble":
        return dict(case=case, ens=pfc.Ensemble(_members(case, seed), dtype=dt))
    shape = (case["nx"], case["ny"], case["nz"])
    if kind == "step":
        st = pfc.Stepper(shape, DX, case["dt"], _eps(case), dtype=dt, namp=_namp(case), seed=seed)
        st.kpsi.copy_(torch.view_as_real(_spectrum(case, _liquid(case, seed))).reshape(-1))
        return dict(case=case, st=st)
    if kind == "loop":
        a = {k: pfc.GPUArray(shape, dt) for k in ("kpsi", "tmp", "psi", "knl", "noise")}
        a["kpsi"].ptr_cmpl().copy_(_spectrum(case, _liquid(case, seed)))
        return dict(case=case, a=a, c2r=pfc.CufftPlan(dt, pfc.C2R, shape), r2c=pfc.CufftPlan(dt, pfc.R2C, shape),
                    rng=pfc.NoiseHostApi(dt, seed))
    if kind == "analysis":
        st = pfc.Stepper(shape, DX, 0.5, _eps(case), dtype=dt)
        psi = pfc.GPUArray(shape, dt)
        field = _crystal(case, seed)
        psi.ptr_real().copy_(field)
        st.kpsi.copy_(torch.view_as_real(_spectrum(case, field)).reshape(-1))
        return dict(case=case, st=st, psi=psi)
    if kind == "adjoint":
        run_ = pfc.AdjointRun(shape, DX, case["dt"], _eps(case), dtype=dt, every=case["every"])
        return dict(case=case, run=run_, psi=_crystal(case, seed).to(_fdtype(case)), s=_target(case, seed))
    ctx = pfc.get_context(shape, dt)
    s = dict(case=case, ctx=ctx, psi=_crystal(case, seed).to(_fdtype(case)).reshape(-1), spectrum=ctx.empty_state(),
             aux=ctx.empty_state(), kgauss=ctx.empty_state())
    ctx.gaussian_init(s["kgauss"], _lens(case), (DX, DX, DX), DIVS)
    return s


# ---- the passes ---------------------------------------------------------------------------------------
def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "step":
        st = state["st"]
        change = st.step(case["steps"], case["prop"])
        return {"kpsi": st.kpsi, "change": change}
    if kind == "ensemble":
        state["ens"].run(case["steps"])
        return {"kpsi": list(state["ens"].kpsi)}
    if kind == "loop":
        a, lens, eps = state["a"], _lens(case), _eps(case)
        namp = _namp(case)
        for _ in range(case["steps"]):
            a["kpsi"] >> a["tmp"]
            state["c2r"].execute(a["tmp"], a["psi"])
            pfc.call_kernel_psi3_split(a["psi"], norm=True)
            state["r2c"].execute(a["psi"], a["knl"])
            if namp:
                state["rng"].fill_kspace(a["noise"])
                pfc.call_kernel_update_eom(a["kpsi"], a["knl"], a["noise"], namp, case["dt"], eps, lens)
            else:
                pfc.call_kernel_update_eom(a["kpsi"], a["knl"], 0.0, case["dt"], eps, lens)
        return {"kpsi": a["kpsi"].buf}
    if kind == "analysis":
        st, psi = state["st"], state["psi"]
        energy = st.free_energy()
        n, recs = pfc.findpeaks_device(psi, THS)
        rows = st.ctx.bond_order(recs, n, st.hh, THS, st.lens[0], RLIM)
        return {"energy": energy, "n": n, "peaks": recs.view(st.ctx.torch_dtype), "rows": rows}
    if kind == "adjoint":
        loss, g, deps, dpsi0 = state["run"].sf_loss_and_grads(state["psi"], case["steps"], state["s"])
        return {"loss": loss, "grad": g, "deps": deps, "dpsi0": dpsi0}
    ctx = state["ctx"]
    ctx.r2c(state["psi"], state["spectrum"])
    ctx.amplitude_lowpass(state["spectrum"], state["aux"], state["kgauss"], _lens(case))
    return {"amplitude": state["aux"][: ctx.n_real], "spectrum": state["spectrum"]}


# ---- what a pass cannot do without --------------------------------------------------------------------
def _transform_flops(shape):
    n = shape[0] * shape[1] * shape[2]
    return 2.5 * n * math.log2(n)


def _state_bytes(shape, fsize):
    return (shape[0] // 2 + 1) * shape[1] * shape[2] * 2 * fsize


def work(case):
    fsize = 4 if case["dtype"] == "f32" else 8
    if case["kind"] == "ensemble":
        shapes = [m["shape"] for m in pfc.ensemble_members(seed=case["members"], n2d=case["n2d"], n3d=case["n3d"])]
        return {"bytes": sum(2 * _state_bytes(s, fsize) for s in shapes) * case["steps"],
                "flops": sum(2 * _transform_flops(s) + 40 * math.prod(s) for s in shapes) * case["steps"]}
    shape = (case["nx"], case["ny"], case["nz"])
    n, S, F = math.prod(shape), _state_bytes(shape, fsize), _transform_flops(shape)
    if case["kind"] == "step":  # every step reads and writes the state
        return {"bytes": 2 * S * case["steps"], "flops": (2 * F + 25 * n) * case["steps"]}
    if case["kind"] == "loop":  # copy, C2R, psi3, R2C, (noise,) update: each call's own inputs and outputs
        return {"bytes": (11 + (2 if case["T"] else 0)) * S * case["steps"], "flops": (2 * F + 40 * n) * case["steps"]}
    if case["kind"] == "analysis":
        return {"bytes": S + n * fsize, "flops": F + 40 * n}
    if case["kind"] == "adjoint":  # forward, recomputed and adjoint steps
        return {"bytes": 8 * S * case["steps"], "flops": 8 * F * case["steps"]}
    return {"bytes": 4 * S, "flops": 4 * F}


# ---- the same in plain FP64 ---------------------------------------------------------------------------
def _k1d(n, half, length):
    m = torch.arange(n // 2 + 1 if half else n, dtype=torch.float64, device="cuda")
    return torch.where(m < n // 2 + 1, m, m - n) * (2 * math.pi / length)


def _ksq(shape, lens):
    kx, ky, kz = _k1d(shape[0], True, lens[0]), _k1d(shape[1], False, lens[1]), _k1d(shape[2], False, lens[2])
    return kz[:, None, None] ** 2 + ky[None, :, None] ** 2 + kx[None, None, :] ** 2


_M32 = 0xFFFFFFFF


def _philox(c, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors holding 32-bit words."""
    x, y, z, w = c
    for r in range(10):
        p0, p1 = x * 0xD2511F53, z * 0xCD9E8D57  # (the low 64 bits: int64 wraps)
        x, y, z, w = (((p1 >> 32) & _M32) ^ y ^ k0, p1 & _M32, ((p0 >> 32) & _M32) ^ w ^ k1, p0 & _M32)
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return x, y, z, w


def _noise(shape, seed, counter, dtype):
    """The k-space noise of a step: complex normal modes, Hermitian on the planes i0 = 0 and
    i0 = nx/2 (keyed by the lower member of a pair), self-conjugate modes real."""
    nx, ny, nz = shape
    nxh = nx // 2 + 1
    i0 = torch.arange(nxh, device="cuda")[None, None, :]
    i1 = torch.arange(ny, device="cuda")[None, :, None]
    i2 = torch.arange(nz, device="cuda")[:, None, None]
    lin = (i2 * ny + i1) * nxh + i0
    plane = (i0 == 0) | ((i0 == nx // 2) if nx % 2 == 0 else (i0 < 0))
    part = torch.where(plane, (((nz - i2) % nz) * ny + (ny - i1) % ny) * nxh + i0, lin)
    canon, conj, self_conj = torch.minimum(lin, part), part < lin, plane & (part == lin)
    zero = torch.zeros_like(canon)
    x, y, z, w = _philox((canon & _M32, canon >> 32, zero + (counter & _M32), zero + (counter >> 32)),
                         seed & _M32, (seed >> 32) & _M32)
    if dtype == "f32":
        u1, u2 = (((a >> 9) * 2 + 1).double() * 2.0 ** -24 for a in (x, y))
    else:
        u1, u2 = (((((a << 20) | (b >> 12)) * 2) + 1).double() * 2.0 ** -53 for a, b in ((x, y), (z, w)))
    rad = torch.sqrt(-2.0 * torch.log(u1))
    g1, g2 = rad * torch.cos(2 * math.pi * u2), rad * torch.sin(2 * math.pi * u2)
    h = math.sqrt(0.5)
    re = torch.where(self_conj, g1, g1 * h)
    im = torch.where(self_conj, torch.zeros_like(g2), torch.where(conj, -g2 * h, g2 * h))
    return torch.complex(re, im)


def _flat(k):
    return torch.view_as_real(k.contiguous()).reshape(-1)


def _advance(k, shape, lens, dt, eps, steps, namp=0.0, seed=0, dtype="f32", prop="conserved"):
    """Steps of the conserved equation (semi-implicit or exponential) or of the relaxation, C = 1."""
    nx, ny, nz = shape
    k2 = _ksq(shape, lens)
    lin = 2.0 - eps - 2.0 * k2 + k2 * k2
    change = 0.0
    if prop == "conserved":
        a = 1.0 / (1.0 + dt * k2 * lin)
        b, g = -dt * k2 * a, dt * torch.sqrt(k2) * a
    elif prop == "conserved_exp":
        L = k2 * lin
        a = torch.exp(-L * dt)
        q = torch.where(L == 0, torch.full_like(L, -dt), torch.expm1(-L * dt) / L)
        b, g = k2 * q, -torch.sqrt(k2) * q
    else:
        a = 1.0 / (1.0 + dt * lin)
        b = -dt * a
    for t in range(steps):
        psi = torch.fft.irfftn(k, s=(nz, ny, nx))
        new = a * k + b * torch.fft.rfftn(psi * psi * psi - psi)
        del psi
        if namp:
            new += (g * (namp * math.sqrt(nx * ny * nz))) * _noise(shape, seed, t, dtype)
        if prop == "relax":
            change = (new - k).abs().max().item()
        else:
            new[0, 0, 0] = k[0, 0, 0]
        k = new
    return k, change


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        out = []
        for m in _members(case, seed):
            shape = m["shape"]
            u = np.random.default_rng(m["seed"]).uniform(-0.01, 0.01, size=shape[::-1])
            psi = torch.from_numpy((m["psi0"] + u).astype(_np(case))).cuda().double()
            k, _ = _advance(torch.fft.rfftn(psi), shape, tuple(n * m["dx"] for n in shape), m["dt"], m["eps"],
                            case["steps"], namp=m["namp"], seed=m["seed"], dtype=case["dtype"])
            out.append(_flat(k))
        return {"kpsi": out}
    shape, lens = (case["nx"], case["ny"], case["nz"]), _lens(case)
    n = math.prod(shape)
    if kind in ("step", "loop"):
        k = _spectrum(case, _liquid(case, seed)).to(torch.complex128)
        k, change = _advance(k, shape, lens, case["dt"], _eps(case), case["steps"], namp=_namp(case),
                             seed=seed, dtype=case["dtype"], prop=case.get("prop", "conserved"))
        return {"kpsi": _flat(k), "change": change} if kind == "step" else {"kpsi": _flat(k)}
    if kind == "analysis":
        k = _spectrum(case, _crystal(case, seed)).to(torch.complex128)
        psi = torch.fft.irfftn(k, s=shape[::-1])
        lin = torch.fft.irfftn(k * ((1.0 - _ksq(shape, lens)) ** 2 - _eps(case)), s=shape[::-1])
        energy = DX ** 3 * float((0.5 * psi * lin + 0.25 * psi ** 4).sum())
        return {"energy": energy, "n": None, "peaks": None, "rows": None}
    if kind == "adjoint":
        s = _target(case, seed).double().view(shape[2], shape[1], -1)
        psi = _crystal(case, seed).to(_fdtype(case)).double().requires_grad_()
        eps = torch.tensor(_eps(case), dtype=torch.float64, device="cuda", requires_grad=True)
        k2, dt = _ksq(shape, lens), case["dt"]
        k = torch.fft.rfftn(psi)
        for _ in range(case["steps"]):
            f = torch.fft.irfftn(k, s=shape[::-1])
            k = (k - dt * k2 * torch.fft.rfftn(f * f * f - f)) / (1.0 + dt * k2 * (1.0 - eps + (1.0 - k2) ** 2))
        w = torch.full((shape[0] // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
        w[0] = 1.0
        if shape[0] % 2 == 0:
            w[-1] = 1.0
        loss = (w * ((k.real ** 2 + k.imag ** 2) / n - s) ** 2).sum()
        loss.backward()
        return {"loss": loss.item(), "grad": psi.grad, "deps": eps.grad.item(), "dpsi0": psi.grad.sum().item()}
    psi = _crystal(case, seed).to(_fdtype(case)).double()
    kx, ky = _k1d(shape[0], True, lens[0]), _k1d(shape[1], False, lens[1])
    e = torch.exp(-0.5 * (1.1 * DIVS * DX) ** 2 * (ky[None, :, None] ** 2 + kx[None, None, :] ** 2))
    high = torch.fft.irfftn(torch.fft.rfftn(psi) * (1.0 - e), s=shape[::-1])
    low = torch.fft.rfftn(high * high) * e
    return {"amplitude": torch.fft.irfftn(low, s=shape[::-1]).reshape(-1), "spectrum": _flat(low)}
