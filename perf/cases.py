"""What the framework's users have it compute, as cases that can be timed and compared.

Kinds of case, each through the calls that a program makes:

  step     RK4 steps of a plan, in place on the half spectrum (Plan.step), 2D and 3D,
           single and batched trajectories, every forcing, with or without the
           physical field of the last state
  step_fn  the drop-in's functional step (u, u_hat) -> (u, u_hat, e_inj)
  nufft    the combined loop's particle update: coarsening of the fine spectrum, type-2
           NUFFT at the particles, Euler shift
  dft      the drop-in's exact spectral interpolation of a coarse field at particles
  sph      the combined loop's SPH relaxation of the particle velocities
  grad     forward steps under autograd and the adjoint sweep back to the initial
           spectrum
  diag     the diagnostics of a log step: kinetic energy, dissipation, spectrum, maxima

``exact`` restates each in 64 bits with torch alone.
"""

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ql-les-data_gb300"))

from l3es import _native, adjoint, integrator, relax, spectral_solver  # noqa: E402

TWO_PI = 2.0 * math.pi
EPS_INJ, KF, DRAG, KOLM_K, KOLM_AMP = 0.1, 2, 0.1, 4, 1.0
U_REF, RELAX_FACTOR, RELAX_DT = 4.0, 2.0, 2e-3  # the reference's hit32 settings


def listed():
    return [
        # the smallest call: one functional step of a 2D field, all launches and latency
        {"name": "step_fn_2d_64", "kind": "step_fn", "dim": 2, "n": 64},
        # 2D Kolmogorov flow at the size of the bench's 2D workload
        {"name": "kolmogorov_2d_256", "kind": "step", "dim": 2, "n": 256, "batch": 1, "steps": 10,
         "forcing": "kolmogorov", "u_out": False},
        # an ensemble of small 2D runs, one viscosity each, stepped as one batched plan
        {"name": "ensemble_2d_128x8", "kind": "step", "dim": 2, "n": 128, "batch": 8, "steps": 10,
         "forcing": "kolmogorov", "u_out": False},
        # the small 3D grid of the validation runs (ten steps)
        {"name": "decay_3d_64", "kind": "step", "dim": 3, "n": 64, "batch": 1, "steps": 10, "forcing": "none",
         "u_out": False},
        # a log step of the reference's energy-pinned forced turbulence: step and physical field
        {"name": "pinned_3d_128_u", "kind": "step", "dim": 3, "n": 128, "batch": 1, "steps": 1,
         "forcing": "ekin_tot", "u_out": True},
        # the headline workload's step: 256^3, constant-power forcing
        {"name": "forced_3d_256", "kind": "step", "dim": 3, "n": 256, "batch": 1, "steps": 1,
         "forcing": "const_power", "u_out": False},
        # the largest grid
        {"name": "decay_3d_512", "kind": "step", "dim": 3, "n": 512, "batch": 1, "steps": 1, "forcing": "none",
         "u_out": False},
        # particle update of the headline workload
        {"name": "nufft_3d_32", "kind": "nufft", "dim": 3, "n_fine": 256, "c": 32, "np": 32768, "width": 6, "batch": 1},
        # the combined driver's default interpolation, on part of a particle set
        {"name": "dft_3d_32", "kind": "dft", "dim": 3, "c": 32, "np": 10007},
        # relaxation step of the reference's own turbulence configuration
        {"name": "sph_3d_32", "kind": "sph", "dim": 3, "n": 32},
        # gradient through two steps at the size of the differentiation workload
        {"name": "grad_3d_128", "kind": "grad", "dim": 3, "n": 128, "steps": 2, "forcing": "const_power"},
        # diagnostics of a log step of the headline workload
        {"name": "diag_3d_256", "kind": "diag", "dim": 3, "n": 256},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step_fn", "nufft", "dft", "sph", "grad", "diag"])
    dim = rng.choice([2, 3])
    if kind == "step":
        forcing = rng.choice(["none", "const_power", "ekin_tot"] + (["kolmogorov"] * 3 if dim == 2 else []))
        if dim == 2:
            n, most = rng.choice([32, 64, 128, 256, 512]), 1 << 19
            batch = _log_int(rng, 1, max(1, min(9, most // n**2)))
            steps = _log_int(rng, 1, 20)
        else:
            n = rng.choice([16, 32, 64, 128, 256])
            batch = rng.choice([1, 1, 1, 2, 3]) if n <= 128 else 1
            steps = _log_int(rng, 1, max(1, min(20, (1 << 26) // (n**3 * batch))))
        return {"kind": kind, "dim": dim, "n": n, "batch": batch, "steps": steps, "forcing": forcing,
                "u_out": rng.random() < 0.3}
    if kind == "step_fn":
        return {"kind": kind, "dim": dim, "n": rng.choice([32, 64, 128, 256] if dim == 2 else [16, 32, 64, 128])}
    if kind == "nufft":
        c = rng.choice([16, 32, 64])
        return {"kind": kind, "dim": dim, "n_fine": c * rng.choice([1, 2, 4]), "c": c, "np": _log_int(rng, 500, 60000),
                "width": rng.choice([4, 6, 6, 6, 8]), "batch": rng.choice([1, 1, 2, 5])}
    if kind == "dft":
        return {"kind": kind, "dim": dim, "c": rng.choice([8, 16, 32]) if dim == 3 else rng.choice([16, 32, 64]),
                "np": _log_int(rng, 300, 12000)}
    if kind == "sph":
        return {"kind": kind, "dim": dim, "n": rng.randint(8, 36) if dim == 3 else rng.randint(12, 160)}
    if kind == "grad":
        return {"kind": kind, "dim": dim, "n": rng.choice([32, 64, 128]), "steps": rng.randint(1, 3),
                "forcing": rng.choice(["none", "const_power", "ekin_tot"])}
    return {"kind": kind, "dim": dim, "n": rng.choice([32, 64, 128, 256])}


# --- inputs ---------------------------------------------------------------------------


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 16 + salt)


def _axes(dim):
    return (-3, -2, -1) if dim == 3 else (-2, -1)


def _wavenumbers(dim, n, dtype):
    """(3, ...) integer wavenumbers of a half spectrum, the Nyquist entry of the half axis positive."""
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=dtype, device="cuda")
    kh = torch.arange(n // 2 + 1, dtype=dtype, device="cuda")
    if dim == 3:
        return torch.stack(torch.meshgrid(k, k, kh, indexing="ij"))
    g = torch.meshgrid(k, kh, indexing="ij")
    return torch.stack([g[0], g[1], torch.zeros_like(g[0])])


def _half_weights(n, dtype):
    w = torch.full((n // 2 + 1,), 2.0, dtype=dtype, device="cuda")
    w[0] = w[-1] = 1.0
    return w


def _flow(dim, n, batch, gen, energy=0.5, kp=4.0):
    """Half spectra (batch, 3, ...) complex64 of solenoidal random fields with a developed
    spectrum (energy-containing range at kp, inertial slope, exponential cutoff) and the
    given kinetic energy; 2D fields have no third component."""
    k = _wavenumbers(dim, n, torch.float32)
    k2 = (k * k).sum(0)
    kk = torch.sqrt(k2)
    slope = 17.0 / 6.0 if dim == 3 else 3.5
    e = kk**4 / (1.0 + (kk / kp) ** 2) ** slope * torch.exp(-8.0 * kk / n)
    amp = torch.sqrt(e / torch.clamp(kk, min=1.0) ** (dim - 1))
    out = torch.empty((batch, 3) + tuple(k2.shape), dtype=torch.complex64, device="cuda")
    w = _half_weights(n, torch.float32)
    for b in range(batch):
        noise = torch.randn((3,) + (n,) * dim, generator=gen, device="cuda")
        if dim == 2:
            noise[2] = 0.0
        a = torch.fft.rfftn(noise, dim=_axes(dim))
        a *= amp
        div = (a * k).sum(0) / torch.clamp(k2, min=1.0)
        a -= div * k
        # fields of a real velocity: the transform there and back drops the rest
        a = torch.fft.rfftn(torch.fft.irfftn(a, s=(n,) * dim, dim=_axes(dim)), dim=_axes(dim))
        ke = 0.5 * float((w * (a.real**2 + a.imag**2)).sum(dtype=torch.float64)) / float(n) ** (2 * dim)
        out[b] = a * math.sqrt(energy / ke)
    return out


def _flow_args(case):
    dim, n, forcing = case["dim"], case["n"], case.get("forcing", "none")
    a = {"dim": dim, "n": n}
    if dim == 3:
        a.update(nu=1.28 / n, dt=1.0 / n)
    else:
        a.update(nu=1e-3 * max(1.0, 256.0 / n), dt=0.25 / n)
    if forcing == "const_power":
        a.update(forcing="const_power", kf=KF, eps_inj=EPS_INJ)
    elif forcing == "ekin_tot":
        a.update(forcing="ekin_tot", kf=KF, e_kin_init=0.5)
    elif forcing == "kolmogorov":
        a.update(drag=DRAG, kolm_k=KOLM_K, kolm_amp=KOLM_AMP)
    return a


def _viscosities(case):
    nu = _flow_args(case)["nu"]
    return [nu * (0.75 + 0.5 * b / max(1, case["batch"] - 1)) for b in range(case["batch"])]


def _positions(dim, count, batch, gen):
    shape = (count, dim) if batch == 1 else (batch, count, dim)
    return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) * TWO_PI


def _lattice(dim, n, gen):
    ax = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * (TWO_PI / n)
    r = torch.stack([g.reshape(-1) for g in torch.meshgrid(*([ax] * dim), indexing="ij")], 1)
    jitter = torch.randn(r.shape, generator=gen, device="cuda", dtype=torch.float64)
    return torch.remainder(r + 0.15 * TWO_PI / n * jitter, TWO_PI).contiguous()


def _inputs(case, seed):
    gen, kind, dim = _gen(seed), case["kind"], case["dim"]
    if kind == "step":
        uh = _flow(dim, case["n"], case["batch"], gen)
        return {"uh": uh if case["batch"] > 1 else uh[0].contiguous()}
    if kind in ("step_fn", "diag"):
        n = case["n"]
        uh = _flow(dim, n, 1, gen)[0].contiguous()
        u = torch.fft.irfftn(uh, s=(n,) * dim, dim=_axes(dim))
        return {"uh": uh, "u": u.contiguous() if dim == 3 else u[..., None].contiguous()}
    if kind == "nufft":
        uh = _flow(dim, case["n_fine"], case["batch"], gen)
        return {"uh": uh if case["batch"] > 1 else uh[0].contiguous(),
                "r": _positions(dim, case["np"], case["batch"], gen)}
    if kind == "dft":
        c = case["c"]
        u = torch.fft.irfftn(_flow(dim, c, 1, gen, kp=3.0)[0], s=(c,) * dim, dim=_axes(dim))
        return {"u": u[:dim].contiguous(), "r": _positions(dim, case["np"], 1, gen)}
    if kind == "sph":
        r = _lattice(dim, case["n"], gen)
        return {"r": r, "u": U_REF * torch.randn(r.shape, generator=gen, device="cuda", dtype=torch.float64)}
    n = case["n"]  # grad
    uh = _flow(dim, n, 1, gen)[0].contiguous()
    # cotangent of a loss on the final real field
    g = _flow(dim, n, 1, gen, energy=1.0)[0] * (_half_weights(n, torch.float32) / float(n) ** dim)
    return {"uh": uh, "g": g.contiguous()}


# --- the cases ------------------------------------------------------------------------


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"], kind, dim = case, case["kind"], case["dim"]
    if kind == "step":
        s["plan"] = _native.Plan(batch=case["batch"], **_flow_args(case))
        if case["batch"] > 1:
            s["plan"].set_nu(_viscosities(case))
        s["u"] = torch.empty(s["plan"].phys_shape, device="cuda") if case["u_out"] else None
    elif kind == "step_fn":
        a = _flow_args(case)
        axes = (1, 2, 3) if dim == 3 else (1, 2)
        rhs = spectral_solver.rhs_wrapper(case["n"], a["nu"], axes)
        s["step"] = spectral_solver.rk4_wrapper(a["dt"], rhs, None, None, "none", axes)
    elif kind == "nufft":
        s["plan"] = _native.InterpPlan(dim=dim, ckp_n=case["c"], n_fine=case["n_fine"], width=case["width"],
                                       np_max=case["np"], batch=case["batch"])
        s["u_r"], s["r_next"] = torch.empty_like(s["r"]), torch.empty_like(s["r"])
    elif kind == "dft":
        s["interp"] = integrator.spectral_interpolator_wrapper(case["c"], (1, 2, 3) if dim == 3 else (1, 2),
                                                               backend="dft")
    elif kind == "sph":
        s["relax"] = relax.relax_velocity_wrapper(case["n"], dim, TWO_PI, U_REF, RELAX_FACTOR)
        s["r_next"] = torch.empty_like(s["r"])
    elif kind == "grad":
        a = _flow_args(case)
        s["plan"] = adjoint.make_plan(a["n"], a["nu"], dim, a["dt"], a.get("forcing", "none"), kf=a.get("kf", 0),
                                      eps_inj=a.get("eps_inj", 0.0), e_kin_init=a.get("e_kin_init", 0.0))
        s["uh"].requires_grad_(True)
    else:
        s["plan"] = _native.Plan(dim=dim, n=case["n"], nu=_flow_args(case)["nu"], dt=1.0)
        for name, count in (("ke", 1), ("eps", 1), ("ek", case["n"]), ("stats", 4)):
            s[name] = torch.empty(count, device="cuda", dtype=torch.float64)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        s["plan"].step(s["uh"], case["steps"], u_out=s["u"])
        return {"u_hat": s["uh"], "u": s["u"]}
    if kind == "step_fn":
        u, u_hat, e_inj = s["step"](s["u"], s["uh"])
        return {"u": u, "u_hat": u_hat, "e_inj": e_inj}
    if kind == "nufft":
        s["plan"].set_spectrum(s["uh"])
        s["plan"].interp(s["r"], s["u_r"], backend="nufft", dt=RELAX_DT, r_out=s["r_next"])
        return {"u_r": s["u_r"], "r": s["r_next"]}
    if kind == "dft":
        return {"u_r": s["interp"](s["u"], s["r"])}
    if kind == "sph":
        return {"u_r": s["relax"](s["r"], s["u"], RELAX_DT, r_out=s["r_next"]), "r": s["r_next"]}
    if kind == "grad":
        y = adjoint.integrate(s["uh"], s["plan"], case["steps"])
        (grad,) = torch.autograd.grad(y, s["uh"], s["g"])
        return {"u_hat": y.detach(), "grad": grad}
    p = s["plan"]
    p.kinetic_energy(s["uh"], s["ke"])
    p.dissipation(s["uh"], p.nu, s["eps"])
    p.energy_spectrum(s["uh"], s["ek"])
    p.field_stats(s["u"], s["stats"])
    return {"ke": s["ke"], "eps": s["eps"], "ek": s["ek"], "stats": s["stats"]}


def work(case):
    kind, dim = case["kind"], case["dim"]
    if kind in ("step", "step_fn", "grad", "diag"):
        n, batch = case["n"], case.get("batch", 1)
        points, modes = n**dim * batch, n ** (dim - 1) * (n // 2 + 1) * batch
        spectrum, field = 24.0 * modes, 12.0 * points
        fft = 2.5 * points * math.log2(n**dim)  # one real transform
        stage = 9 * fft + 12.0 * points + 120.0 * modes
        if kind == "step":
            return {"bytes": 2 * spectrum + (field if case["u_out"] else 0.0),
                    "flops": case["steps"] * 4 * stage + (3 * fft if case["u_out"] else 0.0)}
        if kind == "step_fn":
            return {"bytes": 2 * spectrum + field, "flops": 4 * stage + 3 * fft}
        if kind == "grad":  # forward, inner stages again, and a product of 9 inverse and 6 forward transforms each
            return {"bytes": 4 * spectrum, "flops": case["steps"] * (7 * stage + 4 * (15 * fft + 300.0 * modes))}
        return {"bytes": spectrum + field, "flops": 60.0 * modes + 12.0 * points}
    if kind == "nufft":
        c, batch, width = case["c"], case["batch"], case["width"]
        points, grid = case["np"] * batch, (2 * c) ** dim * batch
        return {"bytes": 24.0 * c ** (dim - 1) * (c // 2 + 1) * batch + 24.0 * dim * points,
                "flops": 3 * 2.5 * grid * math.log2((2 * c) ** dim) + points * dim * (2.0 * width**dim + 20 * width)}
    if kind == "dft":
        c, points = case["c"], case["np"]
        return {"bytes": 4.0 * dim * c**dim + 16.0 * dim * points, "flops": 4.0 * points * dim * c**dim}
    points = case["n"] ** dim  # sph: about 113 neighbours in 3D and 28 in 2D
    return {"bytes": 32.0 * dim * points, "flops": points * (113 if dim == 3 else 28) * 80.0}


# --- the same in 64 bits --------------------------------------------------------------


class _Flow64:
    """Right-hand side and RK4 step in FP64, differentiable by autograd."""

    def __init__(self, dim, n, nu, dt, forcing="none", kf=0, eps_inj=0.0, e_kin_init=0.0, drag=0.0, kolm_k=0,
                 kolm_amp=0.0):
        self.dim, self.n, self.dt, self.forcing = dim, n, dt, forcing
        self.eps_inj, self.e0 = eps_inj, e_kin_init
        self.k = _wavenumbers(dim, n, torch.float64)
        self.k2 = (self.k * self.k).sum(0)
        self.lin = nu * self.k2 + drag
        self.keep = (self.k.abs() < 2.0 / 3.0 * (n // 2 + 1)).all(0).to(torch.float64)
        self.band = ((self.k2 > 0) & (self.k2 <= kf * kf)).to(torch.float64)
        self.w = _half_weights(n, torch.float64)
        self.force = (0, kolm_k, -0.5 * kolm_amp * n * n) if kolm_k else None

    def field(self, a):
        return torch.fft.irfftn(a, s=(self.n,) * self.dim, dim=_axes(self.dim))

    def curl(self, a):
        k = self.k
        return 1j * torch.stack([k[1] * a[2] - k[2] * a[1], k[2] * a[0] - k[0] * a[2], k[0] * a[1] - k[1] * a[0]])

    def energy(self, a):
        return 0.5 * (self.w * (a.real**2 + a.imag**2)).sum() / float(self.n) ** (2 * self.dim)

    def rhs(self, a):
        u, om = self.field(a), self.field(self.curl(a))
        p = torch.stack([u[1] * om[2] - u[2] * om[1], u[2] * om[0] - u[0] * om[2], u[0] * om[1] - u[1] * om[0]])
        del u, om
        du = torch.fft.rfftn(p, dim=_axes(self.dim)) * self.keep
        du = du - ((du * self.k).sum(0) / torch.clamp(self.k2, min=1.0)) * self.k
        du = du - self.lin * a
        if self.force is not None:
            f = torch.zeros_like(a)
            f[0, self.force[0], self.force[1]] = 1j * self.force[2]
            du = du + f
        if self.forcing == "const_power":
            du = du + (self.eps_inj / (2.0 * self.energy(a * self.band) + 1e-30)) * a * self.band
        return du

    def step(self, a):
        dt = self.dt
        k1 = self.rhs(a)
        acc = a + dt / 6 * k1
        k2 = self.rhs(a + 0.5 * dt * k1)
        acc = acc + dt / 3 * k2
        k3 = self.rhs(a + 0.5 * dt * k2)
        acc = acc + dt / 3 * k3
        acc = acc + dt / 6 * self.rhs(a + dt * k3)
        if self.forcing == "ekin_tot":
            low = self.energy(acc * self.band)
            alpha = torch.sqrt(torch.clamp((self.e0 - (self.energy(acc) - low)) / (low + 2.220446049250313e-16), min=0.0))
            acc = acc * (alpha * self.band + (1.0 - self.band))
        return acc


def _exact_flow(case, uh):
    args = _flow_args(case)
    nus = _viscosities(case) if case["batch"] > 1 else [args["nu"]]
    outs, fields = [], []
    for b, nu in enumerate(nus):
        m = _Flow64(**dict(args, nu=nu))
        a = (uh[b] if case["batch"] > 1 else uh).to(torch.complex128)
        for _ in range(case["steps"]):
            a = m.step(a)
        outs.append(a)
        if case["u_out"]:
            f = m.field(a)
            fields.append(f if case["dim"] == 3 else f[..., None])
    pack = (lambda v: torch.stack(v)) if case["batch"] > 1 else (lambda v: v[0])
    return {"u_hat": pack(outs), "u": pack(fields) if fields else None}


def _spectral_sum(h, r):
    """Re sum_k h[k] exp(i k.r) / c^dim of full spectra (comp, c, ..., c) at positions (count, dim)."""
    comp, c, dim = h.shape[0], h.shape[1], r.shape[1]
    k = torch.fft.fftfreq(c, 1.0 / c, dtype=torch.float64, device="cuda")
    out = torch.empty((r.shape[0], comp), dtype=torch.float64, device="cuda")
    mat = h.movedim(-1, 0).reshape(c, -1)  # last axis first
    for lo in range(0, r.shape[0], 2048):
        x = r[lo:lo + 2048]
        ph = [torch.polar(torch.ones((), dtype=torch.float64, device="cuda"), x[:, d, None] * k) for d in range(dim)]
        t = (ph[dim - 1] @ mat).reshape(x.shape[0], comp, *([c] * (dim - 1)))
        for d in range(dim - 2, -1, -1):
            t = (t * ph[d].reshape(x.shape[0], *([1] * (t.dim() - 2)), c)).sum(-1)
        out[lo:lo + 2048] = t.real / float(c) ** dim
    return out


def _coarse_spectrum(uh, dim, n, c):
    """Full spectra (3, c, ..., c) of the real field that the modes [-c/2, c/2 - 1] of uh give."""
    full = torch.fft.fftn(torch.fft.irfftn(uh.to(torch.complex128), s=(n,) * dim, dim=_axes(dim)), dim=_axes(dim))
    idx = torch.fft.fftfreq(c, 1.0 / c, dtype=torch.float64, device="cuda").to(torch.int64) % n
    for d in _axes(dim):
        full = full.index_select(full.dim() + d, idx)
    return torch.fft.fftn(torch.fft.ifftn(full * (float(c) / n) ** dim, dim=_axes(dim)).real, dim=_axes(dim))


def _exact_nufft(case, s):
    dim, n, c = case["dim"], case["n_fine"], case["c"]
    many = case["batch"] > 1
    us, rs = [], []
    for b in range(case["batch"]):
        r = s["r"][b] if many else s["r"]
        u = _spectral_sum(_coarse_spectrum((s["uh"][b] if many else s["uh"])[:dim], dim, n, c), r)
        us.append(u)
        rs.append(torch.remainder(r + RELAX_DT * u, TWO_PI))
    return {"u_r": torch.stack(us) if many else us[0], "r": torch.stack(rs) if many else rs[0]}


def _exact_sph(case, s):
    dim, n = case["dim"], case["n"]
    h = TWO_PI / n
    sigma = 3.0 / (359.0 * math.pi * h**3) if dim == 3 else 7.0 / (478.0 * math.pi * h * h)
    mass, p_ref = h**dim, 100.0 * U_REF * U_REF
    x = torch.remainder(s["r"] + RELAX_DT * s["u"], TWO_PI)
    rho, acc = torch.empty(x.shape[0], dtype=torch.float64, device="cuda"), torch.empty_like(x)

    def pairs(lo):
        d = x[lo:lo + 512, None, :] - x[None, :, :]
        d -= TWO_PI * torch.round(d / TWO_PI)
        dist = torch.sqrt((d * d).sum(-1))
        q = dist / h
        return d, dist, [torch.clamp(a - q, min=0.0) for a in (3.0, 2.0, 1.0)]

    for lo in range(0, x.shape[0], 512):
        _, _, (q3, q2, q1) = pairs(lo)
        rho[lo:lo + 512] = mass * sigma * (q3**5 - 6.0 * q2**5 + 15.0 * q1**5).sum(1)
    p = p_ref * (rho - 1.0)
    for lo in range(0, x.shape[0], 512):
        d, dist, (q3, q2, q1) = pairs(lo)
        ri, pi, rj, pj = rho[lo:lo + 512, None], p[lo:lo + 512, None], rho[None], p[None]
        grad = sigma / h * (-5.0 * q3**4 + 30.0 * q2**4 - 75.0 * q1**4) / (dist + 2.220446049250313e-16)
        f = -mass * (1.0 / ri**2 + 1.0 / rj**2) * ((rj * pi + ri * pj) / (ri + rj) + 0.5 * p_ref) * grad
        acc[lo:lo + 512] = (f[..., None] * d).sum(1)
    moved = torch.remainder(x + (RELAX_FACTOR * RELAX_DT) ** 2 * acc, TWO_PI)
    u = (torch.remainder(moved - s["r"] + math.pi, TWO_PI) - math.pi) / RELAX_DT
    return {"u_r": u, "r": torch.remainder(s["r"] + RELAX_DT * u, TWO_PI)}


def _exact_diag(case, s):
    dim, n = case["dim"], case["n"]
    m = _Flow64(dim, n, _flow_args(case)["nu"], 1.0)
    a, u = s["uh"].to(torch.complex128), s["u"].to(torch.float64)
    shell = torch.floor(torch.sqrt(m.k2) + 0.5).to(torch.int64).reshape(-1)
    w = m.w.expand(m.k2.shape).reshape(-1)
    e = w * (a.real**2 + a.imag**2).sum(0).reshape(-1) / float(n) ** (2 * dim)
    count, total = torch.bincount(shell, w, minlength=n)[:n], torch.bincount(shell, e, minlength=n)[:n]
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    om = m.field(m.curl(a))
    return {"ke": m.energy(a).reshape(1), "eps": (_flow_args(case)["nu"] * (om * om).sum(0).mean()).reshape(1),
            "ek": total * 4.0 * math.pi * k * k / (count + 2.220446049250313e-16),
            "stats": torch.cat([u.abs().flatten(1).amax(1), 0.5 * (u * u).sum(0).mean().reshape(1)])}


def exact(case, seed):
    s, kind = _inputs(case, seed), case["kind"]
    if kind == "step":
        return _exact_flow(case, s["uh"])
    if kind == "step_fn":
        one = _exact_flow(dict(case, batch=1, steps=1, u_out=True), s["uh"])
        return {"u": one["u"], "u_hat": one["u_hat"], "e_inj": None}
    if kind == "nufft":
        return _exact_nufft(case, s)
    if kind == "dft":
        return {"u_r": _spectral_sum(torch.fft.fftn(s["u"].to(torch.float64), dim=_axes(case["dim"])), s["r"])}
    if kind == "sph":
        return _exact_sph(case, s)
    if kind == "grad":
        m = _Flow64(**_flow_args(case))
        x = s["uh"].to(torch.complex128).requires_grad_(True)
        y = x
        for _ in range(case["steps"]):
            y = m.step(y)
        (grad,) = torch.autograd.grad(y, x, s["g"].to(torch.complex128))
        return {"u_hat": y.detach(), "grad": grad}
    return _exact_diag(case, s)
