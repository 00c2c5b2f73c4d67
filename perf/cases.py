"""The work that a user of palinstrophy_gb300 has it do, as measurable cases.

Kinds, each through the package's public entry points:

  run       a stretch of a simulation: Field.step(method, nsteps, update) on a
            field that stays on the GPU, om2 read as a device array
            (run_dns between two of its marks; batch jobs)
  gui       the simulator facade's loop: single steps as dns_step2b, dns_step3,
            dns_step2a, then next_dt and the vorticity frame in host memory
  report    what run_dns and the GUI print and save at a mark: the flow
            diagnostics and the energy-spectrum sample of the current field
  ensemble  many members of several sizes with their own dt, stepped together
            from a CUDA graph, the members' fields read at the end
  adjoint   one value-and-gradient call of PalinstrophyLoss (torch.autograd)

Sizes, methods, CFL numbers and Reynolds numbers are those of the repository's
configurations, tests and benchmark (N = 256 CNAB2, 1024 RK3, 512 adjoint,
256/384/512 ensemble, 4096 and 8192 single fields) and of the grids it
compiles, N = 64 .. 8192 with the radix-3 sizes 384, 768, 1536, 3072 among
them.  Initial fields are random-phase vorticity with the KM3 energy spectrum
(k^4 below K0, k^-3 above), the start of the repository's simulations.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from palinstrophy_gb300.autograd import PalinstrophyLoss
from palinstrophy_gb300.spectrum import compute_energy_spectrum_uv_bins
from palinstrophy_gb300.turbo_simulator import (
    Ensemble,
    Field,
    create_dns_state,
    dns_om2_phys,
    dns_step2a,
    dns_step2b,
    dns_step3,
    next_dt,
)

SIZES = (64, 128, 256, 384, 512, 768, 1024, 1536, 2048, 3072, 4096, 8192)
ENSEMBLE_SIZES = (256, 384, 512)
ADJOINT_SIZES = (64, 128, 256, 512)
ALPHA = (8.0 / 15.0, 5.0 / 12.0, 3.0 / 4.0)
BETA = (0.0, -17.0 / 60.0, -5.0 / 12.0)


def _run(name, N, precision, method, nsteps, update, Re, K0, cfl):
    return {"name": name, "kind": "run", "N": N, "precision": precision, "method": method, "nsteps": nsteps,
            "update": update, "Re": Re, "K0": K0, "cfl": cfl}


def listed():
    return [
        # the smallest call: one time step of a small field, call by call (latency and launches)
        {"name": "calls_n64_fp32", "kind": "gui", "N": 64, "precision": "fp32", "nsteps": 1, "frame": False,
         "Re": 1e3, "K0": 5.0, "cfl": 0.25},
        # the CLI's default kind of run at a small grid, between two diagnostics marks
        _run("run_n256_fp32_cnab2", 256, "fp32", "CNAB2", 40, 20, 1e4, 10.0, 0.25),
        # the GUI at its usual grid: a few steps, then the vorticity frame
        {"name": "gui_n512_fp32", "kind": "gui", "N": 512, "precision": "fp32", "nsteps": 4, "frame": True,
         "Re": 1e4, "K0": 15.0, "cfl": 0.25},
        # an ordinary grid with a radix-3 factor
        _run("run_n1536_fp32_rk3", 1536, "fp32", "LS_IMEX_RK3", 10, 5, 1e4, 15.0, 0.1),
        # the headline configuration
        _run("run_n4096_fp32_rk3", 4096, "fp32", "LS_IMEX_RK3", 4, 100, 1e5, 15.0, 0.1),
        # the largest field
        _run("run_n8192_fp32_rk3", 8192, "fp32", "LS_IMEX_RK3", 2, 100, 1e5, 15.0, 0.1),
        # the plain double-precision form: the small reference configuration, an ordinary grid, the large one
        _run("run_n256_fp64_cnab2", 256, "fp64", "CNAB2", 25, 100, 1e4, 10.0, 0.25),
        _run("run_n1024_fp64_rk3", 1024, "fp64", "LS_IMEX_RK3", 4, 100, 1e4, 15.0, 0.1),
        _run("run_n4096_fp64_rk3", 4096, "fp64", "LS_IMEX_RK3", 1, 100, 1e5, 15.0, 0.1),
        # diagnostics and spectrum sample of a large-ish field at a mark
        {"name": "report_n2048_fp32", "kind": "report", "N": 2048, "precision": "fp32", "Re": 1e5, "K0": 15.0,
         "cfl": 0.1},
        # the 96-member ensemble, dt of every member adapted every step
        {"name": "ensemble_96_fp32", "kind": "ensemble", "N": 512, "precision": "fp32", "members": 32, "sizes": 3,
         "method": "CNAB2", "nsteps": 25, "Re": 1e4, "K0": 10.0, "cfl": 0.5},
        # differentiation: loss and gradient through 20 steps, a checkpoint every 10
        {"name": "adjoint_n512_fp32", "kind": "adjoint", "N": 512, "precision": "fp32", "nsteps": 20, "ckpt": 10,
         "dt": 2e-3, "Re": 5e3, "K0": 12.0},
    ]


def draw(rng):
    kind = rng.choices(("run", "gui", "report", "ensemble", "adjoint"), (62, 8, 10, 10, 10))[0]
    prec = rng.choices(("fp32", "fp64"), (65, 35))[0]
    Re = float(round(10.0 ** rng.uniform(3.0, 5.0)))
    K0 = round(rng.uniform(5.0, 15.0), 2)
    cfl = round(rng.uniform(0.1, 0.25), 3)
    if kind == "run":
        N = rng.choice(SIZES if prec == "fp32" else SIZES[:-1])
        method = rng.choice(("CNAB2", "LS_IMEX_RK3"))
        # from one step to a stretch of about the same length in time as the listed ones
        stages = 1 if method == "CNAB2" else 3
        most = (4096 / N) ** 2 * (12 if prec == "fp32" else 3) / stages
        nsteps = max(1, min(40, int(math.exp(rng.uniform(0.0, math.log(max(1.0, most)))))))
        return _drop_name(_run("", N, prec, method, nsteps, rng.choice((5, 20, 100)), Re, K0, cfl))
    if kind == "gui":
        return {"kind": kind, "N": rng.choice(SIZES[:9]), "precision": prec, "nsteps": rng.randint(1, 8),
                "frame": rng.random() < 0.7, "Re": Re, "K0": K0, "cfl": cfl}
    if kind == "report":
        return {"kind": kind, "N": rng.choice(SIZES[2:-1] if prec == "fp32" else SIZES[2:-2]), "precision": prec, "Re": Re,
                "K0": K0, "cfl": cfl}
    if kind == "ensemble":
        return {"kind": kind, "N": 512, "precision": "fp32", "members": rng.randint(2, 32), "sizes": rng.randint(1, 3),
                "method": rng.choice(("CNAB2", "LS_IMEX_RK3")), "nsteps": rng.randint(5, 25), "Re": Re, "K0": K0,
                "cfl": cfl}
    return {"kind": kind, "N": rng.choice(ADJOINT_SIZES), "precision": prec, "nsteps": rng.randint(5, 20),
            "ckpt": rng.choice((5, 10, 20)), "dt": 1e-3, "Re": max(Re, 2e3), "K0": K0}


def _drop_name(c):
    return {k: v for k, v in c.items() if k != "name"}


# --------------------------------------------------------------------------
# inputs
def _field(N, K0, seed, precision):
    """Random-phase vorticity om2 (N, N/2) with the KM3 energy spectrum, on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + N)
    nh = N // 2
    kx = torch.arange(nh, device="cuda", dtype=torch.float64)[None, :]
    z = torch.arange(N, device="cuda")
    kz = torch.where(z < nh, z, z - N).to(torch.float64)[:, None]
    k2 = kx * kx + kz * kz
    k = torch.sqrt(k2)
    k0 = min(K0, N / 8.0)
    e = torch.where(k < k0, k2 * k2 / k0**7, torch.clamp(k, min=1.0) ** -3)
    # shell energy e(k) over about pi k modes of the half plane; |om|^2 = k^2 |u|^2
    amp = torch.sqrt(e / (math.pi * torch.clamp(k, min=1.0))) * k
    amp = torch.where((k > 0) & (k <= nh), amp, torch.zeros_like(amp))
    jit = 0.75 + 0.5 * torch.rand((N, nh), generator=g, device="cuda", dtype=torch.float64)
    th = 2.0 * math.pi * torch.rand((N, nh), generator=g, device="cuda", dtype=torch.float64)
    om = torch.polar(amp * torch.sqrt(jit), th)
    om[nh] = 0.0
    om[nh + 1:, 0] = torch.conj(torch.flip(om[1:nh, 0], (0,)))  # real field: Hermitian kx = 0 column
    # unit mean square velocity, as the generator's fields have
    w = torch.where(kx == 0, 1.0, 2.0)
    u2 = (w * om.abs() ** 2 / torch.clamp(k2, min=1.0)).sum()
    om = om / torch.sqrt(u2)
    return om.to(torch.complex64 if precision == "fp32" else torch.complex128).contiguous()


def _start(F, om, case):
    """The calls that begin a run: state, viscosity, first transform, dt from the CFL number."""
    torch.cuda.current_stream().synchronize()
    F.set_state_device(om.data_ptr())
    F.set_scalar("visc", 1.0 / case["Re"])
    F.step2a()
    F.set_scalar("dt", case["cfl"] / (F.compute_cflm() * math.pi))
    F.set_scalar("cn", 1.0)
    F.set_scalar("cnm1", 0.0)


def _members(case):
    return [n for n in ENSEMBLE_SIZES[: case["sizes"]] for _ in range(case["members"])]


def prepare(case, seed):
    kind, N = case["kind"], case["N"]
    state = {"case": case}
    if kind in ("run", "report"):
        F = Field(N, case["precision"], case["Re"], case["cfl"])
        _start(F, _field(N, case["K0"], seed, case["precision"]), case)
        state["F"] = F
        state["stream"] = torch.cuda.ExternalStream(F.stream_ptr())
    elif kind == "gui":
        S = create_dns_state(N=N, Re=case["Re"], K0=case["K0"], CFL=case["cfl"], skip_pao=True,
                             precision=case["precision"])
        _start(S.field, _field(N, case["K0"], seed, case["precision"]), case)
        state["S"] = S
        state["stream"] = torch.cuda.ExternalStream(S.field.stream_ptr())
    elif kind == "ensemble":
        ns = _members(case)
        E = Ensemble(ns, case["precision"], case["Re"], case["cfl"])
        for m, n in enumerate(ns):
            E.set_member(m, _field(n, case["K0"], seed * 100 + m, case["precision"]).cpu().numpy())
        E.set_scalar(-1, "visc", 1.0 / case["Re"])
        E.init_dt()
        state["E"], state["ns"] = E, ns
    else:
        state["om0"] = _field(N, case["K0"], seed, case["precision"]).requires_grad_(True)
    return state


# --------------------------------------------------------------------------
# one pass
def _view(F, which, stream):
    """A device array of the field as a tensor, ordered after the field's own stream."""
    t = torch.as_tensor(F.device_array(which), device="cuda")
    torch.cuda.current_stream().wait_stream(stream)
    return t


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        F = state["F"]
        F.step(case["method"], case["nsteps"], update=case["update"])
        return {"om2": _view(F, "om2", state["stream"])}
    if kind == "gui":
        S = state["S"]
        for _ in range(case["nsteps"]):
            dns_step2b(S)
            dns_step3(S)
            dns_step2a(S)
        out = {}
        if case["frame"]:
            next_dt(S)
            dns_om2_phys(S)
            out["frame"] = S.ur_full[2]
        out["om2"] = _view(S.field, "om2", state["stream"])
        return out
    if kind == "report":
        F = state["F"]
        d = F.diagnostics()
        s = compute_energy_spectrum_uv_bins(F)
        # the velocity statistics are as exact as the field's own precision; the spectral sums are FP64
        real = np.float32 if case["precision"] == "fp32" else np.float64
        out = {k: real(d[k]) for k in ("U", "tau_l", "cflm", "energy_joules")}
        out.update({k: d[k] for k in ("E", "L", "Z", "P", "pal_over_ens_kmax2")})
        out["spectrum"], out["count"] = s.energy, s.count
        return out
    if kind == "ensemble":
        E, ns = state["E"], state["ns"]
        E.step(case["method"], case["nsteps"], update=1, graph=True)
        return {str(n): np.stack([E.om2(m) for m in range(len(ns)) if ns[m] == n]) for n in sorted(set(ns))}
    om0 = state["om0"]
    om0.grad = None
    loss = PalinstrophyLoss.apply(om0, case["N"], case["precision"], case["dt"], 1.0 / case["Re"], case["nsteps"],
                                  case["ckpt"])
    loss.backward()
    return {"loss": loss.detach().to(om0.real.dtype), "grad": om0.grad}


# --------------------------------------------------------------------------
# the least work of one pass
def _stage_work(N, cs):
    """Bytes and flops of one stage on an N x N field: om and fnm1 in and out, the four x and z
    transforms of the padded field, products and spectral update."""
    M = 1.5 * N
    lg = math.log2(M)
    flops = 2 * 5 * M * M * lg + (N / 2) * 4 * 5 * M * lg + 4 * M * M + 40 * N * N / 2
    return 4 * (N * N / 2) * cs, flops


def work(case):
    kind, N = case["kind"], case["N"]
    cs = 8 if case["precision"] == "fp32" else 16
    M = 3 * N // 2
    if kind in ("run", "gui"):
        stages = case["nsteps"] * (3 if case.get("method") == "LS_IMEX_RK3" else 1)
        b, f = _stage_work(N, cs)
        b, f = b * stages, f * stages
        if case.get("frame"):
            b += M * M * cs / 2 + N * N / 2 * cs
            f += 5 * M * M * math.log2(M)
        return {"bytes": b, "flops": f}
    if kind == "report":
        return {"bytes": 2 * (N * N / 2) * cs, "flops": 5 * M * M * math.log2(M) + 20 * N * N / 2}
    if kind == "ensemble":
        stages = case["nsteps"] * (3 if case["method"] == "LS_IMEX_RK3" else 1)
        w = [_stage_work(n, cs) for n in _members(case)]
        return {"bytes": stages * sum(x[0] for x in w), "flops": stages * sum(x[1] for x in w)}
    b, f = _stage_work(N, cs)
    # forward, and the reversed stages: the stage's velocity again and the transposed transforms
    return {"bytes": 3 * 2 * case["nsteps"] * b, "flops": 3 * 2.5 * case["nsteps"] * f}


# --------------------------------------------------------------------------
# the same in plain torch, 64 bits
class _Grid:
    def __init__(self, N):
        self.N, self.nh, self.M = N, N // 2, 3 * N // 2
        nh = self.nh
        self.kx = torch.arange(nh, device="cuda", dtype=torch.float64)[None, :]
        z = torch.arange(N, device="cuda")
        self.kz = torch.where(z < nh, z, z - N).to(torch.float64)[:, None]
        self.k2 = self.kx**2 + self.kz**2
        inv = 1.0 / torch.where(self.k2 > 0, self.k2, torch.ones_like(self.k2))
        self.iu, self.iv = -self.kz * inv, self.kx * inv  # u^ = i iu om, v^ = i iv om
        self.iu[0, 0] = 0.0
        self.ga, self.g2 = self.kz * self.kx, self.kz**2 - self.kx**2
        self.ga[nh] = 0.0  # the nonlinear term of the row kz = -N/2 is zero
        self.g2[nh] = 0.0

    def phys(self, band):
        X = torch.zeros((self.M, self.M // 2 + 1), device="cuda", dtype=torch.complex128)
        X[: self.nh, : self.nh] = band[: self.nh]
        X[self.N:, : self.nh] = band[self.nh:]
        return torch.fft.irfft2(X, s=(self.M, self.M), norm="forward")

    def gather(self, spec):
        return torch.cat((spec[: self.nh, : self.nh], spec[self.N:, : self.nh]))

    def velocity(self, om):
        return self.phys(1j * self.iu * om), self.phys(1j * self.iv * om)

    def nonlinear(self, om):
        u, v = self.velocity(om)
        b = self.gather(torch.fft.rfft2(u * v))
        a = self.gather(torch.fft.rfft2(u * u - v * v))
        return (self.ga * a + self.g2 * b) / float(self.M) ** 2

    def cflm(self, om):
        u, v = self.velocity(om)
        return float((u.abs() + v.abs()).max()) * self.N / (2.0 * math.pi)


def _exact_steps(g, om, case, method, nsteps, update, dt=None):
    """om after nsteps steps, NEXTDT after the steps whose number is on the cadence."""
    nu = 1.0 / case["Re"]
    if dt is None:
        dt = case["cfl"] / (g.cflm(om) * math.pi)
    cn, cnm1 = 1.0, 0.0
    f = torch.zeros_like(om)
    for it in range(1, nsteps + 1):
        if method == "CNAB2":
            fn = g.nonlinear(om)
            h = 0.5 * nu * dt
            om = ((1.0 - g.k2 * h) * om + 0.5 * dt * ((2.0 + cnm1) * fn - cnm1 * f)) / (1.0 + g.k2 * h)
            f = fn
            cnm1 = cn
        else:
            for a, b in zip(ALPHA, BETA):
                fn = g.nonlinear(om)
                om = ((1.0 - g.k2 * (b * dt * nu)) * om + a * dt * fn + b * dt * f) / (1.0 + g.k2 * (a * dt * nu))
                f = fn
        if update > 0 and (it % update == 0 or it == 1):
            cn = 0.8 + 0.2 * case["cfl"] / (g.cflm(om) * dt * math.pi)
            dt = dt * cn
    return om


def exact(case, seed):
    kind, N = case["kind"], case["N"]
    if kind == "run":
        om = _field(N, case["K0"], seed, case["precision"]).to(torch.complex128)
        return {"om2": _exact_steps(_Grid(N), om, case, case["method"], case["nsteps"], case["update"])}
    if kind == "gui":
        g = _Grid(N)
        om = _field(N, case["K0"], seed, case["precision"]).to(torch.complex128)
        om = _exact_steps(g, om, case, "CNAB2", case["nsteps"], 0)
        out = {"om2": om}
        if case["frame"]:
            band = om.clone()
            band[N // 2] = 0.0
            out["frame"] = g.phys(band)
        return out
    if kind == "report":
        g = _Grid(N)
        om = _field(N, case["K0"], seed, case["precision"]).to(torch.complex128)
        u, v = g.velocity(om)
        ms = float((u * u + v * v).mean())
        p = om.real**2 + om.imag**2
        w = torch.full((1, N // 2), 2.0, device="cuda", dtype=torch.float64)
        w[0, 0] = w[0, -1] = 1.0
        k2 = torch.where(g.k2 > 0, g.k2, torch.full_like(g.k2, math.inf))
        E = float((w * p / k2).sum())
        L = 2.0 * math.pi * float((w * p / k2**1.5).sum()) / E
        Z = float((w * p).sum() - p[0, 0])
        P = float((w * g.k2 * p).sum())
        nh = N // 2
        nbins, scale = max(32, 2 * N), float(g.M) ** 4
        # in NumPy: a mode on a bin's edge belongs where the correctly rounded quotients put it
        b = np.floor(np.sqrt(g.k2.cpu().numpy()) / (0.5 * N) / math.sqrt(2.0) * nbins)
        bins = torch.from_numpy(np.clip(b, 0, nbins - 1).astype(np.int64)).cuda()
        wt = torch.where(g.kx > 0, 2.0, 1.0) * torch.ones_like(g.k2)
        wt[0, 0] = 0.0
        s = torch.zeros(nbins, device="cuda", dtype=torch.float64)
        s.index_add_(0, bins.flatten(), (wt * p / k2 * scale).flatten())
        U = math.sqrt(ms)
        return {"U": U, "tau_l": L / U, "cflm": float((u.abs() + v.abs()).max()) * N / (2.0 * math.pi),
                "energy_joules": 0.5 * (2.0 * math.pi) ** 2 * ms, "E": E, "L": L, "Z": Z, "P": P,
                "pal_over_ens_kmax2": P / (Z * ((nh - 1.0) ** 2 + float(nh) ** 2)), "spectrum": s, "count": None}
    if kind == "ensemble":
        ns = _members(case)
        grids = {n: _Grid(n) for n in set(ns)}
        got = {n: [] for n in ns}
        for m, n in enumerate(ns):
            om = _field(n, case["K0"], seed * 100 + m, case["precision"]).to(torch.complex128)
            got[n].append(_exact_steps(grids[n], om, case, case["method"], case["nsteps"], 1))
        return {str(n): torch.stack(v) for n, v in got.items()}
    g = _Grid(N)
    om0 = _field(N, case["K0"], seed, case["precision"]).to(torch.complex128).requires_grad_(True)
    om = _exact_steps(g, om0, case, "LS_IMEX_RK3", case["nsteps"], 0, dt=case["dt"])
    w = torch.where(g.kx == 0, 1.0, 2.0)
    loss = 0.5 * (w * g.k2 * (om.real**2 + om.imag**2)).sum()
    loss.backward()
    return {"loss": loss.detach(), "grad": om0.grad}
