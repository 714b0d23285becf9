"""The work that users of this framework time: whole runs through the public
entry points (`SolverFactory` / `Solver`, `BatchSolver`, `adjoint.evolve`).

A case is one run of a simulation: its inputs go in, a number of iterations is
taken, and the final fields come out.

  listed()            the cases by name
  draw(rng)           one more case of the same ranges
  prepare(case, seed) inputs and handles, made from the seed
  run(state)          one run; returns the fields it computes
  work(case)          bytes and operations a run cannot do without
  exact(case, seed)   what run() returns, in 64 bits and plain torch
"""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import phoenix_b200 as pb
from phoenix_b200.adjoint import evolve

# 100 um box, hbar = 0.6582 meV ps, m_eff = 5.6e-4 m_e; units ps / um / meV
BOX = 100.0
PHYS = dict(h_bar_s=0.6582, m_eff=3.1840, gamma_c=0.15, gamma_r=0.225, g_c=6e-6, g_r=1.2e-5, R=0.01)
THRESHOLD = 0.15 * 0.225 / 0.01
TETM = dict(g_pm=-1.2e-6, delta_LT=0.05)
SEED_NOISE = 7


def _case(name, kind, n_c, n_r, dtype, iterations, **more):
    c = dict(name=name, kind=kind, N_c=n_c, N_r=n_r, dtype=dtype, iterations=iterations, periodic_x=True,
             periodic_y=True, potential=True, mask=False, noise=0.0, pulse=False, fma=False)
    c.update(more)
    return c


def listed():
    return [
        # a host program that steps a small grid itself and reads it back
        # (parameter scans on a laptop-sized grid, a live view): launch and
        # call latency; the reference's default zero boundaries and FP64
        _case("iterate_96_f64_host", "host", 96, 72, "f64", 16, periodic_x=False, periodic_y=False, potential=False),
        # the plain polariton run: 256^2 FP64, a pump and nothing else
        _case("rk4_256_f64", "scalar", 256, 256, "f64", 100, potential=False),
        # the benchmark's run: 1024^2 FP32, disorder, k-space mask every 100
        _case("rk4_1024_f32_mask", "scalar", 1024, 1024, "f32", 100, mask=True),
        # the same grid in the default precision
        _case("rk4_1024_f64", "scalar", 1024, 1024, "f64", 50),
        # a sample of its own shape: ragged sides, walls on one axis
        _case("rk4_1310x997_f32_mixed", "scalar", 1310, 997, "f32", 60, periodic_x=False),
        # a large grid with the faster arithmetic switched on
        _case("rk4_4096_f32_fma", "scalar", 4096, 4096, "f32", 8, fma=True),
        # a resonant pulse on a pumped sample: two pump groups, one of them
        # in time, and a complex pulse envelope
        _case("rk4_1024_f32_pulse", "scalar", 1024, 1024, "f32", 24, pulse=True),
        # step-size control
        _case("dp45_1024_f32", "adaptive", 1024, 1024, "f32", 20),
        # the spinor with TE/TM splitting and the stochastic term
        _case("tetm_2048_f32_noise", "tetm", 2048, 2048, "f32", 8, noise=1e-3),
        # split-step Fourier
        _case("ssfm_1024_f32", "ssfm", 1024, 1024, "f32", 16),
        # a pump-power sweep: instances of 128^2 .. 1024^2 advanced together
        _case("batch_24_f32", "batch", 1024, 1024, "f32", 192, instances=24),
        # inverse design: gradients of a density misfit through the run
        _case("adjoint_512_f32", "adjoint", 512, 512, "f32", 200, potential=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "scalar", "scalar", "scalar", "scalar", "pulse", "adaptive", "tetm", "ssfm", "batch",
                       "adjoint"])
    dtype = rng.choice(["f32", "f64"])
    even = lambda n: n + (n & 1)  # noqa: E731  FP32 grids have an even number of columns
    if kind == "host":
        n_c, n_r = _log_int(rng, 32, 160), _log_int(rng, 32, 160)
        return _drawn("host", even(n_c), n_r, dtype, rng.randint(4, 24), periodic_x=rng.random() < 0.5,
                      periodic_y=rng.random() < 0.5, potential=rng.random() < 0.5)
    if kind in ("scalar", "pulse"):
        n_c, n_r = _log_int(rng, 128, 3000), _log_int(rng, 128, 3000)
        if rng.random() < 0.3:
            n_c = n_r = 1 << rng.randint(7, 11)
        if dtype == "f32":
            n_c = even(n_c)
        iterations = max(8, min(200, int(4e7 / (n_c * n_r)) + rng.randint(0, 7)))
        square = n_c == n_r and n_c % 2 == 0
        return _drawn("scalar", n_c, n_r, dtype, iterations, periodic_x=rng.random() < 0.7,
                      periodic_y=rng.random() < 0.7, potential=rng.random() < 0.7, pulse=kind == "pulse",
                      mask=square and kind == "scalar" and rng.random() < 0.5,
                      noise=1e-3 if kind == "scalar" and rng.random() < 0.15 else 0.0,
                      fma=dtype == "f32" and kind == "scalar" and rng.random() < 0.3)
    if kind == "adaptive":
        n_c, n_r = even(_log_int(rng, 128, 1400)), _log_int(rng, 128, 1400)
        periodic = rng.random() < 0.7
        return _drawn("adaptive", n_c, n_r, dtype, rng.randint(8, 20), periodic_x=periodic, periodic_y=periodic,
                      potential=rng.random() < 0.7)
    if kind == "tetm":
        n_c, n_r = even(_log_int(rng, 128, 2200)), _log_int(rng, 128, 2200)
        iterations = max(4, min(60, int(1.5e7 / (n_c * n_r)) + rng.randint(0, 4)))
        return _drawn("tetm", n_c, n_r, dtype, iterations, periodic_x=rng.random() < 0.7,
                      periodic_y=rng.random() < 0.7, noise=1e-3 if rng.random() < 0.5 else 0.0)
    if kind == "ssfm":
        n = 64 * rng.randint(3, 20)
        return _drawn("ssfm", n, n, dtype, rng.randint(8, 24))
    if kind == "batch":
        top = rng.choice([256, 512, 1024])
        return _drawn("batch", top, top, dtype, rng.randint(64, 160), instances=rng.randint(4, 16))
    n = 16 * rng.randint(8, 36)
    return _drawn("adjoint", n, n, dtype, rng.randint(60, 160), potential=rng.random() < 0.5)


def _drawn(*a, **k):
    c = _case("", *a, **k)
    del c["name"]
    return c


# ---------------------------------------------------------------- inputs


def _dt(n):
    """0.02 ps at 1024 columns of 100 um, with dx^2 for other grids, at most 0.04 ps (RK4 stability)."""
    return min(0.04, 0.02 * (1024.0 / n) ** 2)


def _types(dtype):
    return (torch.complex64, torch.float32) if dtype == "f32" else (torch.complex128, torch.float64)


def _gen(seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _axes(n_c, n_r, device):
    x = torch.linspace(-BOX / 2, BOX / 2, n_c, dtype=torch.float64, device=device)
    y = torch.linspace(-BOX / 2, BOX / 2, n_r, dtype=torch.float64, device=device)
    return x[None, :], y[:, None]


def _disorder(n_c, n_r, rms, g):
    """White noise smoothed to 1 um, of the given rms (meV)."""
    w = torch.randn(n_r, n_c, dtype=torch.float64, device=g.device, generator=g)
    kx = 2 * math.pi * torch.fft.fftfreq(n_c, d=BOX / (n_c - 1), dtype=torch.float64, device=g.device)[None, :]
    ky = 2 * math.pi * torch.fft.fftfreq(n_r, d=BOX / (n_r - 1), dtype=torch.float64, device=g.device)[:, None]
    v = torch.fft.ifft2(torch.fft.fft2(w) * torch.exp(-(kx ** 2 + ky ** 2) / 2)).real
    return v * (rms / v.pow(2).mean().sqrt())


def _condensate(n_c, n_r, amplitude, g):
    """A condensate spot with a phase gradient, on white noise of 1e-2."""
    x, y = _axes(n_c, n_r, g.device)
    k = torch.rand(2, dtype=torch.float64, device=g.device, generator=g) - 0.5
    spot = amplitude * torch.exp(-(x ** 2 + y ** 2) / (2 * 12.0 ** 2))
    noise = torch.randn(n_r, n_c, dtype=torch.complex128, device=g.device, generator=g)
    return torch.polar(spot, k[0] * x + k[1] * y) + 1e-2 * noise


def _fields(case, seed):
    """Name -> tensor in the case's precision, every input of the run."""
    g = _gen(seed)
    n_c, n_r = case["N_c"], case["N_r"]
    cdt, rdt = _types(case["dtype"])
    x, y = _axes(n_c, n_r, g.device)
    r2 = x ** 2 + y ** 2
    f = {}
    comps = ("plus", "minus") if case["kind"] == "tetm" else ("plus",)
    ring = torch.exp(-((r2.sqrt() - 20.0) ** 2) / (2 * 3.0 ** 2))
    for comp in comps:
        power = THRESHOLD * (1.2 + 0.6 * torch.rand(1, dtype=torch.float64, device=g.device, generator=g))
        shape = ring if case["kind"] == "tetm" else torch.exp(-r2 / (2 * 10.0 ** 2))
        f["psi_" + comp] = _condensate(n_c, n_r, 4.0, g).to(cdt)
        f["n_" + comp] = (15.0 * torch.exp(-r2 / (2 * 14.0 ** 2))).expand(n_r, n_c).to(rdt).contiguous()
        f["pump_" + comp] = (power * shape).to(rdt).contiguous()
        if case["pulse"]:
            f["pump2_" + comp] = (0.5 * power * ring).to(rdt).contiguous()
            f["pulse_" + comp] = (0.2 * _condensate(n_c, n_r, 1.0, g)).to(cdt)
        if case["potential"]:
            f["potential_" + comp] = _disorder(n_c, n_r, 0.1, g).to(rdt)
    if case["mask"]:
        lx, ly = 2 * x / BOX, 2 * y / BOX
        f["mask"] = torch.exp(-((0.5 * ((lx / 0.8) ** 2 + (ly / 0.8) ** 2)) ** 4)).to(rdt)
    return f


def _instances(case, seed):
    """Sizes and inputs of a batch: powers of two up to the case's size."""
    rng = np.random.default_rng([seed, 11])
    sizes = [s for s in (128, 256, 512, 1024) if s <= case["N_c"]]
    out = []
    for k in range(case["instances"]):
        n = sizes[k % len(sizes)]  # every size as often, so that a batch's work does not depend on the seed
        c = dict(case, N_c=n, N_r=n, kind="scalar")
        f = _fields(c, int(rng.integers(1 << 30)))
        f["pump_plus"] = f["pump_plus"] * float(rng.uniform(0.8, 2.0))
        out.append((c, f))
    return out


#: temporal envelopes of the pulsed cases: the second pump group swells and
#: beats, the pulse is a detuned Gaussian (phoenix's iexp)
PUMP2_T = ("cos", 0.3, 0.6, 4.0)
PULSE_T = ("iexp", 0.25, 0.2, 3.0)


def _system(case, **more):
    t = pb.Temporal
    pumps = [t()] + ([t(*PUMP2_T)] if case["pulse"] else [])
    dt = _dt(max(case["N_c"], case["N_r"]))
    kind = case["kind"]
    p = dict(N_c=case["N_c"], N_r=case["N_r"], L_x=BOX, L_y=BOX, **PHYS, periodic_boundary_x=case["periodic_x"],
             periodic_boundary_y=case["periodic_y"], dtype=case["dtype"], dt=dt, t_max=1e12,
             fft_every=99.5 * dt if case["mask"] else 1e12, pump_temporal=pumps,
             potential_temporal=[t()] if case["potential"] else [], pulse_temporal=[t(*PULSE_T)] if case["pulse"] else [],
             stochastic_amplitude=case["noise"], random_seed=SEED_NOISE, fma=case["fma"])
    if kind == "tetm":
        p.update(TETM, use_twin_mode=True)
    if kind == "adaptive":
        p.update(iterator="DP45", use_adaptive_timestep=True, tolerance=1e-6, dt_min=1e-6, dt_max=0.2)
    if kind == "ssfm":
        p.update(iterator="SSFM")
    p.update(more)
    return pb.SystemParameters(**p)


# ---------------------------------------------------------------- runs


def prepare(case, seed):
    if case["kind"] == "batch":
        inst = _instances(case, seed)
        batch = pb.BatchSolver([_system(c) for c, _ in inst])
        for i, (_, f) in enumerate(inst):
            batch.set_field(i, "psi_plus", f["psi_plus"].cpu().numpy())
            batch.set_field(i, "n_plus", f["n_plus"].cpu().numpy())
            batch.set_field(i, "pump_plus", f["pump_plus"].cpu().numpy())
            if case["potential"]:
                batch.set_field(i, "potential_plus", f["potential_plus"].cpu().numpy())
        return dict(case=case, batch=batch, count=len(inst))
    f = _fields(case, seed)
    system = _system(case)
    solver = pb.SolverFactory.create(system)
    comps = ("plus", "minus") if case["kind"] == "tetm" else ("plus",)
    for comp in comps:
        if case["kind"] == "adjoint":
            break  # evolve() takes them with every call
        solver.set_field_tensor("pump_" + comp, f["pump_" + comp])
        if case["pulse"]:
            solver.set_field_tensor("pump_" + comp, f["pump2_" + comp], 1)
            solver.set_field_tensor("pulse_" + comp, f["pulse_" + comp])
        if case["potential"]:
            solver.set_field_tensor("potential_" + comp, f["potential_" + comp])
    if case["mask"]:
        solver.set_field("fft_mask_plus", f["mask"].cpu().numpy())
    state = dict(case=case, solver=solver, fields=f, comps=comps, dt=system.dt)
    if case["kind"] == "host":
        state["psi"], state["n"] = f["psi_plus"].cpu().numpy(), f["n_plus"].cpu().numpy()
    if case["kind"] == "adjoint":
        g = _gen(seed + 1)
        x, y = _axes(case["N_c"], case["N_r"], g.device)
        state["target"] = _target(x, y).to(_types(case["dtype"])[1])
    return state


def _target(x, y):
    """Seven Gaussian spots of 4 um on a hexagon of 15 um."""
    t = torch.zeros_like(x + y)
    for k in range(7):
        cx = 0.0 if k == 6 else 15.0 * math.cos(k * math.pi / 3)
        cy = 0.0 if k == 6 else 15.0 * math.sin(k * math.pi / 3)
        t = t + 10.0 * torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * 4.0 ** 2))
    return t


def _loss(psi, target):
    return ((psi.real ** 2 + psi.imag ** 2 - target) ** 2).sum() * (BOX / psi.shape[0]) ** 2


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        # a sweep goes on from where it stands
        batch = state["batch"]
        batch.run(case["iterations"])
        return [{name: batch.get_field(i, name) for name in ("psi_plus", "n_plus")} for i in range(state["count"])]
    solver, f = state["solver"], state["fields"]
    if case["kind"] == "adjoint":
        leaves = [f[k].detach().requires_grad_() for k in ("pump_plus", "psi_plus", "n_plus")]
        pot = f["potential_plus"].detach().requires_grad_() if case["potential"] else None
        solver.set_time(0.0, state["dt"])
        psi_T, n_T = evolve(solver, leaves[0], leaves[1], leaves[2], case["iterations"], potential=pot)
        wanted = leaves + ([pot] if pot is not None else [])
        grads = torch.autograd.grad(_loss(psi_T, state["target"]), wanted)
        return dict(zip(("d_pump", "d_psi", "d_n", "d_potential"), grads), psi=psi_T.detach(), n=n_T.detach())
    if case["kind"] == "host":
        solver.set_field("psi_plus", state["psi"])
        solver.set_field("n_plus", state["n"])
        solver.set_time(0.0, state["dt"])
        for _ in range(case["iterations"]):
            solver.iterate()
        return {"psi_plus": solver.get_field("psi_plus"), "n_plus": solver.get_field("n_plus")}
    for comp in state["comps"]:
        solver.set_field_tensor("psi_" + comp, f["psi_" + comp])
        solver.set_field_tensor("n_" + comp, f["n_" + comp])
    if not case["mask"]:  # the filter keeps its own clock; a filtered run's time goes on
        solver.set_time(0.0, state["dt"])
    solver.run(case["iterations"])
    out = {}
    for comp in state["comps"]:
        out["psi_" + comp] = solver.get_field_tensor("psi_" + comp)
        out["n_" + comp] = solver.get_field_tensor("n_" + comp)
    if case["kind"] == "adaptive":
        out["t"] = solver.t
    return out


# ---------------------------------------------------------------- work


def work(case):
    """Operations of the scheme itself (no halo, one per rounded result), and
    every input read and every output written once."""
    if case["kind"] == "batch":
        sizes = [s for s in (128, 256, 512, 1024) if s <= case["N_c"]]
        points = sum(sizes[k % len(sizes)] ** 2 for k in range(case["instances"]))
    else:
        points = case["N_c"] * case["N_r"]
    esz = 4 if case["dtype"] == "f32" else 8
    comps = 2 if case["kind"] == "tetm" else 1
    reals = 6 + 1 + (1 if case["potential"] else 0) + (3 if case["pulse"] else 0)  # psi, n in and out; inputs
    b = points * esz * comps * reals
    # one evaluation of the scalar right-hand side: 45, potential 6, pulse and
    # second pump 12; RK4's sums 12 a stage
    rhs = 45 + (6 if case["potential"] else 0) + (12 if case["pulse"] else 0)
    per = 4 * (rhs + 12)
    if case["kind"] == "adaptive":
        per = 7 * rhs + 22 * 6 + 7 * 9 + 12  # 22 nonzero weights, the updates, the error and norm
    if case["kind"] == "tetm":
        per = 2 * 4 * (rhs + 12 + 26)  # cross terms
    if case["noise"]:
        per += 120 + comps * 4 * 16
    if case["kind"] == "ssfm":
        per = 4 * 5 * math.log2(max(2, points)) + 2 * 40 + 60
    ops = points * case["iterations"] * per
    if case["mask"]:
        ops += (case["iterations"] // 100) * points * (2 * 5 * math.log2(points) + 4)
    if case["kind"] == "adjoint":
        ops = 3.5 * ops  # the run, and its transpose with the stage values it needs
        b = points * esz * (4 + 3 + 4 + (2 if case["potential"] else 0))
    return {"bytes": float(b), "flops": float(ops)}


# ---------------------------------------------------------------- exact

CW = (0.0, 0.5, 0.5, 1.0)
AW = (0.5, 0.5, 1.0)
BW = (1 / 6, 1 / 3, 1 / 3, 1 / 6)
HALO = 8


class _Model:
    """The right-hand side in complex128 on grids padded by `HALO` cells: wrapped
    along periodic axes, zeros that evolve with the rest along the others."""

    def __init__(self, case, f, halo=HALO):
        self.case, self.halo = case, halo
        self.px, self.py = case["periodic_x"], case["periodic_y"]
        p = PHYS
        self.dx, self.dy = BOX / (case["N_c"] - 1), BOX / (case["N_r"] - 1)
        self.dV = self.dx * self.dy
        self.ohb = 1.0 / p["h_bar_s"]
        self.A = self.ohb * (-0.5 * p["h_bar_s"] ** 2 / p["m_eff"])
        self.dt = _dt(max(case["N_c"], case["N_r"]))
        wide = lambda v: v.to(torch.complex128 if v.is_complex() else torch.float64)  # noqa: E731
        self.f = {k: self.pad(wide(v)) for k, v in f.items() if k != "mask"}
        self.mask = f["mask"].double() if "mask" in f else None

    def pad(self, v):
        h = self.halo
        for axis, periodic in ((0, self.py), (1, self.px)):
            if periodic:
                reps = -(-h // v.shape[axis])
                ring = torch.cat([v] * reps, axis) if reps > 1 else v
                n = ring.shape[axis]
                v = torch.cat([ring.narrow(axis, n - h, h), v, ring.narrow(axis, 0, h)], axis)
            else:
                shape = list(v.shape)
                shape[axis] = h
                zero = v.new_zeros(shape)
                v = torch.cat([zero, v, zero], axis)
        return v

    def cut(self, v, ext=0):
        h = self.halo - ext
        return v[h:v.shape[0] - h, h:v.shape[1] - h]

    def amps(self, spec, t, w):
        def at(s):
            kind, t0, sigma, freq = spec
            if kind == "cos":
                return math.exp(-0.5 * ((s - t0) / sigma) ** 2) * (1 + math.cos(freq * (s - t0))) / 2
            a = (s - t0) ** 2 / (2 * sigma ** 2)
            return complex(math.exp(-a) * math.cos(freq * (s - t0)), -math.exp(-a) * math.sin(freq * (s - t0)))

        return at(t) * (1 - w) + at(t + self.dt) * w

    @staticmethod
    def lap_x(v):
        return torch.roll(v, 1, 1) + torch.roll(v, -1, 1) - 2 * v

    @staticmethod
    def lap_y(v):
        return torch.roll(v, 1, 0) + torch.roll(v, -1, 0) - 2 * v

    def rhs(self, y, t, w, noisy):
        """k of {psi_*, n_*}; w: the stage's place between t and t + dt."""
        p, f, out = PHYS, self.f, {}
        comps = ("plus", "minus") if "psi_minus" in y else ("plus",)
        for comp in comps:
            psi, n = y["psi_" + comp], y["n_" + comp]
            norm = psi.real ** 2 + psi.imag ** 2
            lx, ly = self.lap_x(psi) / self.dx ** 2, self.lap_y(psi) / self.dy ** 2
            energy = p["g_c"] * norm + p["g_r"] * n
            if "potential_" + comp in f:
                energy = energy + f["potential_" + comp]
            if noisy:
                energy = energy - p["g_c"] / self.dV
            if len(comps) == 2:
                o = y["psi_minus" if comp == "plus" else "psi_plus"]
                energy = energy + TETM["g_pm"] * (o.real ** 2 + o.imag ** 2)
            k = -1j * (self.A * (lx + ly) + self.ohb * energy * psi) + 0.5 * (p["R"] * n - p["gamma_c"]) * psi
            if len(comps) == 2:
                cross = self.lap_x(o) / self.dx ** 2 - self.lap_y(o) / self.dy ** 2
                down, up = torch.roll(o, -1, 0), torch.roll(o, 1, 0)  # rows + 1 and - 1
                diag = torch.roll(down, -1, 1) + torch.roll(up, 1, 1) - torch.roll(down, 1, 1) - torch.roll(up, -1, 1)
                # the reference's d2/dx2 - d2/dy2 keeps no centre term: the two cancel on square cells only
                cross = cross + 2 * o / self.dx ** 2 - 2 * o / self.dy ** 2
                sign = 1.0 if comp == "plus" else -1.0
                k = k - 1j * self.ohb * TETM["delta_LT"] * (cross + sign * (0.5j / self.dx / self.dy) * diag)
            kn = -(p["gamma_r"] + p["R"] * norm) * n + f["pump_" + comp]
            if self.case["pulse"]:
                kn = kn + f["pump2_" + comp] * self.amps(PUMP2_T, t, w)
                k = k + self.ohb * f["pulse_" + comp] * self.amps(PULSE_T, t, w)
            if noisy:
                kn = kn + p["R"] * n / self.dV
            out["psi_" + comp], out["n_" + comp] = k, kn
        return out

    def rk4(self, y, t, iteration=0):
        dt, p = self.dt, PHYS
        noise = self.case["noise"] > 0
        xi = self.noise(iteration) * (self.case["noise"] * math.sqrt(dt)) if noise else None
        scale = lambda n: torch.sqrt((p["R"] * n + p["gamma_c"]) / (4 * self.dV))  # noqa: E731
        s0 = scale(y["n_plus"]) if noise else None
        cur, acc = y, None
        for s in range(4):
            k = self.rhs(cur, t, CW[s], noise)
            acc = {q: BW[s] * v for q, v in k.items()} if acc is None else {q: acc[q] + BW[s] * v for q, v in k.items()}
            if s < 3:
                cur = {q: y[q] + (dt * AW[s]) * k[q] for q in y}
                if noise:
                    for q in cur:
                        if q.startswith("psi"):
                            cur[q] = cur[q] + AW[s] * xi * s0
        new = {q: y[q] + dt * acc[q] for q in y}
        if noise:
            # the last sum scales the minus component by the new reservoir
            new["psi_plus"] = new["psi_plus"] + xi * s0
            if "psi_minus" in new:
                new["psi_minus"] = new["psi_minus"] + xi * scale(new["n_plus"])
        return new

    def noise(self, iteration):
        """Philox4x32-10 normals of every padded point (periodic images draw their point's)."""
        c, h = self.case, self.halo
        dev = self.f["pump_plus"].device
        rows = torch.arange(-h, c["N_r"] + h, device=dev)
        cols = torch.arange(-h, c["N_c"] + h, device=dev)
        if self.py:
            rows = rows % c["N_r"]
        if self.px:
            cols = cols % c["N_c"]
        m32 = 0xFFFFFFFF
        x0 = ((rows[:, None] + 16) * (c["N_c"] + 32) + cols[None, :] + 16) & m32
        x1 = torch.full_like(x0, iteration & m32)
        x2 = torch.full_like(x0, iteration >> 32)
        x3 = torch.zeros_like(x0)

        def mul(a, v):
            lo, hi = (v & 0xFFFF) * a, (v >> 16) * a  # below 2^48 each
            low = (lo + ((hi & 0xFFFF) << 16)) & m32
            return low, ((lo >> 16) + hi) >> 16

        k0, k1 = SEED_NOISE & m32, SEED_NOISE >> 32
        for _ in range(10):
            l0, h0 = mul(0xD2511F53, x0)
            l1, h1 = mul(0xCD9E8D57, x2)
            x0, x1, x2, x3 = h1 ^ x1 ^ k0, l1, h0 ^ x3 ^ k1, l0
            k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
        u1 = ((x0 >> 8) + 1).double() * 2.0 ** -24
        u2 = (x1 >> 8).double() * 2.0 ** -24
        return torch.polar(torch.sqrt(-2 * torch.log(u1)), 2 * math.pi * u2)

    def filtered(self, psi):
        return torch.fft.ifft2(torch.fft.fft2(psi) * torch.fft.fftshift(self.mask))


def _exact_rk4(case, f):
    m = _Model(case, f)
    y = {q: v for q, v in m.f.items() if q[:2] in ("ps", "n_")}
    t, cached = 0.0, 0.0
    for i in range(case["iterations"]):
        y = m.rk4(y, t, i)
        t += m.dt
        y = {q: m.cut(v) for q, v in y.items()}
        if case["mask"] and t - cached >= 99.5 * m.dt:
            cached = t
            y["psi_plus"] = m.filtered(y["psi_plus"])
        y = {q: m.pad(v) for q, v in y.items()}
    return {q: m.cut(v) for q, v in y.items()}


DP_A = ((1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
        (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
        (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
        (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))
DP_E = (71 / 57600, 0.0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40)


def _exact_adaptive(case, f):
    """Dormand-Prince 5(4) with the reference's norms: sums over the grid padded
    by 7 cells, ring r holding the stages evaluated that far out and ring 7
    the state before the last accepted step."""
    m = _Model(case, f)
    y = {"psi": m.f["psi_plus"], "n": m.f["n_plus"]}
    ab2 = lambda v: v.real ** 2 + v.imag ** 2  # noqa: E731
    both = lambda v: {"psi_plus": v["psi"], "n_plus": v["n"]}  # noqa: E731
    t, dt, ring7 = 0.0, m.dt, 0.0
    for _ in range(case["iterations"]):
        t += dt  # a rejected attempt keeps the increment
        while True:
            ks, stages = [], [y]
            for s in range(7):
                k = m.rhs(both(stages[-1]), t, 0.0, False)
                ks.append({"psi": k["psi_plus"], "n": k["n_plus"]})
                if s < 6:
                    stages.append({q: y[q] + dt * sum(a * kk[q] for a, kk in zip(DP_A[s], ks) if a) for q in y})
            err = nrm = 0.0
            for ring in range(7):  # ring 0: the grid itself
                e = dt * sum(DP_E[j] * ks[j]["psi"] for j in range(7 - ring) if DP_E[j] or j == 0)
                v = stages[6 if ring == 0 else 7 - ring]["psi"]
                for what, arr in (("e", e), ("n", v)):
                    total = ab2(m.cut(arr, ring)).sum() - (ab2(m.cut(arr, ring - 1)).sum() if ring else 0.0)
                    err, nrm = (err + float(total), nrm) if what == "e" else (err, nrm + float(total))
            old7 = float(ab2(m.cut(y["psi"], 7)).sum() - ab2(m.cut(y["psi"], 6)).sum())
            final = abs(err / (nrm + ring7))
            dt = max(1e-6, min(0.2, dt * (1e-6 / 2 / max(final, 1e-300)) ** 0.25))
            if final < 1e-6:
                break
        ring7 = old7
        y = {q: m.pad(m.cut(v)) for q, v in stages[6].items()}
    return {"psi_plus": m.cut(y["psi"]), "n_plus": m.cut(y["n"]), "t": t}


def _exact_ssfm(case, f):
    m = _Model(case, f, halo=0)
    p, pi = PHYS, 3.1415926535
    n = case["N_c"]
    dev = m.f["pump_plus"].device
    j = torch.arange(n, dtype=torch.float64, device=dev)
    k = 2 * pi * torch.where(j <= n // 2, j, j - n) / BOX
    lin = p["h_bar_s"] / 2 / p["m_eff"] * (k[None, :] ** 2 + k[:, None] ** 2)
    step = torch.polar(torch.ones_like(lin), -lin * m.dt / 2)
    psi, res = m.f["psi_plus"], m.f["n_plus"]
    for _ in range(case["iterations"]):
        psi = torch.fft.ifft2(torch.fft.fft2(psi) * step)
        norm = psi.real ** 2 + psi.imag ** 2
        h = torch.complex(p["g_c"] * norm + p["g_r"] * res, 0.5 * p["h_bar_s"] * (p["R"] * res - p["gamma_c"]))
        if "potential_plus" in m.f:
            h = h + m.f["potential_plus"]
        new = res + m.dt * (m.f["pump_plus"] - p["gamma_r"] * res - p["R"] * norm * res)
        psi = torch.fft.ifft2(torch.fft.fft2(psi * torch.exp(-1j * m.ohb * h * m.dt)) * step)
        res = new
    return {"psi_plus": psi, "n_plus": res}


def _exact_adjoint(case, f):
    with torch.enable_grad():
        leaf = {q: v.to(torch.complex128 if v.is_complex() else torch.float64).requires_grad_() for q, v in f.items()}
        m = _Model(case, leaf, halo=0)  # periodic: rolls wrap by themselves

        def one(psi, n, pump, pot):
            m.f["pump_plus"] = pump
            if pot is not None:
                m.f["potential_plus"] = pot
            y = m.rk4({"psi_plus": psi, "n_plus": n}, 0.0)
            return y["psi_plus"], y["n_plus"]

        psi, n, pot = leaf["psi_plus"], leaf["n_plus"], leaf.get("potential_plus")
        for _ in range(case["iterations"]):
            psi, n = checkpoint(one, psi, n, leaf["pump_plus"], pot, use_reentrant=False)
        x, y = _axes(case["N_c"], case["N_r"], psi.device)
        target = _target(x, y).to(_types(case["dtype"])[1]).double()
        wanted = [leaf[q] for q in ("pump_plus", "psi_plus", "n_plus")] + ([pot] if pot is not None else [])
        grads = torch.autograd.grad(_loss(psi, target), wanted)
    return dict(zip(("d_pump", "d_psi", "d_n", "d_potential"), grads), psi=psi.detach(), n=n.detach())


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "batch":
            return [_exact_rk4(c, f) for c, f in _instances(case, seed)]
        f = _fields(case, seed)
        if case["kind"] == "adaptive":
            return _exact_adaptive(case, f)
        if case["kind"] == "ssfm":
            return _exact_ssfm(case, f)
        if case["kind"] == "adjoint":
            return _exact_adjoint(case, f)
        return _exact_rk4(case, f)
