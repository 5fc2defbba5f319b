"""The work this engine is measured on: calls of its public entry points over the sizes and options its users run.

A case is a dict of plain values.  `kind` names the call:
  track     window driver: init_particles + run_windows(persistent), snapshot blocks in a device buffer
  loop      the reference's own interface: init_particles, then run_simulation(next_t) + output_data per window
  sweep     as track, with many parameter sets in one context
  adjoint   init_particles + adjoint_record + adjoint_backward, gradients per particle
  grid      torch autograd through track_spins (a grid of parameter sets, dressing pulse gradients)
  analysis  ensemble statistics, unwrapped phases and spins of the current state
  spectrum  integratorType 6: noise-spectrum aggregators and the covariance spectrum

The physics follows the repository's configurations: a 0.07 x 0.1 x 0.4 m box, B0 = 3 uT along x, E along z, gradients
of order 1e-9 T/m, Maxwell-Boltzmann speeds at 4.2 K (gas off) or 0.4 K (gas on), DOP853 at rtol 1e-12.  The seed sets
the particles' random numbers and the field gradients, so another seed is another ensemble in another field.
"""
from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "spin-tracking_gb300"))

GAMMA, MASS = -2.038e8, 1.20239e-26
BOX = (0.07, 0.1, 0.4)
C2 = 299792458.0 ** 2
GRAVITY = -9.81
W_PULSE = 2 * math.pi * 1000.0
# step attempts per particle-second and trajectory segments per particle-second, for work(): at 3 uT and rtol 1e-12
STEPS_PER_S, WALLS_PER_S, GAS_PER_S = 4630.0, 1480.0, 4700.0
FLOPS = {0: 785, 1: 318, 2: 1191, 3: 497, 4: 318, 5: 361}
# (rtol, simulated seconds of one window, attempts per particle-second) of the other steppers
FAMILY = {1: (1e-12, 5e-5, 2e7), 3: (1e-10, 0.0125, 2e4), 4: (1e-3, 0.005, 3.3e5), 5: (1e-6, 2.5e-4, 1e7)}


def listed():
    return [
        # the smallest call: a quick look at a few particles through the reference's run-one-window interface
        {"name": "small_loop", "kind": "loop", "n": 100, "tf": 0.05, "windows": 2, "dist": "M", "gas": True,
         "diffuse": 0.3, "gravity": True},
        # the reference's validation run: 1,000 particles between specular walls, a snapshot every 50 ms
        {"name": "validation_1000", "kind": "track", "n": 1000, "tf": 0.5, "windows": 10, "dist": "M", "gas": False,
         "diffuse": 0.0, "gravity": True, "integrator": 0, "pulse": False},
        # an ordinary production run of odd size with the reference's default walls and gas, uniform speeds
        {"name": "gas_24571", "kind": "track", "n": 24571, "tf": 0.1, "windows": 2, "dist": "C", "gas": True,
         "diffuse": 0.3, "gravity": True, "integrator": 0, "pulse": False},
        # the headline ensemble: 2^20 particles, cosine-law walls, no gas
        {"name": "ensemble_1M", "kind": "track", "n": 1048576, "tf": 0.1, "windows": 2, "dist": "M", "gas": False,
         "diffuse": 0.1, "gravity": True, "integrator": 0, "pulse": False},
        # spin dressing: 1 kHz pulse, gas, diffuse walls, hmax 1e-4
        {"name": "dressing_65536", "kind": "track", "n": 65536, "tf": 0.05, "windows": 1, "dist": "M", "gas": True,
         "diffuse": 0.5, "gravity": True, "integrator": 0, "pulse": True},
        # the Magnus stepper on the headline physics
        {"name": "magnus_65536", "kind": "track", "n": 65536, "tf": 0.1, "windows": 1, "dist": "M", "gas": False,
         "diffuse": 0.1, "gravity": True, "integrator": 2, "pulse": False},
        # a parameter sweep: fields, walls, run lengths and steppers (DOP853, RK45) differ from set to set
        {"name": "sweep_256x37", "kind": "sweep", "sets": 256, "n": 37, "tf": 0.05, "family": False},
        # the remaining steppers side by side (RK45, RK45 with quaternions, RKF45, RKF45 with quaternions)
        {"name": "steppers_4x4096", "kind": "sweep", "sets": 4, "n": 4096, "tf": 0.0, "family": True},
        # sensitivity of an ensemble: forward with tape, then the gradient of every particle
        {"name": "adjoint_32768", "kind": "adjoint", "n": 32768, "tf": 0.1, "windows": 2, "integrator": 0},
        # an optimiser's step over a small dressing grid (amplitude x frequency) through torch autograd
        {"name": "grid_4x4x24", "kind": "grid", "side": 4, "n": 24, "tf": 0.02},
        # the analysis of one snapshot of a large ensemble
        {"name": "analysis_524288", "kind": "analysis", "n": 524288, "tf": 0.004},
        # the noise spectrum seen by an ensemble
        {"name": "spectrum_4099", "kind": "spectrum", "n": 4099, "tf": 0.02, "windows": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["track", "track", "track", "loop", "sweep", "adjoint", "grid", "analysis", "spectrum"])
    tf = round(rng.uniform(0.02, 0.1), 4)
    if kind == "track":
        gas = rng.random() < 0.5
        pulse = rng.random() < 0.25
        return {"kind": kind, "n": _log_int(rng, 100, 65536 if gas or pulse else 524288), "tf": tf,
                "windows": rng.randint(1, 4), "dist": rng.choice("MMC"), "gas": gas,
                "diffuse": round(rng.choice([0.0, rng.uniform(0.02, 0.6)]), 3), "gravity": rng.random() < 0.85,
                "integrator": rng.choice([0, 0, 0, 2]), "pulse": pulse}
    if kind == "loop":
        return {"kind": kind, "n": _log_int(rng, 32, 20000), "tf": tf, "windows": rng.randint(1, 4),
                "dist": rng.choice("MC"), "gas": rng.random() < 0.5, "diffuse": round(rng.uniform(0.0, 0.5), 3),
                "gravity": rng.random() < 0.85}
    if kind == "sweep":
        if rng.random() < 0.3:
            return {"kind": kind, "sets": 4, "n": _log_int(rng, 64, 4096), "tf": 0.0, "family": True}
        return {"kind": kind, "sets": _log_int(rng, 4, 256), "n": rng.randint(8, 64), "tf": round(tf / 2, 4),
                "family": False}
    if kind == "adjoint":
        return {"kind": kind, "n": _log_int(rng, 200, 32768), "tf": tf, "windows": rng.randint(1, 4),
                "integrator": rng.choice([0, 0, 2])}
    if kind == "grid":
        return {"kind": kind, "side": rng.randint(2, 4), "n": rng.randint(5, 24), "tf": round(rng.uniform(0.005, 0.02), 4)}
    if kind == "analysis":
        return {"kind": kind, "n": _log_int(rng, 500, 524288), "tf": round(rng.uniform(0.002, 0.004), 4)}
    return {"kind": "spectrum", "n": _log_int(rng, 100, 4099), "tf": round(rng.uniform(0.004, 0.02), 4),
            "windows": rng.randint(1, 2)}


# ------------------------------------------------------------------ options
def _fields(case, seed):
    """The options of a one-set case as plain values."""
    g = np.random.default_rng(seed).normal(0.0, 1e-9, 9)
    gas, pulse = bool(case.get("gas", False)), bool(case.get("pulse", False))
    return dict(numParticles=case["n"], dist=case.get("dist", "M"), T=0.4 if gas else 4.2, m=MASS, gamma=GAMMA, V=5.0,
                diffuse=float(case.get("diffuse", 0.0)), gas_coll=gas, gravity=bool(case.get("gravity", True)), L=BOX,
                B0=(3e-6, 0.0, 0.0), E=(0.0, 0.0, 75e5), yi=(0.0, 0.0, 1.0), Gx=tuple(g[0:3]), Gy=tuple(g[3:6]),
                Gz=tuple(g[6:9]), t0=0.0, tf=case["tf"], ioutInt=case["tf"] / case.get("windows", 1), rtol=1e-12,
                atol=1e-12, h=1e-3, hmax=1e-4 if pulse else 1.0, hmin=1e-8, integratorType=case.get("integrator", 0),
                seed=int(seed) & 0x7FFFFFFF, maxPosStep=0.1, a=5e-6 if pulse else 0.0, w=W_PULSE if pulse else 0.0)


def _field_sets(case, seed):
    kind = case["kind"]
    if kind == "sweep" and case["family"]:
        sets = []
        for k, (it, (rtol, tf, _)) in enumerate(FAMILY.items()):
            f = _fields(dict(case, tf=tf, diffuse=0.1), seed + k)
            sets.append(dict(f, integratorType=it, rtol=rtol))
        return sets
    if kind == "sweep":
        r = np.random.default_rng(seed)
        sets = []
        for s in range(case["sets"]):
            dop = s < case["sets"] // 2
            tf = case["tf"] * r.uniform(0.2, 1.0) if dop else r.uniform(1e-5, 5e-5)
            f = _fields(dict(case, tf=tf, gas=True, diffuse=r.uniform(0.0, 0.5)), seed + s * case["n"])
            g = r.uniform(0.0, 1e-8, 9)
            f.update(B0=(r.uniform(1e-6, 1e-5), 0.0, 0.0), E=(0.0, 0.0, 75e5 if r.uniform() < 0.5 else -75e5),
                     Gx=tuple(g[0:3]), Gy=tuple(g[3:6]), Gz=tuple(g[6:9]), integratorType=0 if dop else 1)
            sets.append(f)
        return sets
    if kind == "grid":
        f = _fields(dict(case, gas=True, diffuse=0.5, pulse=True), seed)
        return [dict(f, a=float(a), w=float(w), seed=f["seed"] + 1000 * k) for k, (a, w) in enumerate(
            (a, w) for a in np.linspace(1e-6, 1e-5, case["side"])
            for w in 2 * np.pi * np.linspace(500.0, 2000.0, case["side"]))]
    if kind == "analysis":
        return [_fields(dict(case, diffuse=0.1), seed)]
    if kind == "spectrum":
        return [dict(_fields(dict(case, dist="C", gas=True, diffuse=0.3), seed), h=1e-5, integratorType=6, a=5e-6,
                     w=W_PULSE)]
    return [_fields(case, seed)]


def prepare(case, seed):
    import spintrack as st
    from spintrack import adjoint
    opts = [st.derive(st.make_options(**f)) for f in _field_sets(case, seed)]
    p = st.Particles(opts)
    nw = max(st.num_windows(o) for o in opts)
    s = {"kind": case["kind"], "p": p, "opts": opts, "nw": nw, "n": p.n}
    dev = torch.device("cuda", 0)
    if case["kind"] in ("track", "sweep"):
        # several windows' snapshot blocks in one device buffer, and a view of every field over the windows
        blk = p.snapshot_bytes()
        buf = torch.zeros(blk * nw, dtype=torch.uint8, device=dev)
        s["buf"], s["fields"] = buf, {}
        offs = dict(zip(st.SNAP_FIELDS, p.snapshot_offsets()))
        for name in ("t", "fail", "n_coll", "n_bounce", "n_steps", "turns", "pos", "v", "S"):
            dt = torch.int32 if name in ("fail", "turns") else torch.int64 if name.startswith("n_") else torch.float64
            w = torch.empty(0, dtype=dt).element_size()
            if name in offs:
                s["fields"][name] = buf.view(dt).as_strided((nw, p.n), (blk // w, 1), offs[name] // w)
            else:  # a vector: its three component arrays follow one another
                x, y = offs[name + "_x"], offs[name + "_y"]
                s["fields"][name] = buf.view(dt).as_strided((nw, 3, p.n), (blk // w, (y - x) // w, 1), x // w)
    elif case["kind"] == "adjoint":
        g = torch.Generator(device="cpu").manual_seed(int(seed))
        s["w"] = torch.randn(p.n, 3, dtype=torch.float64, generator=g).to(dev) / p.n
        s["S"] = torch.empty(p.n, 3, dtype=torch.float64, device=dev)
        s["grad"] = torch.empty(p.n, adjoint.NUM_THETA, dtype=torch.float64, device=dev)
        s["tape"] = int(p.n * case["tf"] * 400e3 + p.n * 3e4 + 2 ** 26)
    elif case["kind"] == "grid":
        s["theta"] = torch.tensor([adjoint.theta_of(o) for o in opts], dtype=torch.float64, device=dev)
        s["track"] = adjoint.track_spins
    elif case["kind"] == "analysis":
        p.init_particles()
        p.run_windows(0, nw)
        s["phase"] = torch.empty(p.n, dtype=torch.float64, device=dev)
        s["S"] = torch.empty(p.n, 3, dtype=torch.float64, device=dev)
    torch.cuda.synchronize()
    return s


def _counts(d):
    return {k: (v.view(np.int64) if v.dtype == np.uint64 else v) for k, v in d.items()}


def run(s):
    p, kind = s["p"], s["kind"]
    if kind in ("track", "sweep"):
        p.init_particles()
        p.run_windows(0, s["nw"], snap_ptr=s["buf"].data_ptr())
        return s["fields"]
    if kind == "loop":
        p.init_particles()
        out = []
        for w in range(s["nw"]):
            p.run_simulation((w + 1.0) * s["opts"][0].ioutInt)
            out.append(_counts(p.output_data()))
        return out
    if kind == "adjoint":
        p.init_particles()
        p.adjoint_record(s["nw"], tape_bytes=s["tape"])
        p.gather_spins(s["S"].data_ptr())
        p.adjoint_backward(s["w"].data_ptr(), s["grad"].data_ptr())
        return {"S": s["S"], "grad": s["grad"]}
    if kind == "grid":
        theta = s["theta"].detach().requires_grad_(True)
        S = s["track"](theta, p, s["opts"], s["nw"], pulse=True)
        pol = S.reshape(len(s["opts"]), -1, 3).mean(1).norm(dim=1)
        pol.sum().backward()
        return {"S": S.detach(), "grad": theta.grad}
    if kind == "analysis":
        e = p.ensemble()
        p.gather_phase(s["phase"].data_ptr())
        p.gather_spins(s["S"].data_ptr())
        return {"stats": dict(e, mean_S=np.array(e["mean_S"])), "phase": s["phase"], "S": s["S"]}
    p.init_particles()
    p.run_windows(0, s["nw"])
    cov, ns = p.covariance_spectrum()
    return {"state": _counts(p.output_data()), "agg": p.spectrum_state(), "cov": cov, "samples": ns}


def work(case):
    kind, n = case["kind"], case["n"]
    state = 300.0  # bytes of a particle's state and one snapshot
    if kind == "analysis":
        return {"bytes": n * (8 * 4 + 8 + 8 * 4 + 24.0), "flops": n * 150.0}
    if kind == "sweep" and case["family"]:
        fl = sum(n * tf * (rate * FLOPS[it] + WALLS_PER_S * 150) for it, (_, tf, rate) in FAMILY.items())
        return {"bytes": 4 * n * state, "flops": fl}
    segs = WALLS_PER_S + (GAS_PER_S if case.get("gas") or kind in ("sweep", "grid", "spectrum") else 0.0)
    if kind == "sweep":
        half = case["sets"] / 2 * n
        return {"bytes": 2 * half * state,
                "flops": half * (0.6 * case["tf"] * (1.5 * STEPS_PER_S * 785 + segs * 150) + 3e-5 * 2e7 * 318)}
    if kind == "spectrum":
        return {"bytes": n * (state + 17 * 9 * 8.0), "flops": n * case["tf"] * (1e5 * 17 * 21 + segs * 150)}
    steps = (27400.0 if case.get("pulse") or kind == "grid" else max(STEPS_PER_S, segs)) * case["tf"]
    if kind == "grid":
        n *= case["side"] ** 2
    per = steps * FLOPS[case.get("integrator", 0)] + segs * case["tf"] * 150
    tape = 40.0 * steps + 64.0 * segs * case["tf"]
    if kind in ("adjoint", "grid"):
        return {"bytes": n * (state + 17 * 8 + 2 * tape), "flops": n * (per + 1.5 * per)}
    return {"bytes": n * state * case.get("windows", 1), "flops": n * per}


# ------------------------------------------------------------------ exact values, in plain torch
# The ensemble followed again in float64 without the engine: the reference's random numbers and event rules, and each
# segment's spin rotation by a sixth-order Magnus step (three Gauss nodes) short enough to be exact to rounding.
MASK53 = (1 << 53) - 1


def _shr(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


class _Rng:
    def __init__(self, seed, dev):
        def word(v):  # a 64-bit constant as torch's signed integer
            return v - (1 << 64) if v >= 1 << 63 else v
        s = seed.to(dev) & 0xFFFFFFFF
        outs = []
        for _ in range(2):
            s = s + word(0x9E3779B97F4A7C15)
            z = s
            z = (z ^ _shr(z, 30)) * word(0xBF58476D1CE4E5B9)
            z = (z ^ _shr(z, 27)) * word(0x94D049BB133111EB)
            outs.append(z ^ _shr(z, 31))
        self.x, self.y = outs[0] & 0xFFFFFFFF, _shr(outs[0], 32)
        self.z, self.w = outs[1] & 0xFFFFFFFF, _shr(outs[1], 32)
        self.spare = torch.zeros(len(s), dtype=torch.float64, device=dev)
        self.has = torch.zeros(len(s), dtype=torch.bool, device=dev)
        every = torch.ones_like(self.has)
        for _ in range(3):
            self.next(every)

    def next(self, m):
        out = self.x + self.z
        t = self.y << 17
        z = self.z ^ self.x
        w = self.w ^ self.y
        y = self.y ^ z
        x = self.x ^ w
        z = z ^ t
        w = (z << 45) | _shr(z, 19)
        self.x, self.y = torch.where(m, x, self.x), torch.where(m, y, self.y)
        self.z, self.w = torch.where(m, z, self.z), torch.where(m, w, self.w)
        return out

    def uniform(self, m):
        return _shr(self.next(m), 11).to(torch.float64) * 2.0 ** -53

    def exponential(self, m, tc):
        return -tc * torch.log(1.0 - self.uniform(m))

    def normal(self, m):
        cached = m & self.has
        value = torch.where(cached, self.spare, torch.zeros_like(self.spare))
        self.has = self.has & ~cached
        todo = m & ~cached
        while bool(todo.any()):
            u = self.uniform(todo) * 2.0 - 1.0
            v = self.uniform(todo) * 2.0 - 1.0
            s = u * u + v * v
            ok = todo & (s < 1.0) & (s != 0.0)
            f = torch.sqrt(-2.0 * torch.log(torch.where(ok, s, torch.full_like(s, 0.5))) / torch.where(ok, s, torch.ones_like(s)))
            value = torch.where(ok, u * f, value)
            self.spare = torch.where(ok, v * f, self.spare)
            self.has = self.has | ok
            todo = todo & ~ok
        return value


def _paths(f, dev):
    """Segments (t0, t1, p0, v0) of every particle, window by window, and the position and velocity at window ends."""
    n = f["numParticles"]
    kb = 1.380649e-23
    tc = 1.6e-4 * f["m"] / (kb * f["T"] ** 8)
    sd = math.sqrt(kb * f["T"] / f["m"])
    every = torch.ones(n, dtype=torch.bool, device=dev)
    r = _Rng(torch.arange(n, dtype=torch.int64) + f["seed"], dev)
    L = f["L"]
    p = torch.stack([r.uniform(every) * L[k] - L[k] / 2.0 for k in range(3)], 1)
    gas_at = r.exponential(every, tc) if f["gas_coll"] else torch.full((n,), math.inf, dtype=torch.float64, device=dev)

    def velocity(m, speed):
        d = torch.stack([r.normal(m) for _ in range(3)], 1)
        return d * sd if f["dist"] == "M" else d * speed[:, None] / d.square().sum(1).sqrt()[:, None]
    t = torch.zeros(n, dtype=torch.float64, device=dev)
    v = velocity(every, torch.full_like(t, f["V"]))
    half = torch.tensor(L, dtype=torch.float64, device=dev) / 2.0
    G = GRAVITY if f["gravity"] else 0.0
    windows = []
    for w in range(int(math.floor(f["tf"] / f["ioutInt"]))):
        tw = (w + 1.0) * f["ioutInt"]
        segs, live = [], every.clone()
        while bool(live.any()):
            wall_t = (torch.where(v < 0.0, -half, half) - p) / v
            if G:
                y, vy = p[:, 1], v[:, 1]
                arg = torch.where(vy <= 0.0, -2.0 * G * (y + half[1]) + vy * vy, vy * vy - 2.0 * G * (y - half[1]))
                sq = torch.sqrt(arg)
                ty = torch.minimum(((sq + vy) / G).abs(), ((sq - vy) / G).abs())
                t1 = -vy / G
                apex = y + vy * t1 + 0.5 * G * t1 * t1
                fall = t1 + torch.sqrt((-half[1] - apex) * 2.0 / G)
                under = (vy > 0.0) & (-0.5 * vy * vy / G + y < half[1])
                wall_t[:, 1] = torch.where(under, fall, ty)
            bad = (wall_t < 1e-16) | wall_t.isnan()
            first = bad.cumsum(1) == 1
            wall_t = torch.where(bad & first, torch.full_like(wall_t, 1e6), wall_t)
            tb, axis = wall_t.min(1)
            to_gas = gas_at - t
            gas = to_gas < tb
            to = torch.where(gas, to_gas, tb)
            left = tw - t
            end = left <= f["maxPosStep"]
            free = torch.where(end, left, torch.full_like(left, f["maxPosStep"]))
            hit = live & (to <= free)
            dt = torch.where(live, torch.where(hit, to, free), torch.zeros_like(t))
            gas = gas & hit
            wall = hit & ~gas
            if f["gas_coll"] and bool(gas.any()):
                gas_at = torch.where(gas, gas_at + r.exponential(gas, tc), gas_at)
            segs.append((t, t + dt, p, v))
            t = t + dt
            acc = torch.tensor([0.0, G, 0.0], dtype=torch.float64, device=dev)
            p = p + v * dt[:, None] + 0.5 * acc * dt[:, None] * dt[:, None]
            v = v + acc * dt[:, None]
            speed = v.square().sum(1).sqrt()
            on = torch.nn.functional.one_hot(axis, 3).bool() & wall[:, None]
            p = torch.where(on, torch.where(p < 0.0, -half, half), p)
            if f["diffuse"] > 1.2e-38:
                rough = wall & (r.uniform(wall) < f["diffuse"])
            else:
                rough = torch.zeros_like(wall)
            su = torch.sqrt(r.uniform(rough))
            th = r.uniform(rough) * 2.0 * 3.141592653589793
            phi = torch.acos(su)
            sp, cp = torch.sin(phi), torch.cos(phi)
            a, b = speed * sp * torch.cos(th), speed * sp * torch.sin(th)
            back = -torch.where(v < 0.0, -1.0, 1.0) * (speed * cp)[:, None]
            zero = torch.zeros_like(a)
            side = torch.where((axis == 0)[:, None], torch.stack([zero, -a, b], 1),
                               torch.where((axis == 1)[:, None], torch.stack([a, zero, b], 1),
                                           torch.stack([a, b, zero], 1)))
            v = torch.where(rough[:, None], torch.where(on, back, side), torch.where(on, -v, v))
            if f["gas_coll"] and bool(gas.any()):
                v = torch.where(gas[:, None], velocity(gas, speed), v)
            live = live & ~(end & (~hit | (to == free)))
        windows.append((segs, p, v))
    return windows


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


def _spins(f, windows, S, theta=None):
    """Spins at the window ends; theta: per-particle [n, 17] field parameters (with gradients), default those of f."""
    dev = S.device
    if theta is None:
        row = [*f["Gx"], *f["Gy"], *f["Gz"], *f["B0"], *f["E"], f["a"], f["w"]]
        theta = torch.tensor(row, dtype=torch.float64, device=dev).expand(len(S), 17)
    Gt, B0, E = theta[:, :9].reshape(-1, 3, 3), theta[:, 9:12], theta[:, 12:15]
    a, w = theta[:, 15], theta[:, 16]
    pulse = bool((a != 0).any())
    acc = torch.tensor([0.0, GRAVITY if f["gravity"] else 0.0, 0.0], dtype=torch.float64, device=dev)
    sub = 5e-6 if pulse else 0.5 / (abs(f["gamma"]) * float(B0.detach().abs().max()))
    ends = []
    for segs, _, _ in windows:
        t0, t1 = torch.stack([s[0] for s in segs]), torch.stack([s[1] for s in segs])
        p0, v0 = torch.stack([s[2] for s in segs]), torch.stack([s[3] for s in segs])
        cnt = torch.ceil((t1 - t0) / sub).to(torch.int64)
        ends_at = cnt.cumsum(0)
        total = int(ends_at[-1].max())
        col = torch.arange(t0.shape[1], device=dev)
        upto = ends_at.t().contiguous()
        for k in range(total):
            e = torch.searchsorted(upto, torch.full((upto.shape[0], 1), k, device=dev, dtype=torch.int64),
                                   right=True)[:, 0]
            live = e < len(segs)
            e = e.clamp(max=len(segs) - 1)
            c = cnt[e, col].clamp(min=1)
            j = k - (ends_at[e, col] - cnt[e, col])
            h = torch.where(live, (t1[e, col] - t0[e, col]) / c, torch.zeros_like(t0[0]))
            start = j * h
            q, u, at = p0[e, col], v0[e, col], t0[e, col]
            om = []
            for node in (0.5 - math.sqrt(15) / 10, 0.5, 0.5 + math.sqrt(15) / 10):
                tau = (start + node * h)[:, None]
                pos = q + u * tau + 0.5 * acc * tau * tau
                vel = u + acc * tau
                B = B0 + _cross(vel, E.expand_as(vel)) / C2 + (Gt * pos[:, None, :]).sum(2)
                if pulse:
                    z = torch.zeros_like(a)
                    B = B + torch.stack([z, z, a * torch.cos(w * (at + tau[:, 0]))], 1)
                om.append(f["gamma"] * B)
            hh = h[:, None]
            a1, a2 = hh * om[1], math.sqrt(15) / 3 * hh * (om[2] - om[0])
            a3 = 10.0 / 3 * hh * (om[2] - 2 * om[1] + om[0])
            c1 = -_cross(a1, a2)
            c2 = _cross(a1, 2 * a3 + c1) / 60
            x = a1 + a3 / 12 - _cross(-20 * a1 - a3 + c1, a2 + c2) / 240
            x2 = x.square().sum(1, keepdim=True)
            r = torch.sqrt(x2 + 1e-300)
            sinc = torch.where(r < 1e-3, 1 - x2 / 6 * (1 - x2 / 20), torch.sin(r) / r)
            cosc = torch.where(r < 1e-3, 0.5 - x2 / 24 * (1 - x2 / 30), 2 * (torch.sin(r / 2) / r) ** 2)
            y = _cross(S, x)
            S = S + sinc * y + cosc * _cross(y, x)
        ends.append(S)
    return ends


def exact(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")
    fs = _field_sets(case, seed)
    if kind in ("spectrum", "sweep") or (case.get("pulse") and case["n"] * case["tf"] > 4000):
        return None
    steps = case["tf"] * 200000 if kind == "grid" or case.get("pulse") else case["tf"] * (
        WALLS_PER_S + (GAS_PER_S if case.get("gas") else 0.0))
    if steps * case["n"] * (case["side"] ** 2 if kind == "grid" else 1) > 2.5e8 or steps > 2.5e4:
        return None
    grad = kind in ("adjoint", "grid")
    S_all, P_all, V_all, th_all = [], [], [], []
    for f in fs:
        wins = _paths(f, dev)
        row = [*f["Gx"], *f["Gy"], *f["Gz"], *f["B0"], *f["E"], f["a"], f["w"]]
        th = torch.tensor(row, dtype=torch.float64, device=dev).expand(f["numParticles"], 17).clone()
        S0 = torch.tensor(f["yi"], dtype=torch.float64, device=dev).expand(f["numParticles"], 3)
        th.requires_grad_(grad)
        S_all.append(_spins(f, wins, S0, th))
        P_all.append([w[1] for w in wins])
        V_all.append([w[2] for w in wins])
        th_all.append(th)
    if kind == "track":
        out = dict.fromkeys(("t", "fail", "n_coll", "n_bounce", "n_steps", "turns"))
        for name, rows in (("pos", P_all[0]), ("v", V_all[0]), ("S", S_all[0])):
            out[name] = torch.stack(rows).transpose(1, 2).contiguous()
        return out
    if kind == "loop":
        none = dict.fromkeys(("t", "fail", "n_coll", "n_bounce", "n_steps"))
        return [dict(none, pos=p, v=v, S=s) for p, v, s in zip(P_all[0], V_all[0], S_all[0])]
    if kind == "adjoint":
        g = torch.Generator(device="cpu").manual_seed(int(seed))
        w = torch.randn(case["n"], 3, dtype=torch.float64, generator=g).to(dev) / case["n"]
        S = S_all[0][-1]
        (S * w).sum().backward()
        gr = th_all[0].grad.clone()
        gr[:, 15:] = 0.0  # no pulse, no pulse gradients
        return {"S": S.detach(), "grad": gr}
    if kind == "grid":
        S = [s[-1] for s in S_all]
        sum(s.mean(0).norm() for s in S).backward()
        return {"S": torch.cat(S).detach(), "grad": torch.stack([t.grad.sum(0) for t in th_all])}
    S = S_all[0][-1]
    stats = dict.fromkeys(("t", "n_valid", "n_phase", "mean_S", "polarisation", "phase_mean", "phase_std",
                           "phase_stderr", "phase_expected", "freq_shift", "freq_shift_err", "phase_unwrapped_mean",
                           "phase_unwrapped_std", "freq_shift_unwrapped"))
    m = S.mean(0)
    stats.update(mean_S=m.cpu().numpy(), polarisation=float(m.norm()))
    return {"stats": stats, "phase": None, "S": S}
