"""The work whose speed counts: what a user of this framework has it do, over the range of its uses.

A case is one call pattern on one scene. The scenes are the framework's own (sph2d_gb300/cases.py: dam break,
piston flume, tank ensemble, 3D dam break, adjoint flume) at several sizes, with a seeded smooth velocity field on
the fluid, so that the viscosity meets a moving fluid as it does in the middle of a run. The call patterns:

- "run":     the state is uploaded (a dump, a restart) and advanced to the next data layer: rrsph_upload and
             rrsph_step_download of `steps` steps on page-locked host arrays, as the RRSPH_CUDA backend calls them;
- "step":    the drop-in call on the caller's host arrays, one step at a time: rrsph_step_host on page-locked arrays,
             which the next call reads again;
- "adjoint": a gradient of the piston optimisation: upload, rrsph_adjoint_forward, rrsph_adjoint_reverse.

Positions and everything of the FP64 step come back as the doubles the calls write. The FP32-mixed step's velocity,
density and pressure, whose pair arithmetic is float, go to float32 arrays, as a viewer or a layer of single-precision
fields takes them.
"""

import ctypes as C
import math

import numpy as np
import torch

from sph2d_gb300 import Solver, cases
from sph2d_gb300.capi import check, lib

G = 9.81
DELTA_SPH = 0.1  # density_delta_sph_coef of the delta-SPH cases


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # the smallest ensemble tank (2,000 fluid particles) through the drop-in call: launches and latency
        {"name": "tank_step_mixed", "call": "step", "scene": "tank", "precision": "mixed", "density": 0,
         "nx": 50, "ny": 40, "steps": 1},
        # the 2D dam break of the configurations (5,000 fluid particles), between two data layers
        {"name": "dam2d_run_mixed", "call": "run", "scene": "dam2d", "precision": "mixed", "density": 0,
         "nx": 100, "ny": 50, "steps": 50},
        # the same in the reference's own precision
        {"name": "dam2d_run_fp64", "call": "run", "scene": "dam2d", "precision": "fp64", "density": 0,
         "nx": 100, "ny": 50, "steps": 20},
        # the headline workload: the 409k-particle piston flume
        {"name": "flume_run_mixed", "call": "run", "scene": "flume", "precision": "mixed", "density": 0,
         "nx": 4000, "ny": 100, "steps": 20},
        # the flume in double, one step a call (the backend with RRSPH_CUDA_PRECISION=fp64, layers every step)
        {"name": "flume_step_fp64", "call": "step", "scene": "flume", "precision": "fp64", "density": 0,
         "nx": 4000, "ny": 100, "steps": 1},
        # continuity density with the delta-SPH term, a ragged mid-size dam break, both precisions
        {"name": "dam2d_delta_mixed", "call": "run", "scene": "dam2d", "precision": "mixed", "density": 2,
         "nx": 283, "ny": 141, "steps": 20},
        {"name": "dam2d_delta_fp64", "call": "run", "scene": "dam2d", "precision": "fp64", "density": 2,
         "nx": 283, "ny": 141, "steps": 5},
        # the 3D dam break (continuity density) at twice the configured spacing: about 1M particles
        {"name": "dam3d_run_mixed", "call": "run", "scene": "dam3d", "precision": "mixed", "density": 1,
         "dx": 0.0052, "steps": 5},
        # the same scene in double, coarser
        {"name": "dam3d_run_fp64", "call": "run", "scene": "dam3d", "precision": "fp64", "density": 1,
         "dx": 0.0078, "steps": 2},
        # a packed ensemble of piston tanks of uneven size, each with its own piston
        {"name": "ensemble_run_mixed", "call": "run", "scene": "tanks", "precision": "mixed", "density": 0,
         "tanks": 40, "steps": 10},
        # one gradient of the piston optimisation on a 2 m flume, the piston touching the water
        {"name": "adjoint_flume", "call": "adjoint", "scene": "flume", "precision": "fp64", "density": 0,
         "nx": 400, "ny": 100, "steps": 50, "every": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.randrange(8)
    mixed = {"precision": "mixed"}
    fp64 = {"precision": "fp64"}
    if kind == 0:  # a tank, one step a call
        return {"call": "step", "scene": "tank", "density": 0, "nx": _log(rng, 40, 600), "ny": rng.randint(30, 120),
                "steps": 1, **(mixed if rng.random() < 0.6 else fp64)}
    if kind == 1:  # a dam break between two layers
        ny = _log(rng, 40, 280)
        return {"call": "run", "scene": "dam2d", "density": 0, "nx": 2 * ny + rng.randint(-9, 9), "ny": ny,
                "steps": rng.randint(10, 40), **mixed}
    if kind == 2:
        ny = _log(rng, 40, 200)
        return {"call": "run", "scene": "dam2d", "density": 0, "nx": 2 * ny + rng.randint(-9, 9), "ny": ny,
                "steps": rng.randint(3, 10), **fp64}
    if kind == 3:  # a flume
        return {"call": "run", "scene": "flume", "density": 0, "nx": _log(rng, 500, 4000), "ny": rng.randint(60, 110),
                "steps": rng.randint(8, 20), **mixed}
    if kind == 4:
        return {"call": "step", "scene": "flume", "density": 0, "nx": _log(rng, 500, 4000), "ny": rng.randint(60, 100),
                "steps": 1, **fp64}
    if kind == 5:  # continuity density, with and without the delta-SPH term
        ny = _log(rng, 40, 200)
        p = mixed if rng.random() < 0.5 else fp64
        return {"call": "run", "scene": "dam2d", "density": rng.choice([1, 2]), "nx": 2 * ny + rng.randint(-9, 9),
                "ny": ny, "steps": rng.randint(8, 20) if p is mixed else rng.randint(2, 6), **p}
    if kind == 6:  # 3D
        if rng.random() < 0.5:
            return {"call": "run", "scene": "dam3d", "density": 1, "dx": round(rng.uniform(0.0054, 0.016), 5),
                    "steps": rng.randint(2, 5), **mixed}
        return {"call": "run", "scene": "dam3d", "density": 1, "dx": round(rng.uniform(0.008, 0.016), 5),
                "steps": rng.randint(1, 2), **fp64}
    if rng.random() < 0.5:  # tanks
        return {"call": "run", "scene": "tanks", "density": 0, "tanks": rng.randint(4, 40), "steps": rng.randint(8, 12),
                **mixed}
    steps = rng.randint(30, 50)
    return {"call": "adjoint", "scene": "flume", "density": 0, "nx": _log(rng, 60, 400), "ny": rng.randint(30, 90),
            "steps": steps, "every": rng.randint(5, steps), **fp64}


# ----------------------------------------------------------------- scenes --
def _scene(case, seed):
    """The framework's scene of `case`, jittered by the seed, its fluid set in smooth motion."""
    kind, density = case["scene"], case["density"]
    rng = np.random.default_rng(1000003 * int(seed) + 17)
    jitter = int(rng.integers(1 << 30))
    if kind == "dam2d":
        c = cases.dam_break_2d(seed=jitter, nx=case["nx"], ny=case["ny"], dx=0.5 / case["ny"], density_treatment=density)
    elif kind == "flume":
        c = cases.piston_flume_2d(seed=jitter, nx=case["nx"], ny=case["ny"], density_treatment=density)
    elif kind == "tank":
        c = cases.piston_flume_2d(seed=jitter, nx=case["nx"], ny=case["ny"], tank_height=case["ny"] * 0.005 + 0.3,
                                  density_treatment=density)
    elif kind == "dam3d":
        c = cases.dam_break_3d(seed=jitter, dx=case["dx"], density_treatment=density)
    else:  # tanks: the sizes are the case's, the pistons the seed's
        tanks = cases.ensemble_tanks(ntanks=case["tanks"], seed=4, wave_seed=jitter)
        c = cases.pack_tanks(tanks)
    if case["call"] == "adjoint":  # within reach of the first fluid column, so that the gauge feels it
        c.r[c.particle["nwm_particles_start"]:c.particle["nwm_particles_end"], 0] += 0.08 * c.notes["h"]
    if density == 2:
        c.model["density_delta_sph_coef"] = DELTA_SPH
    fluid = c.itype > 0
    r = c.r[fluid]
    v = np.zeros_like(r)
    for _ in range(4):  # modes of 0.1 to 0.6 m, about 0.2 m/s together
        k = 2.0 * math.pi / rng.uniform(0.1, 0.6, size=r.shape[1])
        ph = rng.uniform(0.0, 2.0 * math.pi, size=r.shape[1])
        a = 0.1 * rng.uniform(0.5, 1.0)
        s, co = np.sin(r * k + ph), np.cos(r * k + ph)
        # 2D: from a stream function (no divergence); 3D adds a shear along z
        v[:, 0] += a * s[:, 0] * co[:, 1]
        v[:, 1] -= a * k[0] / k[1] * co[:, 0] * s[:, 1]
        if r.shape[1] == 3:
            v[:, 2] += a * s[:, 0] * s[:, 1]
    np.clip(v, -0.8, 0.8, out=v)
    c.v = c.v.copy()
    c.v[fluid] = v
    return c


def _adjoint_setup(case, seed):
    """Piston coefficients, gauge and weights of an adjoint case."""
    rng = np.random.default_rng(1000003 * int(seed) + 29)
    n = case["steps"]
    return {"omega": 2.0 * math.pi / 8.0, "coef": rng.uniform(0.005, 0.03, size=8), "gauge_x": 0.01,
            "sample_from": n // 2, "sample_every": 5, "w": rng.standard_normal((n - n // 2) // 5 + 1)}


def _pinned(shape, dtype, value=None):
    t = torch.empty(shape, dtype=dtype, pin_memory=True)
    if value is not None:
        t.copy_(torch.from_numpy(np.ascontiguousarray(value)))
    else:
        t.zero_()
    return t


def _ptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_int32 if t.dtype == torch.int32 else C.c_double))


def prepare(case, seed):
    c = _scene(case, seed)
    solver = Solver(c.params(), case["precision"])
    if c.name == "ensemble_2d":
        solver.set_wave_makers(c.notes["wave_makers"])
    st = {"solver": solver, "case": case}
    if case["call"] == "adjoint":
        a = _adjoint_setup(case, seed)
        solver.set_piston_fourier(a["omega"], a["coef"])
        st.update(a, arrays=(c.r, c.v, c.rho, c.itype))
        return st
    n, dim = c.r.shape
    st["in"] = {"r": _pinned((n, dim), torch.float64, c.r), "v": _pinned((n, dim), torch.float64, c.v),
                "rho": _pinned((n,), torch.float64, c.rho), "itype": _pinned((n,), torch.int32, c.itype)}
    if case["call"] == "step":
        st["out"] = dict(st["in"], p=_pinned((n,), torch.float64))
    else:
        st["out"] = {"r": _pinned((n, dim), torch.float64), "v": _pinned((n, dim), torch.float64),
                     "rho": _pinned((n,), torch.float64), "itype": _pinned((n,), torch.int32),
                     "p": _pinned((n,), torch.float64)}
    i, o = st["in"], st["out"]
    st["t"] = C.c_double(0.0)
    st["upload"] = (_ptr(i["r"]), dim, _ptr(i["v"]), _ptr(i["rho"]), None, _ptr(i["itype"]))
    st["download"] = (_ptr(o["r"]), dim, _ptr(o["v"]), _ptr(o["rho"]), _ptr(o["p"]), _ptr(o["itype"]))
    if case["precision"] == "mixed":
        st["single"] = {k: torch.zeros(o[k].shape, dtype=torch.float32) for k in ("v", "rho", "p")}
    return st


# -------------------------------------------------------------------- run --
def run(st):
    case, s = st["case"], st["solver"]
    if case["call"] == "adjoint":
        s.upload(*st["arrays"][:3], st["arrays"][3])
        gauges, _ = s.adjoint_forward(case["steps"], st["gauge_x"], sample_from=st["sample_from"],
                                      sample_every=st["sample_every"], checkpoint_every=case["every"])
        dcoef, dvx = s.adjoint_reverse(st["w"])
        return {"gauges": gauges, "dcoef": dcoef, "dvx": dvx}
    L, t = lib(), st["t"]
    if case["call"] == "step":
        check(L.rrsph_step_host(s.handle, case["steps"], C.byref(t), *st["download"]))
    else:
        t.value = 0.0
        check(L.rrsph_upload(s.handle, *st["upload"]))
        check(L.rrsph_step_download(s.handle, case["steps"], C.byref(t), *st["download"]))
    o = st["out"]
    if case["precision"] == "mixed":
        f = st["single"]
        return {"r": o["r"], "itype": o["itype"], **{k: f[k].copy_(o[k]) for k in f}}
    return dict(o)


# ------------------------------------------------------------------- work --
def work(case):
    """Each step reads and writes the state (positions, velocities, accelerations; with continuity density also the
    density and its rate) once and evaluates each directed pair once: 68 operations (a kernel value and gradient,
    pressure and viscosity terms, the sums); a call also takes the host arrays in and gives them back. The adjoint's
    cost is a forward run and a reverse run of about twice its arithmetic."""
    c = _scene(case, 0)
    n, dim = c.r.shape
    steps, cont = case["steps"], case["density"] != 0
    pairs = n * (80.0 if dim == 3 else 20.0)
    state = 2 * (3 * dim * 8 + (16 if cont else 0))
    host = (2 * dim * 8 + 8 + 4) + (2 * dim * 8 + 16 + 4)
    times = 3 if case["call"] == "adjoint" else 1
    return {"bytes": float(n * (host + times * steps * state)), "flops": float(times * steps * pairs * 68)}


# ------------------------------------------------------------------ exact --
def _neighbour_pairs(r, cell):
    """Directed pairs (j, i) with |r_i - r_j| < cell, j != i."""
    n, dim = r.shape
    ij = torch.floor((r - r.min(0).values) / cell).long() + 1
    dims = ij.max(0).values + 2
    stride = torch.ones(dim, dtype=torch.long, device=r.device)
    for d in range(1, dim):
        stride[d] = stride[d - 1] * dims[d - 1]
    key = (ij * stride).sum(1)
    order = torch.argsort(key)
    ks = key[order]
    offs = torch.cartesian_prod(*[torch.tensor([-1, 0, 1], device=r.device)] * dim)
    js, is_ = [], []
    for o in offs:
        want = key + (o * stride).sum()
        lo = torch.searchsorted(ks, want)
        cnt = torch.searchsorted(ks, want, right=True) - lo
        j = torch.repeat_interleave(torch.arange(n, device=r.device), cnt)
        first = torch.cumsum(cnt, 0) - cnt
        i = order[lo[j] + torch.arange(j.numel(), device=r.device) - first[j]]
        d = r[i] - r[j]
        keep = ((d * d).sum(1) < cell * cell) & (i != j)
        js.append(j[keep])
        is_.append(i[keep])
    return torch.cat(js), torch.cat(is_)


class _Physics:
    """The method of the scenes' parameters in plain torch, 64 bits."""

    def __init__(self, c):
        m, q = c.model, c.particle
        self.dim, self.h = q["dim"], q["delta"] * m["intf_hsml_coef"]
        self.rho0, self.mass, self.dt = q["rho0"], q["rho0"] * q["delta"] ** q["dim"], m["dt"]
        c2 = 200 * G * q["depth"] * m["eos_sound_vel_coef"]
        self.c, self.B = math.sqrt(c2), c2 * self.rho0 / 7
        self.f = 15 / (7 * math.pi * self.h ** 2) if self.dim == 2 else 3 / (2 * math.pi * self.h ** 3)
        self.alpha, self.beta = m["artificial_shear_visc"], m["artificial_bulk_visc"]
        self.D, self.rr0, self.eta2 = 5 * G * q["depth"], 2 * self.h, (self.h * float(np.float32(0.1))) ** 2
        self.density = m["density_treatment"]
        self.dhc = m.get("density_delta_sph_coef", 0.0) * self.h * self.c

    def p(self, rho):
        return self.B * ((rho / self.rho0) ** 7 - 1)

    def rates(self, r, v, vp, rho, rho_f, itype):
        """(rho or drho, p, a) of one evaluation: density_sum / density_con, the EOS, update_acceleration."""
        j, i = _neighbour_pairs(r.detach(), 2 * self.h)
        d = r[i] - r[j]
        d2 = (d * d).sum(1)
        dist = torch.sqrt(d2)
        q = dist / self.h
        t = 2 - q
        sc = torch.where(q <= 1, self.f / self.h ** 2 * (1.5 * q - 2), -self.f / (self.h * dist) * t * t * 0.5)

        def total(x):
            return torch.zeros(r.shape[:1] + x.shape[1:], dtype=r.dtype, device=r.device).index_add(0, j, x)

        if self.density == 0:
            w = torch.where(q <= 1, self.f * (2 / 3 - q * q + 0.5 * q ** 3), self.f / 6 * t ** 3)
            out = self.mass * (self.f * 2 / 3) + total(self.mass * w)
            rho_f, p = out, self.p(out)
        else:
            term = ((v[i] - v[j]) * d).sum(1) * sc
            if self.density == 2:
                term = term - 2 * self.dhc * (rho[i] - rho[j]) / rho[i] * sc
            out, p = total(self.mass * term), self.p(rho)
        pr2 = p / rho_f ** 2
        vr = -((vp[j] - vp[i]) * d).sum(1)
        mu = torch.where(vr < 0, self.h * vr / (d2 + self.eta2), torch.zeros_like(vr))
        m = self.mass * sc * (pr2[i] + pr2[j] + (self.beta * mu - self.alpha * self.c) * mu * 2 / (rho_f[i] + rho_f[j]))
        rn4 = (self.rr0 / dist) ** 4
        m = m - torch.where((itype[j] > 0) & (itype[i] < 0), self.D * (rn4 ** 3 - rn4) / d2, torch.zeros_like(d2))
        down = torch.zeros(self.dim, dtype=r.dtype, device=r.device)
        down[1] = -G
        return out, p, total(m[:, None] * d) + down


def _pistons(c):
    """(start, end, velocity law) of each piston of the scene."""
    def law(m, depth):
        k = 2 * math.pi / m["wave_length"]
        kd, omega = k * depth, math.sqrt(G * k * math.tanh(k * depth))
        s0 = m["wave_magnitude"] * (math.sinh(kd) * math.cosh(kd) + kd) / (2 * math.sinh(kd) ** 2)
        return lambda t: 0.5 * s0 * omega * math.cos(omega * t)
    if c.name == "ensemble_2d":
        return [(m["particles_start"], m["particles_end"], law(m, m["depth"])) for m in c.notes["wave_makers"]]
    if c.model["nwm"] == 2:
        m = {"wave_length": c.model["nwm_wave_length"], "wave_magnitude": c.model["nwm_wave_magnitude"]}
        return [(c.particle["nwm_particles_start"], c.particle["nwm_particles_end"], law(m, c.particle["depth"]))]
    return []


def _advance(ph, c, steps, laws, watch=None):
    """The time loop from the scene's state, with the piston velocities of `laws`."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    r, v, rho = (torch.tensor(x, dtype=torch.float64, device=dev) for x in (c.r, c.v, c.rho))
    itype = torch.tensor(c.itype, device=dev)
    fluid = (itype > 0)[:, None]
    a, drho, p, time = torch.zeros_like(r), torch.zeros_like(rho), torch.zeros_like(rho), 0.0
    for n in range(steps):
        if watch:
            watch(n, r)
        out, p, new_a = ph.rates(r, v, v + a * ph.dt * 0.5, rho, rho + drho * ph.dt * 0.5, itype)
        a = new_a
        v_dt = ph.dt if n else 0.5 * ph.dt
        if ph.density == 0:
            rho = out
        else:
            drho = out
            rho = rho + drho * v_dt
        v = torch.where(fluid, v + a * v_dt, v)
        r = torch.where(fluid, r + v * ph.dt, r)
        for lo, hi, law in laws:
            vx = law(n, time)
            push = torch.zeros_like(r)
            push[lo:hi, 0] = 1.0
            v = torch.where(push > 0, push * vx, v)
            r = r + push * (vx * ph.dt)
        time += ph.dt
    if watch:
        watch(steps, r)
    return r, v, rho, p


def exact(case, seed):
    c = _scene(case, seed)
    ph = _Physics(c)
    if case["call"] != "adjoint":
        laws = [(lo, hi, lambda n, t, f=f: f(t)) for lo, hi, f in _pistons(c)]
        with torch.no_grad():
            r, v, rho, p = _advance(ph, c, case["steps"], laws)
        return {"r": r, "v": v, "rho": rho, "p": p, "itype": None}
    if case["nx"] * case["ny"] * case["steps"] > 2_500_000:
        return None  # the recorded pairs of every step would not fit the time
    a = _adjoint_setup(case, seed)
    n = case["steps"]
    dt = c.model["dt"]
    ks = np.arange(1, 9)
    times, t = [], 0.0
    for _ in range(n):
        times.append(t)
        t += dt
    vx0 = [float(np.sum(a["coef"] * ks * a["omega"] * np.cos(ks * a["omega"] * t))) for t in times]
    vx = torch.tensor(vx0, dtype=torch.float64, device="cuda" if torch.cuda.is_available() else "cpu", requires_grad=True)
    gauges = []
    fluid = torch.tensor(c.itype == 2, device=vx.device)

    def watch(m, r):
        if m >= a["sample_from"] and (m - a["sample_from"]) % a["sample_every"] == 0:
            near = fluid & ((r[:, 0] - a["gauge_x"]).abs() < 3.0 * ph.h) & (r[:, 1] > 0)
            gauges.append(r[torch.where(near, r[:, 1], torch.zeros_like(r[:, 1])).argmax(), 1])

    laws = [(lo, hi, lambda n, t: vx[n]) for lo, hi, _ in _pistons(c)]
    _advance(ph, c, n, laws, watch)
    g = torch.stack(gauges)
    (g * torch.tensor(a["w"], device=g.device)).sum().backward()
    dvx = vx.grad.cpu().numpy()
    dcoef = np.array([np.sum(dvx * k * a["omega"] * np.cos(k * a["omega"] * np.array(times))) for k in ks])
    return {"gauges": g.detach(), "dcoef": dcoef, "dvx": dvx}
