"""Timed workloads of the finite-volume update, through the package's public calls.

Every case is a whole call (or loop of calls) of a program that uses this
package: it holds a problem on the GPU, advances it and takes the state back
into its host array, as the reference's main loop does between two frames, or
steps a device array that it owns.  Inputs are synthetic and seeded.

Kinds
  step      gk_rk2_step_noalloc on a device array that the caller owns: one RK2
            step per call, the smallest piece of work, bound by latency
  tube      a 1D shock tube of a few hundred cells, the whole run to its end
            time: upload, Sim.run, download (the reference's shock_tube)
  row       a long 1D row (a resolution study), a fixed number of steps
  kh        2D Kelvin-Helmholtz, periodic: the benchmark problem; small grids
            advance to the next output time, large ones a number of steps
  rt        2D Rayleigh-Taylor, RK3, constant gravity, reflecting walls
  box       3D smooth random state with all velocity components, periodic
  blast     3D pressure blast between reflecting / outflow sides
  disk      2D disk around a softened point mass: fixed (type 4) sides and the
            inner reset (the reference's disk setups)
  ensemble  independent KH problems of uneven sizes advanced together
  learned   KH with the learned flux correction at every face
Both arithmetic modes are used in earnest: "parity" (the default, the
reference's bits) and "fast".  Everything the solver computes is FP64.
"""
import ctypes
import math

import numpy as np
import torch

from gaukuk_b200 import _lib, learned
from gaukuk_b200.config import (BC_FIXED, BC_OUTFLOW, BC_PERIODIC, BC_REFLECTIVE, Params)
from gaukuk_b200.ensemble import Ensemble
from gaukuk_b200.sim import MODES, Sim, _descs

P6 = (BC_PERIODIC,) * 6


def listed():
    return [
        # one step of a small grid on the caller's own device array
        {"name": "step 130x94 parity", "kind": "step", "mode": "parity", "nx": 130, "ny": 94},
        # the 1D benchmark configuration, run to t = 0.2
        {"name": "tube 256 parity", "kind": "tube", "mode": "parity", "nx": 256, "tmax": 0.2},
        # a long row of an odd length
        {"name": "row 262143 parity", "kind": "row", "mode": "parity", "nx": 262143, "steps": 48},
        # the 256^2 benchmark configuration at its output cadence
        {"name": "kh 256 parity", "kind": "kh", "mode": "parity", "nx": 256, "ny": 256, "dtout": 0.05},
        # a ragged large grid in the default mode
        {"name": "kh 2001x1503 parity", "kind": "kh", "mode": "parity", "nx": 2001, "ny": 1503, "steps": 32},
        # the headline grid
        {"name": "kh 4096 fast", "kind": "kh", "mode": "fast", "nx": 4096, "ny": 4096, "steps": 64},
        # the Rayleigh-Taylor benchmark configuration
        {"name": "rt 1024x3072 fast", "kind": "rt", "mode": "fast", "nx": 1024, "ny": 3072, "steps": 40},
        # 3D at the size the 3D path is quoted on
        {"name": "box 256 fast", "kind": "box", "mode": "fast", "nx": 256, "ny": 256, "nz": 256, "steps": 8},
        # a 3D blast of uneven extents in the default mode
        {"name": "blast 101x97x90 parity", "kind": "blast", "mode": "parity", "nx": 101, "ny": 97,
         "nz": 90, "steps": 16},
        # point mass, fixed sides, inner reset
        {"name": "disk 384 parity", "kind": "disk", "mode": "parity", "nx": 384, "ny": 384, "steps": 32},
        # 32 problems of 128^2, 256^2 and 512^2 cells together
        {"name": "ensemble 32 fast", "kind": "ensemble", "mode": "fast", "count": 32, "steps": 32},
        # the learned correction at the size it is trained for
        {"name": "learned 256 parity", "kind": "learned", "mode": "parity", "nx": 256, "ny": 256, "steps": 16},
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n | 1 if rng.random() < 0.5 else n


def _steps_for(cells, budget, lo, hi):
    return max(lo, min(hi, budget // max(cells, 1)))


def draw(rng):
    kind = rng.choice(["step", "tube", "row", "kh", "kh", "rt", "box", "blast", "disk", "ensemble"])
    mode = rng.choice(["parity", "fast"])
    c = {"kind": kind, "mode": mode}
    if kind == "step":
        c.update(nx=_log_int(rng, 48, 1200), ny=_log_int(rng, 48, 1200))
    elif kind == "tube":
        c.update(nx=_log_int(rng, 64, 1018), tmax=round(rng.uniform(0.02, 0.2), 3))
    elif kind == "row":
        n = _log_int(rng, 1100, 1 << 20)
        c.update(nx=n, steps=_steps_for(n, 12_000_000, 16, 128))
    elif kind == "kh":
        nx, ny = _log_int(rng, 48, 3000), _log_int(rng, 48, 3000)
        c.update(nx=nx, ny=ny, steps=_steps_for(nx * ny, 128_000_000, 16, 128))
    elif kind == "rt":
        nx, ny = _log_int(rng, 48, 1500), _log_int(rng, 96, 3000)
        c.update(nx=nx, ny=ny, steps=_steps_for(nx * ny, 96_000_000, 12, 96))
    elif kind in ("box", "blast"):
        nx, ny, nz = (_log_int(rng, 20, 200) for _ in range(3))
        c.update(nx=nx, ny=ny, nz=nz, steps=_steps_for(nx * ny * nz, 48_000_000, 6, 64))
    elif kind == "disk":
        nx, ny = _log_int(rng, 64, 1400), _log_int(rng, 64, 1400)
        c.update(nx=nx, ny=ny, steps=_steps_for(nx * ny, 32_000_000, 12, 64))
    else:
        c.update(count=rng.randint(4, 32), steps=16)
    return c


# ------------------------------------------------------------------ problems
# Each problem is (Params, primitives): rho, vx, vy, vz, p as float64 tensors
# of shape (nz, ny, nx) on the GPU, made from the seed alone.

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _centres(p):
    out = []
    for lo, hi, n in ((p.xmin, p.xmax, p.nx), (p.ymin, p.ymax, p.ny), (p.zmin, p.zmax, p.nz)):
        d = (hi - lo) / n
        out.append(lo + d * (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5))
    x, y, z = out
    return x[None, None, :], y[None, :, None], z[:, None, None]


def _kh(nx, ny, seed):
    r = np.random.default_rng(seed)
    ratio, half, amp = r.uniform(1.5, 4.0), r.uniform(0.2, 0.3), r.uniform(0.005, 0.02)
    p = Params(nx=nx, ny=ny, cfl=0.4, integrator=2, bc=P6, tmax=2.0, dtoutput=2.0)
    x, y, _ = _centres(p)
    inside = ((y - 0.5).abs() < half).expand(1, ny, nx)
    one = torch.ones((1, ny, nx), dtype=torch.float64, device="cuda")
    vy = amp * torch.sin(4 * math.pi * x) + 1e-3 * (2 * torch.rand(one.shape, dtype=torch.float64,
                                                                 device="cuda", generator=_gen(seed)) - 1)
    return p, (torch.where(inside, ratio * one, one), torch.where(inside, -0.5 * one, 0.5 * one), vy,
               torch.zeros_like(one), 2.5 * one)


def _rt(nx, ny, seed):
    r = np.random.default_rng(seed)
    amp, up = 0.01 * r.uniform(0.7, 1.3), r.uniform(1.8, 2.2)
    g = -0.1
    p = Params(nx=nx, ny=ny, xmin=-0.25, xmax=0.25, ymin=-0.75, ymax=0.75, zmin=-0.5, zmax=0.5, cfl=0.4,
               integrator=3, bc=(BC_PERIODIC, BC_PERIODIC, BC_REFLECTIVE, BC_REFLECTIVE, BC_PERIODIC,
                                 BC_PERIODIC), grav=(0.0, g, 0.0), tmax=5.0, dtoutput=5.0)
    x, y, _ = _centres(p)
    one = torch.ones((1, ny, nx), dtype=torch.float64, device="cuda")
    rho = torch.where((y > 0).expand_as(one), up * one, one)
    vy = amp * (1 + torch.cos(4 * math.pi * x)) * (1 + torch.cos(3 * math.pi * y)) / 4
    zero = torch.zeros_like(one)
    return p, (rho, zero, vy * one, zero, 2.5 + g * rho * y)


def _tube(nx, seed, tmax):
    r = np.random.default_rng(seed)
    p = Params(nx=nx, cfl=0.4, integrator=2, bc=(BC_OUTFLOW, BC_OUTFLOW) + P6[2:], tmax=tmax, dtoutput=tmax)
    x, _, _ = _centres(p)
    left = x < 0.5
    one = torch.ones((1, 1, nx), dtype=torch.float64, device="cuda")
    rho = torch.where(left, one, 0.125 * r.uniform(0.9, 1.1) * one)
    pre = torch.where(left, one * r.uniform(0.9, 1.1), 0.1 * one)
    zero = torch.zeros_like(one)
    return p, (rho, zero, zero, zero, pre)


def _row(nx, seed):
    r = np.random.default_rng(seed)
    p = Params(nx=nx, cfl=0.4, integrator=2, bc=(BC_OUTFLOW, BC_OUTFLOW) + P6[2:], tmax=1.0, dtoutput=1.0)
    x, _, _ = _centres(p)
    # a train of jumps with smooth waves between them
    k = int(r.integers(20, 60))
    level = torch.tensor(r.uniform(0.3, 2.0, size=(2, k)), device="cuda")
    seg = torch.clamp((x * k).long(), max=k - 1)
    wave = 0.1 * torch.sin(2 * math.pi * 37 * x + r.uniform(0, 6))
    zero = torch.zeros_like(x)
    return p, (level[0][seg] * (1 + wave), 0.5 * wave, zero, zero, level[1][seg] * (1 - wave))


def _box(nx, ny, nz, seed):
    r = np.random.default_rng(seed)
    p = Params(nx=nx, ny=ny, nz=nz, cfl=0.4, integrator=2, bc=P6, tmax=1.0, dtoutput=1.0)
    x, y, z = _centres(p)

    def field(base, ampl):
        f = torch.full((nz, ny, nx), base, dtype=torch.float64, device="cuda")
        for _ in range(3):
            kx, ky, kz = r.integers(1, 4, size=3)
            a, b, c = r.uniform(0, 2 * math.pi, size=3)
            f += float(r.uniform(-ampl, ampl)) * (torch.sin(2 * math.pi * kx * x + a) *
                                                  torch.cos(2 * math.pi * ky * y + b) *
                                                  torch.cos(2 * math.pi * kz * z + c))
        return f

    return p, (field(1.5, 0.3), field(0.0, 0.4), field(0.0, 0.4), field(0.0, 0.4), field(2.0, 0.4))


def _blast(nx, ny, nz, seed):
    r = np.random.default_rng(seed)
    p = Params(nx=nx, ny=ny, nz=nz, cfl=0.4, integrator=2,
               bc=(BC_REFLECTIVE, BC_REFLECTIVE, BC_OUTFLOW, BC_OUTFLOW, BC_REFLECTIVE, BC_OUTFLOW),
               tmax=0.2, dtoutput=0.2)
    x, y, z = _centres(p)
    cx, cy, cz = r.uniform(0.35, 0.65, size=3)
    one = torch.ones((nz, ny, nx), dtype=torch.float64, device="cuda")
    d2 = (x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2
    rho = one * (1 + 0.1 * torch.sin(2 * math.pi * x) * torch.cos(2 * math.pi * (y + z)))
    zero = torch.zeros_like(one)
    return p, (rho, zero, zero, zero, torch.where(d2 < 0.04, 10.0 * one, 0.1 * one))


def _disk(nx, ny, seed):
    r = np.random.default_rng(seed)
    p = Params(nx=nx, ny=ny, xmin=-2.0, xmax=2.0, ymin=-2.0, ymax=2.0, zmin=-2.0, zmax=2.0, cfl=0.4,
               integrator=2, bc=(BC_FIXED,) * 4 + P6[4:], tmax=1.0, dtoutput=1.0)
    x, y, _ = _centres(p)
    r2 = x * x + y * y
    om = (r2 + 0.09) ** -0.75  # circular motion around the softened mass
    rho = (r2 + 0.25) ** -0.5 * (1 + 0.02 * torch.cos(3 * torch.atan2(y, x.expand(1, ny, nx)) +
                                                      float(r.uniform(0, 6))))
    one = torch.ones((1, ny, nx), dtype=torch.float64, device="cuda")
    return p, (rho * one, -om * y * one, om * x * one, torch.zeros_like(one),
               float(r.uniform(0.008, 0.012)) * rho * (r2 + 0.09) ** -0.5)


POINT = (1.0, 0.0, 0.0, 0.0, 0.3)  # gm, x, y, z, softening


def _problem(c, seed):
    k = c["kind"]
    if k in ("step", "kh", "learned"):
        return _kh(c["nx"], c["ny"], seed)
    if k == "rt":
        return _rt(c["nx"], c["ny"], seed)
    if k == "tube":
        return _tube(c["nx"], seed, c["tmax"])
    if k == "row":
        return _row(c["nx"], seed)
    if k == "box":
        return _box(c["nx"], c["ny"], c["nz"], seed)
    if k == "blast":
        return _blast(c["nx"], c["ny"], c["nz"], seed)
    return _disk(c["nx"], c["ny"], seed)


def _instances(c, seed):
    sizes = np.random.default_rng(c["count"]).choice([128, 256, 512], size=c["count"])
    return [_kh(int(n), int(n), seed * 1000 + i) for i, n in enumerate(sizes)]


def _cons_active(p, w):
    """Conserved variables (DEN, MTX, MTY, MTZ, ENG) of the active cells."""
    rho, vx, vy, vz, pre = w
    return torch.stack([rho, rho * vx, rho * vy, rho * vz,
                        pre * (1.0 / (p.gamma - 1.0)) + 0.5 * rho * (vx * vx + vy * vy + vz * vz)])


def _act(p, a):
    g = p.ng
    return a[..., g:g + p.nz, g:g + p.ny, g:g + p.nx]


def _host(p, w):
    """The program's host array in the reference layout: pinned, ghosts zero."""
    t = torch.zeros(p.shape, dtype=torch.float64, pin_memory=True)
    _act(p, t).copy_(_cons_active(p, w))
    return t


# ------------------------------------------------------------------ one case
def prepare(case, seed):
    c = case
    k = c["kind"]
    if k == "ensemble":
        sims, frames = [], []
        for p, w in _instances(c, seed):
            t = _host(p, w)
            sims.append(Sim(p, t.numpy(), mode=c["mode"]))
            frames.append(t)
        return {"case": c, "sims": sims, "frames": frames, "ens": Ensemble(sims)}
    p, w = _problem(c, seed)
    if k == "step":
        # the library's device layout: planes DEN, MTX, MTY, ENG, MTZ, rows of `pitch` doubles
        pitch = (p.lenx + 15) // 16 * 16
        u = torch.zeros((5, p.leny, pitch), dtype=torch.float64, device="cuda")
        a = _cons_active(p, w)[:, 0]
        for slot, v in enumerate((0, 1, 2, 4, 3)):
            u[slot, p.ng:p.ng + p.ny, p.ng:p.ng + p.nx] = a[v]
        gd, pd = _descs(p, MODES[c["mode"]], 0)
        return {"case": c, "p": p, "u": u, "gd": gd, "pd": pd, "lib": _lib.load(), "dt": ctypes.c_double()}
    t = _host(p, w)
    s = {"case": c, "p": p, "frame": t, "host": t.numpy()}
    sim = Sim(p, mode=c["mode"])
    if k == "disk":
        sim.set_fixed_boundary(s["host"], fix_inner=True)
        sim.set_point_gravity([POINT])
    sim.upload(s["host"])
    if k == "tube":
        s["initial"] = s["host"].copy()
    if k == "learned":
        r = np.random.default_rng(seed + 1)
        X = r.normal(size=(4096, learned.NI)).astype(np.float32)
        blob = learned.init_model(X, np.asarray(r.normal(size=(4096, learned.NO)), dtype=np.float32), seed=seed)
        blob[learned.NPARAM + 36:] *= 1e-4  # small corrections: the run stays close to the plain one
        learned.install(sim, blob)
    s["sim"] = sim
    return s


def run(state):
    c = state["case"]
    k = c["kind"]
    if k == "step":
        u, p = state["u"], state["p"]
        _lib.check(state["lib"].gk_rk2_step_noalloc(
            ctypes.byref(state["gd"]), ctypes.byref(state["pd"]), ctypes.c_void_p(u.data_ptr()), 1e300,
            ctypes.byref(state["dt"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {"cons": u[:, p.ng:p.ng + p.ny, p.ng:p.ng + p.nx], "dt": state["dt"].value}
    if k == "ensemble":
        state["ens"].run_steps(c["steps"])
        out = []
        for s, t in zip(state["sims"], state["frames"]):
            s.download(t.numpy(), planes_only=True)
            out.append(_act(s.params, t))
        return out
    sim, p = state["sim"], state["p"]
    if k == "tube":
        sim.upload(state["initial"])
        sim.set_time(0.0, 0)
        sim.run(p.tmax, p.dtoutput)
    elif "dtout" in c:
        sim.advance(c["dtout"])
    else:
        sim.run_steps(c["steps"])
    sim.download(state["host"], planes_only=True)
    return {"cons": _act(p, state["frame"]), "t": sim.get_time()}


def _nsteps(c):
    """Steps of one pass (estimated from the sound speed where it runs to a time)."""
    if c["kind"] == "tube":
        return int(c["tmax"] * c["nx"] / (0.4 / 2.2)) + 1
    if "dtout" in c:
        return int(c["dtout"] * max(c["nx"], c["ny"]) / (0.4 / 2.6)) + 1
    return c.get("steps", 1)


# FP64 operations per cell, stage and direction (conversion share, PLM slopes,
# HLLC, update; a fused multiply-add counts two)
FLOPS = 220


def work(case):
    """One pass: per step the evolved variables are read once and written once
    (1D 3, 2D 4, 3D and point-mass runs 5; a tube fits on chip: once per pass);
    a whole frame goes to the host where the program takes one."""
    c = case
    k = c["kind"]
    if k == "ensemble":
        cells = c["count"] * (128 ** 2 + 256 ** 2 + 512 ** 2) // 3
    else:
        cells = c["nx"] * c.get("ny", 1) * c.get("nz", 1)
    nvar = {"tube": 3, "row": 3, "box": 5, "blast": 5}.get(k, 4)
    dims = {"tube": 1, "row": 1, "box": 3, "blast": 3}.get(k, 2)
    stages = 3 if k == "rt" else 2
    n = _nsteps(c)
    passes = 1 if k == "tube" else n
    frame = 0 if k == "step" else 8 * nvar * cells
    flops = FLOPS * dims * stages * n * cells
    if k == "learned":
        flops += 2 * 5376 * 2 * stages * n * cells
    return {"bytes": 16 * nvar * passes * cells + frame, "flops": flops}


# ------------------------------------------------------------------ 64-bit reference
# The update as plain torch float64: arrays (5, K, J, I) in the order DEN, MTX,
# MTY, MTZ, ENG with two ghost cells in each active direction.

class _Plain:
    def __init__(self, p, w, fixed=False, point=None):
        self.p = p
        self.n = (p.nx, p.ny, p.nz)
        self.g = [2 if n > 1 else 0 for n in self.n]  # x, y, z
        gx, gy, gz = self.g
        self.u = torch.zeros((5, p.nz + 2 * gz, p.ny + 2 * gy, p.nx + 2 * gx), dtype=torch.float64,
                             device="cuda")
        self.inner = (slice(None), slice(gz, gz + p.nz), slice(gy, gy + p.ny), slice(gx, gx + p.nx))
        self.u[self.inner] = _cons_active(p, w)
        self.fix = self.u.clone() if fixed else None
        self.point = point
        d = [(p.xmax - p.xmin) / p.nx, (p.ymax - p.ymin) / p.ny, (p.zmax - p.zmin) / p.nz]
        self.d, self.drmin = d, min(d)
        x, y, z = _centres(p)
        self.x, self.y, self.z = x, y, z
        if fixed:
            keep = (x * x + y * y + z * z) < 0.25
            i = torch.arange(p.nx, device="cuda")[None, None, :] + 2
            j = torch.arange(p.ny, device="cuda")[None, :, None] + 2
            lo = [int(2 + 0.25 * n) for n in (p.nx, p.ny)]
            hi = [int(2 + 0.75 * n) for n in (p.nx, p.ny)]
            self.keep = keep & (i >= lo[0]) & (i < hi[0]) & (j >= lo[1]) & (j < hi[1])
        self.t, self.steps = 0.0, 0
        self.cmax = self._cmax()

    def fill(self, u):
        for d in range(3):
            if self.n[d] <= 1:
                continue
            ax = 3 - d
            e = 2 + self.n[d]
            for side in (0, 1):
                typ = self.p.bc[2 * d + side]
                for g in range(2):
                    gc = g if side == 0 else e + g
                    if typ == BC_PERIODIC:
                        sc = gc + self.n[d] if side == 0 else gc - self.n[d]
                    else:
                        sc = 3 - gc if side == 0 else 2 * e - gc - 1
                    idx = list(self.inner)
                    idx[ax] = gc
                    if typ == BC_FIXED:
                        u[tuple(idx)] = self.fix[tuple(idx)]
                        continue
                    src = list(self.inner)
                    src[ax] = sc
                    q = u[tuple(src)].clone()
                    if typ == BC_REFLECTIVE:
                        q[1 + d] = -q[1 + d]
                    elif typ == BC_OUTFLOW:
                        m = q[1 + d]
                        mc = torch.clamp(m, max=0.0) if side == 0 else torch.clamp(m, min=0.0)
                        rho = torch.clamp(q[0], min=self.p.dfloor)
                        eint = torch.clamp(q[4] - 0.5 * m * m / rho, min=1e-16)
                        q[0], q[1 + d], q[4] = rho, mc, eint + 0.5 * mc * mc / rho
                    u[tuple(idx)] = q
        if self.fix is not None:
            a = u[self.inner]
            u[self.inner] = torch.where(self.keep, self.fix[self.inner], a)

    def prim(self, u):
        rho = torch.clamp(u[0], min=self.p.dfloor)
        v = u[1:4] / rho
        ke = 0.5 * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) / rho
        pre = torch.clamp((self.p.gamma - 1.0) * (u[4] - ke), min=self.p.pfloor)
        return torch.cat([rho[None], v, pre[None]])

    def _cmax(self):
        w = self.prim(self.u[self.inner])
        cs = torch.sqrt(self.p.gamma * w[4] / w[0])
        dims = 1 + (self.p.ny > 1) + (self.p.nz > 1)
        return max(float((w[1 + d].abs() + cs).max()) for d in range(3 if dims == 3 else 2))

    @staticmethod
    def half_slope(w, ax):
        a = w - torch.roll(w, 1, ax)
        b = torch.roll(a, -1, ax)
        m = a * b
        return torch.where(m > 0, m / torch.where(m > 0, a + b, torch.ones_like(m)), torch.zeros_like(m))

    def hllc(self, l, r, n):
        gam = self.p.gamma
        rl, vl, pl, rr, vr, pr = l[0], l[1 + n], l[4], r[0], r[1 + n], r[4]
        al, ar = torch.sqrt(gam * pl / rl), torch.sqrt(gam * pr / rr)
        ps = torch.clamp(0.5 * (pl + pr) - 0.125 * (vr - vl) * (rl + rr) * (al + ar), min=0.0)
        cq = 0.5 * (1 + 1 / gam)
        sl = vl - al * torch.sqrt(1 + cq * torch.clamp(ps / pl - 1, min=0.0))
        sr = vr + ar * torch.sqrt(1 + cq * torch.clamp(ps / pr - 1, min=0.0))
        ss = (pr - pl + rl * vl * (sl - vl) - rr * vr * (sr - vr)) / (rl * (sl - vl) - rr * (sr - vr))
        left = ss >= 0
        w = torch.where(left, l, r)
        s = torch.where(left, sl, sr)
        s0 = torch.where(left, torch.clamp(sl, max=0.0), torch.clamp(sr, min=0.0))
        v = w[1 + n]
        c = s0 * (ss - v) / (s - ss)
        e = w[4] / (gam - 1) + 0.5 * w[0] * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3])
        f1 = w[0] * (v + c)
        f = [f1] + [f1 * w[1 + d] for d in range(3)] + [(e + w[4]) * (v + c) + w[0] * c * ss * (s - v)]
        f[1 + n] = w[0] * (v * v + c * s) + w[4]
        return torch.stack(f)

    def flux_difference(self, u, dt):
        w = self.prim(u)
        total = 0.0
        hy = self.half_slope(w, 2) if self.n[1] > 1 else None
        for d in range(3):
            if self.n[d] <= 1:
                continue
            ax = 3 - d
            h = self.half_slope(w, 3) if d == 0 else hy  # the z sweep slopes along y too
            f = self.hllc(torch.roll(w + h, 1, ax), w - h, d)
            total = total + (torch.roll(f, -1, ax) - f)[self.inner] * (dt / self.d[d])
        return total

    def floors(self, a):
        low = a[0] < self.p.dfloor
        ke = 0.5 * (a[1] * a[1] + a[2] * a[2] + a[3] * a[3]) / torch.where(low, torch.ones_like(a[0]), a[0])
        pre = (self.p.gamma - 1.0) * (a[4] - ke)
        a[4] = torch.where(pre < self.p.pfloor, self.p.pfloor / (self.p.gamma - 1.0) + ke, a[4])
        if bool(low.any()):
            empty = torch.zeros_like(a)
            empty[0], empty[4] = self.p.dfloor, self.p.pfloor / (self.p.gamma - 1.0)
            a = torch.where(low, empty, a)
        return a

    def kick(self, h):
        a = self.u[self.inner]
        for d in range(3):
            gd = self.p.grav[d]
            if gd:
                a[4] += a[1 + d] * gd * h
                a[1 + d] += a[0] * gd * h
        if self.point is not None:
            gm, x0, y0, z0, rs = self.point
            dx, dy, dz = self.x - x0, self.y - y0, self.z - z0
            k = -gm * h * (dx * dx + dy * dy + dz * dz + rs * rs) ** -1.5
            a[4] += k * (a[1] * dx + a[2] * dy + a[3] * dz)
            for d, q in enumerate((dx, dy, dz)):
                a[1 + d] += a[0] * k * q

    def step(self, limit=math.inf):
        dt = min(self.p.cfl * self.drmin / self.cmax, limit)
        self.kick(0.5 * dt)
        self.fill(self.u)
        u0 = self.u[self.inner].clone()

        def stage(a, b, c):  # the new state from a u0 + b u - c dF
            self.fill(self.u)
            df = self.flux_difference(self.u, dt)
            self.u[self.inner] = self.floors(a * u0 + b * self.u[self.inner] - c * df)

        stage(0.0, 1.0, 1.0)
        if self.p.integrator == 3:
            stage(0.75, 0.25, 0.25)
            stage(1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0)
        else:
            stage(0.5, 0.5, 0.5)
        self.kick(0.5 * dt)
        self.t += dt
        self.steps += 1
        self.cmax = self._cmax()
        return dt

    def advance(self, dtout):
        end = self.t + dtout
        while abs(end - self.t) > 1e-12:
            self.step(end - self.t)

    def cons(self):
        return self.u[self.inner]


def exact(case, seed):
    c = case
    k = c["kind"]
    if k == "learned":
        return None  # the correction is a 16-bit network's output
    if k == "ensemble":
        out = []
        for p, w in _instances(c, seed):
            s = _Plain(p, w)
            for _ in range(c["steps"]):
                s.step()
            out.append(s.cons())
        return out
    p, w = _problem(c, seed)
    s = _Plain(p, w, fixed=k == "disk", point=POINT if k == "disk" else None)
    if k == "step":
        dt = s.step()
        return {"cons": s.cons()[[0, 1, 2, 4, 3], 0], "dt": dt}
    if k == "tube":
        s.advance(c["tmax"])
    elif "dtout" in c:
        s.advance(c["dtout"])
    else:
        for _ in range(c["steps"]):
            s.step()
    return {"cons": s.cons(), "t": s.t}
