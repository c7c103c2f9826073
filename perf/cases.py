"""The work a user has this framework do, as timed cases.

Three kinds of pass, each through the public API:

- ``run``: the time loop of one run, as ``KHRun.run`` drives it: some steps,
  then the energy check (and, where the run records it, the k = 1 amplitude).
- ``batch``: some steps of a ``KHBatch``, the form campaigns and the server
  advance many runs in.
- ``diag``: the on-device diagnostics a run takes at an export: energy,
  amplitudes (plain and shear-weighted) and the Gauss-law residual.

``exact`` restates the step and the diagnostics in plain torch at 64 bits,
without this repository's code.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from kh_simulations_b200.batch import KHBatch
from kh_simulations_b200.config import loads
from kh_simulations_b200.run import KHRun

DEV = "cuda"
TWO_PI = 2.0 * math.pi

# The grids of the uneven parameter sweep (NX x NZ), drawn uniformly.
SWEEP_NX = (128, 256, 512, 1024)
SWEEP_NZ = (256, 512, 1024, 2048)


def listed():
    return [
        # the smallest grid in use (the smoke run's), unfiltered: launch latency
        {"name": "run_64x96", "kind": "run", "nz": 64, "nx": 96, "steps": 10, "stages": "plain"},
        # ragged and bounded: wall boundaries in x, odd NX and NZ (no row is 16-byte aligned)
        {"name": "run_walls_243x371", "kind": "run", "nz": 243, "nx": 371, "steps": 10, "stages": "walls"},
        # the benchmark's small run: modes above NZ/3 subtracted every step, energy every 10 steps
        {"name": "run_256x512_dft", "kind": "run", "nz": 256, "nx": 512, "steps": 10, "stages": "dft"},
        # the resolution study's baseline: every stage (sponge, z-mean, band, hyperdiffusion), amplitude recorded
        {"name": "run_256x768_production", "kind": "run", "nz": 256, "nx": 768, "steps": 20, "stages": "production"},
        # an ordinary run with the kz = 0 modes removed
        {"name": "run_512x1024_kz0", "kind": "run", "nz": 512, "nx": 1024, "steps": 10, "stages": "kz0"},
        # the filter benchmark's grid, both filter engines, kz = 0 removed
        {"name": "run_1024x2048_dft", "kind": "run", "nz": 1024, "nx": 2048, "steps": 2, "stages": "dft_kz0"},
        {"name": "run_1024x2048_tf32", "kind": "run", "nz": 1024, "nx": 2048, "steps": 4, "stages": "tf32_kz0"},
        # the headline benchmark's grid: far larger than L2
        {"name": "run_4096x8192", "kind": "run", "nz": 4096, "nx": 8192, "steps": 4, "stages": "plain"},
        # an uneven parameter sweep in one batch, kz = 0 removed in half the runs
        {"name": "batch_sweep_16", "kind": "batch", "runs": 16, "mix": 1, "steps": 10},
        # a campaign at the default grid: many small runs with every stage
        {"name": "batch_campaign_24", "kind": "batch", "runs": 24, "nz": 64, "nx": 768, "steps": 10},
        # what a run measures at an export, at the study's grid and at a large one
        {"name": "diag_256x768", "kind": "diag", "nz": 256, "nx": 768},
        {"name": "diag_1024x2048", "kind": "diag", "nz": 1024, "nx": 2048},
    ]


STAGES = ("plain", "walls", "warm", "dft", "dft_kz0", "kz0", "production", "tf32", "tf32_kz0")


def _grid(rng, cells_lo, cells_hi, nz_multiple, pow2, odd):
    cells = math.exp(rng.uniform(math.log(cells_lo), math.log(cells_hi)))
    aspect = 2.0 ** rng.uniform(0.0, 2.0)  # NX / NZ
    nz = math.sqrt(cells / aspect)
    nz = 2 ** round(math.log2(nz)) if pow2 else max(nz_multiple, round(nz / nz_multiple) * nz_multiple)
    nx = max(64, round(cells / nz))
    if odd:
        return nz | 1, nx | 1
    return nz, nx - nx % 2


def draw(rng):
    while True:
        case = _draw(rng)
        cells = sum(r["nz"] * r["nx"] for r in _runs_of(case, 0))
        if case.get("steps", 1) * cells <= 4 * 4096 * 8192:  # no more work than the largest listed case
            return case


def _draw(rng):
    kind = rng.choice(("run", "run", "run", "run", "batch", "batch", "diag"))
    if kind == "batch":
        if rng.random() < 0.5:
            return {"kind": "batch", "runs": rng.randint(4, 16), "mix": rng.randrange(1 << 20), "steps": rng.choice((4, 10))}
        return {"kind": "batch", "runs": rng.randint(8, 30), "nz": rng.choice((64, 128)),
                "nx": 2 * rng.randint(96, 500), "steps": rng.choice((4, 10))}
    if kind == "diag":
        nz, nx = _grid(rng, 64 * 96, 2048 * 4096, 1, False, rng.random() < 0.3)
        return {"kind": "diag", "nz": nz, "nx": nx}
    stages = rng.choice(STAGES)
    banded = stages.startswith(("dft", "tf32")) or stages == "production"
    pow2 = stages.endswith("kz0") or stages == "production"
    hi = {"dft": 1 << 20, "dft_kz0": 1 << 20, "tf32": 1 << 23, "tf32_kz0": 1 << 23, "production": 1 << 20}
    top = hi.get(stages, 1 << 24)
    odd = not banded and not pow2 and rng.random() < 0.3
    if odd:
        top = 1 << 21
    nz, nx = _grid(rng, 64 * 96, top, 32 if banded else 1, pow2, odd)
    return {"kind": "run", "nz": nz, "nx": nx, "steps": rng.choice((2, 4, 10)), "stages": stages}


# ------------------------------------------------------------------ set-up
def _runs_of(case, seed):
    """Per run of the case: its grid, stages and physical parameters."""
    rng = random.Random(seed)
    if case["kind"] == "batch":
        if "mix" in case:
            sizes = random.Random(case["mix"])
            grids = [(sizes.choice(SWEEP_NZ), sizes.choice(SWEEP_NX), "kz0" if i % 2 else "plain")
                     for i in range(case["runs"])]
        else:
            grids = [(case["nz"], case["nx"], "production")] * case["runs"]
    else:
        grids = [(case["nz"], case["nx"], case.get("stages", "plain"))]
    out = []
    for i, (nz, nx, stages) in enumerate(grids):
        prod = stages == "production"
        lx = 6.0 * math.pi if prod else 20.0
        dx, dz = lx / nx, TWO_PI / nz
        # CFL-safe: dt sqrt(dx^-2 + dz^-2) <= 0.1 with dt = courant dx, and dt <= 0.00025, the
        # resolution study's baseline, so that a coarse run stays regular over many thousand steps
        courant = min(0.1, 0.1 / (dx * math.sqrt(dx ** -2 + dz ** -2)), 0.00025 / dx)
        out.append({
            "nz": nz, "nx": nx, "stages": stages, "prod": prod, "seed": seed * 1000 + i,
            "V0": 0.05 if prod else round(rng.uniform(0.02, 0.1), 4),
            "eps": 0.15 if prod else round(rng.uniform(0.5, 2.0), 4),
            "amp": 0.001 if prod else round(rng.uniform(0.05, 0.2), 4),
            "courant": round(courant, 6) if not prod else min(0.04, round(courant, 6)),
        })
    return out


def _ini(r):
    s = r["stages"]
    text = (f"k_mode = 1\nalpha_YM = 1.0\nrun_mode = {0 if s == 'walls' else 6}\nV0 = {r['V0']}\n"
            f"eps_override = {r['eps']}\nperturb_amp = {r['amp']}\ncourant_override = {r['courant']}\n"
            f"nz_override = {r['nz']}\nnx_override = {r['nx']}\n")
    if r["prod"]:
        text += "xi_sponge = 10\nsigma_sponge = 5\nsuppress_kz0 = 1\nhyp_diff = 5e-5\nkz_suppress_hi = 14\n"
    else:
        text += "lx_override = 20\n"
    if s == "warm":
        text += "warm_T = 0.01\n"
    if s.endswith("kz0"):
        text += "suppress_kz0 = 1\n"
    if s.startswith(("dft", "tf32")):
        text += f"kz_keep_max = {r['nz'] // 3}\n"
    if s.startswith("tf32"):
        text += "filter_engine = tf32x3\n"
    return text


def _initial(r):
    """A shear layer of two counter-streaming beams with a seeded k = 1
    perturbation and field noise: [24, NZ, NX]."""
    nz, nx = r["nz"], r["nx"]
    lx = 6.0 * math.pi if r["prod"] else 20.0
    g = torch.Generator(device=DEV).manual_seed(r["seed"] & 0x7FFFFFFF)
    st = torch.zeros((24, nz, nx), dtype=torch.float64, device=DEV)
    x = torch.arange(nx, dtype=torch.float64, device=DEV) * (lx / nx)
    z = (torch.arange(nz, dtype=torch.float64, device=DEV) * (TWO_PI / nz))[:, None]
    xi = (x - lx / 2) / r["eps"]
    env = r["amp"] * r["V0"] * torch.exp(-0.5 * r["V0"] * xi * xi)
    vz = r["V0"] * torch.tanh(xi)
    for f in range(9):  # E and B noise
        st[f] = 1e-6 * torch.randn((nz, nx), dtype=torch.float64, device=DEV, generator=g)
    st[9] = -r["V0"] * (xi.abs() - math.log(2.0) + torch.log1p(torch.exp(-2.0 * xi.abs())))  # Az1: -V0 log cosh xi
    st[10] = 1.2 * env * torch.cos(z)  # both helicities, 11 : 1
    st[11] = env * torch.sin(z)
    for b, sgn in ((12, 1.0), (18, -1.0)):
        st[b] = 1.0
        st[b + 2] = sgn * vz
        st[b + 3] = sgn
    return st


def _weight(r):
    lx = 6.0 * math.pi if r["prod"] else 20.0
    x = np.arange(r["nx"]) * (lx / r["nx"])
    w = 1.0 / np.cosh((x - lx / 2.0) / r["eps"])
    return w / w.sum()


def prepare(case, seed):
    runs = []
    specs = _runs_of(case, seed)
    for i, r in enumerate(specs):
        run = KHRun(loads(_ini(r), f"run{i}"), device=DEV)
        run.set_state(_initial(r))
        runs.append(run)
    s = {"case": case, "runs": runs}
    if case["kind"] == "batch":
        s["batch"] = KHBatch(device=DEV)
        for run in runs:
            s["batch"].add(run)
    if case["kind"] == "diag":
        s["weight"] = _weight(specs[0])
    return s


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
        return {"states": [r.state for r in state["runs"]]}
    r = state["runs"][0]
    if case["kind"] == "diag":
        g = r.gauss()
        return {"energy": r.energy(), "amp": list(r.mode_amp()), "by": list(r.circ_amp("By", k=1, weight=state["weight"])),
                "gauss": [float(v) for k in ("G", "div_E", "nonabelian", "rho", "lhs") for v in g[k]],
                "scale": float(g["Etot_scale"])}
    r.step(case["steps"])
    out = {"energy": r.energy()}
    if case["stages"] == "production":
        out["amp"] = r.mode_amp()[0]
    out["state"] = r.state
    return out


# -------------------------------------------------------------------- work
def _band_modes(r):
    s, nz = r["stages"], r["nz"]
    if s == "production":
        return 2, 14
    if s.startswith(("dft", "tf32")):
        return nz // 3 + 1, nz // 2
    return 1, 0


def work(case):
    """Compulsory traffic: per step the 24 FP64 arrays read and 23 written
    (Az1 is frozen); 15 arrays per energy, 2 per amplitude, 17 per Gauss
    residual.  FP64 operations per cell and step: about 1100 for the 24
    flux-corrected sweeps with their sources, 250 for the field update, and
    4 per filtered array and band coefficient."""
    if case["kind"] == "diag":
        n = case["nz"] * case["nx"]
        return {"bytes": 8 * n * (15 + 2 + 2 + 17), "flops": n * (35 + 16 + 16 + 120)}
    b = f = 0
    for r in _runs_of(case, 0):
        n = r["nz"] * r["nx"]
        lo, hi = _band_modes(r)
        arrs = 18 if r["stages"].endswith("kz0") or r["prod"] else 21
        b += case["steps"] * 376 * n
        f += case["steps"] * n * (1350 + 4 * 2 * (hi - lo + 1) * arrs)
        if case["kind"] == "run":
            b += 8 * n * (17 if r["prod"] else 15)
            f += 35 * n
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------- exact
# The state's arrays in order: Ex1-3, Ez1-3, By1-3, Az1-3, then n, px, pz,
# Q1-3 of beam A and of beam B.
def _pad(a, dim, periodic):
    n = a.shape[dim]
    if periodic:
        return torch.cat([a.narrow(dim, n - 3, 3), a, a.narrow(dim, 0, 3)], dim)
    lo, hi = a.narrow(dim, 0, 1), a.narrow(dim, n - 1, 1)
    return torch.cat([lo, lo, lo, a, hi, hi, hi], dim)


def _sweep(v, u, src, dt, d, dim, periodic):
    """One flux-corrected transport sweep of v along dim with velocity u."""
    n = v.shape[dim]
    lo = lambda a: a.narrow(dim, 0, a.shape[dim] - 1)  # noqa: E731
    hi = lambda a: a.narrow(dim, 1, a.shape[dim] - 1)  # noqa: E731
    U, V = _pad(u, dim, periodic), _pad(v, dim, periodic)
    e = 0.5 * (lo(U) + hi(U)) * (dt / d)
    c = e.abs().clamp(max=1.0 / 6.0)
    c = (1.0 / 3.0) * c * c
    nu = 1.0 / 6.0 + (1.0 / 3.0) * (e * e - c * c)
    mu = 0.25 - 0.5 * nu
    f = 0.5 * e * (lo(V) + hi(V))
    dif = nu * (hi(V) - lo(V))
    lor = V.narrow(dim, 1, n + 4)
    if src is not None:
        lor = lor + dt * _pad(src, dim, periodic).narrow(dim, 1, n + 4)
    lor = lor - (hi(f) - lo(f))
    lnr = lor + (hi(dif) - lo(dif))
    fad = (mu.narrow(dim, 1, n + 3) * (hi(lor) - lo(lor))).narrow(dim, 1, n + 1)
    del U, V, e, c, nu, mu, f, dif, lor
    dl = hi(lnr) - lo(lnr)
    d0 = dl.narrow(dim, 1, n + 1)
    s = torch.copysign(torch.ones_like(d0), d0)
    lim = torch.minimum(torch.minimum(s * dl.narrow(dim, 0, n + 1), fad.abs()), s * dl.narrow(dim, 2, n + 1))
    fl = s * lim.clamp(min=0.0)
    return lnr.narrow(dim, 2, n) - (hi(fl) - lo(fl))


def _back(a, dim, wall):
    """The neighbour at index - 1 (periodic, or the edge itself at a wall)."""
    if not wall:
        return torch.roll(a, 1, dim)
    return torch.cat([a.narrow(dim, 0, 1), a.narrow(dim, 0, a.shape[dim] - 1)], dim)


def _ahead(a, dim, wall):
    if not wall:
        return torch.roll(a, -1, dim)
    n = a.shape[dim]
    return torch.cat([a.narrow(dim, 1, n - 1), a.narrow(dim, n - 1, 1)], dim)


class _Exact:
    def __init__(self, r):
        f32 = lambda v: float(np.float32(v))  # noqa: E731  (a configuration holds float32 values)
        s = r["stages"]
        self.prod = r["prod"]
        self.nx, self.nz = r["nx"], r["nz"]
        lx = 6.0 * math.pi if self.prod else 20.0
        self.dx, self.dz = lx / self.nx, TWO_PI / self.nz
        self.dt = f32(r["courant"]) * self.dx
        self.eps, self.wall, self.warm = f32(r["eps"]), s == "walls", f32(0.01) if s == "warm" else 0.0
        self.kz0 = self.prod or s.endswith("kz0")
        self.hyp = f32(5e-5) if self.prod else 0.0
        self.st = _initial(r)
        lo, hi = _band_modes(r)
        self.W = None
        if hi >= lo:
            m = torch.arange(lo, hi + 1, device=DEV).float()
            z = torch.arange(self.nz, device=DEV).float()
            ph = (torch.tensor(math.pi, dtype=torch.float32, device=DEV) * 2.0 * m)[:, None] * z / float(self.nz)
            self.W = torch.cat([torch.cos(ph), torch.sin(ph)]).double()  # float32 twiddles
            self.inv2 = float(np.float32(2.0) / np.float32(self.nz))

    def _beam(self, b):
        st, dt, dx, dz, wall = self.st, self.dt, self.dx, self.dz, self.wall
        n, px, pz, q = st[b], st[b + 1], st[b + 2], [st[b + 3 + a] for a in range(3)]
        ns = n.clamp(min=0.05)
        ux, uz = px / ns, pz / ns
        sx, sz = torch.zeros_like(n), torch.zeros_like(n)
        for a in range(3):
            by = st[6 + a]
            bym = torch.roll(by, 1, 0)
            byc = 0.25 * (by + _back(by, 1, wall) + bym + _back(bym, 1, wall))
            sx -= q[a] * (0.5 * (st[a] + _back(st[a], 1, wall)) + uz * byc)
            sz -= q[a] * (0.5 * (st[3 + a] + torch.roll(st[3 + a], 1, 0)) - ux * byc)
        if self.warm > 0:
            sx -= self.warm * (_ahead(n, 1, wall) - _back(n, 1, wall)) / (2 * dx)
            sz -= self.warm * (torch.roll(n, -1, 0) - torch.roll(n, 1, 0)) / (2 * dz)
        az = [0.5 * (st[9 + a] + torch.roll(st[9 + a], 1, 0)) for a in range(3)]
        sq = [uz * (q[(a + 1) % 3] * az[(a + 2) % 3] - q[(a + 2) % 3] * az[(a + 1) % 3]) for a in range(3)]
        srcs = ((None, None), (sx, None), (None, sz), (None, sq[0]), (None, sq[1]), (None, sq[2]))
        new = []
        for k, (s1, s2) in enumerate(srcs):
            v = _sweep(st[b + k], ux, s1, dt, dx, 1, not wall)
            new.append(_sweep(v, uz, s2, dt, dz, 0, False))
        new[0].clamp_(min=0.05)
        if wall:
            new[1][:, 0] = 0.0
            new[1][:, -1] = 0.0
        return new

    def _fields(self):
        st, dt, dx, dz, wall = self.st, self.dt, self.dx, self.dz, self.wall
        if wall:
            st[3:6, :, 0] = 0.0
            st[3:6, :, -1] = 0.0
        jx, jz = [0.0] * 3, [0.0] * 3
        for b in (12, 18):
            n = st[b]
            nm = n.clamp(min=1e-10)
            vx, vz = st[b + 1] / nm, st[b + 2] / nm
            vx, vz = 0.5 * (vx + _ahead(vx, 1, wall)), 0.5 * (vz + torch.roll(vz, -1, 0))
            for a in range(3):
                nq = n * st[b + 3 + a]
                jx[a] = jx[a] - 0.5 * (nq + _ahead(nq, 1, wall)) * vx
                jz[a] = jz[a] - 0.5 * (nq + torch.roll(nq, -1, 0)) * vz
        cross = lambda p, q: [p[(a + 1) % 3] * q[(a + 2) % 3] - p[(a + 2) % 3] * q[(a + 1) % 3] for a in range(3)]  # noqa: E731
        k = cross([st[9], st[10], st[11]], [st[6], st[7], st[8]])
        for a in range(3):
            by = st[6 + a]
            st[a] += dt * (-(by - torch.roll(by, 1, 0)) / dz - k[a] - jx[a])
            st[3 + a] += dt * ((by - _back(by, 1, wall)) / dx - jz[a])
        for a in range(1 if not wall else 0, 3):  # Az1 is frozen but in the wall run
            st[9 + a] -= dt * st[3 + a]
        k = cross([st[9], st[10], st[11]], [st[0], st[1], st[2]])
        for a in range(3):
            dex = (torch.roll(st[a], -1, 0) - st[a]) / dz
            dez = (_ahead(st[3 + a], 1, wall) - st[3 + a]) / dx
            st[6 + a] -= dt * (dex - dez - k[a])

    def step(self):
        st = self.st
        fluid = self._beam(12) + self._beam(18)
        for k, v in enumerate(fluid):
            st[12 + k] = v
        del fluid
        self._fields()
        two_three = (7, 8, 1, 2, 4, 5, 10, 11, 16, 17, 22, 23)  # colours 2 and 3 of By, Ex, Ez, Az and Q
        if self.prod:
            xi = ((torch.arange(self.nx, device=DEV, dtype=torch.float64) * self.dx - self.nx * self.dx / 2) / self.eps).abs()
            dec = torch.where(xi > 10.0, torch.exp(-5.0 * (xi - 10.0) * self.dt), torch.ones_like(xi))
            for k in two_three:
                st[k] *= dec
        if self.kz0:
            for k in two_three:
                st[k] -= st[k].mean(0)
        if self.W is not None:
            for k in (6, 0, 3) + two_three + (14, 20, 13, 19, 12, 18):
                st[k] -= self.W.T @ (self.inv2 * (self.W @ st[k]))
        if self.hyp > 0:
            for k in two_three:
                a = st[k]
                st[k] = a - self.hyp * (torch.roll(a, 2, 0) - 4 * torch.roll(a, 1, 0) + 6 * a - 4 * torch.roll(a, -1, 0) + torch.roll(a, -2, 0))
        if self.kz0:
            for k in (6, 0, 3):
                st[k] = 0.0

    def energy(self):
        st = self.st
        e = 0.5 * (st[0:9] ** 2).sum(0)
        for b in (12, 18):
            e += 0.5 * (st[b + 1] ** 2 + st[b + 2] ** 2) / st[b].clamp(min=1e-10)
        return float(e.sum())

    def amps(self, re, im, w=None):
        ph = -TWO_PI / self.nz * torch.arange(self.nz, device=DEV, dtype=torch.float64)[:, None]
        c, s = torch.cos(ph), torch.sin(ph)
        a, b = self.st[re], self.st[im]
        p = torch.hypot((a * c - b * s).sum(0), (a * s + b * c).sum(0)) / self.nz
        q = torch.hypot((a * c + b * s).sum(0), (a * s - b * c).sum(0)) / self.nz
        if w is None:
            return [float(p.mean()), float(q.mean())]
        w = torch.as_tensor(w, device=DEV)
        return [float((p * w).sum()), float((q * w).sum())]

    def gauss(self):
        st, n = self.st, self.nx * self.nz
        rms = lambda a: math.sqrt(float((a * a).sum()) / n)  # noqa: E731
        ezc = [0.5 * (st[3 + a] + torch.roll(st[3 + a], 1, 0)) for a in range(3)]
        rows = [[], [], [], [], []]
        for a in range(3):
            i, j = (a + 1) % 3, (a + 2) % 3
            div = (st[a] - torch.roll(st[a], 1, 1)) / self.dx + (st[3 + a] - torch.roll(st[3 + a], 1, 0)) / self.dz
            nab = st[9 + i] * ezc[j] - st[9 + j] * ezc[i]
            rho = st[15 + a] * st[12] + st[21 + a] * st[18]
            for row, v in zip(rows, (div + nab - rho, div, nab, rho, div + nab)):
                row.append(rms(v))
        return [v for row in rows for v in row], rms(st[0:6].abs().sum(0)) / self.dx + 1e-30


def exact(case, seed):
    specs = _runs_of(case, seed)
    if case["kind"] == "batch":
        states = []
        for r in specs:
            x = _Exact(r)
            for _ in range(case["steps"]):
                x.step()
            states.append(x.st)
        return {"states": states}
    x = _Exact(specs[0])
    if case["kind"] == "diag":
        g, scale = x.gauss()
        return {"energy": x.energy(), "amp": x.amps(10, 11), "by": x.amps(7, 8, _weight(specs[0])), "gauss": g, "scale": scale}
    for _ in range(case["steps"]):
        x.step()
    out = {"energy": x.energy()}
    if case["stages"] == "production":
        out["amp"] = x.amps(10, 11)[0]
    out["state"] = x.st
    return out
