"""The performance cases of penguin_b200: what a user's program has it do.

Each case is a simulation in the hands of such a program: ``prepare`` builds the
disk, tube, box, ensemble or gradient model and its seeded state, ``run`` is one
stretch of the program's step loop through the public API, and its outputs are the
whole state the stretch leaves (for the gradient model, the final field and every
gradient).  A run goes on from where the last one on the same state ended, as a
simulation does between two outputs; the shock tube and the gradient model start
again from their initial state each time.

``exact`` is the same step in plain torch, 64 bits, written from the scheme itself:
PPM on the cubic fit of four cell averages, HLLC, Strang-ordered sweeps, orbital
advection, viscosity, planet, damping, drag and the CFL step.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from penguin_b200 import params as P
from penguin_b200.adjoint import DiskAdjoint, evolve_sigma
from penguin_b200.disk import Disk
from penguin_b200.disk3 import Disk3
from penguin_b200.ensemble import Ensemble

T0 = 70.0  # past the ten orbits over which the planet's mass is ramped up


# ------------------------------------------------------------------ the cases
def listed() -> list:
    return [
        # a shock tube solved whole: the smallest call, all latency (the 1D verification run)
        {"name": "tube_1024", "kind": "tube", "n": 1024, "t_end": 0.2},
        # a coarse disk of a parameter study, sizes that no tile divides
        {"name": "disk_126x389", "kind": "disk", "nr": 126, "nphi": 389, "q": 1e-3, "alpha": 1e-3, "h": 0.05,
         "steps": 40},
        # the planet-disk at its production size, device-resident loop
        {"name": "disk_1024x3072", "kind": "disk", "nr": 1024, "nphi": 3072, "q": 1e-3, "alpha": 1e-3, "h": 0.05,
         "steps": 20},
        # an ideal-gas disk with cooling, stepped from the host as main.cu does (dt read back every step)
        {"name": "cooled_host_512x1536", "kind": "host", "nr": 512, "nphi": 1536, "cool": 1, "steps": 20},
        # gas and dust in FP64
        {"name": "dust_384x1024", "kind": "dust", "nr": 384, "nphi": 1024, "stokes": 0.01, "steps": 20},
        # the FP32-mixed form of one large disk
        {"name": "mixed_1024x3072", "kind": "mixed", "members": 1, "nr": 1024, "seed": 0, "dust": 0, "steps": 100},
        # an ensemble of uneven disks with uneven parameters, one launch per pass for all
        {"name": "ensemble_12", "kind": "mixed", "members": 12, "nr": 0, "seed": 2024, "dust": 0, "steps": 100},
        # gas and dust in the FP32-mixed form
        {"name": "mixed_dust_682x2046", "kind": "mixed", "members": 1, "nr": 682, "seed": 0, "dust": 1, "steps": 100},
        # the spherical 3D preset at a third of its production resolution per axis
        {"name": "sphere_128x256x72", "kind": "sphere", "nr": 128, "nphi": 256, "ntheta": 72, "steps": 30},
        # a small Cartesian box, ideal gas with the total energy
        {"name": "box_48x40x36", "kind": "box", "nx": 48, "ny": 40, "nz": 36, "steps": 40},
        # the gradient of a profile misfit through 64 steps
        {"name": "gradient_256x768", "kind": "gradient", "nr": 256, "nphi": 768, "steps": 64},
        # and on a coarse disk, where the launches count
        {"name": "gradient_64x190", "kind": "gradient", "nr": 64, "nphi": 190, "steps": 64},
    ]


def _logu(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng) -> dict:
    even = lambda x: 2 * max(4, round(x / 2))  # noqa: E731
    kind = rng.choice(["tube", "disk", "disk", "host", "dust", "mixed", "mixed", "sphere", "box", "gradient"])
    if kind == "tube":
        return {"kind": kind, "n": even(_logu(rng, 128, 4096)), "t_end": round(rng.uniform(0.1, 0.2), 3)}
    if kind == "disk":
        nr = even(_logu(rng, 64, 1024))
        return {"kind": kind, "nr": nr, "nphi": int(nr * rng.uniform(2.0, 3.0)), "q": _logu(rng, 1e-5, 1e-3),
                "alpha": rng.choice([0.0, _logu(rng, 1e-4, 1e-2)]), "h": rng.uniform(0.04, 0.08), "steps": 20}
    if kind == "host":
        nr = even(_logu(rng, 64, 512))
        return {"kind": kind, "nr": nr, "nphi": int(nr * rng.uniform(2.0, 3.0)), "cool": rng.choice([0, 1, 2]),
                "steps": 20}
    if kind == "dust":
        nr = even(_logu(rng, 64, 512))
        return {"kind": kind, "nr": nr, "nphi": int(nr * rng.uniform(2.0, 3.0)), "stokes": _logu(rng, 0.005, 0.2),
                "steps": 20}
    if kind == "mixed":
        members = rng.choice([1, 1, 2, 5, 9, 16])
        return {"kind": kind, "members": members, "nr": even(_logu(rng, 96, 1024)) if members == 1 else 0,
                "seed": rng.randrange(1, 10000), "dust": rng.choice([0, 0, 1]), "steps": 50}
    if kind == "sphere":
        nr = 2 * round(_logu(rng, 32, 128) / 2)
        return {"kind": kind, "nr": nr, "nphi": 2 * nr, "ntheta": max(16, int(nr * rng.uniform(0.5, 0.5625))),
                "steps": 30}
    if kind == "box":
        return {"kind": kind, "nx": even(_logu(rng, 16, 96)), "ny": int(_logu(rng, 16, 96)),
                "nz": int(_logu(rng, 16, 96)), "steps": 40}
    nr = even(_logu(rng, 64, 256))
    return {"kind": "gradient", "nr": nr, "nphi": int(nr * rng.uniform(2.5, 3.0)), "steps": rng.randrange(24, 65)}


# --------------------------------------------------------- parameters, states
def _params(case) -> list:
    k = case["kind"]
    if k == "tube":
        return [P.sod_tube(case["n"])]
    if k == "disk":
        p = P.planet_disk(case["nr"], case["nphi"], q=case["q"], alpha=case["alpha"], h=case["h"])
        return [p.replace(visc_flag=int(case["alpha"] > 0.0))]
    if k == "host":
        return [P.adiabatic_disk(case["nr"], case["nphi"], cool_flag=case["cool"], beta_cool=0.5)]
    if k == "dust":
        return [P.dust_disk(case["nr"], case["nphi"], stokes=case["stokes"])]
    if k == "mixed":
        if case["members"] == 1:
            ps = [P.planet_disk(case["nr"], 3 * case["nr"])]
        else:
            ps = P.disk_ensemble(case["members"], case["seed"])
        if case["dust"]:
            ps = [p.replace(dust_flag=1, Stokes=0.01, D_G_ratio=0.01) for p in ps]
        return ps
    if k == "sphere":
        return [P.spherical_disk(case["nr"], case["nphi"], case["ntheta"])]
    if k == "box":
        return [P.cartesian_box(case["nx"], case["ny"], case["nz"])]
    return [P.adjoint_disk(case["nr"], case["nphi"])]


def _profiles(p, x):
    cs2 = lambda r: p.sc_h**2 * r ** (-p.p_beta)  # noqa: E731
    rho = lambda r: r ** (-p.p_alpha)  # noqa: E731
    pre = lambda r: cs2(r) * rho(r)  # noqa: E731
    dr = 1.1514178e-7
    return rho(x), cs2(x), np.sqrt(1.0 / x + x / rho(x) * (pre(x + dr) - pre(x - dr)) / (2.0 * dr))


def _states(case, seed) -> list:
    """The seeded initial state of every member: a disk some orbits old, that is a
    smooth spiral of a per cent or so over the equilibrium, and noise on it."""
    rng = np.random.default_rng([seed, 17])
    out = []
    for p in _params(case):
        if p.ndim == 1:
            # Sod's tube, the two states jittered by a per cent
            x = (np.arange(p.xres) + 0.5) / p.xres
            a = 1.0 + 0.01 * rng.uniform(-1, 1, 4)
            left = x < 0.5
            out.append({"r": np.where(left, a[0], 0.125 * a[1])[None], "p": np.where(left, a[2], 0.1 * a[3])[None],
                        "u": np.zeros((1, p.xres)), "v": np.zeros((1, p.xres))})
            continue
        (xf, _), (yf, _) = _axis(p, 0), _axis(p, 1)
        x, y = 0.5 * (xf[4:-3] + xf[3:-4]), 0.5 * (yf[4:-3] + yf[3:-4])
        if p.ndim == 2:
            s0, c2, v0 = _profiles(p, x)
            cs = np.sqrt(c2)
            ph = rng.uniform(0, 2 * math.pi, 4)
            wave = np.cos(2 * y[:, None] + 6.0 * np.log(x)[None] + ph[0])
            r = s0 * (1.0 + 0.01 * wave + 1e-4 * rng.uniform(-1, 1, (p.yres, p.xres)))
            out.append({"r": r, "p": c2 * r, "u": 0.01 * cs * np.cos(3 * y[:, None] + 5.0 * np.log(x)[None] + ph[1]),
                        "v": v0 + 0.01 * cs * np.cos(y[:, None] - 7.0 * np.log(x)[None] + ph[2])})
            continue
        zf, _ = _axis(p, 2)
        z = 0.5 * (zf[4:-3] + zf[3:-4])
        X, Y, Z = x[None, None], y[None, :, None], z[:, None, None]
        shape = (p.zres, p.yres, p.xres)
        noise = rng.uniform(-1, 1, (5,) + shape)
        ph = rng.uniform(0, 2 * math.pi, 4)
        if p.geomx == 0:
            # a blast in a turbulent box
            blob = 2.0 * np.exp(-((X - 0.3) ** 2 + (Y - 0.6) ** 2 + (Z - 0.2) ** 2) / 0.02)
            out.append({"r": 1.0 + 0.2 * noise[0], "p": 1.0 + 0.2 * noise[1] + blob,
                        "u": 0.1 * noise[2], "v": 0.1 * noise[3], "w": 0.1 * noise[4]})
            continue
        rho, c2, v0 = _sphere_state(p, X, Z)
        cs = np.sqrt(c2)
        r = rho * (1.0 + 0.01 * np.cos(2 * Y + 6.0 * np.log(X) + ph[0]) + 1e-4 * noise[0])
        out.append({"r": r, "p": np.broadcast_to(c2, shape) * r,
                    "u": 0.01 * cs * np.cos(3 * Y + 5.0 * np.log(X) + ph[1]),
                    "v": v0 + 0.01 * cs * np.cos(Y - 7.0 * np.log(X) + ph[2]),
                    "w": 0.01 * cs * np.cos(2 * Y + 20.0 * (Z - 0.5 * math.pi) + ph[3])})
    return [{k: np.ascontiguousarray(v, dtype=np.float64) for k, v in s.items()} for s in out]


def _dust(p, s) -> dict:
    """Dust at a hundredth of the gas density, drifting with the gas."""
    return {"r": p.D_G_ratio * s["r"], "u": s["u"] - 0.01 * p.sc_h * p.sc_h, "v": s["v"]}


class _Cells:
    """The disk's device state as a tensor's memory: 5 FP64 values a cell, ghosts
    included.  The tensor holds this object, and this object the disk that owns it."""

    def __init__(self, disk):
        self.disk = disk
        shape = (disk.params.yarr, disk.params.xarr, 5)
        self.__cuda_array_interface__ = {"data": (disk.state_ptr(), False), "shape": shape, "typestr": "<f8", "version": 2}


def prepare(case, seed):
    k = case["kind"]
    ps, ss = _params(case), _states(case, seed)
    s = {"case": case, "kind": k, "params": ps}
    if k in ("tube", "disk", "host", "dust"):
        s["disk"] = Disk(ps[0])
        s["init"] = ss[0]
        if k != "tube":
            s["disk"].set_state(T0, ss[0])
        if k == "dust":
            s["disk"].set_dust(_dust(ps[0], ss[0]))
    elif k == "mixed":
        s["ens"] = Ensemble(ps)
        for n, (p, st) in enumerate(zip(ps, ss)):
            s["ens"].set_state(n, T0, st)
            if p.dust_flag:
                s["ens"].set_dust(n, _dust(p, st))
    elif k in ("sphere", "box"):
        s["disk"] = Disk3(ps[0])
        s["disk"].set_state(T0, ss[0])
    else:
        p = ps[0]
        s["model"] = DiskAdjoint(p, nsteps=case["steps"], t0=T0)
        s["sigma0"] = torch.tensor(ss[0]["r"], device="cuda").requires_grad_(True)
        s["theta"] = torch.tensor(_theta(p), dtype=torch.float64, device="cuda").requires_grad_(True)
        s["target"] = torch.tensor(_target(p), dtype=torch.float64, device="cuda")
    return s


def _theta(p):
    return [p.planet_mass, p.ss_alpha, p.sc_h]


def _target(p):
    x = _axis(p, 0)[0]
    x = 0.5 * (x[4:-3] + x[3:-4])
    return _profiles(p, x)[0] * (1.0 + 0.05 * np.cos(9.0 * np.log(x)))


def _misfit(sigma, target):
    return ((sigma.mean(0) - target) ** 2).sum()


def run(s):
    k, case = s["kind"], s["case"]
    if k == "tube":
        s["disk"].set_state(0.0, s["init"])
        s["disk"].run(8 * case["n"], end_time=case["t_end"])
        out = s["disk"].get_state()
        return {"r": out["r"], "p": out["p"], "u": out["u"]}
    if k in ("disk", "host", "dust"):
        d = s["disk"]
        if k == "host":
            d.step_host(case["steps"])
        else:
            d.run(case["steps"])
        cells = torch.as_tensor(_Cells(d), device="cuda")
        out = {"cells": cells[3:-3, 3:-3, :4]}  # r, p, u, v of the interior
        if k == "dust":
            out["dust"] = d.get_dust()
        return out
    if k == "mixed":
        s["ens"].run(case["steps"])
        out = []
        for n, p in enumerate(s["params"]):
            g = s["ens"].get_state(n)
            out.append({"r": g["r"], "u": g["u"], "v": g["v"]})
            if p.dust_flag and len(s["params"]) <= 10:
                out[-1]["dust"] = s["ens"].get_dust(n)
        return out
    if k in ("sphere", "box"):
        s["disk"].run(case["steps"])
        out = s["disk"].get_state()
        return {f: out[f] for f in "rpuvw"}
    s["sigma0"].grad = s["theta"].grad = None
    sigma = evolve_sigma(s["sigma0"], s["theta"], s["model"])
    _misfit(sigma, s["target"]).backward()
    return {"sigma": sigma.detach(), "grad_sigma0": s["sigma0"].grad, "grad_theta": s["theta"].grad}


def work(case) -> dict:
    """Per step, each cell's state read and written once, and the arithmetic of the
    scheme counted once per cell: about 400 operations a sweep (five parabolas, two
    traced edge states, one HLLC flux, the update), 120 for the residual advection,
    100 for each half-kick with its stress."""
    k = case["kind"]
    ps = _params(case)
    cells = sum(p.cells for p in ps)
    p = ps[0]
    if k == "tube":
        steps, fields, flops, size = 1.0 * case["n"] * case["t_end"] * 4.5, 3, 400, 8
    else:
        steps, size = case["steps"], 4 if k == "mixed" else 8
        sweeps = 3 if p.ndim == 3 else 2
        fields = {2: 3, 3: 4}[p.ndim] + int(p.EOS_flag == 2) + 3 * p.dust_flag
        flops = 400 * sweeps + 200 + (120 if p.ndim == 2 else 0) + 300 * p.dust_flag
    if k == "gradient":  # the forward, its recomputation between checkpoints and the transposed passes
        flops, fields = 5 * flops, 3 * fields
    return {"bytes": 2.0 * size * fields * cells * steps, "flops": 1.0 * flops * cells * steps}


def tolerance(case) -> dict:
    """About four times what this package and the plain step below, two evaluations of
    one scheme in other orders, were seen to differ by over the listed and drawn cases.
    Most of it is no rounding of the step itself: the reconstruction weights carry the
    rounding of their grid moments, v_phi a numerical pressure derivative, and the
    planet's tight pull and the limiters carry both on."""
    return {
        "tube": {"rel": 5e-8, "max": 1e-6},  # seen 1.1e-8, 1.7e-7
        "disk": {"rel": 8e-7, "max": 6e-5},  # 1.8e-7, 1.4e-5
        "host": {"rel": 5e-7, "max": 2e-5},  # 1.3e-7, 4.9e-6
        "dust": {"rel": 2e-7, "max": 5e-5},  # 3.7e-8, 1.1e-5
        "mixed": {"rel": 4e-4, "max": 6e-2},  # 9.1e-5, 1.5e-2: 32-bit residuals, the worst in v_r
        "sphere": {"rel": 5e-3, "max": 1e-1},  # 1.3e-3, 2.2e-2: cells of 1e-3 of the coordinate
        "box": {"rel": 2e-11, "max": 2e-9},  # 4.2e-12, 4.2e-10
        "gradient": {"rel": 2.5e-3, "max": 2e-1},  # 5.9e-4: the flattening at pressure extrema
    }[case["kind"]]


# ------------------------------------------------------------ the plain step
PAD = 3


def _axis(p, axis):
    """Faces with three ghosts a side, and cell volumes, of one axis."""
    amin, amax, n, grid, geom = ((p.xmin, p.xmax, p.xres, p.gridx, p.geomx), (p.ymin, p.ymax, p.yres, p.gridy, p.geomy),
                                 (p.zmin, p.zmax, p.zres, p.gridz, p.geomz))[axis]
    i = np.arange(-PAD, n + PAD + 1, dtype=np.float64)
    if grid == 1:
        a = amin * np.exp(math.log(amax / amin) * i / n)
    elif grid == 0:
        a = amin + (amax - amin) * i / n
    else:
        a = np.zeros(n + 7)
        a[3:-3] = _stretched(p, grid, amin, amax, n)
    if grid != 1:  # the ghosts mirror the cells at the edge
        a[2::-1] = 2 * a[3] - a[4:7]
        a[-3:] = 2 * a[-4] - a[-5:-8:-1]
    d = np.diff(a)
    if geom == 1:
        v = d * (a[:-1] + d / 2)
    elif geom == 2:
        v = d * (a[:-1] ** 2 + a[:-1] * d + d * d / 3)
    elif geom == 5:
        v = np.where(d < 1e-4, np.sin(a[:-1] + 0.5 * d) * d, np.cos(a[:-1]) - np.cos(a[:-1] + d))
    else:
        v = d
    return a, v


def _stretched(p, grid, amin, amax, n):
    """The non-uniform axes: cells grow as a power law away from the middle (2, 4)
    or from the upper end (3) over the extent L with the smallest cell dmin."""
    def half(L, N, dmin, dmax):
        k = math.log(1 - (dmax - dmin) / (L - N * dmin)) / math.log(1 - 1 / N)
        m = np.arange(N + 1)
        return m * dmin + (L - N * dmin) * (m / N) ** k

    mid = 0.5 * (amin + amax)
    if grid == 2:
        N, L = n // 2, 0.5 * (amax - amin)
        g = half(L, N, L / N / 32, (math.pi - L) / N)
        return np.concatenate([mid - g[:0:-1], mid + g])
    if grid == 3:
        g = half(amax - amin, n, (p.xmax - p.xmin) / p.xres / 32, p.sc_h / 16)
        return amax - g[::-1]
    N = p.xres // 2
    N2, L = (n - 2 * N) // 2, 0.5 * (p.xmax - p.xmin)
    L2 = 0.5 * (amax - amin - 2 * L)
    g = half(L, N, L / N / 32, L2 / N2)
    side = np.arange(N2 + 1) * (L2 / N2)
    return np.concatenate([amin + side[:-1], mid - g[:0:-1], mid + g, amin + 2 * L + L2 + side[1:]])


def _weights(a, geom):
    """Per cell, the weights on the differences of neighbouring averages that give
    the jumps from the cell's average to its two faces of the cubic that has the
    averages of four cells (two below and one above for the left face, and the
    mirror of that).  Moments by 5-point Gauss quadrature on scaled coordinates."""
    n = len(a) - 1
    w = np.zeros((n, 6))
    gx, gw = np.polynomial.legendre.leggauss(5)
    i = np.arange(2, n - 2)
    for side, first in ((0, -2), (1, -1)):
        face = a[i + side]
        h = a[i + 1] - a[i]
        M = np.zeros((len(i), 4, 4))
        for c in range(4):
            lo, hi = a[i + first + c], a[i + first + c + 1]
            x = 0.5 * (lo + hi)[:, None] + 0.5 * (hi - lo)[:, None] * gx
            jac = gw * (x if geom == 1 else x * x if geom == 2 else np.ones_like(x))
            xi = (x - face[:, None]) / h[:, None]
            for m in range(4):
                M[:, c, m] = (jac * xi**m).sum(1) / jac.sum(1)
        k = np.linalg.solve(np.swapaxes(M, 1, 2), np.broadcast_to(np.array([1.0, 0, 0, 0])[:, None], (len(i), 4, 1)))
        k = k[..., 0]  # the face value's weights on the four averages
        if side == 0:
            k = -k
            k[:, 2] += 1.0
        else:
            k[:, 1] -= 1.0
        w[i, 3 * side:3 * side + 3] = -np.cumsum(k, 1)[:, :3]
    return w


def _sh(a, k, n):
    return a[..., k:k + n]


def _where(c, a, b):
    return torch.where(c, a, b)


def _recon(w, a, flat, n):
    """Limited slopes (sL, a, sR) of cells 2 .. n+1 of the last axis of n + 4."""
    q = [_sh(a, k, n) for k in range(5)]
    d = [q[k + 1] - q[k] for k in range(4)]
    sL = w[0] * d[0] + w[1] * d[1] + w[2] * d[2]
    sR = w[3] * d[1] + w[4] * d[2] + w[5] * d[3]
    sL = _where(sL.abs() < d[1].abs(), sL.abs(), d[1].abs()) * torch.sign(d[1])
    sR = _where(sR.abs() < d[2].abs(), sR.abs(), d[2].abs()) * torch.sign(d[2])
    keep = (sR * sL > 0).to(sL.dtype) * (1.0 - flat)
    sL, sR = sL * keep, sR * keep
    t = sR + sL
    t2, t1 = t * t, t * 3.0 * (sL - sR)
    return _where(t2 < t1, 2.0 * sR, sL), q[2], _where((t2 >= t1) & (t2 < -t1), 2.0 * sL, sR)


def _aveL(x, s):
    return s[1] - s[0] + 0.5 * x * (s[2] + s[0] + (1.0 - x / 1.5) * 3.0 * (s[0] - s[2]))


def _aveR(y, s):
    return s[1] + s[2] - 0.5 * y * (s[2] + s[0] - (1.0 - y / 1.5) * 3.0 * (s[0] - s[2]))


def _exp(x):
    return torch.clamp(1.0 + x, min=1e-6)


def _fluxes(g, ax, sdt, F, ie, eos):
    """PPM, characteristic tracing and HLLC along the last axis: F are r, p, u and the
    two transverse fields on n + 6 cells; the seven fluxes on n + 1 faces."""
    N = F[0].shape[-1] - 4
    w, dx = ax["w"][:, 2:-2], ax["dx"][2:-2]
    r, p, u = F[:3]
    pm2, pm1, p0, pp1, pp2 = (_sh(p, k, N) for k in range(5))
    um1, u0, up1 = (_sh(u, k, N) for k in (1, 2, 3))
    f1, f2, b1, b2 = pp1 - p0, pp2 - pm1, p0 - pm1, pp1 - pm2
    shock = ((u0 - up1 > 0) | (um1 - u0 > 0)) & (f2 != 0) & (b2 != 0)
    one = torch.ones_like(f2)
    steep = lambda a, b: 10.0 * torch.clamp((a / _where(b != 0, b, one) - 0.5).abs() - 0.25, min=0.0)  # noqa: E731
    sf, sb = steep(f1, f2), steep(b1, b2)
    big = _where(f1.abs() > b1.abs(), f1.abs(), b1.abs())
    flat = _where(sf > sb, sf, sb) * big / p0
    flat = _where(shock, torch.clamp(flat, max=0.5), torch.zeros_like(flat))
    S = [_recon(w, a, flat, N) for a in F]
    r0 = _sh(r, 2, N)
    cs0 = torch.sqrt(g * p0 / r0)
    half = []
    for ave, sg in ((_aveL, 1.0), (_aveR, -1.0)):  # state at the left edge, then at the right edge
        # the swept fraction of the cell at a speed, and the speed towards the edge
        frac = lambda v: torch.clamp(v * sdt / dx, 0.0, 1.0)  # noqa: E731
        away = lambda q: torch.clamp(-sg * q, min=0.0)  # noqa: E731
        ue = ave(frac(away(u0) + cs0), S[2])
        x1 = frac(away(ue))
        rr, pp, uu = (ave(x1, S[m]) for m in (0, 1, 2))
        rr = _where(rr > r0 * 1e-10, rr, r0 * 1e-10)
        pp = _where(pp > p0 * 1e-10, pp, p0 * 1e-10)
        c = torch.sqrt(g * pp / rr)
        x2 = frac(away(ue) + c)
        du, dp = sg * (ave(x2, S[2]) - uu) / c, sg * (ave(x2, S[1]) - pp) / c
        half.append((rr * _exp(-du), pp * _exp(-g * du), uu - dp / rr, ave(x2, S[3]), ave(x2, S[4])))
    L = [a[..., :-1] for a in half[1]]
    R = [a[..., 1:] for a in half[0]]
    cl, cr = torch.sqrt(g * L[1] / L[0]), torch.sqrt(g * R[1] / R[0])
    pm = 0.5 * (L[1] + R[1]) * _exp(0.5 * g * (L[2] - R[2]) / (0.5 * (cl + cr)))
    ql, qr = torch.sqrt(L[0]), torch.sqrt(R[0])
    um = (ql * L[2] + qr * R[2]) / (ql + qr)
    cc = torch.sqrt((cl * cl * ql + cr * cr * qr) / (ql + qr) + 0.5 * ql * qr / (ql + qr) ** 2 * (R[2] - L[2]) ** 2)
    sl, sr = um - cc, um + cc
    sm = (L[0] * L[2] * cl + R[0] * R[2] * cr) / (L[0] * cl + R[0] * cr)
    sm = sm + (L[1] - R[1]) / ((L[0] + R[0]) * 0.5 * (cl + cr))
    left = (sl >= 0) | ((sr >= 0) & (sm >= 0))
    U = [_where(left, a, b) for a, b in zip(L, R)]
    fast = (sl >= 0) | (sr < 0)
    s = _where(left, sl, sr)
    inv = 1.0 / _where(fast, torch.ones_like(s), s - sm)
    fr = _where(fast, U[0] * U[2], sm * U[0] * (s - U[2]) * inv)
    pres = _where(fast, U[1], (s * pm - sm * U[1]) * inv)
    fp = uprs = torch.zeros_like(fr)
    if eos == 2:
        e = U[1] / ((g - 1.0) * U[0])
        if ie:
            den = _where(fast, torch.ones_like(s), s * pm - sm * U[1])
            uprs = _where(fast, U[2], sm * (s * pm - U[2] * U[1]) / den)
        else:  # the total energy's flux carries the sweep's own kinetic energy
            e = e + 0.5 * U[2] ** 2
            uprs = _where(fast, U[2] * U[1], sm * (s * pm - U[2] * U[1]) * inv)
        fp = e * fr
    return fr, fp, U[2] * fr, U[3] * fr, U[4] * fr, pres, uprs


def _net(fl, gf, eos, ie):
    """Flux differences and pressure sources of each cell (face areas gf)."""
    a, b = slice(0, -1), slice(1, None)
    D = [f[..., a] * gf[a] - f[..., b] * gf[b] for f in fl[:5]]
    p0, p1 = fl[5][..., a], fl[5][..., b]
    D[2] = D[2] + 0.5 * (gf[a] + gf[b]) * (p0 - p1)
    if eos == 2:
        t = fl[6][..., a] * gf[a] - fl[6][..., b] * gf[b]
        D[1] = D[1] + (0.5 * (p0 + p1) * t if ie else t)
    return D


def _update(p, c2, Q, D):
    """Conservative update of (r, p, u, v, w)."""
    r, pr, vel = Q[0], Q[1], Q[2:]
    rn = r + D[0]
    vn = [(a * r + d) / rn for a, d in zip(vel, D[2:])]
    if p.EOS_flag != 2:
        return [rn, c2 * rn] + vn
    gm = p.gam - 1.0
    if p.internal_e_flag:
        pn = (pr / gm + D[1]) * gm
    else:
        e = pr / gm + 0.5 * r * sum(a * a for a in vel)
        pn = (e + D[1]) * gm - gm * rn * sum(a * a for a in vn) / 2.0
    return [rn, pn] + vn


class _Step:
    """Grid, tables and the pieces shared by the two- and three-dimensional steps."""

    def __init__(self, p, dev, theta=None):
        self.p, self.dev = p, dev
        self.q, self.al, self.h = theta if theta is not None else (self.t(v) for v in _theta(p))
        self.ax = []
        for axis in range(p.ndim):
            a, v = _axis(p, axis)
            geom = (p.geomx, p.geomy, p.geomz)[axis]
            w = _weights(a, geom)
            self.ax.append({"a": self.t(a), "v": self.t(v), "dx": self.t(np.diff(a)), "c": self.t(0.5 * (a[1:] + a[:-1])),
                            "w": self.t(w.T.copy())})

    def t(self, v):
        return torch.as_tensor(v, dtype=torch.float64, device=self.dev)

    def ramp(self, x):
        """Damping rate of each interior radius: (sin^2 ramp) / r^1.5 at either end."""
        p = self.p
        h0 = lambda r: self.h * r  # noqa: E731  (flat aspect ratio)
        din, dout = h0(p.xmin) * p.kill_width, h0(p.xmax) * p.kill_width_out
        f = lambda y: torch.sin(0.5 * math.pi * torch.clamp(y, min=0.0)) ** 2  # noqa: E731
        return (f((p.xmin + din - x) / din) + f((x - p.xmax + dout) / dout)) / x**1.5

    def planet(self, t):
        p = self.p
        m = self.q * math.sin(0.5 * math.pi * t / p.ramp_time) if t < p.ramp_time else self.q
        return m, math.fmod(t, 2 * math.pi) - math.fmod(p.frame_omega * t, 2 * math.pi) + math.pi


def _pad_x(Q, lft, rgh, init):
    """Radial ghosts of (r, p, u, ...): 0 the analytic state, 1 zero gradient, 2 mirror."""
    out = []
    for m, a in enumerate(Q):
        sg = -1.0 if m == 2 else 1.0
        shape = a.shape[:-1] + (PAD,)
        lo = {0: lambda: init[m][..., :PAD].expand(shape), 1: lambda: a[..., :1].expand(shape),
              2: lambda: sg * a[..., :PAD].flip(-1)}[lft]()
        hi = {0: lambda: init[m][..., -PAD:].expand(shape), 1: lambda: a[..., -1:].expand(shape),
              2: lambda: sg * a[..., -PAD:].flip(-1)}[rgh]()
        out.append(torch.cat([lo, a, hi], -1))
    return out


def _wrap(a):
    """Periodic ghosts on the first axis, which is then moved to the end."""
    return torch.cat([a[-PAD:], a, a[:PAD]], 0).transpose(0, -1)


def _tube(p, s, t_end, dev):
    S = _Step(p, dev)
    ax = S.ax[0]
    Q = [S.t(s[k]) for k in "rpu"]
    Q += [torch.zeros_like(Q[0]), torch.zeros_like(Q[0])]
    one = torch.ones(p.xres + 1, dtype=torch.float64, device=dev)
    t, cap = 0.0, t_end
    while t < t_end:
        rate = ((Q[2].abs() + torch.sqrt(p.gam * Q[1] / Q[0])) / ax["dx"][3:-3]).max().item()
        dt = min(p.CFL / rate, 1.1 * cap)
        last = t + dt > t_end
        dt = t_end - t if last else dt
        fl = _fluxes(p.gam, ax, dt, _pad_x(Q, p.bound_lft, p.bound_rgh, None), p.internal_e_flag, 2)
        D = _net(fl, one, 2, p.internal_e_flag)
        Q = _update(p, None, Q, [d * dt / ax["v"][3:-3] for d in D])
        t, cap = t + dt, dt
        if last:
            break
    return Q


class _Polar(_Step):
    """The two-dimensional polar step."""

    def __init__(self, p, dev, theta=None):
        super().__init__(p, dev, theta)
        x = self.ax[0]["c"]
        self.x, self.xi = x, x[3:-3]
        cs2 = lambda r: self.h**2 * r ** (-p.p_beta)  # noqa: E731
        rho = lambda r: r ** (-p.p_alpha)  # noqa: E731
        dr = 1.1514178e-7
        dP = (cs2(x + dr) * rho(x + dr) - cs2(x - dr) * rho(x - dr)) / (2 * dr)
        # pressure gradient in closed form for derivatives with respect to h
        dP = dP if theta is None else -(p.p_alpha + p.p_beta) * cs2(x) * rho(x) / x
        self.cs2 = cs2(x)
        self.nu = self.al * self.h**2 * x**p.p_alpha if p.visc_flag else torch.zeros_like(x)
        v0 = torch.sqrt(1.0 / x + x / rho(x) * dP)
        u0 = -1.5 * self.nu / x
        self.init = [rho(x), self.cs2 * rho(x), u0, v0, torch.zeros_like(x)]
        self.rot = v0 - x * p.frame_omega
        self.yc = self.ax[1]["c"][3:-3]
        self.damp = self.ramp(self.xi) if p.kill_flag else None
        if p.dust_flag:
            f = v0 * torch.sqrt(x)
            st = p.Stokes
            b = st * st * f
            Lr = (1 + b) / b * (1 - torch.sqrt(1 - 2 * b * (1 - f) / (1 + b) ** 2))
            uu = (1 - torch.sqrt(1 - 2 * st * (st * (Lr * Lr - 2 * Lr)))) / st
            Lr = (1 - f + st * uu / 2) / (1 + st * uu / 2)
            uu = (1 - torch.sqrt(1 - 2 * st * (st * (Lr * Lr - 2 * Lr)))) / st
            self.dinit = [p.D_G_ratio * rho(x), None, uu * torch.sqrt(1 / x), torch.sqrt(1 / x)]

    def stress(self, Q):
        """Viscous force density of the interior from (r, u, v) with ghosts all round."""
        p = self.p
        if not p.visc_flag:
            return None
        r, u, v = (torch.cat([a[-1:], a, a[:1]], 0)[:, 2:-2] for a in (Q[0], Q[2], Q[3]))
        x = self.x[2:-2]
        n = r * self.nu[2:-2]
        y = self.ax[1]["c"][2:-2]
        x0, x1, x2 = x[:-2], x[1:-1], x[2:]
        y0, y1, y2 = y[:-2, None], y[1:-1, None], y[2:, None]

        def at(a, i, j):
            return a[1 + j:a.shape[0] - 1 + j, 1 + i:a.shape[1] - 1 + i]

        def dx(a, j=0):
            return (at(a, 1, j) - at(a, -1, j)) / (x2 - x0)

        def dy(a):
            return (at(a, 0, 1) - at(a, 0, -1)) / (y2 - y0) / x1

        def dxx(a):
            return ((at(a, 1, 0) - at(a, 0, 0)) / (x2 - x1) - (at(a, 0, 0) - at(a, -1, 0)) / (x1 - x0)) / (0.5 * (x2 - x0))

        def dyy(a):
            return ((at(a, 0, 1) - at(a, 0, 0)) / (y2 - y1) - (at(a, 0, 0) - at(a, 0, -1)) / (y1 - y0)) / (0.5 * (y2 - y0)) / x1 / x1

        def dxy(a):
            return (at(a, 1, 1) - at(a, -1, 1) - at(a, 1, -1) + at(a, -1, -1)) / (x2 - x0) / (y2 - y0) / x1

        N, U, V = at(n, 0, 0), at(u, 0, 0), at(v, 0, 0)
        sxx = 2 * N * dx(u)
        syy = 2 * N * (dy(v) + U / x1)
        sxy = N * (dy(u) + dx(v) - V / x1)
        fx = 2 * dx(n) * dx(u) + 2 * N * dxx(u) + sxx / x1 + dy(n) * (dy(u) + dx(v)) + N * (dyy(u) + dxy(v)) \
            - dy(n) * V / x1 - N * dy(v) / x1 - syy / x1
        fy = 2 * dy(n) * dy(v) + 2 * N * dyy(v) + 2 * N * dy(u) / x1 + 2 * dy(n) * U / x1 + dx(n) * (dy(u) + dx(v)) \
            + N * (dxy(u) + dxx(v)) - dx(n) * V / x1 - N * dx(v) / x1 + N * V / x1 / x1 + 2 * sxy / x1
        return fx, fy

    def gravity(self, body):
        p, (m, y) = self.p, body
        x, a = self.xi, p.planet_radius
        rs = p.rs_fac * self.h * a
        s, c = torch.sin(self.yc - y)[:, None], torch.cos(self.yc - y)[:, None]
        f = (x * x + a * a - 2 * a * x * c + rs * rs) ** -1.5
        return -1.0 / x**2 - m * (x - a * c) * f - m * c / a**2, -m * a * s * f + m * s / a**2

    def kick(self, Q, g, vis, hdt, mdt):
        """Velocities after hdt, with the centrifugal term at the mdt prediction; the prediction too."""
        vx, vy = (0.0, 0.0) if vis is None else (vis[0] / Q[0], vis[1] / Q[0])
        u, v = Q[2], Q[3]
        if mdt:
            u = Q[2] + (Q[3] ** 2 / self.xi + vx + g[0]) * mdt
            v = Q[3] + (vy + g[1]) * mdt
        return Q[2] + (v * v / self.xi + vx + g[0]) * hdt, Q[3] + (vy + g[1]) * hdt, u, v

    def cool(self, Q, dt):
        p = self.p
        if not p.cool_flag:
            return Q[1]
        e, e0 = Q[1] / Q[0], self.cs2[3:-3]
        tc = p.beta_cool * self.xi**1.5 if p.cool_flag == 1 else p.beta_cool / Q[0] * torch.sqrt(e) / self.h
        return Q[0] * (e0 + (e - e0) * torch.exp(-dt / tc))

    def drag(self, D, Q, Tu, Tv, Tp, g, hdt, mdt):
        p = self.p
        ts = p.Stokes * self.h / torch.sqrt(p.gam * Q[1] / Q[0]) / Q[0]
        fx, fy = D[3] ** 2 / self.xi * ts + Q[2] - D[2], Q[3] - D[3]
        if mdt:
            e = -torch.expm1(-mdt / ts)
            v = D[3] + (fy + g[1] * ts) * e
            ts = p.Stokes * self.h / torch.sqrt(p.gam * Tp / Q[0]) / Q[0]
            fx, fy = v * v / self.xi * ts + Tu - D[2], Tv - D[3]
        e = -torch.expm1(-hdt / ts)
        return [D[0], None, D[2] + (fx + g[0] * ts) * e, D[3] + (fy + g[1] * ts) * e]

    def rate(self, Q, D):
        p = self.p
        cs = torch.sqrt(p.gam * Q[1] / Q[0])
        su, sv = Q[2].abs() + cs, (Q[3] - self.init[3][3:-3]).abs() + cs
        if D is not None:
            su = torch.maximum(su, D[2].abs())
            sv = torch.maximum(sv, (D[3] - self.init[3][3:-3]).abs())
        return max((su / self.ax[0]["dx"][3:-3]).max().item(),
                   (sv / self.ax[1]["dx"][3:-3, None] / self.xi).max().item())

    def pad(self, Q):
        return _pad_x(Q, self.p.bound_lft, self.p.bound_rgh, self.init)

    def advance(self, Q, D, t, dt):
        p = self.p
        ax, ay = self.ax
        x, xi, c2 = self.x, self.xi, self.cs2[3:-3]
        now, then = self.planet(t), self.planet(t + dt)
        hdt = 0.5 * dt
        # first half-kick
        g = self.gravity(now)
        vis = self.stress(self.pad(Q))
        u, v, _, _ = self.kick(Q, g, vis, hdt, 0.0)
        D = None if D is None else self.drag(D, Q, None, None, None, g, hdt, 0.0)
        Q = [Q[0], self.cool(Q, hdt), u, v, Q[4]]
        # radial sweep on the angular momentum
        F = self.pad(Q)
        F[3] = F[3] * x
        dD = _net(_fluxes(p.gam, ax, dt, F, p.internal_e_flag, p.EOS_flag), ax["a"][3:-3], p.EOS_flag, p.internal_e_flag)
        dD = [d * dt / ax["v"][3:-3] for d in dD]
        dD[3] = dD[3] / xi
        Q = _update(p, c2, Q, dD)
        # azimuthal sweep in the frame of the disk's rotation, then the shift by whole cells
        v0 = self.rot[3:-3] + xi * p.frame_omega
        F = [_wrap(a) for a in (Q[0], Q[1], Q[3] - v0, Q[4], Q[2])]
        one = torch.ones(p.yres + 1, dtype=torch.float64, device=self.dev)
        dD = _net(_fluxes(p.gam, ay, (dt / xi)[:, None], F, p.internal_e_flag, p.EOS_flag), one, p.EOS_flag, p.internal_e_flag)
        dD = [(d * dt / ay["v"][3:-3]).transpose(0, 1) / xi for d in dD]
        dD = [dD[0], dD[1], dD[4], dD[2] + v0 * dD[0], dD[3]]
        Qs = _update(p, c2, Q, dD)
        dy = (p.ymax - p.ymin) / p.yres * xi
        shift = torch.floor(self.rot[3:-3].detach() * dt / dy + 0.5)
        res = self.rot[3:-3] - shift * dy / dt
        rows = (torch.arange(p.yres, device=self.dev)[:, None] - shift.to(torch.int64)) % p.yres
        roll = lambda a: torch.gather(a, 0, rows)  # noqa: E731
        Qs = [roll(a) for a in Qs]
        # residual advection
        fl = self.upwind([_wrap(Qs[m]) for m in (0, 1, 2, 3, 4)], res, dt)
        dq = [((f[..., :-1] - f[..., 1:]) * dt / ay["v"][3:-3]).transpose(0, 1) / xi for f in fl]
        rn = Qs[0] + dq[0]
        Qn = [rn, Qs[1] + dq[1] if p.EOS_flag == 2 else c2 * rn] + [(Qs[m] * Qs[0] + dq[m]) / rn for m in (2, 3, 4)]
        if D is not None:
            D = self.dust_sweeps(D, v0, roll, res, dt)
        Q = Qn
        # second half-kick: predictor, its stress, corrector
        g = self.gravity(then)
        if vis is not None:
            u, v, _, _ = self.kick(Q, g, vis, hdt, hdt)
            vis = self.stress(self.pad([Q[0], Q[1], u, v, Q[4]]))
        u, v, Tu, Tv = self.kick(Q, g, vis, hdt, hdt)
        pr = self.cool(Q, hdt)
        D = None if D is None else self.drag(D, Q, Tu, Tv, pr, g, hdt, hdt)
        Q = [Q[0], pr, u, v, Q[4]]
        if self.damp is not None:
            Q = [a + self.damp * dt * (i[3:-3] - a) for a, i in zip(Q, self.init)]
        return Q, D

    def upwind(self, F, res, dt):
        """Mass and momentum carried through each face by the residual speed."""
        N = F[0].shape[-1] - 4
        ay = self.ax[1]
        S = [_recon(ay["w"][:, 2:-2], a, 0.0, N) for a in F]
        x = torch.clamp(res.abs() * dt / self.xi, min=0.0)[:, None] / ay["dx"][2:-2]
        up = (res > 0)[:, None]
        side = lambda s: _where(up, _aveR(x, s)[..., :-1], _aveL(x, s)[..., 1:])  # noqa: E731
        f = [side(s) for s in S]
        return [f[0] * res[:, None], f[1] * res[:, None]] + [f[0] * a * res[:, None] for a in f[2:]]

    def dust_flux(self, ax, sdt, F):
        """Upwind PPM fluxes of the pressureless fluid: F = r, u, and one more velocity.
        No face takes more than its upwind cell holds."""
        N = F[0].shape[-1] - 4
        S = [_recon(ax["w"][:, 2:-2], a, 0.0, N) for a in F]
        dx, u0 = ax["dx"][2:-2], _sh(F[1], 2, N)
        frac = lambda v: torch.clamp(v * sdt / dx, 0.0, 1.0)  # noqa: E731
        out = []
        for ave, sg, edge in ((_aveL, 1.0, S[1][1] - S[1][0]), (_aveR, -1.0, S[1][1] + S[1][2])):
            away = lambda q: torch.clamp(-sg * q, min=0.0)  # noqa: E731
            d = away(edge) * sdt
            ue = ave(frac(away(edge)), S[1])
            comp = sg * sdt * (ue - u0) / (dx - d)
            x = frac(away(ue))
            out.append([ave(x, S[0]) * _exp(comp), ave(x, S[1])] + [ave(x, s) for s in S[2:]])
        L = [a[..., :-1] for a in out[1]]
        R = [a[..., 1:] for a in out[0]]
        rc, n = F[0], F[0].shape[-1]
        a = torch.minimum(rc[..., 2:n - 3] * sdt / ax["dx"][2:-3], torch.clamp(L[1] * L[0], min=0.0))
        b = torch.maximum(-rc[..., 3:n - 2] * sdt / ax["dx"][3:-2], torch.clamp(R[1] * R[0], max=0.0))
        return [a + b] + [a * l + b * r for l, r in zip(L[1:], R[1:])]

    def dust_sweeps(self, D, v0, roll, res, dt):
        p, (ax, ay), xi = self.p, self.ax, self.xi

        def upd(D, d):
            rmin = torch.clamp(D[0] * 1e-10, min=p.D_G_ratio * 1e-10)
            rn = D[0] + d[0]
            ok = rn >= rmin
            vel = [_where(ok, (a * D[0] + e) / rn, a) for a, e in ((D[2], d[1]), (D[3], d[2]))]
            return [_where(ok, rn, rmin), None] + vel

        ghost = lambda m: torch.cat([self.dinit[m][:PAD].expand(p.yres, PAD), D[m],  # noqa: E731
                                     self.dinit[m][-PAD:].expand(p.yres, PAD)], -1)
        gf = ax["a"][3:-3]
        fl = self.dust_flux(ax, dt, [ghost(0), ghost(2), ghost(3) * self.x])
        d = [(f[..., :-1] * gf[:-1] - f[..., 1:] * gf[1:]) * dt / ax["v"][3:-3] for f in fl]
        D = upd(D, [d[0], d[1], d[2] / xi])
        sdt = (dt / xi)[:, None]
        fl = self.dust_flux(ay, sdt, [_wrap(D[0]), _wrap(D[3] - v0), _wrap(D[2])])
        d = [((f[..., :-1] - f[..., 1:]) * dt / ay["v"][3:-3]).transpose(0, 1) / xi for f in fl]
        D = upd(D, [d[0], d[2], d[1] + v0 * d[0]])
        D = [None if a is None else roll(a) for a in D]
        fl = self.upwind([_wrap(D[0]), _wrap(D[0]), _wrap(D[2]), _wrap(D[3])], res, dt)
        d = [((f[..., :-1] - f[..., 1:]) * dt / ay["v"][3:-3]).transpose(0, 1) / xi for f in fl]
        return upd(D, [d[0], d[2], d[3]])


def _polar_run(p, s, steps, dev):
    S = _Polar(p, dev)
    Q = [S.t(s[k]) for k in "rpuv"]
    if p.EOS_flag != 2:
        Q[1] = S.cs2[3:-3] * Q[0]
    Q.append(torch.zeros_like(Q[0]))
    D = None
    if p.dust_flag:
        d = _dust(p, s)
        D = [S.t(d["r"]), None, S.t(d["u"]), S.t(d["v"])]
    t, cap = T0, 1e30
    for _ in range(steps):
        dt = min(p.CFL / S.rate(Q, D), 1.1 * cap)
        Q, D = S.advance(Q, D, t, dt)
        t, cap = t + dt, dt
    return Q, D


def _sphere_state(p, X, Z):
    """The spherical disk in vertical balance: density, sound speed squared, v_phi."""
    cs2 = lambda x: p.sc_h**2 * (x * np.sin(Z)) ** (-p.p_beta)  # noqa: E731

    def rho(x):
        r = x * np.sin(Z)
        return r ** (-p.p_alpha) * np.exp((1.0 / x - 1.0 / r) / cs2(x))

    dr = 1.1514178e-7
    dP = (cs2(X + dr) * rho(X + dr) - cs2(X - dr) * rho(X - dr)) / (2 * dr)
    return rho(X), cs2(X), np.sqrt(1.0 / X + X / rho(X) * dP)


class _Solid(_Step):
    """The three-dimensional step: spherical (r, phi, theta) or Cartesian."""

    def __init__(self, p, dev):
        super().__init__(p, dev)
        self.sph = p.geomx == 2
        x, z = self.ax[0]["c"], self.ax[2]["c"]
        self.X = x[3:-3]
        self.sin = torch.sin(z[3:-3])[:, None, None] if self.sph else 1.0
        self.rad = self.X if self.sph else 1.0
        self.damp = None
        self.cs2 = None
        if self.sph:
            f = _sphere_state(p, x.cpu().numpy()[None, None], z.cpu().numpy()[:, None, None])
            r, c2, v = (self.t(a) for a in f)
            self.init = [a[3:-3] for a in (r, c2 * r, torch.zeros_like(r), v, torch.zeros_like(r))]
            self.cs2 = c2[3:-3, :, 3:-3]
            self.damp = self.ramp(self.X) if p.kill_flag else None
        else:
            self.init = None

    def forces(self, Q, body):
        p = self.p
        if not self.sph:
            return [0.0] * 3, lambda v, w: (0.0, 0.0)
        m, y = body
        x, a = self.X, p.planet_radius
        rs = p.rs_fac * (p.planet_mass / 3.0) ** (1.0 / 3.0) * a
        yc, z = self.ax[1]["c"][3:-3][None, :, None] - y, self.ax[2]["c"][3:-3][:, None, None]
        s, c, sp, cp = torch.sin(yc), torch.cos(yc), torch.sin(z), torch.cos(z)
        R = torch.sqrt(x * x + a * a - 2 * a * x * c * sp)
        f = torch.clamp(4.0 - 3.0 * R / rs, min=1.0) / torch.clamp(R**3, min=rs**3)
        g = [-1.0 / x**2 - m * (x - a * c * sp) * f - m * sp * c / a**2, -m * a * s * f + m * sp * s / a**2,
             m * a * c * cp * f - m * cp * c / (sp * a * a)]
        return g, lambda v, w: ((v * v + w * w) / x, v * v / x / torch.tan(z))

    def sweep(self, Q, axis, dt):
        """One direction: fields to the sweep's order, fluxes along the last axis, and back."""
        p, ax = self.p, self.ax[axis]
        r, pr, u, v, w = Q
        if axis == 0:
            F = _pad_x(Q, p.bound_lft, p.bound_rgh, self.init)
            if self.sph:
                F[3] = F[3] * self.ax[0]["c"] * self.sin
                F[4] = F[4] * self.ax[0]["c"]
            fl = _fluxes(p.gam, ax, dt, F, p.internal_e_flag, p.EOS_flag)
            gf = ax["a"][3:-3] ** 2 if self.sph else torch.ones_like(ax["a"][3:-3])
            D = [d * dt / ax["v"][3:-3] for d in _net(fl, gf, p.EOS_flag, p.internal_e_flag)]
            D = [D[0], D[1], D[2], D[3] / (self.rad * self.sin), D[4] / self.rad]
        elif axis == 1:
            rc = self.rad * self.sin if self.sph else torch.ones((1, 1, 1), dtype=torch.float64, device=self.dev)
            om = rc * p.frame_omega if self.sph else 0.0 * rc
            mv = lambda a: torch.cat([a[:, -PAD:], a, a[:, :PAD]], 1).transpose(1, 2)  # noqa: E731
            fl = _fluxes(p.gam, ax, dt / rc.transpose(1, 2), [mv(a) for a in (r, pr, v - om, w, u)], p.internal_e_flag, p.EOS_flag)
            D = _net(fl, torch.ones_like(ax["a"][3:-3]), p.EOS_flag, p.internal_e_flag)
            D = [(d * dt / ax["v"][3:-3]).transpose(1, 2) / rc for d in D]
            D = [D[0], D[1], D[4], D[2] + om * D[0], D[3]]
        else:
            zc = self.ax[2]["c"]

            def mv(a, sg=1.0):
                lo = a[:PAD].flip(0) * sg if p.bound_bom == 2 else a[:1].expand((PAD,) + a.shape[1:])
                hi = a[-PAD:].flip(0) * sg if p.bound_top == 2 else a[-1:].expand((PAD,) + a.shape[1:])
                return torch.cat([lo, a, hi], 0).permute(1, 2, 0)

            rd = (self.rad if self.sph else torch.ones(1, dtype=torch.float64, device=self.dev))
            F = [mv(r), mv(pr), mv(w, -1.0), mv(u), mv(v)]
            if self.sph:
                F[4] = F[4] * rd[None, :, None] * torch.sin(zc)
            fl = _fluxes(p.gam, ax, dt / rd[None, :, None], F, p.internal_e_flag, p.EOS_flag)
            gf = torch.sin(ax["a"][3:-3]) if self.sph else torch.ones_like(ax["a"][3:-3])
            D = [(d * dt / ax["v"][3:-3]).permute(2, 0, 1) / rd for d in _net(fl, gf, p.EOS_flag, p.internal_e_flag)]
            D = [D[0], D[1], D[3], D[4] / (rd * self.sin), D[2]]
        return _update(p, self.cs2, Q, D)

    def rate(self, Q):
        p = self.p
        cs = torch.sqrt(p.gam * Q[1] / Q[0])
        rc, om = self.rad * self.sin, (self.rad * self.sin * p.frame_omega if self.sph else 0.0)
        return max(((Q[2].abs() + cs) / self.ax[0]["dx"][3:-3]).max().item(),
                   (((Q[3] - om).abs() + cs) / (self.ax[1]["dx"][3:-3][None, :, None] * rc)).max().item(),
                   ((Q[4].abs() + cs) / (self.ax[2]["dx"][3:-3][:, None, None] * self.rad)).max().item())

    def advance(self, Q, t, dt):
        hdt = 0.5 * dt
        g, fict = self.forces(Q, self.planet(t))
        fx, fz = fict(Q[3], Q[4])
        Q = [Q[0], Q[1], Q[2] + (fx + g[0]) * hdt, Q[3] + g[1] * hdt, Q[4] + (fz + g[2]) * hdt]
        for axis in range(3):
            Q = self.sweep(Q, axis, dt)
        g, fict = self.forces(Q, self.planet(t + dt))
        _, fz = fict(Q[3], Q[4])  # the corrector's forces at the predicted velocities
        fx, fz = fict(Q[3] + g[1] * hdt, Q[4] + (fz + g[2]) * hdt)
        Q = [Q[0], Q[1], Q[2] + (fx + g[0]) * hdt, Q[3] + g[1] * hdt, Q[4] + (fz + g[2]) * hdt]
        if self.damp is not None:
            Q = [a + self.damp * dt * (i[..., 3:-3] - a) for a, i in zip(Q, self.init)]
        return Q


def _gradient(p, s, steps, dev):
    """The final field and the misfit's gradients by torch's own differentiation of
    the plain step, dt as the CFL condition gives it and held fixed."""
    from torch.utils.checkpoint import checkpoint

    s0 = torch.as_tensor(s["r"], dtype=torch.float64, device=dev).requires_grad_(True)
    th = torch.tensor(_theta(p), dtype=torch.float64, device=dev).requires_grad_(True)

    def one(r, u, v, th, t, dt):
        S = _Polar(p, dev, (th[0], th[1], th[2]))
        Q, _ = S.advance([r, S.cs2[3:-3] * r, u, v, torch.zeros_like(r)], None, t, dt)
        return Q[0], Q[2], Q[3]

    S = _Polar(p, dev, (th[0], th[1], th[2]))
    r, u, v = s0, torch.zeros_like(s0), S.init[3][3:-3].expand(s0.shape)
    t, cap = T0, 1e30
    for _ in range(steps):
        with torch.no_grad():
            dt = min(p.CFL / S.rate([r, S.cs2[3:-3] * r, u, v], None), 1.1 * cap)
        r, u, v = checkpoint(one, r, u, v, th, t, dt, use_reentrant=False)
        t, cap = t + dt, dt
    _misfit(r, torch.as_tensor(_target(p), device=dev)).backward()
    return {"sigma": r.detach(), "grad_sigma0": s0.grad, "grad_theta": th.grad}


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    k = case["kind"]
    ps, ss = _params(case), _states(case, seed)
    if k == "gradient":
        return _gradient(ps[0], ss[0], case["steps"], dev)
    with torch.no_grad():
        if k == "tube":
            if case["n"] > 2048:
                return None
            Q = _tube(ps[0], ss[0], case["t_end"], dev)
            return {"r": Q[0], "p": Q[1], "u": Q[2]}
        if k in ("disk", "host", "dust"):
            Q, D = _polar_run(ps[0], ss[0], case["steps"], dev)
            out = {"cells": torch.stack(Q[:4], -1)}
            if D is not None:
                out["dust"] = {"r": D[0], "u": D[2], "v": D[3]}
            return out
        if k == "mixed":
            if case["members"] > 12:
                return None
            out = []
            for p, s in zip(ps, ss):
                Q, D = _polar_run(p, s, case["steps"], dev)
                out.append({"r": Q[0], "u": Q[2], "v": Q[3]})
                if D is not None and len(ps) <= 10:
                    out[-1]["dust"] = {"r": D[0], "u": D[2], "v": D[3]}
            return out
        p, s = ps[0], ss[0]
        S = _Solid(p, dev)
        Q = [S.t(s[f]) for f in "rpuvw"]
        t, cap = T0, 1e30
        for _ in range(case["steps"]):
            dt = min(p.CFL / S.rate(Q), 1.1 * cap)
            Q = S.advance(Q, t, dt)
            t, cap = t + dt, dt
        return dict(zip("rpuvw", Q))
