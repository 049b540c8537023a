"""Performance cases of the projection library: what a user's program calls, over the range of sizes and options it uses.

Each case is one pass through the Python mirror of the C ABI on device data: a projection (with or without new coefficients), its
vector-Jacobian product, a differentiated chain of projections, a fluid step, an EM induction step with its source pass, or the
reference algorithm.  Geometries are the workloads of ``mhdproj.synth`` (cylinder, two-phase jet with a nozzle, liquid column, driven
ring), made on the GPU from the seed and stretched to the case's grid.  ``exact`` restates each pass in FP64 torch operations.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mhd-simulator_gb300"))
import mhdproj  # noqa: E402

RHO_L, RHO_A = 6440.0, 1.2
SIGMA_RING = 40.0 / 0.75e-6  # S/m
EPISODE = 16                 # fluid steps before a state starts again from its first velocity


def _project(name, nx, ny, nz, geometry, precision, tol, outlet, periodic, rebuild):
    return {"name": name, "kind": "project", "nx": nx, "ny": ny, "nz": nz, "geometry": geometry, "precision": precision, "tol": tol,
            "outlet": outlet, "periodic": periodic, "rebuild": rebuild}


def listed():
    return [
        # a probe-sized domain with ragged extents, the smallest projection: launches and latency
        _project("cylinder_30x22x17", 30, 22, 17, "cylinder", "fp32", 1e-6, True, 0, False),
        # the single-phase 64^3 configuration, FP32 levels, fixed coefficients
        _project("cylinder_64", 64, 64, 64, "cylinder", "fp32", 1e-6, True, 0, False),
        # 128^3 two-phase jet in the reference's closed box, BF16 levels, a tight tolerance (two refinement passes)
        _project("jet_128_closed", 128, 128, 128, "jet", "bf16", 1e-8, False, 0, True),
        # the benchmark configuration: 256^3 two-phase jet, new coefficients every step, FP16 levels
        _project("jet_256", 256, 256, 256, "jet", "fp16", 1e-6, True, 0, True),
        # a liquid column through periodic x and y walls, extents that are no powers of two
        _project("column_160x120x96_periodic", 160, 120, 96, "column", "fp16", 1e-6, False, 3, True),
        # the elongated domain, the largest grid of the configurations
        _project("column_512x256x256", 512, 256, 256, "column", "fp16", 1e-6, True, 0, True),
        # backward pass of one projection on an uneven grid
        {"name": "vjp_192x160x132", "kind": "vjp", "nx": 192, "ny": 160, "nz": 132, "geometry": "jet", "precision": "fp16", "tol": 1e-6},
        # the differentiated chain: forward of 8 steps with checkpoints every 4, and the gradient of the force
        {"name": "chain_128", "kind": "chain", "nx": 128, "ny": 128, "nz": 128, "geometry": "jet", "precision": "fp16", "tol": 1e-6,
         "steps": 8, "every": 4},
        # one liquid: advection, viscosity, gravity, the warm-started projection
        {"name": "step_one_phase_128", "kind": "step", "nx": 128, "ny": 128, "nz": 128, "geometry": "jet", "precision": "fp16",
         "tol": 1e-6, "two_phase": False},
        # a moving interface: stress diffusion, capillary force, face densities, the projection, cell records for the display
        {"name": "step_two_phase_144x112x160", "kind": "step", "nx": 144, "ny": 112, "nz": 160, "geometry": "jet", "precision": "fp16",
         "tol": 1e-6, "two_phase": True},
        # a coil driving a conducting ring: the source pass for the new current, then the induction step
        {"name": "em_coil_96", "kind": "em", "nx": 96, "ny": 96, "nz": 96, "segments": 128},
        # the reference algorithm (FP32 aggregation-multigrid CG) on the 96^3 closed jet
        {"name": "reference_jet_96", "kind": "reference", "nx": 96, "ny": 96, "nz": 96, "geometry": "jet", "tol": 1e-5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi, cells):
    while True:
        d = [_log(rng, lo, hi) for _ in range(3)]
        if rng.random() < 0.5:  # half of the programs take extents that divide well
            d = [max(lo, (v + 4) // 8 * 8) for v in d]
        if d[0] * d[1] * d[2] <= cells:
            return dict(zip(("nx", "ny", "nz"), d))


def draw(rng):
    kind = rng.choice(("project", "project", "project", "vjp", "chain", "step", "step", "em", "reference"))
    if kind == "project":
        geometry = rng.choice(("cylinder", "jet", "jet", "column"))
        boundary = rng.choice(("outlet", "outlet", "closed", "periodic")) if geometry == "column" else rng.choice(("outlet", "outlet", "closed"))
        c = {"kind": kind, **_dims(rng, 16, 320, 20_000_000), "geometry": geometry, "precision": rng.choice(("fp16", "fp16", "bf16", "fp32")),
             "tol": rng.choice((1e-6, 1e-6, 1e-7, 1e-8)), "outlet": boundary == "outlet", "periodic": 3 if boundary == "periodic" else 0,
             "rebuild": geometry != "cylinder"}
        if boundary == "periodic":  # a checkerboard needs even periodic extents in most programs
            c["nx"], c["ny"] = c["nx"] // 2 * 2, c["ny"] // 2 * 2
        return c
    if kind == "vjp":
        return {"kind": kind, **_dims(rng, 16, 256, 8_000_000), "geometry": rng.choice(("jet", "column")),
                "precision": rng.choice(("fp16", "bf16", "fp32")), "tol": 1e-6}
    if kind == "chain":
        return {"kind": kind, **_dims(rng, 16, 160, 2_200_000), "geometry": "jet", "precision": rng.choice(("fp16", "bf16")), "tol": 1e-6,
                "steps": rng.randint(2, 6), "every": rng.randint(1, 4)}
    if kind == "step":
        return {"kind": kind, **_dims(rng, 20, 200, 4_000_000), "geometry": "jet", "precision": rng.choice(("fp16", "fp32")), "tol": 1e-6,
                "two_phase": rng.random() < 0.5}
    if kind == "em":
        n = _log(rng, 20, 112)
        return {"kind": kind, "nx": n, "ny": n, "nz": max(18, n - rng.randint(0, n // 4)), "segments": rng.choice((0, 0, _log(rng, 24, 256)))}
    return {"kind": "reference", **_dims(rng, 16, 128, 1_200_000), "geometry": "jet", "tol": rng.choice((1e-4, 3e-5))}  # above its FP32 noise floor


# ------------------------------------------------------------------ inputs
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _normal(shape, seed, salt):
    return torch.randn(shape, generator=_gen(seed, salt), device="cuda", dtype=torch.float32)


def _centres(c):
    mk = lambda n: torch.arange(n, device="cuda", dtype=torch.float64) + 0.5  # noqa: E731
    return mk(c["nz"])[:, None, None], mk(c["ny"])[None, :, None], mk(c["nx"])[None, None, :]


def _shapes(c):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    return (nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)


def _geometry(c, seed):
    """Liquid fraction, solid mask and cell size."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    z, y, x = _centres(c)
    s = min(nx, ny) / 128.0
    off = torch.rand(20, generator=_gen(seed, 1), device="cuda", dtype=torch.float64).tolist()
    soft = lambda d, w: 0.5 * (1.0 - torch.tanh(d / w))  # noqa: E731
    if c["geometry"] == "cylinder":  # one liquid inside a cylinder of 7/8 of the width
        r = torch.sqrt((x - nx / 2) ** 2 + (y - ny / 2) ** 2)
        solid = (r > 0.4375 * min(nx, ny)).expand(nz, ny, nx)
        return torch.ones((nz, ny, nx), device="cuda"), solid.to(torch.uint8).contiguous(), 1e-4 * 64 / min(nx, ny)
    if c["geometry"] == "jet":  # a jet along z, a drop, and a tapered annular nozzle round the inlet
        cx, cy = nx / 2 + (8 * off[0] - 4) * s, ny / 2 + (8 * off[1] - 4) * s
        sx, sy, sz = nx / 2 + (16 * off[2] - 8) * s, ny / 2 + (16 * off[3] - 8) * s, nz * (0.625 + 0.1 * (off[4] - 0.5))
        alpha = torch.maximum(soft(torch.sqrt((x - cx) ** 2 + (y - cy) ** 2) - 10 * s, 1.5 * max(s, 0.5)),
                              soft(torch.sqrt((x - sx) ** 2 + (y - sy) ** 2 + (z - sz) ** 2) - 16 * s, 1.5 * max(s, 0.5)))
        r = torch.sqrt((x - nx / 2) ** 2 + (y - ny / 2) ** 2)
        inner = 24 * s - 12 * s * torch.clamp(z / (0.25 * nz), 0, 1)
        solid = (z < 0.25 * nz) & (r >= inner) & (r <= inner + 8 * s)
        return alpha.float().contiguous(), solid.to(torch.uint8).contiguous(), 5e-5 if c["kind"] == "step" else 5e-5 * 128 / min(nx, ny)
    s = min(ny, nz) / 256.0  # a column along x with four satellite drops
    alpha = soft(torch.sqrt((y - ny / 2) ** 2 + (z - nz / 2) ** 2) - 20 * s, 3 * max(s, 0.3)).expand(nz, ny, nx)
    for k in range(4):
        px, py, pz = off[4 * k] * nx, (0.2 + 0.6 * off[4 * k + 1]) * ny, (0.2 + 0.6 * off[4 * k + 2]) * nz
        d = torch.sqrt((x - px) ** 2 + (y - py) ** 2 + (z - pz) ** 2) - (8 + 6 * off[4 * k + 3]) * s
        alpha = torch.maximum(alpha, soft(d, 3 * max(s, 0.3)))
    return alpha.float().contiguous(), torch.zeros((nz, ny, nx), dtype=torch.uint8, device="cuda"), 2.5e-5 * 256 / min(ny, nz)


def _low(a, axis):
    """The value of the low neighbour along torch axis `axis`, wrapped."""
    return torch.roll(a, 1, axis)


def _open_low(c, solid):
    """Per axis x, y, z: whether the low face of a cell is open (periodic axes wrap)."""
    fluid = solid == 0
    out = []
    for a in range(3):
        o = fluid & _low(fluid, 2 - a)
        if not c.get("periodic", 0) >> a & 1:
            o.select(2 - a, 0).zero_()
        out.append(o)
    return out


def _to_faces(c, low, top=None):
    """Cell-shaped low-face arrays to face arrays; the last face of a periodic axis repeats the first one, of another it is 0 (or `top`)."""
    out = []
    for a, v in enumerate(low):
        last = v.select(2 - a, 0) if c.get("periodic", 0) >> a & 1 else torch.zeros_like(v.select(2 - a, 0))
        if a == 2 and top is not None:
            last = top
        out.append(torch.cat([v, last.unsqueeze(2 - a)], 2 - a))
    return out


def _noise(c, alpha, solid, seed):
    """Face velocities N(0, 0.2 m/s) in the liquid and N(0, 0.02 m/s) in the air, 0 on closed faces."""
    op, top = _open_low(c, solid), (solid[-1] == 0) if c.get("outlet", True) else None
    fa = [0.5 * (alpha + _low(alpha, 2 - a)) for a in range(3)]
    sd = [torch.where(f >= 0.5, 0.2, 0.02) * o for f, o in zip(fa, op)]
    tops = torch.where(alpha[-1] >= 0.5, 0.2, 0.02) * top if top is not None else None
    sd = _to_faces(c, sd, tops)
    out = []
    for a, s in enumerate(sd):
        v = _normal(s.shape, seed, 10 + a) * s
        if c.get("periodic", 0) >> a & 1:
            v.select(2 - a, -1).copy_(v.select(2 - a, 0))
        out.append(v.float().contiguous())
    return out


def _flow(c, solid, seed):
    """A smooth flow of up to about 0.3 m/s (0.15 m/s with an interface) with 5 % noise, 0 on closed faces and at the outlet."""
    z, y, x = _centres(c)
    ph = (2 * math.pi * torch.rand(3, generator=_gen(seed, 5), device="cuda", dtype=torch.float64)).tolist()
    kx, ky, kz = (2 * math.pi * m / n for m, n in ((1, c["nx"]), (2, c["ny"]), (1, c["nz"])))
    s = 0.3 if c["two_phase"] else 0.6
    v = [0.2 * torch.sin(ky * y + ph[0]) * torch.cos(kz * z), 0.2 * torch.sin(kz * z + ph[1]) * torch.cos(kx * x),
         0.3 * torch.sin(kx * x + ph[2]) * torch.cos(ky * y)]
    op = _open_low(c, solid)
    v = [s * (a.expand(o.shape) + 0.01 * _normal(o.shape, seed, 20 + k)) * o for k, (a, o) in enumerate(zip(v, op))]
    return [f.float().contiguous() for f in _to_faces(c, v)]


def _context(c, h, **kw):
    return mhdproj.PressureProjection((c["nx"], c["ny"], c["nz"]), h, periodic=[bool(c.get("periodic", 0) >> a & 1) for a in range(3)],
                                      outlet=c.get("outlet", True), precision=c.get("precision", "fp16"), rel_tol=c["tol"], **kw)


def _rho_air(c):
    return RHO_L if c.get("geometry") == "cylinder" or c.get("two_phase") is False else RHO_A


def _ring(c):
    """Cell materials of a conducting annulus about the z axis, the cell size, the low corner."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    z, y, x = _centres(c)
    r = torch.sqrt((x - nx / 2) ** 2 + (y - ny / 2) ** 2)
    m = (r >= 0.19 * nx) & (r <= 0.38 * nx) & (z > nz // 3) & (z < nz - nz // 3)
    return m, 1e-3, (-0.5e-3 * nx, -0.5e-3 * ny, -0.5e-3 * nz)


def _edge_points(c):
    """Edge midpoints (x, y, z) of the x-, y- and z-edge blocks, as broadcastable FP64 arrays."""
    n, (_, h, origin) = (c["nx"], c["ny"], c["nz"]), _ring(c)
    out = []
    for a in range(3):
        p = []
        for k in range(3):
            q = torch.arange(n[k] + (k != a), device="cuda", dtype=torch.float64) + (0.5 if k == a else 0.0)
            p.append((np.float32(origin[k]) + q * np.float32(h)).reshape([-1 if 2 - j == k else 1 for j in range(3)]))
        out.append(p)
    return out


def _drive(seed):
    return 50.0 + 100.0 * float(torch.rand(1, generator=_gen(seed, 9), device="cuda"))  # amperes


def _coil(c, seed):
    """A closed wire loop of straight elements round the ring, 12 floats each."""
    k, h = c["segments"], 1e-3
    ang = 2 * np.pi * np.arange(k + 1) / k
    pts = np.stack([0.44 * c["nx"] * h * np.cos(ang), 0.44 * c["ny"] * h * np.sin(ang), np.full(k + 1, 0.03 * c["nz"] * h)], 1)
    el = np.zeros((k, 12), np.float32)
    el[:, 0:3], el[:, 4:7], el[:, 8], el[:, 10] = pts[:-1], pts[1:], h, 100.0 * _drive(seed)
    return el


def _uniform(c, seed):
    """A_s of a uniform field B_z at every edge (x-, y-, then z-edges)."""
    b = 2e-4 * _drive(seed)
    blocks = [(-0.5 * b * p[1], 0.5 * b * p[0], 0.0 * p[0])[a] for a, p in enumerate(_edge_points(c))]
    return torch.cat([(v + 0 * p[0] + 0 * p[1] + 0 * p[2]).reshape(-1) for v, p in zip(blocks, _edge_points(c))]).float()


def _wave(k):
    return math.sin(2 * math.pi * 1e3 * 1e-5 * k)  # 1 kHz, 10 us steps


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "em":
        ring, h, origin = _ring(c)
        em = mhdproj.EmInduction((c["nx"], c["ny"], c["nz"]), h, dt_s=1e-5, origin_m=origin)
        em.set_materials(ring.to(torch.int32).reshape(-1), np.array([[0.0, 1.0], [SIGMA_RING, 1.0]], np.float32))
        s = {"c": c, "em": em, "k": 0}
        if c["segments"]:
            s["coil"] = _coil(c, seed)
        else:
            s["uniform"] = _uniform(c, seed)
        em.advance(0.0, initial=True, applied=_applied(s))
        for _ in range(2):
            _em_step(s)
        return s
    alpha, solid, h = _geometry(c, seed)
    s = {"c": c, "alpha": alpha, "solid": solid}
    if c["kind"] == "reference":
        c["outlet"] = False
        s["u"] = _noise(c, alpha, solid, seed)
        s["proj"] = _context(c, h, solver="reference")
    elif c["kind"] == "step":
        s["proj"] = _context(c, h)
        s["proj"].set_coefficients(alpha, solid, RHO_L, _rho_air(c))
        s["u0"], s["p"], _ = s["proj"].project(_flow(c, solid, seed), _step_dt(c))
        s["u"] = [v.clone() for v in s["u0"]]
        s["k"] = 0
        if c["two_phase"]:
            s["curvature"] = _curvature(c, seed)
            s["cells"] = torch.empty((c["nz"], c["ny"], c["nx"], 16), device="cuda")
        return s
    else:
        s["u"] = _noise(c, alpha, solid, seed)
        s["proj"] = _context(c, h, gauge=0 if c["kind"] in ("vjp", "chain") else -1)
    s["proj"].set_coefficients(alpha, solid, RHO_L, _rho_air(c))
    s["out"] = tuple(torch.empty_like(v) for v in s["u"])
    if c["kind"] == "vjp":
        s["gp"] = _normal((c["nz"], c["ny"], c["nx"]), seed, 30) * 1e-6 * (solid == 0)
    if c["kind"] == "chain":
        s["f"] = _force(c, alpha, solid, seed)
    return s


def _force(c, alpha, solid, seed):
    """A face force N(0, 1e5 N/m^3) inside the liquid."""
    op = _open_low(c, solid)
    keep = _to_faces(c, [o & (0.5 * (alpha + _low(alpha, 2 - a)) >= 0.5) for a, o in enumerate(op)])
    return [_normal(k.shape, seed, 40 + a) * 1e5 * k for a, k in enumerate(keep)]


def _curvature(c, seed):
    z, y, x = _centres(c)
    phase = float(torch.rand(1, generator=_gen(seed, 6), device="cuda"))
    return (2000.0 + 100.0 * torch.sin(2 * math.pi * (z / c["nz"] + phase)) + 0 * x + 0 * y).float().contiguous()


def _step_dt(c):
    return 2e-6 if c["two_phase"] else 8e-6


def _step_options(c):
    o = {"acceleration": (0.0, 0.0, -9.81), "viscosity": 3.7e-7, "advection": True}
    return {**o, "surface_tension": 0.5, "air_viscosity": 1.8e-5} if c["two_phase"] else o


def _applied(s):
    if "uniform" in s:
        return s["uniform"] * _wave(s["k"])
    el = s["coil"].copy()
    el[:, 10] *= np.float32(_wave(s["k"]))
    return s["em"].evaluate_sources(el)


def _em_step(s):
    s["k"] += 1
    s["em"].advance(s["k"] * 1e-5, applied=_applied(s))


def run(s):
    c = s["c"]
    if c["kind"] == "project":
        if c["rebuild"]:
            s["proj"].set_coefficients(s["alpha"], s["solid"], RHO_L, _rho_air(c))
        out, p, _ = s["proj"].project(s["u"], 1e-5, out=s["out"])
        return {"u": out, "p": p}
    if c["kind"] == "reference":
        s["proj"].set_coefficients(s["alpha"], s["solid"], RHO_L, RHO_A)
        out, p, st = s["proj"].project(s["u"], 1e-5, out=s["out"])
        return {"u": out, "p": p, "iterations": st.iterations}
    if c["kind"] == "vjp":
        return {"g": s["proj"].vjp(s["u"], s["gp"], 1e-5)[0]}
    if c["kind"] == "chain":
        u, objective, _ = s["proj"].chain_forward(s["u"], s["f"], 1e-6, c["steps"], c["every"])
        return {"u": u, "objective": objective, "g": s["proj"].chain_backward(s["u"])[0]}
    if c["kind"] == "step":
        if s["k"] % EPISODE == 0:
            for v, v0 in zip(s["u"], s["u0"]):
                v.copy_(v0)
        s["k"] += 1
        s["proj"].fluid_step(s["u"], _step_dt(c), p_out=s["p"], cells=s.get("cells"), curvature=s.get("curvature"), **_step_options(c))
        out = {"u": s["u"], "p": s["p"]}
        return {**out, "cells": s["cells"]} if c["two_phase"] else out
    _em_step(s)
    return {"cells": s["em"].copy("cells"), "reaction": s["em"].copy("reaction")}


def work(case):
    """Each input read once and each output written once; a multigrid solve to 1e-6 taken as 1200 flops a cell, an induction step as
    100 iterations of 40 flops an edge, a wire element as 60 flops an edge."""
    n = case["nx"] * case["ny"] * case["nz"]
    solve = 1200.0 * n * -math.log10(case.get("tol", 1e-6)) / 6
    if case["kind"] == "em":
        e = 3 * n
        return {"bytes": 4.0 * 5 * e + 64.0 * n, "flops": (4000.0 + 60.0 * case["segments"]) * e}
    if case["kind"] == "chain":
        return {"bytes": 53.0 * n, "flops": 2 * case["steps"] * solve}
    if case["kind"] == "step":
        return {"bytes": (33.0 + (68.0 if case["two_phase"] else 0.0)) * n, "flops": solve + 600.0 * n}
    return {"bytes": 33.0 * n, "flops": solve}


# ------------------------------------------------------------ FP64 restatement
class _Exact:
    """The discrete projection of one case in FP64: mobilities, operator, Jacobi-CG solve."""

    def __init__(self, c, alpha, solid, h, rho_air):
        self.c, self.h, self.rho_air = c, h, rho_air
        self.fluid = solid == 0
        self.open = _open_low(c, solid)
        a = alpha.double()
        self.rho = rho_air * (1 - a) + RHO_L * a
        self.face_rho = [0.5 * (self.rho + _low(self.rho, 2 - k)) for k in range(3)]
        self.beta = [RHO_L / r * o for r, o in zip(self.face_rho, self.open)]
        self.top = (2 * RHO_L / self.rho[-1] * self.fluid[-1]) if c.get("outlet", True) else None
        d = sum(b + torch.roll(b, -1, 2 - k) for k, b in enumerate(self.beta))
        if self.top is not None:
            d[-1] += self.top
        self.inv = torch.where(d > 0, 1 / d, 0.0)

    def apply(self, x):
        y = torch.zeros_like(x)
        for k, b in enumerate(self.beta):
            f = b * (x - _low(x, 2 - k))
            y += f
            y -= torch.roll(f, -1, 2 - k)
        if self.top is not None:
            y[-1] += self.top * x[-1]
        return y

    def solve(self, b):
        x, r = torch.zeros_like(b), b.clone()
        z = self.inv * r
        p, rz, bb = z.clone(), (r * z).sum(), (b * b).sum()
        for k in range(20000):
            q = self.apply(p)
            al = rz / (p * q).sum()
            x += al * p
            r -= al * q
            if k % 50 == 49 and float((r * r).sum()) <= 1e-22 * float(bb):
                break
            z = self.inv * r
            rz, old = (r * z).sum(), rz
            p = z + (rz / old) * p
        if self.top is None:  # one closed component: zero at its first cell
            first = int(torch.nonzero(self.fluid.reshape(-1))[0])
            x = torch.where(self.fluid, x - x.reshape(-1)[first], 0.0)
        return x

    def low(self, faces):
        """Low-face cell arrays of face arrays."""
        return [v.double().narrow(2 - k, 0, v.shape[2 - k] - 1) for k, v in enumerate(faces)]

    def project(self, faces):
        lo = [v * o for v, o in zip(self.low(faces), self.open)]
        top = faces[2][-1].double() * self.fluid[-1] if self.top is not None else None
        div = sum(torch.roll(v, -1, 2 - k) - v for k, v in enumerate(lo))
        if top is not None:
            div[-1] += top
        phi = self.solve(-self.h * div * self.fluid)
        lo = [v - b * (phi - _low(phi, 2 - k)) / self.h for k, (v, b) in enumerate(zip(lo, self.beta))]
        if top is not None:
            top = top + self.top * phi[-1] / self.h
        return _to_faces(self.c, lo, top), phi

    def transpose(self, grads, gp, dt):
        """The transposed projection of face gradients and a pressure gradient (no periodic axes)."""
        lo = [g * o for g, o in zip(self.low(grads), self.open)]
        top = grads[2][-1].double() * self.fluid[-1]
        s = sum((torch.roll(b * g, -1, 2 - k) - b * g) / self.h for k, (b, g) in enumerate(zip(self.beta, lo)))
        s[-1] += self.top * top / self.h
        if gp is not None:
            s = s + RHO_L / dt * gp.double()
        psi = self.solve(s * self.fluid)
        lo = [(g + self.h * (psi - _low(psi, 2 - k))) * o for k, (g, o) in enumerate(zip(lo, self.open))]
        return _to_faces(self.c, lo, (top - self.h * psi[-1]) * self.fluid[-1])

    def mobility_dt(self, dt):
        """dt / rho on every face, 0 on closed ones."""
        return _to_faces(self.c, [dt / r * o for r, o in zip(self.face_rho, self.open)], dt / self.rho[-1] * self.fluid[-1])


class _Box:
    """Arrays of a grid in a frame of zeros (two low, three high), so that shifts need no edge cases; position p sits at p + 2."""

    def __init__(self, c):
        self.shape = (c["nz"] + 5, c["ny"] + 5, c["nx"] + 5)

    def put(self, v):
        b = torch.zeros(self.shape, dtype=v.dtype, device="cuda")
        b[2:2 + v.shape[0], 2:2 + v.shape[1], 2:2 + v.shape[2]] = v
        return b

    @staticmethod
    def at(b, axis, d):
        return torch.roll(b, -d, 2 - axis)

    @staticmethod
    def get(b, shape):
        return b[2:2 + shape[0], 2:2 + shape[1], 2:2 + shape[2]]


def _sample(box, b, comp, pos):
    """Trilinear value at `pos` (x, y, z in cells) of the face grid of component `comp`, 0 outside."""
    q = [p - (0.0 if k == comp else 0.5) for k, p in enumerate(pos)]
    base = [torch.floor(v) for v in q]
    fr = [v - w for v, w in zip(q, base)]
    nz, ny, nx = box.shape
    out = torch.zeros_like(pos[0])
    flat = b.reshape(-1)
    for k in range(8):
        t = (k & 1, k >> 1 & 1, k >> 2)
        w = math.prod(fr[a] if t[a] else 1 - fr[a] for a in range(3))
        ix, iy, iz = (torch.clamp((base[a] + t[a]).long() + 2, 0, n - 1) for a, n in enumerate((nx, ny, nz)))
        out += w * flat[ix + nx * (iy + ny * iz)]
    return out


def _exact_step(c, e, u):
    """predict, stresses or viscosity, forcing, projection and cell records of one step from the divergence-free faces u."""
    box, h, dt, o = _Box(c), e.h, _step_dt(c), _step_options(c)
    shapes, g = _shapes(c), o["acceleration"]
    opens = [box.put(f) for f in _to_faces(c, e.open)]                    # the top faces count as closed in these passes
    vel = [box.put(v.double()) * f for v, f in zip(u, opens)]
    if not c["two_phase"]:
        pred = []
        for a in range(3):
            pos = [torch.arange(n, device="cuda", dtype=torch.float64) for n in reversed(shapes[a])]
            pos = [p + (0.0 if k == a else 0.5) for k, p in enumerate(pos)]
            at = [v.expand(shapes[a]) for v in (pos[0][None, None, :], pos[1][None, :, None], pos[2][:, None, None])]
            mid = [p - _sample(box, vel[k], k, at) * (0.5 * dt / h) for k, p in enumerate(at)]
            back = [p - _sample(box, vel[k], k, mid) * (dt / h) for k, p in enumerate(at)]
            pred.append(box.put(_sample(box, vel[a], a, back)) * opens[a])
        star = []
        for a in range(3):
            lap = torch.zeros_like(pred[a])
            for d in range(3):
                for s in (-1, 1):
                    nb, op = box.at(pred[a], d, s), box.at(opens[a], d, s)
                    lap += (torch.where(op, nb, -pred[a]) if d != a else nb) - pred[a]
            star.append((pred[a] + o["viscosity"] * dt / h ** 2 * lap + dt * g[a]) * opens[a])
    else:
        fluid, alpha = box.put(e.fluid), box.put(e.alpha.double())
        mu = (o["air_viscosity"] * (1 - alpha) + o["viscosity"] * RHO_L * alpha) * fluid
        rho = e.rho_air * (1 - alpha) + RHO_L * alpha
        normal = [2 * mu * (box.at(vel[a], a, 1) - vel[a]) / h for a in range(3)]

        def shear(i, j):
            ui1, ui0, uj1, uj0 = vel[i], box.at(vel[i], j, -1), vel[j], box.at(vel[j], i, -1)
            oi1, oi0, oj1, oj0 = opens[i], box.at(opens[i], j, -1), opens[j], box.at(opens[j], i, -1)
            a1, a0 = torch.where(~oi1 & oi0, -ui0, ui1), torch.where(~oi0 & oi1, -ui1, ui0)
            b1, b0 = torch.where(~oj1 & oj0, -uj0, uj1), torch.where(~oj0 & oj1, -uj1, uj0)
            tot, cnt = 0.0, 0.0
            for p in (0, -1):
                for q in (0, -1):
                    tot = tot + box.at(box.at(mu, i, p), j, q)
                    cnt = cnt + box.at(box.at(fluid, i, p), j, q).double()
            return tot / torch.clamp(cnt, min=1.0) * (a1 - a0 + b1 - b0) / h

        star = []
        kap = box.put(e.curvature.double())
        for a in range(3):
            div = normal[a] - box.at(normal[a], a, -1)
            for j in range(3):
                if j != a:
                    s = shear(a, j)
                    div = div + box.at(s, j, 1) - s
            fr = 0.5 * (rho + box.at(rho, a, -1))
            al, kl = box.at(alpha, a, -1), box.at(kap, a, -1)
            wl, wr = al * (1 - al), alpha * (1 - alpha)
            k = torch.where(wl + wr > 1e-6, (wl * kl + wr * kap) / torch.clamp(wl + wr, min=1e-20), 0.5 * (kl + kap))
            acc = g[a] + o["surface_tension"] * k * (alpha - al) / h / fr
            star.append(torch.where(opens[a], vel[a] + dt * div / (h * fr) + dt * acc, 0.0))
    out, phi = e.project([box.get(v, s) for v, s in zip(star, shapes)])
    p = RHO_L * phi / dt
    res = {"u": out, "p": p * e.fluid}
    if c["two_phase"]:
        vel = [box.put(v) * f for v, f in zip(out, opens)]
        lo, hi = [box.get(v, p.shape) for v in vel], [box.get(box.at(v, a, 1), p.shape) for a, v in enumerate(vel)]
        v = [0.5 * (a + b) for a, b in zip(lo, hi)]
        div, zero = sum(b - a for a, b in zip(lo, hi)) / h, torch.zeros_like(p)
        lanes = v + [torch.sqrt(sum(x * x for x in v)), p, div, zero, zero] + [zero + RHO_L * x for x in g] + [zero, zero + 1, zero + 1]
        lanes = [x * e.fluid for x in lanes] + [e.alpha.double(), e.curvature.double()]
        res["cells"] = torch.stack(lanes, 3)
    return res


def _exact_em(c, seed):
    """Three induction steps after the initial field; the cell records and the reaction potential of the last one."""
    n, (ring, h, _) = (c["nx"], c["ny"], c["nz"]), _ring(c)
    h, dt, mu0 = float(np.float32(h)), 1e-5, 4e-7 * math.pi
    box = _Box(c)
    at = box.at
    edge = [tuple(n[k] + (k != a) for k in (2, 1, 0)) for a in range(3)]
    inner, cond = [], box.put(ring)
    for a in range(3):
        m = torch.zeros(edge[a], dtype=torch.bool, device="cuda")
        m[tuple(slice(None) if k == a else slice(1, n[k]) for k in (2, 1, 0))] = True
        inner.append(box.put(m))
    is_edge = [box.put(torch.ones(s, dtype=torch.bool, device="cuda")) for s in edge]
    is_face = [box.put(torch.ones(tuple(n[k] + (k == a) for k in (2, 1, 0)), dtype=torch.bool, device="cuda")) for a in range(3)]
    air = torch.zeros((n[2] + 1, n[1] + 1, n[0] + 1), dtype=torch.bool, device="cuda")
    air[1:-1, 1:-1, 1:-1] = True
    air = box.put(air)
    near = torch.zeros_like(air)
    for k in range(8):
        near = near | at(at(at(cond, 0, -(k & 1)), 1, -(k >> 1 & 1)), 2, -(k >> 2))
    air = (air & ~near).double()
    sig_c = SIGMA_RING * cond
    sig = []
    for a in range(3):
        i, j = (a + 1) % 3, (a + 2) % 3
        sig.append(0.25 * sum(at(at(sig_c, i, -p), j, -q) for p in (0, 1) for q in (0, 1)) * is_edge[a])
    m = [mu0 * s * h * h / dt for s in sig]

    def curl(v):
        out = []
        for f in range(3):
            a, b = (f + 1) % 3, (f + 2) % 3
            out.append((at(v[b], a, 1) - v[b] - at(v[a], b, 1) + v[a]) * is_face[f])
        return out

    def stiff(v):  # curl-curl and the nodal gauge
        f, out = curl(v), []
        d = sum(v[a] - at(v[a], a, -1) for a in range(3)) * air
        for w in range(3):
            a, b = (w + 1) % 3, (w + 2) % 3
            out.append((f[b] - at(f[b], a, -1) - f[a] + at(f[a], b, -1) + d - at(d, w, 1)) * inner[w])
        return out

    dot = lambda x, y: sum((p * q).sum() for p, q in zip(x, y))  # noqa: E731

    def solve(b):
        x, r = [torch.zeros_like(v) for v in b], [v.clone() for v in b]
        diag = [4.0 + mm + air + at(air, a, 1) for a, mm in enumerate(m)]
        z = [v / d for v, d in zip(r, diag)]
        p, rz, bb = [v.clone() for v in z], dot(r, z), float(dot(b, b))
        for k in range(4000):
            q = [s + mm * v for s, mm, v in zip(stiff(p), m, p)]
            al = rz / dot(p, q)
            x = [v + al * w for v, w in zip(x, p)]
            r = [v - al * w for v, w in zip(r, q)]
            if k % 20 == 19 and float(dot(r, r)) <= 1e-22 * bb:
                break
            z = [v / d for v, d in zip(r, diag)]
            rz, old = dot(r, z), rz
            p = [v + (rz / old) * w for v, w in zip(z, p)]
        return x

    pts = _edge_points(c)
    if c["segments"]:
        base, el = [], torch.from_numpy(_coil(c, seed)).double()
        for a in range(3):
            v = torch.zeros(edge[a], dtype=torch.float64, device="cuda")
            for t in el.tolist():
                d = [t[4 + k] - t[k] for k in range(3)]
                ln = math.sqrt(sum(x * x for x in d))
                d = [x / ln for x in d]
                if d[a] == 0.0:
                    continue
                r = [pts[a][k] - t[k] for k in range(3)]
                s = sum(x * y for x, y in zip(r, d))
                rad = torch.sqrt(sum((x - y * s) ** 2 for x, y in zip(r, d)) + t[8] ** 2)
                v += d[a] * 1e-7 * t[10] * (torch.asinh(s / rad) - torch.asinh((s - ln) / rad))
            base.append(box.put(v))
    else:
        flat, base, o = _uniform(c, seed).double(), [], 0
        for s in edge:
            base.append(box.put(flat[o:o + math.prod(s)].reshape(s)))
            o += math.prod(s)
    prev, asp = [torch.zeros_like(v) for v in base], [_wave(0) * v for v in base]
    for k in range(1, 4):
        now = [_wave(k) * v for v in base]
        change = [p - q for p, q in zip(now, asp)]
        b = [(-mm * d) * i - s for mm, d, i, s in zip(m, change, inner, stiff(prev))]
        x = solve(b)
        if k == 3:
            total = curl([p + q + r for p, q, r in zip(prev, x, now)])
            ext = curl(now)
            mid = lambda f: [0.5 * (f[a] + at(f[a], a, 1)) / h for a in range(3)]  # noqa: E731
            mag, app = mid(total), mid(ext)
            j, heat = [], 0.0
            for a in range(3):
                i, l = (a + 1) % 3, (a + 2) % 3
                ee = -(x[a] + change[a]) / dt * is_edge[a]
                four = [at(at(ee, i, p), l, q) for p in (0, 1) for q in (0, 1)]
                j.append(sig_c * 0.25 * sum(four))
                heat = heat + sig_c * 0.25 * sum(v * v for v in four)
            f = [j[1] * mag[2] - j[2] * mag[1], j[2] * mag[0] - j[0] * mag[2], j[0] * mag[1] - j[1] * mag[0]]
            ln = lambda v: torch.sqrt(sum(q * q for q in v))  # noqa: E731
            lanes = mag + [ln(mag)] + j + [ln(j)] + f + [heat] + app + [ln(app)]
            cells = torch.stack([box.get(v, (n[2], n[1], n[0])).reshape(-1) for v in lanes], 1)
        prev = [p + q for p, q in zip(prev, x)]
        asp = now
    return {"cells": cells, "reaction": torch.cat([box.get(v, s).reshape(-1) for v, s in zip(prev, edge)])}


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "em":
        return _exact_em(c, seed)
    if c["kind"] == "reference":
        c["outlet"] = False
    alpha, solid, h = _geometry(c, seed)
    e = _Exact(c, alpha, solid, float(np.float32(h)), RHO_L if _rho_air(c) == RHO_L else float(np.float32(RHO_A)))
    if c["kind"] == "step":
        e.alpha = alpha
        e.curvature = _curvature(c, seed) if c["two_phase"] else None
        return _exact_step(c, e, e.project(_flow(c, solid, seed))[0])
    u = _noise(c, alpha, solid, seed)
    if c["kind"] == "vjp":
        return {"g": e.transpose(u, _normal((c["nz"], c["ny"], c["nx"]), seed, 30) * 1e-6 * (solid == 0), 1e-5)}
    if c["kind"] == "chain":
        w = [v * f.double() for v, f in zip(e.mobility_dt(1e-6), _force(c, alpha, solid, seed))]
        for _ in range(c["steps"]):
            u = e.project([v.double() + d for v, d in zip(u, w)])[0]
        lam = [torch.zeros_like(u[0]), torch.zeros_like(u[1]), torch.zeros_like(u[2])]
        lam[2][-1] = 2 * u[2][-1]
        grad = [torch.zeros_like(v) for v in lam]
        for _ in range(c["steps"]):
            lam = e.transpose(lam, None, 1e-6)
            grad = [g + d * v for g, d, v in zip(grad, e.mobility_dt(1e-6), lam)]
        return {"u": u, "objective": float((u[2][-1] ** 2).sum()), "g": grad}
    out, phi = e.project(u)
    res = {"u": out, "p": RHO_L * phi / 1e-5}
    return {**res, "iterations": None} if c["kind"] == "reference" else res
