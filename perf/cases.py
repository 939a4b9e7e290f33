"""The work that users of this framework have it do, as cases that can be timed.

Four kinds, each through the public entry points of mortontrie_amr_b200:

  uniform  a periodic Morton cube (DenseCase): FP64 fields in from pinned host
           buffers, the time steps, FP64 fields back into pinned host buffers
  flow     a multi-level flow (LBM_Manager): start from equilibrium at the
           initial velocity, coarse steps, the fields of every level, the force
  request  one served request from its specification: lattice classified on
           the device, the case built, stepped and released
  batch    independent uneven cases stepped together (Batch)

Sizes are those of this repository's configurations, tests and benchmark
(the 2-level sphere of 64x32x32, the 256^3 Taylor-Green cube, the 4-level
cumulant sphere of 192x96x96, the served direct-forcing spheres, the seeded
list of uneven instances) or generic ones around them, odd extents included.

A run returns the fields as one array per case, rows rho - 1, u_x, u_y, u_z
over the cells of all its levels, in the precision the case is stored in
(double, float, half), and the mean force on the body where there is one.
"""
import itertools

import numpy as np
import torch

from mortontrie_amr_b200.case import cavity_case, sphere_case, uniform_box_case
from mortontrie_amr_b200.lbm import Batch, Context, DenseCase, LBM_Manager
from mortontrie_amr_b200.mesh import estimate_cells
from mortontrie_amr_b200.serving import Request, build_template, request_case, template_key
from mortontrie_amr_b200.workloads import batched_uneven_cases

DTYPE = {"f64": torch.float64, "f32": torch.float32, "f16": torch.float16, "bf16": torch.float16}
BYTES = {"f64": 8, "f32": 4, "f16": 2, "bf16": 2}
#: arithmetic of one cell update (collision with its macros)
FLOPS = {(19, "LBGK"): 260.0, (27, "LBGK"): 370.0, (27, "Cumulant"): 600.0}
U0 = 0.02  # Taylor-Green amplitude


def listed():
    return [
        # the drop-in run as a user of the reference starts it: FP64, the
        # reference's phase order, the 2-level sphere (small: launches count)
        {"name": "sphere-2l-plain-f64", "kind": "flow", "body": "sphere", "q": 19, "collision": "LBGK", "nx": 64, "ny": 32,
         "nz": 32, "levels": 1, "radius": 4.0, "re": 20.0, "u": 0.05, "storage": "f64", "schedule": "phases",
         "scaling": "reference", "itime": "reference", "shift": "none", "steps": 50},
        # the same sphere in the fast form, the smallest call: a few hundred steps between two looks at the flow
        {"name": "sphere-2l-f16", "kind": "flow", "body": "sphere", "q": 19, "collision": "LBGK", "nx": 64, "ny": 32,
         "nz": 32, "levels": 1, "radius": 4.0, "re": 20.0, "u": 0.05, "storage": "f16", "schedule": "fused",
         "scaling": "standard", "itime": "reference", "shift": "far_field", "steps": 200},
        # a lid-driven cavity of odd extents, walls on every face, FP32
        {"name": "cavity-odd-f32", "kind": "flow", "body": "cavity", "q": 19, "collision": "LBGK", "nx": 45, "ny": 37,
         "nz": 41, "levels": 2, "radius": 0.0, "re": 100.0, "u": 0.05, "storage": "f32", "schedule": "fused",
         "scaling": "standard", "itime": "hold", "shift": "none", "steps": 60},
        # the uniform headline job: 500 steps of the 256^3 cube, fields in and out
        {"name": "tgv-256-f16", "kind": "uniform", "q": 19, "collision": "LBGK", "n": 256, "storage": "f16",
         "tau": 0.6, "steps": 500},
        # the same flow in the reference's precision on a cube that a convergence study uses
        {"name": "tgv-128-f64", "kind": "uniform", "q": 19, "collision": "LBGK", "n": 128, "storage": "f64",
         "tau": 0.6, "steps": 100},
        # cumulant cubes: a small one where the launches count, and a large one
        {"name": "tgv-64-cumulant-f32", "kind": "uniform", "q": 27, "collision": "Cumulant", "n": 64, "storage": "f32",
         "tau": 0.55, "steps": 400},
        {"name": "tgv-128-cumulant-f16", "kind": "uniform", "q": 27, "collision": "Cumulant", "n": 128,
         "storage": "f16", "tau": 0.55, "steps": 200},
        # the 4-level cumulant sphere, the largest multi-level case (under the
        # interface options that keep it finite)
        {"name": "sphere-4l-cumulant-f16", "kind": "flow", "body": "sphere", "q": 27, "collision": "Cumulant",
         "nx": 192, "ny": 96, "nz": 96, "levels": 3, "radius": 6.0, "re": 200.0, "u": 0.04, "storage": "f16",
         "schedule": "fused", "scaling": "standard", "itime": "hold", "shift": "none", "steps": 40},
        # half its size in FP32, the accurate fast form
        {"name": "sphere-4l-cumulant-f32", "kind": "flow", "body": "sphere", "q": 27, "collision": "Cumulant",
         "nx": 96, "ny": 48, "nz": 48, "levels": 3, "radius": 3.0, "re": 200.0, "u": 0.04, "storage": "f32",
         "schedule": "fused", "scaling": "standard", "itime": "hold", "shift": "none", "steps": 40},
        # bit-exact FP64 under the fused schedule, periodic sides of odd extent
        {"name": "sphere-3l-cumulant-f64", "kind": "flow", "body": "sphere", "q": 27, "collision": "Cumulant",
         "nx": 50, "ny": 26, "nz": 27, "levels": 2, "radius": 2.0, "re": 100.0, "u": 0.04, "storage": "f64",
         "schedule": "fused", "scaling": "standard", "itime": "hold", "shift": "none", "steps": 20},
        # a served request, from its specification to its drag and its flow
        {"name": "request-f16", "kind": "request", "radius": 5.4, "levels": 2, "re": 100.0, "oscillating": True,
         "storage": "f16", "steps": 125},
        # a batch of uneven instances, each too small to fill the GPU
        {"name": "batch-8-f16", "kind": "batch", "members": 8, "list_seed": 4, "most_cells": 65536, "most_levels": 2,
         "most_re": 120.0, "storage": "f16", "steps": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    """A case of the same ranges: any kind, storage, model and option, extents of any parity."""
    kind = rng.choice(["uniform", "flow", "flow", "flow", "request", "batch"])
    if kind == "uniform":
        q, coll = rng.choice([(19, "LBGK"), (27, "LBGK"), (27, "Cumulant")])
        return {"kind": kind, "q": q, "collision": coll, "n": rng.choice([16, 32, 64, 128]),
                "storage": rng.choice(["f64", "f32", "f16", "bf16"]), "tau": round(rng.uniform(0.53, 0.9), 4),
                "steps": _log_int(rng, 20, 100)}
    if kind == "request":
        return {"kind": kind, "radius": round(rng.uniform(3.0, 8.0), 3), "levels": rng.choice([1, 2]),
                "re": round(rng.uniform(20.0, 200.0), 2), "oscillating": rng.random() < 0.5,
                "storage": rng.choice(["f16", "f16", "f32"]), "steps": _log_int(rng, 20, 125)}
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(3, 8), "list_seed": 4, "most_cells": 65536,
                "most_levels": 2, "most_re": round(rng.uniform(100.0, 120.0), 2),
                "storage": rng.choice(["f16", "f16", "f32"]), "steps": _log_int(rng, 6, 20)}
    q, coll = rng.choice([(19, "LBGK"), (27, "Cumulant")])
    storage = rng.choice(["f64", "f32", "f16", "bf16"])
    c = {"kind": kind, "body": rng.choice(["sphere", "sphere", "cavity"]), "q": q, "collision": coll,
         "storage": storage, "schedule": "fused", "scaling": "standard", "itime": "hold",
         "shift": "none", "u": 0.05, "steps": _log_int(rng, 6, 20)}
    if storage == "f64" and rng.random() < 0.5:
        c["schedule"] = "phases"
    if c["body"] == "cavity":
        c.update(nx=_log_int(rng, 28, 90), ny=_log_int(rng, 28, 70), nz=_log_int(rng, 32, 70),
                 levels=rng.choice([1, 2]), radius=0.0, re=round(rng.uniform(50.0, 150.0), 2))
    else:
        r = rng.choice([2.0, 3.0, 4.0, 5.0])
        ny = _log_int(rng, 8.2 * r + 4, 14 * r)
        c.update(radius=r, ny=ny, nz=ny + rng.randint(-1, 2), nx=_log_int(rng, 12 * r + 6, 28 * r),
                 levels=rng.choice([1, 2, 3]), re=round(rng.uniform(20.0, 100.0 if q == 27 else 50.0), 2))
        if storage in ("f16", "bf16") and rng.random() < 0.3:
            c["shift"] = "far_field"
    return c


# ---- what a user's program has in hand ----------------------------------------

_context = []


def _ctx():
    if not _context:
        _context.append(Context(0))
    return _context[0]


class _State:
    """A prepared case; its device memory goes with it."""

    def __init__(self, **kw):
        self.batch = None
        self.managers = []
        self.__dict__.update(kw)

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        for m in self.managers:
            m.close()


def _flow_case(c):
    cells = (c["nx"], c["ny"], c["nz"])
    if c["body"] == "cavity":
        return cavity_case(q=c["q"], collision=c["collision"], coarse=cells, max_level=c["levels"], re=c["re"],
                           u_lid=c["u"], mesh="device")
    # nested boxes around a sphere in the front third of a channel
    r, levels = c["radius"], c["levels"]
    center = (int(max(c["nx"] // 3, 4 * r + 2)) if levels > 1 else max(c["nx"] // 4, int(3 * r) + 2), c["ny"] // 2,
              c["nz"] // 2)
    if levels == 1:
        half = [(3.0 * r, 2.0 * r, 2.0 * r)]
    else:
        half = [(h * r,) * 3 for h in (4.0, 2.5, 1.75)[:levels]]
    refine = [(tuple(int(round((center[a] - h[a]) * 2 ** l)) for a in range(3)),
               tuple(int(round((center[a] + h[a]) * 2 ** l)) for a in range(3))) for l, h in enumerate(half)]
    return sphere_case(q=c["q"], collision=c["collision"], coarse=cells, max_level=levels, refine=refine,
                       center=center, radius=r, u=c["u"], re=c["re"], mesh="device")


def _request(c, rng=None):
    re = c["re"] if rng is None else c["re"] * rng.uniform(0.8, 1.2)
    return Request(rid=0, arrival=0.0, radius=c["radius"], levels=c["levels"], re=re, oscillating=c["oscillating"],
                   finest_steps=c["steps"] << c["levels"])


def _batch_specs(c):
    few = [s for s in batched_uneven_cases(seed=c["list_seed"], n=64)
           if s.coarse[0] * s.coarse[1] * s.coarse[2] <= c["most_cells"] and s.levels <= c["most_levels"]
           and s.re <= c["most_re"]]
    return few[:c["members"]]


def _start_velocity(rng, u):
    return (u * rng.uniform(0.2, 1.0), 0.1 * u * rng.uniform(-1, 1), 0.1 * u * rng.uniform(-1, 1))


def _coordinates(n, device):
    """(x, y, z) of each cell of an n^3 cube in Morton order, x at bit 3i."""
    i = torch.arange(n ** 3, device=device)
    out = []
    for a in range(3):
        v = torch.zeros_like(i)
        for b in range(n.bit_length() - 1):
            v |= ((i >> (3 * b + a)) & 1) << b
        out.append(v)
    return out


def _tgv_fields(c, seed, device="cuda"):
    """rho, u, v, w in Morton order: the Taylor-Green vortex at seeded phases
    with a weak second harmonic, and its pressure in the density."""
    rng = np.random.default_rng(seed)
    n = c["n"]
    k = 2.0 * np.pi / n
    X, Y, Z = (k * (v.double() + 0.5) + float(p) for v, p in zip(_coordinates(n, device), rng.uniform(0, 2 * np.pi, 3)))
    e = 0.2 * float(rng.uniform(0.5, 1.0))
    u = U0 * (torch.sin(X) * torch.cos(Y) * torch.cos(Z) + e * torch.sin(2 * Y + 1.0))
    v = -U0 * (torch.cos(X) * torch.sin(Y) * torch.cos(Z) - e * torch.cos(2 * Z))
    w = U0 * e * torch.sin(2 * X) * torch.cos(Y)
    rho = 1.0 + 3.0 * (U0 * U0 / 16.0) * (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0)
    return rho, u, v, w


def prepare(case, seed):
    c, ctx = case, _ctx()
    rng = np.random.default_rng(seed)
    if c["kind"] == "uniform":
        d = DenseCase(ctx, uniform_box_case(q=c["q"], n=(c["n"],) * 3, collision=c["collision"],
                                            nu=(c["tau"] - 0.5) / 3.0, u_ref=U0, mesh="device"), c["storage"])
        given = torch.empty(4, d.n, dtype=torch.float64, pin_memory=True)
        for row, f in zip(given, _tgv_fields(c, seed)):
            row.copy_(f)
        got = torch.empty(4, d.n, dtype=torch.float64, pin_memory=True)
        return _State(case=c, managers=[d], given=given, got=got)
    if c["kind"] == "request":
        req = _request(c, rng)
        return _State(case=c, req=req, template=build_template(template_key(req), "device"),
                      u0=_start_velocity(rng, 0.1))
    if c["kind"] == "batch":
        ms = [LBM_Manager(ctx, s.build(mesh="device"), c["storage"], schedule="fused", scaling="standard",
                          interface_time="hold") for s in _batch_specs(c)]
        return _State(case=c, managers=ms, batch=Batch(ctx, ms), u0=[_start_velocity(rng, 0.05) for _ in ms])
    shift = None if c["shift"] == "none" else c["shift"]
    m = LBM_Manager(ctx, _flow_case(c), c["storage"], schedule=c["schedule"], scaling=c["scaling"],
                    storage_shift=shift, interface_time=c["itime"])
    return _State(case=c, managers=[m], u0=_start_velocity(rng, c["u"]))


# ---- one pass -------------------------------------------------------------------

def _fields(mgr, storage):
    """Density deviation and velocity of every level's cells, [4, cells]."""
    sizes = [mgr.size(l) for l in range(mgr.L + 1)]
    out = torch.empty(4, sum(sizes), dtype=DTYPE[storage])
    at = 0
    for l, n in enumerate(sizes):
        if n:
            rho, u = mgr.macros(l)
            rho -= 1.0
            out[0, at:at + n] = torch.from_numpy(rho)
            out[1:, at:at + n] = torch.from_numpy(u)
            at += n
    return out


def _mean_force(mgr, storage):
    f = mgr.force()
    return torch.from_numpy(f[:3] / max(f[3], 1.0)).to(DTYPE[storage])


def run(state):
    c = state.case
    st = c["storage"]
    if c["kind"] == "uniform":
        d, given, got = state.managers[0], state.given, state.got
        d.init_fields_ptr(*(row.data_ptr() for row in given))
        d.step(c["steps"])
        d.macros_ptr(got[0].data_ptr(), got[1].data_ptr())
        got[0] -= 1.0
        return {"fields": got if st == "f64" else got.to(DTYPE[st])}
    if c["kind"] == "request":
        m = LBM_Manager(_ctx(), request_case(state.req, state.template), st, schedule="fused", scaling="standard",
                        interface_time="hold")
        m.initial_equilibrium(1.0, state.u0)
        m.fluidSimulate(c["steps"])
        out = {"force": _mean_force(m, st), "fields": _fields(m, st)}
        m.close()
        return out
    if c["kind"] == "batch":
        for m, u in zip(state.managers, state.u0):
            m.reset_force()
            m.initial_equilibrium(1.0, u)
        state.batch.step(c["steps"])
        return [_fields(m, st) for m in state.managers]
    m = state.managers[0]
    m.reset_force()
    m.initial_equilibrium(1.0, state.u0)
    m.fluidSimulate(c["steps"])
    out = {"fields": _fields(m, st)}
    if c["body"] == "sphere":
        out["force"] = _mean_force(m, st)
    return out


# ---- what a pass cannot do without ------------------------------------------------

def _flow_work(case, storage, steps):
    p = case.params
    cells = estimate_cells(case.mesh.spec)
    updates = sum(n << l for l, n in enumerate(cells)) * steps
    return {"bytes": updates * 2.0 * p.q * BYTES[storage] + sum(cells) * 4.0 * 8.0,
            "flops": updates * FLOPS[(p.q, p.collision)]}


def work(case):
    c = case
    if c["kind"] == "uniform":
        n = c["n"] ** 3
        return {"bytes": c["steps"] * n * 2.0 * c["q"] * BYTES[c["storage"]] + n * 64.0,
                "flops": c["steps"] * n * FLOPS[(c["q"], c["collision"])]}
    if c["kind"] == "request":
        req = _request(c)
        one = [request_case(req, build_template(template_key(req), "device"))]
    elif c["kind"] == "batch":
        one = [s.build(mesh="device") for s in _batch_specs(c)]
    else:
        one = [_flow_case(c)]
    w = [_flow_work(x, c["storage"], c["steps"]) for x in one]
    return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}


# ---- the uniform cubes in 64 bits ---------------------------------------------------

def _directions(q):
    """(e, weight) of D3Q19 / D3Q27."""
    out = []
    for e in itertools.product((-1, 0, 1), repeat=3):
        s = sum(v * v for v in e)
        if q == 19 and s == 3:
            continue
        w = {19: (1 / 3, 1 / 18, 1 / 36), 27: (8 / 27, 2 / 27, 1 / 54, 1 / 216)}[q][s]
        out.append((e, w))
    return out


def _moments(f, dirs):
    rho = sum(f)
    return rho, [sum(e[a] * g for (e, _), g in zip(dirs, f) if e[a]) / rho for a in range(3)]


def _equilibrium(e, w, rho, u, uu):
    eu = sum(e[a] * u[a] for a in range(3) if e[a]) if any(e) else torch.zeros_like(rho)
    return w * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu)


def _cumulant(f, dirs, omega):
    """Second-order cumulants relaxed (shear omega, bulk 1), the higher ones
    set to zero; the moments (2,1,0), (1,0,2), (0,2,1) keep their values."""
    rho, u = _moments(f, dirs)
    orders = list(itertools.product(range(3), repeat=3))
    need = [o for o in orders if sum(o) <= 2] + [(2, 1, 0), (1, 0, 2), (0, 2, 1)]
    need = [o for o in need if max(o) <= 2]
    m = {o: torch.zeros_like(rho) for o in orders}
    for (e, _), g in zip(dirs, f):
        d = [e[a] - u[a] for a in range(3)]
        for o in need:
            t = g
            for a in range(3):
                for _ in range(o[a]):
                    t = t * d[a]
            m[o] += t
    xx, yy, zz, xy, xz, yz = m[2, 0, 0], m[0, 2, 0], m[0, 0, 2], m[1, 1, 0], m[1, 0, 1], m[0, 1, 1]
    dx = -(omega * (2 * xx - yy - zz) + (xx + yy + zz - m[0, 0, 0])) / rho / 2
    dy = dx + 1.5 * omega * (xx - yy) / rho
    dz = dx + 1.5 * omega * (xx - zz) / rho
    u2 = [v * v for v in u]
    a1 = (1 - omega) * (xx - yy) - 3 * rho * (1 - omega / 2) * (u2[0] * dx - u2[1] * dy)
    a2 = (1 - omega) * (xx - zz) - 3 * rho * (1 - omega / 2) * (u2[0] * dx - u2[2] * dz)
    a3 = m[0, 0, 0] - 1.5 * rho * (u2[0] * dx + u2[1] * dy + u2[2] * dz)
    xx = (a1 + a2 + a3) / 3
    yy, zz = xx - a1, xx - a2
    xy, xz, yz = (1 - omega) * xy, (1 - omega) * xz, (1 - omega) * yz
    m[2, 0, 0], m[0, 2, 0], m[0, 0, 2], m[1, 1, 0], m[1, 0, 1], m[0, 1, 1] = xx, yy, zz, xy, xz, yz
    m[2, 1, 1] = (xx * yz + 2 * xy * xz) / rho
    m[1, 2, 1] = (yy * xz + 2 * yz * xy) / rho
    m[1, 1, 2] = (zz * xy + 2 * xz * yz) / rho
    m[2, 2, 0] = (xx * yy + 2 * xy * xy) / rho
    m[0, 2, 2] = (yy * zz + 2 * yz * yz) / rho
    m[2, 0, 2] = (zz * xx + 2 * xz * xz) / rho
    m[1, 2, 2] = (yy * m[1, 0, 2] + 2 * xz * m[0, 2, 1]) / rho
    m[2, 1, 2] = (zz * m[2, 1, 0] + 2 * xy * m[1, 0, 2]) / rho
    m[2, 2, 1] = (xx * m[0, 2, 1] + 2 * yz * m[2, 1, 0]) / rho
    m[2, 2, 2] = (xx * m[0, 2, 2] + yy * m[2, 0, 2] + zz * m[2, 2, 0]
                  + 4 * (yz * m[2, 1, 1] + xz * m[1, 2, 1] + xy * m[1, 1, 2])) / rho \
        - (16 * xy * xz * yz + 4 * (xz * xz * yy + yz * yz * xx + xy * xy * zz) + 2 * xx * yy * zz) / rho ** 2
    for a in range(3):  # central moments to populations, one axis at a time
        v, p = u[a], {}
        for o in itertools.product(range(3), repeat=2):
            k = [o[:a] + (i,) + o[a:] for i in range(3)]
            s0, s1, s2 = (m[x] for x in k)
            p[k[0]] = (s0 * (v * v - v) + s1 * (2 * v - 1) + s2) / 2
            p[k[1]] = s0 * (1 - v * v) - 2 * s1 * v - s2
            p[k[2]] = (s0 * (v * v + v) + s1 * (2 * v + 1) + s2) / 2
        m = p
    return [m[tuple(v + 1 for v in e)] for e, _ in dirs]


def exact(case, seed):
    """The uniform cubes in plain torch, FP64, on a (x, y, z) grid: collide,
    then f_e(x) takes the value of x + e (the reference's pull).  The
    multi-level cases have no such value: their lattices and interface
    transfers are the framework itself."""
    c = case
    if c["kind"] != "uniform":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n, dirs, omega = c["n"], _directions(c["q"]), 1.0 / c["tau"]
    at = _coordinates(n, dev)
    grid = []
    for f in _tgv_fields(c, seed, dev):
        g = torch.empty(n, n, n, dtype=torch.float64, device=dev)
        g[at[0], at[1], at[2]] = f
        grid.append(g)
    rho, u = grid[0], grid[1:]
    uu = sum(v * v for v in u)
    f = [_equilibrium(e, w, rho, u, uu) for e, w in dirs]
    for _ in range(c["steps"]):
        if c["collision"] == "Cumulant":
            f = _cumulant(f, dirs, omega)
        else:
            rho, u = _moments(f, dirs)
            uu = sum(v * v for v in u)
            for k, (e, w) in enumerate(dirs):
                f[k] = f[k] + omega * (_equilibrium(e, w, rho, u, uu) - f[k])
        f = [torch.roll(g, tuple(-v for v in e), (0, 1, 2)) if any(e) else g for g, (e, _) in zip(f, dirs)]
    rho, u = _moments(f, dirs)
    out = torch.stack([v[at[0], at[1], at[2]] for v in (rho - 1.0, *u)])
    return {"fields": out.cpu()}
