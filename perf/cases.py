"""Workloads of the framework as its users run them, for timing and comparing builds.

A simulation run is "one output interval": the world is uploaded from pinned
host memory (a resume, or a host program handing its world over), advanced by
a few steps, and downloaded, brick-sorted, for output. The other workloads are
the projection driven by a host integrator (speed fields in, pressure and
speeds out), the drop-in CSC linear solver in its two forms, and the learned
preconditioner's network forward and in training.

    listed()            the workloads that are always timed
    draw(rng)           one more of the same ranges
    prepare(case, seed) what a program holds before the call
    run(state)          one pass through the public entry points
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   run's outputs in 64-bit torch where a direct form exists
"""
from __future__ import annotations

import ctypes
import dataclasses
import functools
import os

import numpy as np
import torch

from mac_b200.gpu import Context, HostState, load
from mac_b200.state import FLUID, Params, jet_world, lateral_jet_world, pool_spheres_world
from mac_b200.unet import UNet
from mac_b200.world import setup_passes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WEIGHTS = os.path.join(ROOT, "mac_b200", "weights", "unet_pool64.npz")
_P = ctypes.POINTER
_OFF = 1 << 20


# ------------------------------------------------------------------ the workloads
def _jet(name, nx, ny, nz, h, r, w, pool, solver, steps, dt_max=0.01, viscosity=0.0, depth=0, pipeline=0):
    c = dict(kind="jet", nx=nx, ny=ny, nz=nz, h=h, r=r, w=w, pool=pool, solver=solver, steps=steps, dt_max=dt_max,
             viscosity=viscosity, depth=depth, pipeline=pipeline)
    return dict(c, name=name) if name else c


def _lateral(name, nx, ny, nz, r, solver, steps):
    c = dict(kind="lateral", nx=nx, ny=ny, nz=nz, h=0.01, r=r, solver=solver, steps=steps)
    return dict(c, name=name) if name else c


def _named(name, **c):
    return dict(c, name=name) if name else c


def listed():
    return [
        # the small vertical jet of the reference's own experiments (32x32x64 at 5 cm, FP64), where launches and
        # host round trips count
        _jet("jet32_fp64", 32, 32, 64, 0.05, 4.0, 1.0, 8, "mgpcg64", 10, dt_max=0.1),
        # an ordinary run: a box that no brick edge divides, FP32 multigrid inside the FP64 solve
        _jet("jet100_mixed", 100, 84, 150, 0.01, 12.0, 2.0, 37, "mixed", 10),
        # the full-size jet: 8M fluid cells and 64M particles
        _jet("jet256_mixed", 256, 256, 512, 0.01, 24.0, 2.0, 122, "mixed", 10),
        # the lateral jet: a stream through the air, drops and a thin layer on the floor, with the boundary-condition
        # extrapolation that the experiment runs before each output (every five steps)
        _lateral("lateral384_mixed", 384, 192, 192, 16.0, "mixed", 5),
        # the viscous composition (viscous forces, Dirichlet air pressures)
        _jet("viscous_fp64", 60, 44, 72, 0.02, 5.0, 1.0, 20, "mgpcg64", 5, viscosity=1e-3),
        # the depth composition stepped by the four-stage integrator over grid and particles (pipeline B)
        _jet("pipeline_b_fp64", 56, 48, 64, 0.02, 5.0, 1.0, 30, "mgpcg64", 3, viscosity=1e-3, depth=1, pipeline=1),
        # the standalone Poisson problem, 128^3 pool with 12 spheres to 1e-10, driven by a host integrator
        _named("project128_fp64", kind="project", n=128, solver="mgpcg64", rtol=1e-10),
        # the same call at the smallest size: latency only
        _named("project20_mixed", kind="project", n=20, solver="mixed", rtol=1e-8),
        # one application of the learned preconditioner on the 128^3 grid
        _named("unet_forward128", kind="unet", n=1, d=128, h=128, w=128),
        # one training gradient: batch 16 of 64^3 patches, energy loss
        _named("unet_grad64", kind="grad", n=16, d=64, h=64, w=64),
        # the linear-solver policy on matrices handed over by the reference's assembly: factorise, solve, clean
        _named("csc_policy", kind="csc", nx=32, ny=32, nz=20, spheres=4),
        # the allocation-free solve of a system already on the device
        _named("csc_device", kind="csc_device", nx=44, ny=40, nz=37, spheres=3),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["jet", "jet", "jet", "lateral", "viscous", "b", "project", "project", "unet", "grad", "csc",
                       "csc_device"])
    solver = rng.choice(["mgpcg64", "mixed"])
    if kind == "jet":
        nx, ny, nz = _log(rng, 24, 180), _log(rng, 24, 180), _log(rng, 32, 300)
        r = max(2.0, min(nx, ny) * (0.05 + 0.1 * rng.random()))
        return _jet(None, nx, ny, nz, rng.choice([0.01, 0.02, 0.05]), r, 0.5 + 2.0 * rng.random(),
                    max(4, int(nz * (0.12 + 0.25 * rng.random()))), solver, rng.choice([5, 10]),
                    dt_max=rng.choice([0.01, 0.1]))
    if kind == "lateral":
        nx, ny, nz = _log(rng, 96, 384), _log(rng, 64, 192), _log(rng, 64, 192)
        return _lateral(None, nx, ny, nz, max(3.0, min(ny, nz) / 12.0), solver, 5)
    if kind in ("viscous", "b"):
        nx, ny, nz = _log(rng, 24, 90), _log(rng, 24, 90), _log(rng, 32, 96)
        b = kind == "b"
        return _jet(None, nx, ny, nz, 0.02, max(2.0, min(nx, ny) / 10.0), 0.5 + rng.random(),
                    max(8, int(nz * (0.2 + 0.3 * rng.random()))), solver, 2 if b else 5,
                    viscosity=10.0 ** (-4 + 2 * rng.random()), depth=int(b), pipeline=int(b))
    if kind == "project":
        return dict(kind="project", n=_log(rng, 16, 150), solver=solver, rtol=rng.choice([1e-8, 1e-10, 1e-12]))
    if kind in ("unet", "grad"):
        top = 136 if kind == "unet" else 72
        d, h, w = (4 * max(4, _log(rng, 16, top) // 4) for _ in range(3))
        return dict(kind=kind, n=1 if kind == "unet" else rng.choice([1, 2, 4, 8, 16]), d=d, h=h, w=w)
    if kind == "csc":
        return dict(kind="csc", nx=_log(rng, 8, 36), ny=_log(rng, 8, 36), nz=_log(rng, 8, 36),
                    spheres=rng.randrange(1, 6))
    return dict(kind="csc_device", nx=_log(rng, 8, 40), ny=_log(rng, 8, 40), nz=_log(rng, 8, 40),
                spheres=rng.randrange(1, 6))


# ------------------------------------------------------------------ simulation runs
@functools.lru_cache(maxsize=3)
def _walls(kind, nx, ny, nz, h, r, w, dt_max):
    """Walls and inflow of a jet world after the one-time set-up passes (no seed in it; not to be changed)."""
    if kind == "jet":
        s = jet_world(nx, ny, nz, h=h, r_inflow=r, w_inflow=w, dt_max=dt_max)
    else:
        s = lateral_jet_world(nx, ny, nz, h=h, r_inflow=r)
    return setup_passes(s)


def _fluid_cells(case):
    """Keys (n, 3) of the cells that start filled (the case's, whatever the seed), on the GPU."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    m = torch.zeros((nz, ny, nx), dtype=torch.bool, device="cuda")
    if case["kind"] == "jet":
        m[:case["pool"]] = True
    else:
        m[:3] = True  # a thin layer on the floor
        z, y, x = (torch.arange(k, device="cuda", dtype=torch.float64) for k in (nz, ny, nx))
        vx, vz, _ = _stream(case)
        t = x / vx  # the stream: cells within the inflow's radius of the ballistic path
        path = nz / 4.0 + vz * t - 0.5 * (9.81 / case["h"]) * t * t
        d2 = (z[:, None, None] - path[None, None, :]) ** 2 + (y[None, :, None] - (ny - 1) / 2.0) ** 2
        m |= d2 <= (0.9 * case["r"]) ** 2
        lim = torch.tensor([nx, ny, nz], dtype=torch.float64, device="cuda")
        rng = np.random.default_rng(11)
        for k in range(48):  # drops
            c = (torch.from_numpy(rng.random(3)).cuda() * 0.7 + 0.15) * lim
            rad = 1.5 + 3.0 * rng.random()
            m |= ((z[:, None, None] - c[2]) ** 2 + (y[None, :, None] - c[1]) ** 2 + (x[None, None, :] - c[0]) ** 2) \
                <= rad * rad
    return m.nonzero().flip(1)  # (x, y, z), z-major order


def _stream(case):
    a = np.deg2rad(15.0)
    return 3.0 * np.cos(a) / case["h"], 3.0 * np.sin(a) / case["h"], 3.0 * np.cos(a)


def _particles(cells, h, g):
    """Eight jittered particles a cell, cell-major: (8 n, 3) FP64 on the GPU."""
    o = torch.tensor([[0.25 if (s >> i) & 1 else -0.25 for i in range(3)] for s in range(8)], dtype=torch.float64,
                     device="cuda")
    j = torch.rand((cells.shape[0], 8, 3), generator=g, device="cuda", dtype=torch.float64)
    j -= 0.5
    j *= 0.499
    j += o[None]
    j += cells[:, None, :]
    j *= h
    return j.view(-1, 3)


def _sort_bricks(host, out):
    """The downloaded world with its bricks in (z, y, x) key order, into the arrays of `out` (0 past the last)."""
    nb = host.nbricks
    k = torch.from_numpy(host.keys[:3 * nb]).view(nb, 3)
    q = k.long() + _OFF
    order = torch.argsort((q[:, 2] << 42) | (q[:, 1] << 21) | q[:, 0])
    torch.index_select(k, 0, order, out=out["keys"][:nb])
    arrays = dict(host.f64, exists=host.exists, flags=host.flags, type=host.type, layer=host.layer)
    if host.depth is not None:
        arrays["depth"] = host.depth
    for n, a in arrays.items():
        torch.index_select(torch.from_numpy(a[:nb * 512]).view(nb, 512), 0, order, out=out[n][:nb])
    for a in out.values():
        a[nb:].zero_()
    return out


def _sorted_buffers(host):
    nb = host.cap_bricks
    out = {"keys": torch.empty((nb, 3), dtype=torch.int32)}
    arrays = dict(host.f64, exists=host.exists, flags=host.flags, type=host.type, layer=host.layer)
    if host.depth is not None:
        arrays["depth"] = host.depth
    for n, a in arrays.items():
        out[n] = torch.zeros((nb, 512), dtype=torch.from_numpy(a[:1]).dtype)
    return out


def _prepare_run(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    h = case["h"]
    lateral = case["kind"] == "lateral"
    s = _walls(case["kind"], case["nx"], case["ny"], case["nz"], h, case["r"], case.get("w", 0.0),
               case.get("dt_max", 0.01))
    pr = dataclasses.replace(s.params, viscosity=case.get("viscosity", 0.0))
    if case.get("depth"):
        pr = dataclasses.replace(pr, depth_mode=1, depth_max=4, depth_interior=3, depth_remove=3, refill_cube=1,
                                 pipeline=case["pipeline"])
    depth = bool(pr.depth_mode)
    cells = _fluid_cells(case)
    pos = _particles(cells, h, g)
    first = HostState(s.nbricks, pos.shape[0], pinned=True, depth=depth, stage_buffers=False)
    s0 = dataclasses.replace(s, params=pr)
    first.fill(s0)
    first.nparticles = pos.shape[0]
    torch.from_numpy(first.pos)[:pos.numel()].copy_(pos.view(-1))
    # room for the bricks around the fluid and for what the inflow adds
    extra = 3000 + 60 * int(case["r"] ** 2 + 1) * (case["steps"] + 2) * (4 if depth else 1)
    b = cells // 8
    fluid_bricks = torch.unique((b[:, 2] << 20) | (b[:, 1] << 10) | b[:, 0]).numel()
    max_bricks = 2048 + s.nbricks + (12 * fluid_bricks if lateral else fluid_bricks * 5 // 4)
    max_bricks = min(max_bricks, (case["nx"] // 8 + 6) * (case["ny"] // 8 + 6) * (case["nz"] // 8 + 6))
    del cells, pos, b
    ctx = Context(pr, max_bricks=max_bricks, max_particles=int(first.nparticles * 1.02) + extra,
                  solver=case["solver"], rtol=1e-8)
    # the reference's first init on the device; the world it leaves is what the run starts from
    ctx.upload(None, host=first)
    ctx.first_init_topology()
    nb, npart = ctx.sizes()
    raw = ctx.download(host=HostState(nb, npart, pinned=True, depth=depth, stage_buffers=False), to_state=False)
    srt = _sort_bricks(raw, _sorted_buffers(raw))
    # a smooth speed field (plus the stream's ballistic speed) on every face that is not const
    key = srt["keys"].cuda().to(torch.float64)[:, None, :] * 8
    o = torch.arange(512, device="cuda")
    c = [(key[..., 0] + (o % 8)) * h, (key[..., 1] + (o // 8 % 8)) * h, (key[..., 2] + o // 64) * h]
    ph = torch.rand((3, 3), generator=g, device="cuda", dtype=torch.float64) * 6.2831853
    size = [case[k] * h for k in ("nx", "ny", "nz")]
    flags, ex = srt["flags"].cuda(), srt["exists"].cuda() != 0
    amp = 0.2 * (case.get("w") or 2.0)
    for i, n in enumerate(("u0x", "u0y", "u0z")):
        v = amp * torch.sin(c[0] * (6.0 / size[0]) + ph[i, 0]) * torch.sin(c[1] * (6.0 / size[1]) + ph[i, 1]) \
            * torch.cos(c[2] * (6.0 / size[2]) + ph[i, 2])
        if lateral and i != 1:
            vx, vz, ux = _stream(case)
            up = vz * h - 9.81 * (c[0] / ux) if i == 2 else torch.full_like(c[0], ux)
            v = torch.where(c[2] >= 6 * h, up, v)
        free = ex & ((flags >> i) & 1 == 0)
        srt[n].copy_(torch.where(free, v, srt[n].cuda()))
    for n, a in raw.f64.items():
        torch.from_numpy(a[:nb * 512]).view(nb, 512).copy_(srt[n])
    torch.from_numpy(raw.keys[:3 * nb]).view(nb, 3).copy_(srt["keys"])
    for n, a in (("exists", raw.exists), ("flags", raw.flags), ("type", raw.type), ("layer", raw.layer)):
        torch.from_numpy(a[:nb * 512]).view(nb, 512).copy_(srt[n])
    if depth:
        torch.from_numpy(raw.depth[:nb * 512]).view(nb, 512).copy_(srt["depth"])
    out = HostState(max(nb + 256, int(nb * 1.05)), npart + extra - 2500, pinned=True, depth=depth, stage_buffers=False)
    return dict(kind="run", ctx=ctx, host=raw, out=out, sorted=_sorted_buffers(out), steps=case["steps"],
                boundary=lateral)


def _run_run(st):
    ctx = st["ctx"]
    ctx.upload(None, host=st["host"])
    for _ in range(st["steps"]):
        ctx.step()
    if st["boundary"]:
        ctx.extrapolate_boundary_condition(0)
    host = ctx.download(host=st["out"], to_state=False)
    res = dict(_sort_bricks(host, st["sorted"]))
    if host.depth is not None:
        # the depth composition removes particles and leaves the others in no order: sorted for output
        pos = torch.from_numpy(host.pos[:3 * host.nparticles]).view(-1, 3)
        q = pos.cuda()
        for i in (2, 1, 0):
            q = q[torch.argsort(q[:, i], stable=True)]
        pos.copy_(q)
    host.pos[3 * host.nparticles:] = 0.0
    return dict(res, pos=host.pos, t=host.t, dt=host.dt, nbricks=host.nbricks, nparticles=host.nparticles)


# ------------------------------------------------------------------ projection alone
@functools.lru_cache(maxsize=3)
def _pool(n):
    return setup_passes(pool_spheres_world(n, r_range=(6.0 * n / 128, 20.0 * n / 128)))


_SPEEDS = ("u0x", "u0y", "u0z")


def _pool_speeds(s, seed):
    """Face speeds uniform in [-1, 1] on the faces that are not const, (nb, 512) on the GPU, and those faces."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    ex = torch.from_numpy(s.exists).cuda() != 0
    fl = torch.from_numpy(s.flags).cuda()
    free = [ex & ((fl >> i) & 1 == 0) for i in range(3)]
    return [torch.where(f, torch.rand(f.shape, generator=g, device="cuda", dtype=torch.float64) * 2 - 1, 0.0)
            for f in free], free


def _prepare_project(case, seed):
    s = _pool(case["n"])
    u, _ = _pool_speeds(s, seed)
    nc = s.nbricks * 512
    pin = lambda: torch.empty(nc, dtype=torch.float64, pin_memory=True)
    src, dst = [pin() for _ in range(3)], [pin() for _ in range(4)]
    for a, b in zip(src, u):
        a.copy_(b.view(-1))
    ctx = Context(s.params, max_bricks=int(s.nbricks * 1.1) + 64, max_particles=1024, solver=case["solver"],
                  rtol=case["rtol"], max_iters=1000)
    ctx.upload(s)
    return dict(kind="project", ctx=ctx, src=src, dst=dst)


def _run_project(st):
    ctx, lib = st["ctx"], st["ctx"].lib
    fields = [Context.FIELDS.index(n) for n in _SPEEDS]
    ptr = lambda a: ctypes.cast(a.data_ptr(), _P(ctypes.c_double))
    for f, a in zip(fields, st["src"]):
        ctx._check(lib.mac_upload_field(ctx.h, f, ptr(a)), "mac_upload_field")
    ctx.pressure_init()
    ctx.divergence_projection(0)
    ctx.pressure_end()
    for f, a in zip(fields + [Context.FIELDS.index("p")], st["dst"]):
        ctx._check(lib.mac_download_field(ctx.h, f, ptr(a)), "mac_download_field")
    return dict(zip(_SPEEDS + ("p",), st["dst"]))


def _shift(a, axis, by):
    """a(c + by e_axis), 0 outside the grid."""
    r = torch.zeros_like(a)
    d = 2 - axis
    n = a.shape[d]
    if by > 0:
        r.narrow(d, 0, n - 1).copy_(a.narrow(d, 1, n - 1))
    else:
        r.narrow(d, 1, n - 1).copy_(a.narrow(d, 0, n - 1))
    return r


def _cg(apply, b, dinv, tol=1e-15, most=6000):
    x, r = torch.zeros_like(b), b.clone()
    z = dinv * r
    p, rz, bb = z.clone(), (r * z).sum(), (b * b).sum()
    for it in range(most):
        q = apply(p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        z = dinv * r
        new = (r * z).sum()
        if it % 20 == 19 and float((r * r).sum() / bb) <= tol * tol:
            break
        p = z + (new / rz) * p
        rz = new
    return x


def _exact_project(case, seed):
    s = _pool(case["n"])
    u, free = _pool_speeds(s, seed)
    m = case["n"] + 6  # the box with its shell and the cells that the set-up passes add beyond it
    key = torch.from_numpy(s.keys).cuda().long()[:, None, :] * 8
    o = torch.arange(512, device="cuda")
    c = [key[..., 0] + (o % 8) + 1, key[..., 1] + (o // 8 % 8) + 1, key[..., 2] + o // 64 + 1]
    ins = (c[0] >= 0) & (c[0] < m) & (c[1] >= 0) & (c[1] < m) & (c[2] >= 0) & (c[2] < m)
    at = (c[2] * m + c[1]) * m + c[0]

    def dense(a):
        r = torch.zeros(m * m * m, dtype=a.dtype, device="cuda")
        r[at[ins]] = a[ins]
        return r.view(m, m, m)
    dom = dense((torch.from_numpy(s.exists).cuda() != 0) & (torch.from_numpy(s.type).cuda() == FLUID))
    U, F = [dense(a) for a in u], [dense(f) for f in free]
    ih = 1.0 / s.params.h[0]
    div = sum((_shift(U[i], i, 1) - U[i]) * ih for i in range(3)) * dom
    # a face carries a pressure difference where it is not const
    diag = sum(F[i].double() + _shift(F[i].double(), i, 1) for i in range(3)) * dom
    w = [F[i] & dom & _shift(dom.double(), i, -1).bool() for i in range(3)]

    def apply(p):
        q = diag * p
        for i in range(3):
            q -= w[i] * _shift(p, i, -1) + _shift(w[i].double(), i, 1) * _shift(p, i, 1)
        return q * (ih * ih)
    dinv = torch.where(diag > 0, 1.0 / (diag.clamp(min=1.0) * ih * ih), torch.zeros_like(diag))
    p = _cg(apply, -div, dinv) * dom
    near = [F[i] & (dom | _shift(dom.double(), i, -1).bool()) for i in range(3)]
    res = [U[i] - near[i] * (p - _shift(p, i, -1)) * ih for i in range(3)] + [p]
    back = lambda d: torch.where(ins, d.reshape(-1)[at.clamp(0, m ** 3 - 1)], 0.0).view(-1)
    return {n: back(a) for n, a in zip(_SPEEDS + ("p",), res)}


# ------------------------------------------------------------------ drop-in linear solver
def _system(case, seed):
    """The pressure matrix of a pool with spheres in a walled box, as the reference assembles it (CSC, rows sorted),
    and the right-hand side of random face speeds."""
    rng = np.random.default_rng(11)  # the geometry is the case's, the right-hand side the seed's
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    m = z < max(2, 0.75 * nz)
    for _ in range(case["spheres"]):
        c, r = rng.random(3) * (nx, ny, nz), 1.0 + 0.15 * min(nx, ny, nz) * rng.random()
        m |= (x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2 <= r * r
    m[-1, ny // 2, nx // 2] = False  # the box is never full
    h = 0.05
    ident = np.full(m.shape, -1, np.int64)
    ident[m] = np.arange(int(m.sum()))
    me = ident[m]
    diag = np.zeros(len(me))
    rows, cols = [me], [me]
    for ax in range(3):
        for sg in (-1, 1):
            pad = np.pad(ident, [(1, 1)] * 3, constant_values=-2)  # -2: wall (Neumann), -1: air (Dirichlet)
            nb = pad[tuple(slice(1 + (sg if a == 2 - ax else 0), 1 + (sg if a == 2 - ax else 0) + m.shape[a])
                           for a in range(3))][m]
            diag -= (nb != -2) / (h * h)
            rows.append(nb[nb >= 0])
            cols.append(me[nb >= 0])
    diag[diag == 0] = -1.0 / (h * h)
    vals = np.concatenate([diag] + [np.full(len(r), 1.0 / (h * h)) for r in rows[1:]])
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((rows, cols))
    off = np.zeros(len(me) + 1, np.int32)
    off[1:] = np.cumsum(np.bincount(cols, minlength=len(me)))
    return off, rows[order].astype(np.int32), vals[order], \
        np.random.default_rng(seed).uniform(-1.0, 1.0, len(me)) / h


def _prepare_csc(case, seed):
    off, ind, val, b = _system(case, seed)
    if case["kind"] == "csc":
        ctx = Context(Params(h=(0.05, 0.05, 0.05)), max_bricks=64, max_particles=1024, rtol=1e-12, max_iters=5000)
        return dict(kind="csc", ctx=ctx, system=(off, ind, val, b))
    dev = [torch.from_numpy(a).cuda() for a in (off, ind, val, b)]
    lib = load()
    lib.mac_csc_solve_noalloc(None, 0, None, None, None, None, None, 1e-12, 0, None, None)  # the one-time set-up
    return dict(kind="csc_device", lib=lib, dev=dev, x=torch.empty_like(dev[3]))


def _run_csc(st):
    if st["kind"] == "csc":
        return st["ctx"].csc_solve(*st["system"])
    off, ind, val, b = st["dev"]
    rc = st["lib"].mac_csc_solve_noalloc(torch.cuda.current_stream().cuda_stream, b.numel(), off.data_ptr(),
                                         ind.data_ptr(), val.data_ptr(), b.data_ptr(), st["x"].data_ptr(), 1e-12,
                                         5000, None, None)
    if rc != 0:
        raise RuntimeError(f"mac_csc_solve_noalloc: {rc}")
    return st["x"]


def _exact_csc(case, seed):
    off, ind, val, b = (torch.from_numpy(a).cuda() for a in _system(case, seed))
    A = torch.sparse_csr_tensor(off.long(), ind.long(), -val)  # symmetric: the columns read as rows
    n = b.numel()
    col = torch.repeat_interleave(torch.arange(n, device="cuda"), (off[1:] - off[:-1]).long())
    d = torch.zeros(n, dtype=torch.float64, device="cuda")
    d[col[ind.long() == col]] = -val[ind.long() == col]
    return _cg(lambda p: A @ p, -b, 1.0 / d)


# ------------------------------------------------------------------ the network
def _patches(case, seed):
    """Masks (pool below 0.4 of the height, spheres, some solid), residuals and errors of a batch, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, d, h, w = case["n"], case["d"], case["h"], case["w"]
    z = torch.arange(d, device="cuda").view(1, d, 1, 1)
    y = torch.arange(h, device="cuda").view(1, 1, h, 1)
    x = torch.arange(w, device="cuda").view(1, 1, 1, w)
    m = (z < 0.4 * d).expand(n, d, h, w).clone()
    for _ in range(12):
        q = torch.rand((n, 4), generator=g, device="cuda").view(n, 4, 1, 1, 1)
        rad = (0.05 + 0.1 * q[:, 3]) * min(d, h, w)
        m |= (z - q[:, 0] * d) ** 2 + (y - q[:, 1] * h) ** 2 + (x - q[:, 2] * w) ** 2 <= rad * rad
    mask = m.to(torch.int8)
    mask[:, :, :, -1] = -1
    r = torch.randn((n, d, h, w), generator=g, device="cuda")
    smooth = torch.nn.functional.avg_pool3d(r[:, None], 5, 1, 2)[:, 0]
    r = (0.3 * r + 3.0 * smooth) * (mask == 1)
    e = (2.0 * smooth + 0.05 * torch.randn((n, d, h, w), generator=g, device="cuda")) * (mask == 1)
    return r, mask, e


def _prepare_unet(case, seed):
    r, m, e = (t.cpu().numpy() for t in _patches(case, seed))
    net = UNet(0)
    if case["kind"] == "unet":
        net.load(WEIGHTS)
    else:
        net._check(net.lib.mac_unet_init(net.h, 5), "mac_unet_init")
        net.set_loss("energy")
    return dict(kind=case["kind"], net=net, r=r, m=m, e=e)


def _run_unet(st):
    if st["kind"] == "unet":
        return st["net"].forward(st["r"], st["m"])
    loss, grad = st["net"].loss_grad(st["r"], st["m"], st["e"])
    return {"loss": loss, "grad": grad}


#: cin, cout, taps, relu of each layer as stored, and the channels it uses
_LAYERS = [(16, 16, 27, 1, 2, 16), (16, 16, 27, 1, 16, 16), (16, 32, 27, 1, 16, 32), (32, 32, 27, 1, 32, 32),
           (32, 64, 27, 1, 32, 64), (64, 64, 27, 1, 64, 64), (64, 32, 1, 0, 64, 32), (64, 32, 27, 1, 64, 32),
           (32, 32, 27, 1, 32, 32), (32, 16, 1, 0, 32, 16), (32, 16, 27, 1, 32, 16), (16, 16, 27, 1, 16, 16),
           (16, 16, 1, 0, 16, 1)]
_LEVEL = [0, 0, 1, 1, 2, 2, 2, 1, 1, 1, 0, 0, 0]


def _net64(p, r, mask):
    """The network in FP64 on one sample [1, d, h, w]; p: the flat parameters, FP64 on the GPU."""
    ws, o = [], 0
    for cin, cout, taps, relu, rin, rout in _LAYERS:
        k = 3 if taps == 27 else 1
        w = p[o:o + taps * cout * cin].view(taps, cout, cin)[:, :rout, :rin]
        ws.append((w.permute(1, 2, 0).reshape(rout, rin, k, k, k), p[o + taps * cout * cin:][:rout], relu))
        o = (o + taps * cout * cin + cout + 7) // 8 * 8

    def conv(l, v):
        w, b, relu = ws[l]
        k = w.shape[2] // 2
        q = torch.nn.functional.pad(v[0], (k, k) * 3)
        d, hh, ww = v.shape[2:]
        y = b.view(-1, 1).expand(-1, d * hh * ww)
        for a in range(2 * k + 1):  # one product a tap: plain FP64 arithmetic, whatever the library has
            for c in range(2 * k + 1):
                for e in range(2 * k + 1):
                    y = y + w[:, :, a, c, e] @ q[:, a:a + d, c:c + hh, e:e + ww].reshape(v.shape[1], -1)
        y = y.view(1, -1, d, hh, ww)
        return y.relu() if relu else y
    pool = lambda v: torch.nn.functional.avg_pool3d(v, 2)
    up = lambda v: v.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
    fl = mask == 1
    rms = (r[fl] ** 2).mean().sqrt() if bool(fl.any()) else torch.ones((), device=r.device, dtype=r.dtype)
    rms = torch.where(rms > 0, rms, torch.ones_like(rms))
    s1 = conv(1, conv(0, torch.stack([r / rms * fl, mask.double()], 1)))
    s2 = conv(3, conv(2, pool(s1)))
    b3 = conv(5, conv(4, pool(s2)))
    d2 = conv(8, conv(7, torch.cat([s2, up(conv(6, b3))], 1)))
    d1 = conv(11, conv(10, torch.cat([s1, up(conv(9, d2))], 1)))
    return conv(12, d1)[:, 0], rms, fl


def _exact_unet(case, seed):
    if case["n"] * case["d"] * case["h"] * case["w"] > 5_000_000:
        return None
    r, mask, e = _patches(case, seed)
    st = _prepare_unet(dict(case, n=1, d=16, h=16, w=16), 0)
    p, tscale = st["net"].params()
    st["net"].close()
    p = torch.from_numpy(p).cuda().double()
    if case["kind"] == "unet":
        res = []
        with torch.no_grad():
            for k in range(case["n"]):
                out, rms, fl = _net64(p, r[k:k + 1].double(), mask[k:k + 1])
                res.append(torch.where(fl, out * rms * tscale, 0.0))
        return torch.cat(res)
    p.requires_grad_(True)
    total, count = 0.0, int((mask == 1).sum())
    for k in range(case["n"]):
        out, rms, fl = _net64(p, r[k:k + 1].double(), mask[k:k + 1])
        dd = torch.where(fl, out - e[k:k + 1].double() / (rms * tscale), 0.0)
        loss = 0.0
        for ax in (1, 2, 3):  # sum over faces between non-solid cells of (d_i - d_j)^2, air at 0
            n = dd.shape[ax] - 1
            a, b = dd.narrow(ax, 0, n), dd.narrow(ax, 1, n)
            open_ = (mask[k:k + 1].narrow(ax, 0, n) != -1) & (mask[k:k + 1].narrow(ax, 1, n) != -1)
            loss = loss + ((a - b) ** 2 * open_).sum()
        loss = loss / count
        loss.backward()
        total += float(loss)
    return {"loss": total, "grad": p.grad.float().double()}


# ------------------------------------------------------------------ dispatch
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("jet", "lateral"):
        return _prepare_run(case, seed)
    if kind == "project":
        return _prepare_project(case, seed)
    if kind in ("csc", "csc_device"):
        return _prepare_csc(case, seed)
    return _prepare_unet(case, seed)


def run(state):
    kind = state["kind"]
    if kind == "run":
        return _run_run(state)
    if kind == "project":
        return _run_project(state)
    if kind in ("csc", "csc_device"):
        return _run_csc(state)
    return _run_unet(state)


def exact(case, seed):
    kind = case["kind"]
    if kind == "project":
        return _exact_project(case, seed)
    if kind in ("csc", "csc_device"):
        return _exact_csc(case, seed)
    if kind in ("unet", "grad"):
        return _exact_unet(case, seed)
    return None  # whole runs: a step's cell types follow from every bit of the steps before it


def work(case):
    """Each input read once and each output written once; of a simulation, once a step."""
    kind = case["kind"]
    if kind in ("jet", "lateral"):
        nx, ny, nz, k = case["nx"], case["ny"], case["nz"], case["steps"]
        fluid = nx * ny * case["pool"] if kind == "jet" else nx * ny * 3 + int(2.5 * case["r"] ** 2 * nx / 2)
        walls = 2 * (nx + ny) * nz + nx * ny
        cells = fluid + 5 * nx * ny + walls
        # host transfer: 39 B a cell and 24 B a particle each way; a step: speeds in and out, pressure out, flags,
        # positions in and out
        return {"bytes": 2.0 * (39 * cells + 24 * 8 * fluid) + k * (60.0 * cells + 48.0 * 8 * fluid),
                "flops": k * (8 * fluid * 400.0 + fluid * 1500.0)}
    if kind == "project":
        return {"bytes": 7 * 8.0 * (case["n"] + 2) ** 3, "flops": 700.0 * 0.45 * case["n"] ** 3}
    if kind in ("csc", "csc_device"):
        n = 0.8 * case["nx"] * case["ny"] * case["nz"]
        return {"bytes": n * (7 * 12 + 4 + 16), "flops": n * 14 * 60}
    v = case["n"] * case["d"] * case["h"] * case["w"]
    fl = sum(2.0 * t * ri * ro * v / 8 ** lv for (_, _, t, _, ri, ro), lv in zip(_LAYERS, _LEVEL))
    if kind == "unet":
        return {"bytes": 9.0 * v, "flops": fl}
    return {"bytes": 9.0 * v, "flops": 3 * fl}
