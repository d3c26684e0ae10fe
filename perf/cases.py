"""Performance cases: the calls a user of this library makes, over the range of sizes they are made at.

    frame      load a narrow-band state held on the device, advance it some steps, read the
               whole state back into device buffers (a solver coupled to a renderer or to
               other GPU code; also how a divided grid's ranks step their leaves)
    host       one host-resident step: page-locked leaves in, stepped leaves out
    adjoint    forward and backward pass of the differentiable advection through a staggered
               field, on device buffers (a GPU training loop) or on host arrays
    adjoint_ls forward and backward pass of a level set's own step
    crate      the crate's own step on resident grids: find_zero_crossings of the interface, then
               advect_level_set and rebuild_narrow_band, read by sample_trilinear at probe points
    mesh       volume_to_mesh of a resident grid into host arrays
    particles  advect_particles on a PointDataGrid (RK4 and re-binning), host particles

Inputs are made here with plain torch and numpy (unions of spheres, as in the benchmark), so
that ``exact`` can restate each path in 64 bits without the library.
"""
import math

import numpy as np
import torch

from sharc.volrus_b200 import (PARTICLE, Context, DeviceGrid, PointDataGrid, VelocityField, advect_level_set,
                               advect_particles, advect_particles_euler, find_zero_crossings, make_uniform_velocity,
                               rebuild_narrow_band, sample_trilinear, volume_to_mesh)
from sharc.volrus_b200.adjoint import AdvectionFunction
from sharc.volrus_b200.method import LevelSet

HW = 3.0           # narrow-band half width of every case, voxels
MARGIN = 256       # voxels a velocity's tables cover beyond the domain
EXACT_LEAVES = 45000  # largest state restated in 64 bits
F64 = torch.float64


def listed():
    return [
        # the smallest call: one small sphere, one step (an interactive tool, a unit test's grid)
        {"name": "frame-small", "kind": "frame", "velocity": "constant", "spheres": 1, "domain": 64, "rmin": 10.0,
         "rmax": 10.0, "precision": "f32", "integrator": 1, "iters": 2, "mode": 0, "steps": 1},
        # the deformation test at 512^3 in FP16, a frame of 8 steps: launch-bound, resident in L2
        {"name": "frame-deformation512", "kind": "frame", "velocity": "vortex", "spheres": 1, "domain": 512,
         "rmin": 76.8, "rmax": 76.8, "precision": "f16", "integrator": 2, "iters": 2, "mode": 0, "steps": 8},
        # tens of spheres in curl noise, FP32, subcell reinitialisation: a medium simulation
        {"name": "frame-curl-f32", "kind": "frame", "velocity": "curl", "spheres": 100, "domain": 1901, "rmin": 6.0,
         "rmax": 40.0, "precision": "f32", "integrator": 3, "iters": 2, "mode": 1, "steps": 2},
        # the headline configuration (random spheres, 3-octave curl noise, SSP-RK3, FP16) at an eighth of its size
        {"name": "frame-curl-f16-large", "kind": "frame", "velocity": "curl", "spheres": 1000, "domain": 4096,
         "rmin": 6.0, "rmax": 40.0, "precision": "f16", "integrator": 3, "iters": 2, "mode": 0, "steps": 2},
        # a Rust caller whose grid lives on the host: leaves up, one step, leaves down
        {"name": "host-curl-f16", "kind": "host", "velocity": "curl", "spheres": 120, "domain": 2020, "rmin": 6.0,
         "rmax": 40.0, "precision": "f16", "integrator": 3, "iters": 2, "mode": 0, "steps": 1},
        # the adjoint configuration: sphere r = 32 in 256^3, K = 64, device buffers
        {"name": "adjoint256", "kind": "adjoint", "domain": 256, "radius": 32.0, "stag": 128, "steps": 64,
         "every": 8, "scale": 1.0, "io": "device"},
        # a small inverse problem driven from numpy: new phi_0 and V each pass
        {"name": "adjoint64-host", "kind": "adjoint", "domain": 64, "radius": 13.0, "stag": 32, "steps": 16,
         "every": 4, "scale": 1.0, "io": "host"},
        # gradients through a level set's own curl-noise steps, a band of several million voxels
        {"name": "adjoint-curl", "kind": "adjoint_ls", "spheres": 160, "domain": 2224, "rmin": 6.0, "rmax": 40.0,
         "precision": "f16", "steps": 16, "every": 4},
        # the crate's parity configuration: sphere r = 32, uniform velocity, resident grids
        {"name": "crate-sphere128", "kind": "crate", "radius": 32.0, "field": "uniform", "probes": 4096},
        # the crate's step on a large sphere through three sampled velocity grids
        {"name": "crate-sphere512", "kind": "crate", "radius": 200.0, "field": "grids", "probes": 200000},
        # the benchmark's mesh: sphere r = 96
        {"name": "mesh96", "kind": "mesh", "radius": 96.0, "wave": 0.0},
        # a particle cloud through a sampled field, re-binned
        {"name": "particles", "kind": "particles", "n": 300000, "cells": 64, "rk4": True},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "host", "adjoint", "adjoint_ls", "crate", "crate", "mesh",
                       "particles"])
    if kind in ("frame", "host"):
        vel = rng.choice(["constant", "vortex", "curl", "curl"])
        c = {"kind": kind, "velocity": vel, "precision": rng.choice(["f16", "f32"]),
             "integrator": rng.choice([1, 2, 3]) if vel != "curl" else rng.choice([2, 3]),
             "iters": rng.choice([1, 2, 2, 2]), "mode": rng.choice([0, 0, 1])}
        if vel == "vortex":
            dom = int(_log(rng, 64, 512))
            c.update(spheres=1, domain=dom, rmin=0.15 * dom, rmax=0.15 * dom)
        else:
            n = int(_log(rng, 1, 900 if kind == "frame" else 120))
            c.update(spheres=n, domain=int(8192 * (n / 8000.0) ** (1 / 3)) + 1, rmin=6.0, rmax=rng.uniform(12.0, 40.0))
        k = rng.choice([1, 2, 4, 8]) if kind == "frame" else 1
        c["steps"] = max(1, min(k, 1500 // c["spheres"]))
        return c
    if kind == "adjoint":
        dom = int(_log(rng, 48, 256))
        k = int(_log(rng, 6, 64))
        return {"kind": kind, "domain": dom, "radius": dom * rng.uniform(0.1, 0.2), "stag": max(8, dom // 2),
                "steps": k, "every": max(1, int(math.sqrt(k))), "scale": rng.choice([1.0, 1.0, 3.3]),
                "io": rng.choice(["device", "host"])}
    if kind == "adjoint_ls":
        n = int(_log(rng, 1, 150))
        k = rng.randint(4, 16)
        return {"kind": kind, "spheres": n, "domain": int(8192 * (n / 8000.0) ** (1 / 3)) + 1, "rmin": 6.0,
                "rmax": rng.uniform(12.0, 40.0), "precision": rng.choice(["f16", "f32"]), "steps": k,
                "every": max(1, int(math.sqrt(k)))}
    if kind == "crate":
        r = round(_log(rng, 5, 190), 2)
        return {"kind": kind, "radius": r, "field": rng.choice(["uniform", "grids"]),
                "probes": int(_log(rng, 100, 190000))}
    if kind == "mesh":
        return {"kind": kind, "radius": round(_log(rng, 5, 95), 2), "wave": rng.choice([0.0, 0.5])}
    return {"kind": "particles", "n": int(_log(rng, 1000, 290000)), "cells": rng.choice([16, 33, 64]),
            "rk4": rng.choice([True, True, False])}


# ------------------------------------------------------------------ inputs


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _sphere_list(case, seed=None):
    """(n, 4) centres and radii, f64: uniform in the domain (curl, constant) or the deformation test's one sphere.
    The layout belongs to the case; a seed moves every sphere by up to 3 voxels."""
    dom = float(case["domain"])
    n = case["spheres"]
    rng = np.random.default_rng([17, n, case["domain"], int(1000 * case["rmax"])])
    if case.get("velocity") == "vortex":
        c = np.full((1, 3), 0.35 * dom)
    elif n == 1:
        c = np.full((1, 3), 0.5 * dom)
    else:
        c = rng.uniform(0.0, dom, (n, 3))
    r = rng.uniform(case["rmin"], case["rmax"], n)
    if seed is not None:
        c = c + np.random.default_rng([19, seed]).uniform(-3.0, 3.0, c.shape)
    return np.column_stack([c, r])


def _capacity(case):
    """Leaf capacity for this layout, whatever the seed and a few steps make of it."""
    r = _sphere_list(case)[:, 3]
    return int((4.0 * math.pi * (r + 8.0) ** 2 * 2 * HW / 110.0).sum()) + 64


_OFF = [(q >> 6, (q >> 3) & 7, q & 7) for q in range(512)]


def _rel(dev):
    return torch.tensor(_OFF, device=dev)


def _pack(on):
    """(n, 512) bool -> (n, 8) int64 mask words, bit x * 64 + y * 8 + z."""
    sh = torch.arange(64, device=on.device)
    return (on.reshape(-1, 8, 64).long() << sh).sum(-1)


def _unpack(m):
    sh = torch.arange(64, device=m.device)
    return ((m[:, :, None] >> sh) & 1).bool().reshape(-1, 512)


def _union(sph, pad=2.0, wave=0.0):
    """Leaves of the narrow band of a union of spheres, sorted by (x, y, z): origins (n, 3) int32, masks (n, 8)
    int64 and values (n, 512) f32 in voxels; leaves reached by |phi| < HW + pad are allocated.  `wave` adds a
    bumpy displacement of that many voxels to the surface."""
    dev = _dev()
    s = torch.tensor(sph, dtype=F64, device=dev)
    w = HW + pad + wave + 7.0
    half = int((float(s[:, 3].max()) + w) // 8 + 2)
    g = torch.arange(-half, half + 1, device=dev)
    lat = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    keys, who = [], []
    step = max(1, (1 << 24) // len(lat))
    for a in range(0, len(s), step):
        t = s[a:a + step]
        l0 = torch.floor(t[:, :3] / 8).long()
        leaf = l0[:, None, :] + lat[None]
        d = (leaf.double() * 8 + 3.5 - t[:, None, :3]).norm(dim=-1) - t[:, None, 3]
        i, j = torch.nonzero(d < w, as_tuple=True)
        q = leaf[i, j] + (1 << 20)
        keys.append((q[:, 0] << 42) | (q[:, 1] << 21) | q[:, 2])
        who.append(i + a)
    keys, who = torch.cat(keys), torch.cat(who)
    uniq, inv = torch.unique(keys, return_inverse=True)
    org = (torch.stack([uniq >> 42, (uniq >> 21) & ((1 << 21) - 1), uniq & ((1 << 21) - 1)], 1) - (1 << 20)) * 8
    order = torch.argsort(inv, stable=True)
    inv, who = inv[order], who[order]
    first = torch.searchsorted(inv, torch.arange(len(uniq) + 1, device=dev))
    rel = _rel(dev).double()
    keep, vals = [], []
    chunk = 1 << 15
    for a in range(0, len(uniq), chunk):
        b = min(len(uniq), a + chunk)
        p0, p1 = int(first[a]), int(first[b])
        phi = torch.full((b - a, 512), math.inf, dtype=F64, device=dev)
        for c in range(p0, p1, 1 << 16):
            e = min(p1, c + (1 << 16))
            pos = org[inv[c:e]].double()[:, None, :] + rel[None]
            t = s[who[c:e]]
            d = (pos - t[:, None, :3]).norm(dim=-1) - t[:, None, 3]
            if wave:
                d = d + wave * torch.sin(0.37 * pos[..., 0]) * torch.sin(0.41 * pos[..., 1]) * torch.sin(0.29 * pos[..., 2])
            phi.scatter_reduce_(0, (inv[c:e] - a)[:, None].expand(-1, 512), d, "amin")
        k = (phi.abs() < HW + pad).any(1)
        keep.append(org[a:b][k])
        vals.append(phi[k].float())
    org, phi = torch.cat(keep), torch.cat(vals)
    on = phi.abs() < HW
    phi = torch.where(on, phi, torch.copysign(torch.full_like(phi, HW), phi))
    return org.int().contiguous(), _pack(on), phi.contiguous()


def _curl(seed, extent, octaves=3):
    """3-octave divergence-free noise of at most 1 voxel per unit time, as the benchmark's."""
    rng = np.random.default_rng([23, seed])
    w = np.array([2.0 ** -o for o in range(octaves)])
    w /= w.sum()
    octs = []
    for o in range(octaves):
        k = 2.0 * math.pi * 2 ** o / extent
        e = rng.normal(size=3)
        e /= np.linalg.norm(e)
        ph = rng.uniform(0, 2 * math.pi, 3)
        octs.append((float(w[o] / (4.0 * k) * 2.0), float(k), tuple(map(float, ph)), tuple(map(float, e))))
    return octs


def _velocity(case, seed):
    """The library's velocity description and the time step."""
    dom = case["domain"]
    kind = case.get("velocity", "curl")
    if kind == "constant":
        u = np.random.default_rng([29, seed]).uniform(-0.7, 0.7, 3)
        return {"kind": "constant", "c": tuple(map(float, u))}, 1.0
    if kind == "vortex":
        return {"kind": "vortex", "vs": 1.0 / dom, "period": 3.0}, 0.25 / dom
    return {"kind": "curl", "octaves": _curl(seed, float(max(dom, 256))),
            "domain": ((-MARGIN,) * 3, (dom + MARGIN,) * 3)}, 1.0


def _curl_at(octs, p):
    """Curl noise at points p (..., 3) in 64 bits."""
    u = torch.zeros_like(p)
    for A, k, ph, e in octs:
        s = [torch.sin(k * p[..., a] + ph[a]) for a in range(3)]
        c = [torch.cos(k * p[..., a] + ph[a]) for a in range(3)]
        g = [A * k * c[0] * s[1] * s[2], A * k * s[0] * c[1] * s[2], A * k * s[0] * s[1] * c[2]]
        u = u + torch.stack([g[1] * e[2] - g[2] * e[1], g[2] * e[0] - g[0] * e[2], g[0] * e[1] - g[1] * e[0]], -1)
    return u


def _stored(phi, case):
    return phi.half().float() if case["precision"] == "f16" else phi


def _level_set(case, seed, org, masks, phi, capacity):
    """A level set for states of this case: its pool holds `capacity` leaves; the state itself is loaded by
    upload_device."""
    vel, dt = _velocity(case, seed)
    one = slice(0, 1)
    return LevelSet.from_leaves(org[one].cpu().numpy(), masks[one].cpu().numpy().view(np.uint64),
                                phi[one].cpu().numpy(), vel, dt, half_width=HW,
                                precision=1 if case["precision"] == "f16" else 0,
                                integrator=case.get("integrator", 3), reinit_iters=case.get("iters", 2),
                                capacity=capacity, reinit_mode=case.get("mode", 0))


def _stag_field(case, seed):
    """The deformation field at t = 0 on a staggered grid (voxels per unit time), with a seeded smooth part."""
    n, dom = case["stag"], case["domain"]
    cell = dom / n
    rng = np.random.default_rng([31, seed])
    i = np.arange(n, dtype=np.float64)
    face, mid = i * cell / dom, (i + 0.5) * cell / dom
    s, pi = np.sin, math.pi
    V = np.zeros((3, n, n, n), np.float32)
    for a in range(3):
        ax = [mid, mid, mid]
        ax[a] = face
        x, y, z = np.meshgrid(*ax, indexing="ij", sparse=True)
        if a == 0:
            f = 2 * s(pi * x) ** 2 * s(2 * pi * y) * s(2 * pi * z)
        elif a == 1:
            f = -s(2 * pi * x) * s(pi * y) ** 2 * s(2 * pi * z)
        else:
            f = -s(2 * pi * x) * s(2 * pi * y) * s(pi * z) ** 2
        ph = rng.uniform(0, 2 * pi, 3)
        f = 0.9 * f + 0.2 * s(2 * pi * x + ph[0]) * s(2 * pi * y + ph[1]) * s(2 * pi * z + ph[2])
        V[a] = (f * dom).astype(np.float32)
    dt = case["scale"] * 0.25 / dom  # half a voxel per step at scale 1
    return V, cell, dt


def _adjoint_inputs(case, seed):
    c = 0.5 * case["domain"] + np.array([0.3, -0.4, 0.1])
    org, masks, phi = _union(np.array([[*c, case["radius"]]]))
    V, cell, dt = _stag_field(case, seed)
    return org, masks, phi, V, cell, dt


def _crate_inputs(case, seed):
    """A sphere's leaves, three velocity components on those leaves (or one constant), probe points."""
    rng = np.random.default_rng([41, seed])
    org, masks, phi = _union(np.array([[0.3, -1.4, 2.1, case["radius"]]]), pad=0.0)
    k = torch.from_numpy(rng.integers(0, len(org), case["probes"])).to(org.device)
    pts = org[k].double().cpu().numpy() + rng.uniform(0.0, 8.0, (case["probes"], 3))
    if case["field"] == "uniform":
        return org, masks, phi, tuple(np.float32(rng.uniform(-1.0, 1.0, 3)).tolist()), pts
    octs = _curl(seed, 512.0)
    comps = torch.empty((3, len(org), 512), dtype=torch.float32, device=org.device)
    rel = _rel(org.device).double()
    for a in range(0, len(org), 1 << 14):
        u = _curl_at(octs, org[a:a + (1 << 14)].double()[:, None, :] + rel[None])
        for q in range(3):
            comps[q, a:a + (1 << 14)] = u[..., q].float()
    return org, masks, phi, comps, pts


def _device_grid(org, masks, vals, background):
    return DeviceGrid.from_device(org.data_ptr(), masks.data_ptr(), vals.data_ptr(), len(org), background, 1.0)


def _particle_field(case):
    """The deformation field on a cells^3 lattice over the unit cube: (3, c, c, c) f32, c = cells + 1."""
    c = case["cells"] + 1
    x = torch.arange(c, dtype=F64, device=_dev()) / case["cells"]
    x, y, z = torch.meshgrid(x, x, x, indexing="ij")
    s, pi = torch.sin, math.pi
    return torch.stack([2 * s(pi * x) ** 2 * s(2 * pi * y) * s(2 * pi * z),
                        -s(2 * pi * x) * s(pi * y) ** 2 * s(2 * pi * z),
                        -s(2 * pi * x) * s(2 * pi * y) * s(pi * z) ** 2]).float()


def _particles(case, seed):
    rng = np.random.default_rng([43, seed])
    p = np.zeros(case["n"], PARTICLE)
    p["position"] = rng.uniform(0.02, 0.98, (case["n"], 3))
    p["velocity"] = rng.normal(size=(case["n"], 3))
    p["id"] = np.arange(case["n"])
    return p


def _dense_leaves(field):
    """A dense (c, c, c) lattice as leaves: every leaf that holds a lattice voxel, lattice voxels active."""
    c = field.shape[0]
    n = (c + 7) // 8
    d = torch.zeros((8 * n,) * 3, dtype=torch.float32, device=field.device)
    on = torch.zeros((8 * n,) * 3, dtype=torch.bool, device=field.device)
    d[:c, :c, :c] = field
    on[:c, :c, :c] = True

    def cut(t):
        return t.reshape(n, 8, n, 8, n, 8).permute(0, 2, 4, 1, 3, 5).reshape(n ** 3, 512).contiguous()
    g = torch.arange(n, device=field.device, dtype=torch.int32) * 8
    org = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3).contiguous()
    return org, _pack(cut(on)), cut(d)


class State:
    pass


def prepare(case, seed):
    ctx = Context.default()
    s = State()
    s.case, s.ctx = case, ctx
    kind = case["kind"]
    if kind in ("frame", "host"):
        org, masks, phi = _union(_sphere_list(case, seed))
        phi = _stored(phi, case)
        cap = _capacity(case)
        s.ls = _level_set(case, seed, org, masks, phi, cap)
        if kind == "frame":
            s.org, s.masks, s.phi = org, masks, phi
            s.out = [torch.zeros((cap, k), dtype=t, device=org.device)
                     for k, t in ((3, torch.int32), (8, torch.int64), (512, torch.float32))]
            s.cap = cap
        else:
            s.host = [ctx.pinned((len(org), k), t) for k, t in ((3, np.int32), (8, np.uint64), (512, np.float32))]
            for h, t in zip(s.host, (org, masks, phi)):
                torch.from_numpy(h.view(np.int64) if h.dtype == np.uint64 else h).copy_(t)
            s.out = tuple(ctx.pinned((cap, k), t) for k, t in ((3, np.int32), (8, np.uint64), (512, np.float32)))
            for h in s.out:
                h[:] = 0
    elif kind in ("adjoint", "adjoint_ls"):
        if kind == "adjoint":
            org, masks, phi, V, cell, dt = _adjoint_inputs(case, seed)
            s.fn = AdvectionFunction(org.cpu().numpy(), masks.cpu().numpy().view(np.uint64), phi.cpu().numpy(), V,
                                     cell, dt, 2.0, case["steps"], case["every"], half_width=HW)
        else:
            org, masks, phi = _union(_sphere_list(case))
            phi = _stored(phi, case)
            s.ls = _level_set(case, seed, org, masks, phi, len(org) + 64)
            torch.cuda.synchronize()
            s.ls.upload_device(org.data_ptr(), masks.data_ptr(), phi.data_ptr(), len(org))
            s.fn = AdvectionFunction.from_level_set(s.ls, case["steps"], case["every"])
        on = _unpack(masks)
        n = s.fn.n_band
        g = torch.Generator(device=org.device).manual_seed(seed)
        grad = torch.randn(n, generator=g, device=org.device)
        if case.get("io", "device") == "host":
            s.phi0, s.V, s.grad = phi[on].cpu().numpy(), V, grad.cpu().numpy()
        else:
            s.grad = grad
            s.phik, s.g0 = torch.empty(n, device=org.device), torch.empty(n, device=org.device)
            s.gv = torch.empty((3,) + (case["stag"],) * 3, device=org.device) if kind == "adjoint" else None
    elif kind == "crate":
        org, masks, phi, field, s.pts = _crate_inputs(case, seed)
        torch.cuda.synchronize()
        s.grid = _device_grid(org, masks, phi, HW)
        if case["field"] == "uniform":
            u = make_uniform_velocity(1.0, field)
            s.vel = VelocityField(*[DeviceGrid.upload(q) for q in (u.vx, u.vy, u.vz)])
        else:
            s.vel = VelocityField(*[_device_grid(org, masks, q.contiguous(), 0.0) for q in field])
    elif kind == "mesh":
        org, masks, phi = _mesh_inputs(case, seed)
        torch.cuda.synchronize()
        s.grid = _device_grid(org, masks, phi, HW)
    else:
        h = 1.0 / case["cells"]
        grids = []
        for q in _particle_field(case):
            org, masks, vals = _dense_leaves(q)
            torch.cuda.synchronize()
            grids.append(DeviceGrid.from_device(org.data_ptr(), masks.data_ptr(), vals.data_ptr(), len(org), 0.0, h))
        s.vel = VelocityField(*grids)
        s.points = PointDataGrid(h)
        s.points.insert_batch(_particles(case, seed))
        s.leaves = np.zeros(((case["cells"] // 8 + 2) ** 3, 4), np.int64)
    torch.cuda.synchronize()
    return s


def _mesh_inputs(case, seed):
    """A sphere's band, its values scaled by a smooth positive factor that depends on the seed: another surface
    of the same cells."""
    org, masks, phi = _union(np.array([[1.3, -2.4, 0.6, case["radius"]]]), pad=0.0, wave=case["wave"])
    k = np.random.default_rng([47, seed]).uniform(0.1, 0.5, 3)
    p = org.double()[:, None, :] + _rel(org.device).double()[None]
    f = 1.0 - 0.3 * torch.sin(k[0] * p[..., 0]) * torch.sin(k[1] * p[..., 1] + 1.0) * torch.sin(k[2] * p[..., 2] + 2.0)
    return org, masks, torch.where(_unpack(masks), phi.double() * f.abs(), phi.double()).float()


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "frame":
        s.ls.set_step(0)
        s.ls.upload_device(s.org.data_ptr(), s.masks.data_ptr(), s.phi.data_ptr(), len(s.org))
        s.ls.step(case["steps"])
        s.ls.download_device(s.out[0].data_ptr(), s.out[1].data_ptr(), s.out[2].data_ptr(), s.cap)
        return s.out  # rows past the leaf count stay zero
    if kind == "host":
        s.ls.set_step(0)
        k = len(s.ls.step_host(*s.host, n_steps=case["steps"], out=s.out)[0])
        for h in s.out:
            h[k:len(s.host[0])] = 0  # rows past the leaf count are zero
        return [s.out[0], s.out[1].view(np.int64), s.out[2]]
    if kind in ("adjoint", "adjoint_ls"):
        if case.get("io", "device") == "host":
            phik = s.fn.forward(s.phi0, s.V)
            g0, gv = s.fn.backward(s.grad)
            return [phik, g0, gv]
        s.fn.forward_device(s.phik.data_ptr())
        s.fn.backward_device(s.grad.data_ptr(), s.g0.data_ptr(), s.gv.data_ptr() if s.gv is not None else 0)
        return [s.phik, s.g0] + ([s.gv] if s.gv is not None else [])
    if kind == "crate":
        cross = find_zero_crossings(s.grid)
        out = advect_level_set(s.grid, s.vel, 1.0)
        rebuild_narrow_band(out, HW)
        probe = sample_trilinear(out, s.pts)
        out.close()
        return [cross, probe]
    if kind == "mesh":
        m = volume_to_mesh(s.grid, 0.0)
        return [m.vertices, m.triangles.astype(np.int64)]
    pg = PointDataGrid(s.points.voxel_size)
    pg.particles, pg.leaf_origins, pg.leaf_start = s.points.particles, s.points.leaf_origins, s.points.leaf_start
    (advect_particles if case["rk4"] else advect_particles_euler)(pg, s.vel, 0.005)
    k = len(pg.leaf_origins)
    s.leaves[:] = 0
    s.leaves[:k, :3] = pg.leaf_origins
    s.leaves[:k, 3] = pg.leaf_start[1:]
    return [pg.particles["position"], pg.particles["id"].view(np.int64), s.leaves]


def work(case):
    """Bytes and operations of one pass.  Band voxels: 2 HW per unit of surface; a leaf holds about 155 of them
    and about 233 voxels of the dilated band."""
    kind = case["kind"]
    pi4 = 4.0 * math.pi
    if kind in ("frame", "host", "adjoint_ls"):
        a, b = case["rmin"], case["rmax"]
        r2 = (a * a + a * b + b * b) / 3.0
        band = case["spheres"] * pi4 * r2 * 2 * HW
        leaves = band / 155.0
        if kind == "adjoint_ls":
            return {"bytes": case["steps"] * band * (24.0 + 24.0 + 56.0), "flops": case["steps"] * band * 160.0}
        vb = 2 if case["precision"] == "f16" else 4
        vel = {"constant": 6.0, "vortex": 60.0, "curl": 100.0}[case["velocity"]] * case["integrator"]
        per_leaf = 233.0 * (vel + 40.0 + 60.0 * case["iters"])
        return {"bytes": leaves * (2 * (2048 + 76) + case["steps"] * 2 * (512 * vb + 64)),
                "flops": case["steps"] * leaves * per_leaf}
    if kind == "adjoint":
        band = pi4 * case["radius"] ** 2 * 2 * HW
        return {"bytes": case["steps"] * band * (24.0 + 24.0 + 56.0) + 12.0 * case["stag"] ** 3,
                "flops": case["steps"] * band * 200.0}
    band = pi4 * case.get("radius", 1.0) ** 2 * 2 * HW
    leaves = band / 130.0
    if kind == "crate":
        grids = 2 if case["field"] == "uniform" else 5
        return {"bytes": leaves * (2112.0 * (grids + 2)) + 12.0 * band / HW + 28.0 * case["probes"],
                "flops": band * 300.0 + 60.0 * case["probes"]}
    if kind == "mesh":
        area = pi4 * case["radius"] ** 2
        return {"bytes": leaves * 2112.0 + area * 3.0 * (24 + 12 * 2), "flops": leaves * 512.0 * 20.0 + area * 60.0}
    return {"bytes": case["n"] * 112.0 + 12.0 * (case["cells"] + 1) ** 3,
            "flops": case["n"] * (4 if case["rk4"] else 1) * 150.0}


# --------------------------------------------------------- 64-bit restatements


def _neighbours(org):
    """(n, 3, 3, 3) index of the leaf at each leaf offset, -1 if absent."""
    c = (org.long() >> 3) + (1 << 20)

    def key(q):
        return (q[..., 0] << 42) | (q[..., 1] << 21) | q[..., 2]
    ks, order = torch.sort(key(c))
    g = torch.arange(-1, 2, device=org.device)
    d = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), -1)
    want = key(c[:, None, None, None, :] + d[None])
    at = torch.searchsorted(ks, want).clamp(max=len(ks) - 1)
    return torch.where(ks[at] == want, order[at], torch.full_like(at, -1))


def _tile(vals, nb, halo, absent=None):
    """Values on the (8 + 2 halo)^3 tile around each leaf; voxels of absent leaves hold `absent`, or by default
    HW with the sign of the leaf's own value at the clamped position."""
    dev = vals.device
    c = torch.arange(-halo, 8 + halo, device=dev)
    ax = torch.where(c < 0, 0, torch.where(c > 7, 2, 1))
    lo = c & 7
    cl = c.clamp(0, 7)
    slot = nb[:, ax][:, :, ax][:, :, :, ax]
    off = (lo[:, None, None] << 6) | (lo[None, :, None] << 3) | lo[None, None, :]
    own = (cl[:, None, None] << 6) | (cl[None, :, None] << 3) | cl[None, None, :]
    got = vals.reshape(-1)[slot.clamp(min=0) * 512 + off]
    if absent is None:
        mine = vals[:, own.reshape(-1)].reshape(got.shape)
        return torch.where(slot >= 0, got, torch.copysign(torch.full_like(mine, HW), mine))
    return torch.where(slot >= 0, got, torch.full_like(got, absent))


def _blend(c, w):
    """Trilinear blend of corners c[i][j][k] with fractions w (..., 3)."""
    x, y, z = w.unbind(-1)
    c00 = c[0] * (1 - x) + c[4] * x
    c01 = c[1] * (1 - x) + c[5] * x
    c10 = c[2] * (1 - x) + c[6] * x
    c11 = c[3] * (1 - x) + c[7] * x
    return (c00 * (1 - y) + c10 * y) * (1 - z) + (c01 * (1 - y) + c11 * y) * z


def _velocity_at(case, vel, p, t):
    if vel["kind"] == "constant":
        return torch.tensor(vel["c"], dtype=F64, device=p.device).expand_as(p)
    if vel["kind"] == "curl":
        return _curl_at(vel["octaves"], p)
    q = p * vel["vs"]
    s, pi = torch.sin, math.pi
    x, y, z = q.unbind(-1)
    f = math.cos(pi * t / vel["period"]) / vel["vs"]
    return f * torch.stack([2 * s(pi * x) ** 2 * s(2 * pi * y) * s(2 * pi * z),
                            -s(2 * pi * x) * s(pi * y) ** 2 * s(2 * pi * z),
                            -s(2 * pi * x) * s(2 * pi * y) * s(pi * z) ** 2], -1)


def _foot(case, vel, p, t1, dt):
    """Backtrace displacement over one step ending at t1."""
    def u(q, t):
        return _velocity_at(case, vel, q, t)
    k = case.get("integrator", 3)
    if k == 1:
        return -dt * u(p, t1)
    if k == 2:
        return -dt * u(p - 0.5 * dt * u(p, t1), t1 - 0.5 * dt)
    a = -dt * u(p, t1)
    b = 0.25 * (a - dt * u(p + a, t1 - dt))
    return (2.0 / 3.0) * (b - dt * u(p + b, t1 - 0.5 * dt))


def _six(tile):
    i = slice(1, -1)
    return [tile[:, :-2, i, i], tile[:, 2:, i, i], tile[:, i, :-2, i], tile[:, i, 2:, i], tile[:, i, i, :-2],
            tile[:, i, i, 2:]]


def _reinit(phi1, phi, nb, D, mode):
    """One sweep phi -> phi' on the voxels of D (phi1: the field before reinitialisation)."""
    def near(f):
        t = _tile(f, nb, 1, absent=math.nan)
        c = f.reshape(-1, 8, 8, 8)
        return c, [torch.where(torch.isnan(q), torch.copysign(torch.full_like(c, HW), c), q) for q in _six(t)]
    p1, n1 = near(phi1)
    p, n = near(phi)
    s = p1 / torch.sqrt(p1 * p1 + 1.0)
    sg = torch.where(s >= 0, 1.0, -1.0)
    g2 = sum(torch.maximum(sg * p - torch.minimum(sg * n[2 * a], sg * n[2 * a + 1]), torch.zeros_like(p)) ** 2
             for a in range(3))
    new = p - 0.5 * s * (torch.sqrt(g2) - 1.0)
    if mode:
        cut = torch.stack([p1 * q < 0 for q in n1]).any(0)
        m2 = 0
        for a in range(3):
            lo, hi = n1[2 * a], n1[2 * a + 1]
            m = torch.maximum(torch.maximum((hi - lo).abs() * 0.5, (hi - p1).abs()), (p1 - lo).abs().clamp(min=1e-6))
            m2 = m2 + m * m
        d = p1 / torch.sqrt(m2)
        new = torch.where(cut, p - 0.5 * (torch.copysign(p.abs(), p1) - d), new)
    return torch.where(D, new.reshape(-1, 512), phi)


def _method_step(case, vel, dt, step, org, on, phi, slack):
    """One step of the narrow-band method in 64 bits; leaves in list order.  `slack` moves the trim threshold."""
    dev = org.device
    nb = _neighbours(org)
    act = _tile(on.to(F64), nb, 1, absent=0.0)
    D = torch.nn.functional.max_pool3d(act[:, None], 3, 1)[:, 0].reshape(-1, 512) > 0
    leaf, off = torch.nonzero(D, as_tuple=True)
    rel = _rel(dev).double()
    f = _foot(case, vel, org[leaf].double() + rel[off], (step + 1) * dt, dt)
    E = 14
    tile = _tile(phi, nb, 3).reshape(len(org), -1)
    q = rel[off] + 3 + f
    b = torch.floor(q)
    w = q - b
    b = b.long().clamp(0, E - 2)
    base = (b[:, 0] * E + b[:, 1]) * E + b[:, 2]
    flat = tile.reshape(-1)
    corners = [flat[leaf * E ** 3 + base + (i >> 2) * E * E + ((i >> 1) & 1) * E + (i & 1)] for i in range(8)]
    phi1 = torch.copysign(torch.full_like(phi, HW), phi)
    phi1[leaf, off] = _blend(corners, w)
    v = phi1
    for _ in range(case["iters"]):
        v = _reinit(phi1, v, nb, D, case["mode"])
    on = D & (v.abs() < HW + slack)
    v = torch.where(on, v, torch.copysign(torch.full_like(v, HW), v))
    # re-track: leaves an active voxel touches, in list order, each followed by the new leaves it owns
    a = on.reshape(-1, 8, 8, 8)
    pick = [slice(0, 1), slice(0, 8), slice(7, 8)]
    spill = torch.stack([a[:, pick[d // 9], pick[(d // 3) % 3], pick[d % 3]].flatten(1).any(1) for d in range(27)], 1)
    nbf = nb.reshape(-1, 27)
    keep = torch.zeros(len(org), dtype=torch.bool, device=dev)
    i, d = torch.nonzero(spill & (nbf >= 0), as_tuple=True)
    keep[nbf[i, d]] = True
    i, d = torch.nonzero(spill & (nbf < 0), as_tuple=True)
    step3 = torch.tensor([[q // 9 - 1, (q // 3) % 3 - 1, q % 3 - 1] for q in range(27)], device=dev) * 8
    no = org[i].long() + step3[d]
    c = (no >> 3) + (1 << 20)
    key = (c[:, 0] << 42) | (c[:, 1] << 21) | c[:, 2]
    if len(key):
        uk, inv = torch.unique(key, return_inverse=True)
        best = torch.full((len(uk),), -1, dtype=torch.long, device=dev).scatter_reduce_(0, inv, d, "amax")
        win = d == best[inv]
        i, d, no = i[win], d[win], no[win]
    cx = (torch.tensor(_OFF, device=dev)[None] + step3[d][:, None, :]).clamp(0, 7)
    src = (cx[..., 0] << 6) | (cx[..., 1] << 3) | cx[..., 2]
    nv = v[i[:, None], src] if len(i) else v[:0]
    nv = torch.copysign(torch.full_like(nv, HW), nv)
    old = torch.nonzero(keep).reshape(-1)
    rank = torch.cat([old * 32, i * 32 + 1 + d])
    order = torch.argsort(rank)
    org = torch.cat([org[old].long(), no])[order].int()
    on = torch.cat([on[old], torch.zeros((len(i), 512), dtype=torch.bool, device=dev)])[order]
    v = torch.cat([v[old], nv])[order]
    return org, on, v


def _exact_frame(case, seed):
    org, masks, phi = _union(_sphere_list(case, seed))
    if len(org) > EXACT_LEAVES:
        return None
    vel, dt = _velocity(case, seed)
    # a voxel within rounding of the half width can decide whether a leaf exists, and a leaf more moves every row
    # behind it: there is a value only where the threshold's last digits leave the leaves as they are
    tol = 1e-2 if case["precision"] == "f16" else 2e-5
    start, ends = (org, _unpack(masks), _stored(phi, case).double()), []
    for slack in (-tol, tol, 0.0):
        org, on, v = start
        for k in range(case["steps"]):
            org, on, v = _method_step(case, vel, dt, k, org, on, v, slack)
        ends.append(org)
    if not all(torch.equal(q, org) for q in ends):
        return None
    if case["kind"] == "host":
        c = (org.long() >> 3) + (1 << 20)
        v = v[torch.argsort((c[:, 0] << 42) | (c[:, 1] << 21) | c[:, 2])]
    return [None, None, torch.nn.functional.pad(v, (0, 0, 0, _capacity(case) - len(v)))]


def _frozen(case, org, masks, phi, feet, grad, inputs):
    """Frozen-band advection phi_0 -> phi_K by the feet of each step and its gradients, in 64 bits."""
    dev = org.device
    nb = _neighbours(org).reshape(-1, 27)
    leaf, off = torch.nonzero(_unpack(masks), as_tuple=True)
    rel = torch.tensor(_OFF, device=dev)[off]
    at = leaf * 512 + off
    full = phi.double().reshape(-1)
    p0 = full[at].clone().requires_grad_(True)
    cur = full.clone().index_put((at,), p0)
    for k in range(case["steps"]):
        f = feet(k)
        b = torch.floor(f.detach())
        w = f - b
        base = rel + b.long()
        corners = []
        for i in range(8):
            q = base + torch.tensor([i >> 2, (i >> 1) & 1, i & 1], device=dev)
            ax = torch.where(q < 0, 0, torch.where(q > 7, 2, 1))
            s = nb[leaf, ax[:, 0] * 9 + ax[:, 1] * 3 + ax[:, 2]]
            lo, cl = q & 7, q.clamp(0, 7)
            here = cur[s.clamp(min=0) * 512 + ((lo[:, 0] << 6) | (lo[:, 1] << 3) | lo[:, 2])]
            mine = cur.detach()[leaf * 512 + ((cl[:, 0] << 6) | (cl[:, 1] << 3) | cl[:, 2])]
            corners.append(torch.where(s >= 0, here, torch.copysign(torch.full_like(mine, HW), mine)))
        cur = cur.index_put((at,), _blend(corners, w))
    phik = cur[at]
    got = torch.autograd.grad(phik, [p0] + inputs, grad.double())
    return [phik.detach()] + [g.detach() for g in got]


def _exact_adjoint(case, seed):
    org, masks, phi, Vn, cell, dt = _adjoint_inputs(case, seed)
    dev = org.device
    n = case["stag"]
    V = torch.tensor(Vn, dtype=F64, device=dev, requires_grad=True)
    leaf, off = torch.nonzero(_unpack(masks), as_tuple=True)
    if len(leaf) * case["steps"] > 6_000_000:
        return None
    p = org[leaf].double() + _rel(dev).double()[off]
    ub = []
    for a in range(3):
        g = p / cell
        sh = torch.full((3,), 0.5, dtype=F64, device=dev)
        sh[a] = 0.0
        g = g - sh
        b = torch.floor(g)
        w, b = g - b, b.long()
        ub.append(_blend([V[a][tuple((b[:, q] + ((i >> (2 - q)) & 1)).clamp(0, n - 1) for q in range(3))]
                          for i in range(8)], w))
    ub = torch.stack(ub, -1)
    gen = torch.Generator(device=dev).manual_seed(seed)
    grad = torch.randn(len(leaf), generator=gen, device=dev)
    return _frozen(case, org, masks, phi, lambda k: -dt * math.cos(math.pi * (k + 1) * dt / 2.0) * ub, grad, [V])


def _exact_adjoint_ls(case, seed):
    org, masks, phi = _union(_sphere_list(case))
    leaf, off = torch.nonzero(_unpack(masks), as_tuple=True)
    if len(leaf) * case["steps"] > 6_000_000:
        return None
    dev = org.device
    vel, dt = _velocity(case, seed)
    f = _foot(case, vel, org[leaf].double() + _rel(dev).double()[off], 0.0, dt)
    gen = torch.Generator(device=dev).manual_seed(seed)
    grad = torch.randn(len(leaf), generator=gen, device=dev)
    return _frozen(case, org, masks, _stored(phi, case), lambda k: f, grad, [])


def _dense(org, masks, vals, fill, ring):
    """Leaves as dense arrays over their bounding box widened by `ring` voxels: values, activity, lower corner."""
    lo = org.long().min(0).values - ring
    n = (org.long().max(0).values + 8 + ring - lo).tolist()
    d = torch.full(n, fill, dtype=F64, device=org.device)
    on = torch.zeros(n, dtype=torch.bool, device=org.device)
    p = (org.long() - lo)[:, None, :] + torch.tensor(_OFF, device=org.device)[None]
    d[p[..., 0], p[..., 1], p[..., 2]] = vals.double()
    on[p[..., 0], p[..., 1], p[..., 2]] = _unpack(masks)
    return d, on, lo


def _sample_dense(d, lo, p, fill):
    """Trilinear sample of a dense array at points p; `fill` outside it."""
    q = p - lo
    b = torch.floor(q)
    w, b = q - b, b.long()
    top = torch.tensor(d.shape, device=d.device) - 1
    out = []
    for i in range(8):
        c = b + torch.tensor([i >> 2, (i >> 1) & 1, i & 1], device=d.device)
        ok = ((c >= 0) & (c <= top)).all(-1)
        c = torch.minimum(c.clamp(min=0), top)
        out.append(torch.where(ok, d[c[..., 0], c[..., 1], c[..., 2]], fill))
    return _blend(out, w)


def _exact_crate(case, seed):
    org, masks, phi, field, pts = _crate_inputs(case, seed)
    dev = org.device
    d, on, lo = _dense(org, masks, phi, HW, 4)
    at = torch.nonzero(on)
    p = (at + lo).double()
    if case["field"] == "uniform":
        u = torch.tensor(field, dtype=F64, device=dev).expand_as(p)
    else:
        leaf, off = torch.nonzero(_unpack(masks), as_tuple=True)
        dense = [_dense(org, masks, q, 0.0, 4)[0] for q in field]
        u = torch.stack([q[at[:, 0], at[:, 1], at[:, 2]] for q in dense], -1)
    adv = torch.full_like(d, HW)
    adv[on] = _sample_dense(d, lo, p - u, torch.tensor(HW, dtype=F64, device=dev)).float().double()
    # crossings of the advected band, then the signed distance to the nearest within the band
    i = slice(1, -1)
    padded = torch.nn.functional.pad(torch.where(on, adv, 0.0), (1,) * 6)
    cross = torch.zeros_like(on)
    for a, b, c in ((slice(2, None), i, i), (slice(0, -2), i, i), (i, slice(2, None), i), (i, slice(0, -2), i),
                    (i, i, slice(2, None)), (i, i, slice(0, -2))):
        cross |= adv * padded[a, b, c] < 0
    cross = on & (cross | (adv == 0))
    if not bool(cross.any()):
        return None
    R = int(math.ceil(HW)) - 1
    cp = torch.nn.functional.pad(cross, (R,) * 6)
    best = torch.full_like(d, math.inf)
    X, Y, Z = d.shape
    for dx in range(-R, R + 1):
        for dy in range(-R, R + 1):
            for dz in range(-R, R + 1):
                h = cp[R + dx:R + dx + X, R + dy:R + dy + Y, R + dz:R + dz + Z]
                best = torch.where(h, torch.minimum(best, torch.full_like(best, float(dx * dx + dy * dy + dz * dz))), best)
    dist = torch.sqrt(best)
    new = torch.where(on & (dist < HW), torch.where(adv >= 0, dist, -dist), HW)
    q = torch.from_numpy(pts).to(dev)
    return [None, _sample_dense(new, lo, q, torch.tensor(HW, dtype=F64, device=dev))]


def _exact_mesh(case, seed):
    """Vertices in order of the cell that visits their edge first: tiles (leaves and their face neighbours) in
    (x, y, z) order, the tile's cells in (x, y, z) order, the cell's 12 edges in table order."""
    org, masks, phi = _mesh_inputs(case, seed)
    dev = org.device
    d, _, lo = _dense(org, masks, phi, HW, 16)
    T = [s // 8 for s in d.shape]
    tiles = torch.zeros(T, dtype=torch.bool, device=dev)
    c = (org.long() - lo) >> 3
    for e in ((0, 0, 0), (-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)):
        q = c + torch.tensor(e, device=dev)
        tiles[q[:, 0], q[:, 1], q[:, 2]] = True
    rank = torch.cumsum(tiles.reshape(-1).long(), 0).reshape(T) - 1
    corner = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
    ends = [(0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7)]
    none = torch.iinfo(torch.int64).max
    keys, pos = [], []
    inside = d < 0.0
    for axis in range(3):
        step = torch.tensor([int(axis == a) for a in range(3)], device=dev)
        lowc = torch.nonzero(inside.narrow(axis, 0, d.shape[axis] - 1) != inside.narrow(axis, 1, d.shape[axis] - 1))
        best = torch.full((len(lowc),), none, device=dev)
        flip = torch.zeros(len(lowc), dtype=torch.bool, device=dev)
        for e, (a, b) in enumerate(ends):
            low = [min(corner[a][k], corner[b][k]) for k in range(3)]
            if corner[a][axis] == corner[b][axis]:
                continue
            cell = lowc - torch.tensor(low, device=dev)
            t = cell >> 3
            loc = cell & 7
            key = (rank[t[:, 0], t[:, 1], t[:, 2]] * 512 + loc[:, 0] * 64 + loc[:, 1] * 8 + loc[:, 2]) * 12 + e
            key = torch.where(tiles[t[:, 0], t[:, 1], t[:, 2]], key, none)
            better = key < best
            best = torch.where(better, key, best)
            flip = torch.where(better, torch.tensor(corner[a][axis] > corner[b][axis], device=dev), flip)
        va = d[tuple(lowc.T)]
        vb = d[tuple((lowc + step).T)]
        t = (0.0 - va) / (vb - va)
        keys.append(best)
        pos.append((lowc + lo).double() + t[:, None] * step.double())
    keys, pos = torch.cat(keys), torch.cat(pos)
    ok = keys != none
    return [pos[ok][torch.argsort(keys[ok])], None]


def _exact_particles(case, seed):
    f = _particle_field(case).double()
    h = 1.0 / case["cells"]
    pg = _particles(case, seed)
    pos = pg["position"]
    dev = f.device

    def bins(p):
        i = torch.floor(p / h + 0.5).long() & ~7
        return i
    p = torch.from_numpy(np.ascontiguousarray(pos)).to(dev)

    def by_leaf(q):
        i = bins(q) >> 3
        i = i - i.min(0).values
        return torch.argsort((i[:, 0] << 42) | (i[:, 1] << 21) | i[:, 2], stable=True)
    p = p[by_leaf(p)]
    zero = torch.zeros((), dtype=F64, device=dev)
    lo = torch.zeros(3, dtype=torch.long, device=dev)

    def u(q):
        return torch.stack([_sample_dense(f[a], lo, q / h, zero) for a in range(3)], -1)
    dt = 0.005
    if case["rk4"]:
        k1 = dt * u(p)
        k2 = dt * u(p + 0.5 * k1)
        k3 = dt * u(p + 0.5 * k2)
        k4 = dt * u(p + k3)
        p = p + (k1 + 2 * k2 + 2 * k3 + k4) / 6.0
    else:
        p = p + dt * u(p)
    return [p[by_leaf(p)], None, None]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("frame", "host"):
        return _exact_frame(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind == "adjoint_ls":
        return _exact_adjoint_ls(case, seed)
    if kind == "crate":
        return _exact_crate(case, seed)
    if kind == "mesh":
        return _exact_mesh(case, seed)
    return _exact_particles(case, seed)
