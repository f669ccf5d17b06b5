"""Performance cases of the SPH step library: what its users have it do, with
sizes, inputs, the work each pass cannot do without, and 64-bit results.

Every case goes through the Python mirror of the C ABI (World, Batch).  A step
case is one fed step, as a host application drives it: the step's input state
is written from device memory, the world steps, and the state (and the density
where the call reports it) is read back into the caller's device memory.  One
step from a given state keeps the work per pass what the workload states; a
free rollout of these parameter sets blows up within a few steps.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG_DIR = os.path.join(ROOT, "particle-fluid-simulation_b200")


def _package():
    """The package (its directory name is not an identifier), as pfs_b200."""
    if "pfs_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            "pfs_b200", os.path.join(PKG_DIR, "__init__.py"), submodule_search_locations=[PKG_DIR])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["pfs_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["pfs_b200"]


# ---- cases --------------------------------------------------------------------

def listed():
    return [
        # a small interactive scene: launches and latency are the whole cost
        {"name": "small_2k", "kind": "step", "scene": "dam", "n": 2047, "h": 0.07, "precision": "fp32"},
        # the dam break of the parity workload: 3 substeps per step
        {"name": "dam_break_16k", "kind": "step", "scene": "dam", "n": 16384, "h": 0.035, "precision": "fp32"},
        # one frame of the reference application: its particle count (a sparse
        # key mask: 4096 table slots), its parameters, step and point splats
        {"name": "reference_frame_300k", "kind": "frame", "scene": "reference", "n": 300000, "width": 1280, "height": 720},
        # the headline workload: a million particles, a full key mask
        {"name": "slab_1m", "kind": "step", "scene": "slab", "n": 1 << 20, "precision": "fp32"},
        # the same in the bandwidth form
        {"name": "slab_1m_fp16", "kind": "step", "scene": "slab", "n": 1 << 20, "precision": "fp16"},
        # a particle count nobody rounded, in the fused-arithmetic form
        {"name": "slab_odd_fast", "kind": "step", "scene": "slab", "n": 654321, "precision": "fast"},
        # the largest single scene, in both storage forms
        {"name": "blocks_4m", "kind": "step", "scene": "blocks", "n": 1 << 22, "precision": "fp32"},
        {"name": "blocks_4m_fp16", "kind": "step", "scene": "blocks", "n": 1 << 22, "precision": "fp16"},
        # many scenes of uneven sizes and parameters stepped together
        {"name": "batch_32", "kind": "batch", "count": 32, "lo": 2048, "hi": 262144, "sizes": 3, "precision": "fp32"},
        # one dense request of the serving stream, 3 substeps
        {"name": "request_150k_fp16", "kind": "step", "scene": "dam", "n": 150001, "h": 0.03, "precision": "fp16"},
        # the two ray-marched render modes at 720p: density map, light volume
        # and march of the reference's scene; map and refraction of the slab
        {"name": "volumetric_300k", "kind": "volumetric", "scene": "reference", "n": 300000, "width": 1280, "height": 720, "cells_per_h": 2.0},
        {"name": "refractive_1m", "kind": "refractive", "scene": "slab", "n": 1 << 20, "width": 1280, "height": 720, "cells_per_h": 1.0},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def _draw_n(rng, lo, hi):
    """A particle count: mostly whatever a caller has, sometimes a power of two."""
    n = _log_int(rng, lo, hi)
    return 1 << (n.bit_length() - 1) if rng.random() < 0.35 else n


def draw(rng):
    r = rng.random()
    if r < 0.62:
        scene = rng.choice(["dam", "dam", "slab", "slab", "blocks", "reference"])
        precision = rng.choice(["fp32", "fp32", "fast", "fp16"])
        if scene == "dam":
            n = _draw_n(rng, 1500, 300000)
            h = round(rng.uniform(1.2, 3.2) * (0.32 / n) ** (1.0 / 3.0), 5)
            return {"kind": "step", "scene": scene, "n": n, "h": h, "precision": precision}
        hi = {"slab": 1 << 20, "blocks": 1 << 22, "reference": 300000}[scene]
        return {"kind": "step", "scene": scene, "n": _draw_n(rng, 20000, hi), "precision": precision}
    if r < 0.72:
        return {"kind": "batch", "count": rng.randint(3, 32), "lo": 2048, "hi": _log_int(rng, 8192, 131072),
                "sizes": rng.randint(4, 10**6), "precision": rng.choice(["fp32", "fp32", "fp16"])}
    width = _log_int(rng, 320, 1280)
    size = {"width": width, "height": max(1, width * 9 // 16 + rng.randint(-3, 3))}
    if r < 0.8:
        return {"kind": "frame", "scene": "reference", "n": _draw_n(rng, 20000, 300000), **size}
    scene = rng.choice(["slab", "reference"])
    n = _draw_n(rng, 60000, 1 << 20 if scene == "slab" else 300000)
    return {"kind": rng.choice(["volumetric", "refractive"]), "scene": scene, "n": n,
            "cells_per_h": rng.choice([1.0, 1.25, 1.6]), **size}


# ---- inputs --------------------------------------------------------------------

def _precision(name):
    pfs = _package()
    return {"fp32": pfs.PFS_FP32, "fp16": pfs.PFS_FP16_CELL, "fast": pfs.PFS_FP32_FAST}[name]


def _scene(case, seed):
    """(params, pos, vel) of a case's scene; sizes by the case, values by the seed."""
    pfs = _package()
    from pfs_b200 import scenes
    n = case["n"]
    precision = _precision(case.get("precision", "fp32"))
    flags = pfs.PFS_FLAG_COLORS if case["kind"] == "frame" else 0
    if case["scene"] == "dam":
        sc = scenes.dam_break(n=n, seed=seed, h=case["h"], precision=precision, flags=flags)
    elif case["scene"] == "slab":
        sc = scenes.slab_1m(n=n, seed=seed, precision=precision, flags=flags)
        sc.params.h = 0.02 * ((1 << 20) / n) ** (1.0 / 3.0)  # the same neighbour count at every size
    elif case["scene"] == "blocks":
        sc = scenes.colliding_blocks(n=n, seed=seed, precision=precision, flags=flags)
        sc.params.h = 0.015 * ((1 << 22) / n) ** (1.0 / 3.0)
    else:
        # the reference's parameters and start: a centred slab falling at 100
        p = pfs.reference_default()
        p.precision, p.flags = precision, flags
        if n != 300000:
            p.h = 2.5 * (300000 / n) ** (1.0 / 3.0)
        rng = np.random.default_rng(seed)
        pos, vel = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
        pos[:, :3] = rng.uniform(np.array(p.box_min[:]) * 0.3, np.array(p.box_max[:]) * 0.3, (n, 3))
        vel[:, 2] = -100.0
        return p, pos, vel
    return sc.params, sc.pos, sc.vel


def _batch_scenes(case, seed):
    from pfs_b200 import scenes
    spec = np.random.default_rng(case["sizes"])
    sizes = np.exp(spec.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), case["count"])).astype(np.int64)
    out = []
    for k, n in enumerate(np.clip(sizes, case["lo"], case["hi"])):
        out.append(scenes.dam_break(int(n), seed=seed * 1000 + k, h=float(spec.uniform(0.015, 0.04)),
                                    target_density=float(spec.uniform(800.0, 1200.0)),
                                    pressure_multiplier=float(spec.uniform(100.0, 300.0)),
                                    viscosity=float(spec.uniform(0.01, 0.1)), precision=_precision(case["precision"])))
    return out


def _camera(p):
    """The camera of the render cases: in front of the box, looking along +y."""
    lo, hi = np.array(p.box_min[:], np.float64), np.array(p.box_max[:], np.float64)
    c = (lo + hi) / 2
    return (float(c[0]), float(lo[1] - 1.2 * (hi[1] - lo[1])), float(c[2]))


def _view(case, p):
    """Ray-march settings in units of h: map voxels, half-h steps, light voxels of 2h."""
    pfs = _package()
    h = float(p.h)
    ext = (0.4, 0.4, 0.2) if case["kind"] == "refractive" else (0.01, 0.01, 0.005)
    return pfs.volume_view(position=_camera(p), forward=(0, 1, 0), right=(1, 0, 0), up=(0, 0, 1),
                           density_cell_size=h / case["cells_per_h"], step_size=h / 2, light_step_size=2 * h,
                           extinction=ext)


def _float4(n):
    return torch.empty((n, 4), dtype=torch.float32, device="cuda")


def prepare(case, seed):
    pfs = _package()
    if case["kind"] == "batch":
        scs = _batch_scenes(case, seed)
        total = sum(s.n for s in scs)
        b = pfs.Batch(total, len(scs), _precision(case["precision"]), scs[0].params.substeps)
        ids = [b.add(s.params, s.pos, s.vel) for s in scs]
        b.set_feed(True)  # every step runs the scenes' input states
        pos, vel = _float4(total), _float4(total)
        reads, off = [], 0
        for i, s in zip(ids, scs):
            reads.append((i, pos[off:].data_ptr(), vel[off:].data_ptr()))
            off += s.n
        return {"case": case, "batch": b, "reads": reads, "pos": pos, "vel": vel}
    p, pos, vel = _scene(case, seed)
    w = pfs.World(p, pos, vel)
    st = {"case": case, "world": w}
    if case["kind"] in ("step", "frame"):
        st["in"] = (torch.from_numpy(pos).cuda(), torch.from_numpy(vel).cuda())
        st["pos"], st["vel"] = _float4(case["n"]), _float4(case["n"])
        st["density"] = torch.empty(case["n"], dtype=torch.float32, device="cuda")
    else:
        w.step(1)  # the frames show a stepped state
        w.sync()
        st["view"] = _view(case, p)
    if case["kind"] == "frame":
        st["splats"] = pfs.splat_view(_camera(p), (0, 1, 0), case["width"], case["height"], 0.3)
    if case["kind"] != "step":
        st["rgba"] = torch.empty((case["height"], case["width"], 4), dtype=torch.float32, device="cuda")
        st["depth"] = torch.empty((case["height"], case["width"]), dtype=torch.float32, device="cuda")
    if case["kind"] == "refractive":
        # the iso-surface at half the density of the undisturbed fluid
        st["refraction"] = pfs.refraction(surface_density_threshold=0.5 * _mean_density(case, p))
    return st


def _mean_density(case, p):
    """Number density of the scene's fluid times the particle mass."""
    return _number_density(case, p) * float(p.particle_mass)


def _number_density(case, p):
    n = case["n"]
    if case["scene"] == "dam":
        return n / 0.32
    if case["scene"] == "slab":
        return n / (0.8 * 1.6 * 2.0)
    if case["scene"] == "blocks":
        return n / (2 * 1.4 * 2.0 * 2.0)
    return n / float(np.prod((np.array(p.box_max[:]) - np.array(p.box_min[:])) * 0.3))


# ---- one pass ------------------------------------------------------------------

def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(1)
        for sid, pos, vel in state["reads"]:
            b.read_ptr(sid, pos, vel)
        return {"pos": state["pos"], "vel": state["vel"]}
    pfs, w = _package(), state["world"]
    if case["kind"] in ("step", "frame"):
        w.write_ptr(state["in"][0].data_ptr(), state["in"][1].data_ptr())
        w.step(1)
        out = {"pos": state["pos"], "vel": state["vel"], "density": state["density"]}
        if case["kind"] == "frame":
            w.render_splats_ptr(state["splats"], case["width"], case["height"], state["rgba"].data_ptr(),
                                state["depth"].data_ptr())
            out["rgba"], out["depth"] = state["rgba"], state["depth"]
        ptr = ctypes.c_void_p
        pfs.check(pfs.lib().pfs_world_read(w.handle, ptr(out["pos"].data_ptr()), ptr(out["vel"].data_ptr()),
                                           ptr(out["density"].data_ptr()), None, None), "pfs_world_read")
        return out
    if case["kind"] == "volumetric":
        w.render_volumetric_ptr(state["view"], case["width"], case["height"], state["rgba"].data_ptr())
    else:
        w.render_refractive_ptr(state["view"], state["refraction"], case["width"], case["height"],
                                state["rgba"].data_ptr())
    return {"rgba": state["rgba"]}


def _step_work(n, neighbours, substeps):
    """State in and out, density out; per in-range pair the distance and its
    two kernel sums (16 operations) and the force terms (60)."""
    return {"bytes": n * (32 + 32 + 4), "flops": n * neighbours * 76 * substeps}


def work(case):
    if case["kind"] == "batch":
        by = fl = 0
        for s in _batch_specs(case):
            w = _step_work(s[0], s[0] / 0.32 * 4.19 * s[1] ** 3, 3)
            by, fl = by + w["bytes"], fl + w["flops"]
        return {"bytes": by, "flops": fl}
    n = case["n"]
    p = _scene_params(case)
    h = float(p.h)
    near = _number_density(case, p) * 4.19 * h ** 3
    px = case.get("width", 0) * case.get("height", 0)
    if case["kind"] in ("step", "frame"):
        w = _step_work(n, near, int(p.substeps))
        if case["kind"] == "frame":
            # colours in, image and depth out; a disc's coverage test per pixel it touches
            w["bytes"] += n * 16 + px * 20
            w["flops"] += n * 60
        return w
    # positions and keys in, image out; each voxel's sum over its sphere; a
    # trilinear sample (30 operations) per march step of each ray
    cs = h / case["cells_per_h"]
    ext = np.array(p.box_max[:], np.float64) - np.array(p.box_min[:], np.float64)
    fluid = n / _number_density(case, p)
    steps = float(ext[1]) / (h / 2)
    return {"bytes": n * 20 + px * 16, "flops": fluid / cs ** 3 * near * 14 + px * 0.25 * steps * 30}


def _batch_specs(case):
    """(n, h) of the batch's scenes."""
    spec = np.random.default_rng(case["sizes"])
    sizes = np.exp(spec.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), case["count"])).astype(np.int64)
    out = []
    for n in np.clip(sizes, case["lo"], case["hi"]):
        out.append((int(n), float(spec.uniform(0.015, 0.04))))
        spec.uniform(size=3)
    return out


def _scene_params(case):
    """The scene's parameters without its particles."""
    small = dict(case, n=8)
    p = _scene(small, 0)[0]
    n = case["n"]
    if case["scene"] == "slab":
        p.h = 0.02 * ((1 << 20) / n) ** (1.0 / 3.0)
    elif case["scene"] == "blocks":
        p.h = 0.015 * ((1 << 22) / n) ** (1.0 / 3.0)
    elif case["scene"] == "reference":
        p.h = 2.5 * (300000 / n) ** (1.0 / 3.0)
    return p


# ---- 64-bit results --------------------------------------------------------------
# One substep of the reference's equations in 64 bits.  What is discrete (cell
# coordinates, keys, the sort, which sample points lie in the box) follows the
# float32 values, as the equations define them; all sums and the state are in
# 64 bits.  A candidate counts once for every sample cell that hashes to its
# key, so pairs are found by distance and weighted by that number.

def _cells(x32, lo, h):
    # h as a tensor of x's shape: a device division by a plain number multiplies by its reciprocal
    return torch.floor((x32 - lo) / torch.full_like(x32, h)).to(torch.int64)


def _slots(c, mask):
    m = 0xFFFFFFFF
    k = ((c[..., 0] * 73856093) & m) ^ ((c[..., 1] * 19349663) & m) ^ ((c[..., 2] * 83492791) & m)
    k = ((k ^ (k >> 16)) * 0x7FEB352D) & m
    k = ((k ^ (k >> 15)) * 0x846CA68B) & m
    return (k ^ (k >> 16)) & mask


def _offsets(dev):
    r = torch.arange(27, device=dev)
    return torch.stack([r % 3 - 1, (r // 3) % 3 - 1, r // 9 - 1], 1)


def _pairs(q, x, radius, most=1 << 22):
    """Chunks (i, j) of the pairs |q_i - x_j| < radius, by a grid of x."""
    side = radius * 1.0001
    lo = torch.minimum(q.min(0).values, x.min(0).values) - side
    cx, cq = ((x - lo) / side).long(), ((q - lo) / side).long()
    dims = torch.maximum(cx.max(0).values, cq.max(0).values) + 2
    flat = lambda c: c[:, 0] + dims[0] * (c[:, 1] + dims[1] * c[:, 2])  # noqa: E731
    key, order = torch.sort(flat(cx))
    qkey = flat(cq)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            row = qkey + dims[0] * (dy + dims[1] * dz)
            a, b = torch.searchsorted(key, row - 1), torch.searchsorted(key, row + 2)
            ends = torch.cumsum(b - a, 0)
            total, start = int(ends[-1]), 0
            for base in range(0, total, most):
                t = torch.arange(base, min(base + most, total), device=q.device)
                i = torch.searchsorted(ends, t, right=True)
                j = order[a[i] + t - (ends[i] - (b - a)[i])]
                near = ((q[i] - x[j]) ** 2).sum(1) < radius * radius
                yield i[near], j[near]


def _weights(slots, valid, i, j, key):
    """How many of point i's sample cells have candidate j's key."""
    return ((slots[i] == key[j][:, None]) & valid[i]).sum(1).double()


def _f64(a, dev):
    return torch.tensor(np.array(a, np.float32).astype(np.float64), device=dev)


def _walls(x, v, p, margin, dev):
    lo, hi = _f64(p.box_min[:], dev) + margin, _f64(p.box_max[:], dev) - margin
    rest = _f64(p.restitution[:], dev).view(3, 2)
    under, over = x < lo, x > hi
    v = torch.where(under, -v * rest[:, 0], torch.where(over, -v * rest[:, 1], v))
    return torch.minimum(torch.maximum(x, lo), hi), v


def _exact_step(p, pos, vel, dev):
    """(positions, velocities, densities, keys) after one substep, in sort order."""
    f = np.float32
    n, h, h32, m = pos.shape[0], float(p.h), float(p.h), float(p.particle_mass)
    lo32 = torch.tensor(np.array(p.box_min[:], f), device=dev)
    hi32 = torch.tensor(np.array(p.box_max[:], f), device=dev)
    x32, v32 = torch.from_numpy(pos[:, :3]).to(dev), torch.from_numpy(vel[:, :3]).to(dev)
    key, perm = torch.sort(_slots(_cells(x32, lo32, h32), n - 1), stable=True)
    x32, v32 = x32[perm], v32[perm]
    g, dt = _f64(p.gravity[:], dev), float(p.dt)
    # predicted positions: the float32 ones give the cells, the 64-bit ones the sums
    xs, vs = x32.double(), v32.double()
    vp = vs + g * dt
    xp, vp = _walls(xs + vp * dt, vp, p, float(p.margin_predict), dev)
    gdt = torch.tensor([float(f(f(a) * f(dt))) for a in p.gravity[:]], dtype=torch.float32, device=dev)
    vp32 = v32 + gdt
    xp32 = x32 + vp32 * torch.tensor(dt, dtype=torch.float32, device=dev)
    mp = torch.tensor(f(p.margin_predict), device=dev)
    xp32 = torch.minimum(torch.maximum(xp32, lo32 + mp), hi32 - mp)
    off = _offsets(dev)
    samples = xp32[:, None, :] + off.float()[None] * torch.tensor(h32, dtype=torch.float32, device=dev)
    valid = ((samples >= lo32) & (samples <= hi32)).all(2)
    slots = _slots(_cells(samples, lo32, h32), n - 1).int()
    cell = _cells(xp32, lo32, h32)
    fslots = _slots(cell[:, None, :] + off[None], n - 1).int()
    every = torch.ones_like(valid)
    key32 = key.int()
    rho = torch.zeros(n, dtype=torch.float64, device=dev)
    near = torch.zeros_like(rho)
    for i, j in _pairs(xp, xp, h):
        a = (h - (xp[i] - xp[j]).norm(dim=1)) * 1.0
        wgt = m * _weights(slots, valid, i, j, key32)
        rho.index_add_(0, i, wgt * a * a)
        near.index_add_(0, i, wgt * a * a * a)
    volume = float(p.volume) if p.volume > 0 else 2.0 * math.pi * h ** 5 / 15.0
    rho = torch.clamp(rho / volume, min=float(f(0.01)))
    near = torch.clamp(near * 15.0 / (math.pi * h ** 6), min=float(f(0.01)))
    press = (rho - float(p.target_density)) * float(p.pressure_multiplier)
    npress = near * float(p.near_pressure_multiplier)
    force = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    for i, j in _pairs(xp, xp, h):
        d = xp[j] - xp[i]
        dist = d.norm(dim=1)
        keep = (i != j) & (dist >= 1e-7)
        i, j, d, dist = i[keep], j[keep], d[keep], dist[keep]
        wgt = m * _weights(fslots, every, i, j, key32)
        a = h - dist
        pc = 0.5 * (press[i] + press[j]) * (-a * 15.0 / (math.pi * h ** 5)) / rho[j]
        pc += 0.5 * (npress[i] + npress[j]) * (a * a * -45.0 / (math.pi * h ** 6)) / near[j]
        term = (wgt * pc / dist)[:, None] * d
        term += float(p.viscosity) * (wgt * a * a / rho[j])[:, None] * (vs[j] - vp[i])
        force.index_add_(0, i, term)
    v = vs + force / rho[:, None] * dt + g * dt
    x, v = _walls(xs + v * dt, v, p, float(p.margin_integrate), dev)
    return x, v, rho, key32


def _exact_map(p, x, key, n, cs, dev):
    """The density map of positions x (64 bits) with the keys of the last sort."""
    f = np.float32
    cs, h = float(f(cs)), float(p.h)
    lo, hi = np.array(p.box_min[:], f), np.array(p.box_max[:], f)
    dims = [int(math.ceil(float(f(f(b - a) * f(1.0 / f(cs)))))) for a, b in zip(lo, hi)]
    bound = torch.tensor([int(math.ceil(float(f(f(b - a) / f(cs))))) for a, b in zip(lo, hi)], device=dev)
    c = torch.stack(torch.meshgrid(*[torch.arange(d, device=dev) for d in dims[::-1]], indexing="ij"), 3)
    c = c.flip(3).reshape(-1, 3)
    lo32, hi32 = torch.tensor(lo, device=dev), torch.tensor(hi, device=dev)
    centre32 = lo32 + (c.float() + 0.5) * torch.tensor(cs, dtype=torch.float32, device=dev)
    inside = ((centre32 >= lo32) & (centre32 <= hi32)).all(1)
    cell = torch.where(inside[:, None], _cells(centre32, lo32, h), torch.full_like(c, -1))
    out_of = lambda k: ((k < 0) | (k > bound)).any(-1) | (k == bound).all(-1)  # noqa: E731
    centre = _f64(lo, dev) + (c.double() + 0.5) * cs
    grid = torch.zeros(c.shape[0], dtype=torch.float64, device=dev)
    box_lo, box_hi = x.min(0).values - h, x.max(0).values + h
    some = torch.nonzero(((centre >= box_lo) & (centre <= box_hi)).all(1) & ~out_of(c)).view(-1)
    around = cell[some][:, None, :] + _offsets(dev)[None]
    slots, valid = _slots(around, n - 1).int(), ~out_of(around)
    q = centre[some]
    sums = torch.zeros(some.shape[0], dtype=torch.float64, device=dev)
    for i, j in _pairs(q, x, h):
        a = h - (q[i] - x[j]).norm(dim=1)
        sums.index_add_(0, i, float(p.particle_mass) * _weights(slots, valid, i, j, key) * a * a)
    volume = float(p.volume) if p.volume > 0 else 2.0 * math.pi * h ** 5 / 15.0
    grid[some] = sums / volume
    return grid.view(dims[2], dims[1], dims[0])


def _sample(img, uvw):
    """Trilinear samples at normalised coordinates, clamped to the edge."""
    d = torch.tensor(img.shape[::-1], device=img.device)
    u = uvw * d - 0.5
    k = torch.floor(u)
    f = u - k
    k = k.long()
    a, b = torch.minimum(k.clamp(min=0), d - 1), torch.minimum((k + 1).clamp(min=0), d - 1)
    r = 0.0
    for s in range(8):
        w, at = 1.0, []
        for ax in range(3):
            up = (s >> ax) & 1
            w = w * (f[:, ax] if up else 1 - f[:, ax])
            at.append((b if up else a)[:, ax])
        r = r + w * img[at[2], at[1], at[0]]
    return r


def _ray_box(lo, hi, o, d):
    a, b = (lo - o) / d, (hi - o) / d
    t0, t1 = torch.minimum(a, b).max(1).values, torch.maximum(a, b).min(1).values
    return t0, t1, (t0 <= t1) & (t1 >= 0)


def _exact_volumetric(case, p, x, key, dev):
    view = _view(case, p)
    lo, hi = _f64(p.box_min[:], dev), _f64(p.box_max[:], dev)
    size = hi - lo
    dmap = _exact_map(p, x, key, case["n"], view.density_cell_size, dev)
    ls, step = float(view.light_step_size), float(view.step_size)
    sun = _f64(view.dir_to_sun[:], dev)[None]
    f = np.float32
    ldims = [int(math.ceil(float(f(f(b - a) * f(1.0 / f(ls)))))) for a, b in zip(p.box_min[:], p.box_max[:])]
    c = torch.stack(torch.meshgrid(*[torch.arange(d, device=dev) for d in ldims[::-1]], indexing="ij"), 3)
    c = c.flip(3).reshape(-1, 3).double()
    o = lo + (c + 0.5) * ls
    t0, t1, hit = _ray_box(lo, hi, o, sun.expand_as(o))
    hit &= ~(c > size).any(1)
    t, t1 = (t0 - 1.0).clamp(min=0), t1 + 1.0
    light = torch.zeros(c.shape[0], dtype=torch.float64, device=dev)
    while True:
        live = torch.nonzero(hit & (t < t1)).view(-1)
        if not live.numel():
            break
        light[live] += _sample(dmap, (o[live] + t[live, None] * sun - lo) / size) * ls
        t[live] += ls
    light = light.view(ldims[2], ldims[1], ldims[0])
    w, hgt = case["width"], case["height"]
    half_h = math.tan(0.5 * float(view.fov))
    half_w = half_h * w / hgt
    px = torch.arange(w * hgt, device=dev)
    u = ((px % w).double() + 0.5) / w * 2 - 1
    v = ((px // w).double() + 0.5) / hgt * 2 - 1
    fwd, right, up = (_f64(a[:], dev) for a in (view.forward, view.right, view.up))
    d = fwd + (u * half_w)[:, None] * right - (v * half_h)[:, None] * up
    d = d / d.norm(dim=1, keepdim=True)
    pos = _f64(view.position[:], dev)[None]
    t0, t1, hit = _ray_box(lo, hi, pos, d)
    t, t1 = (t0 + 1.0).clamp(min=0) + step, t1 - 1.0 - step
    ext = _f64(view.extinction[:], dev)
    ext = ext / ext.norm()
    amb = torch.tensor([0.529, 0.808, 0.922], dtype=torch.float64, device=dev)
    rgb = torch.zeros((w * hgt, 3), dtype=torch.float64, device=dev)
    depth = torch.zeros(w * hgt, dtype=torch.float64, device=dev)
    while True:
        live = torch.nonzero(hit & (t < t1)).view(-1)
        if not live.numel():
            break
        uvw = ((pos + t[live, None] * d[live] - lo) / size).clamp(0, 1)
        dens = _sample(dmap, uvw) * 0.05
        depth[live] += dens * step
        tr = torch.exp(-depth[live, None] * ext)
        thick = tr.max(1).values < 0.01
        glow = torch.exp(-_sample(light, uvw)[:, None] * ext) * amb * dens[:, None] * ext
        rgb[live] += torch.where(thick[:, None], torch.zeros_like(glow), glow * tr)
        hit[live[thick]] = False
        t[live] += step
    rgb += 0.05 * (rgb > 1e-5).all(1, keepdim=True)
    return torch.cat([rgb, torch.ones_like(rgb[:, :1])], 1).view(hgt, w, 4)


def exact(case, seed):
    """64-bit results of one-substep cases and of the volumetric image.  None
    where there are none to compare with: three substeps (a change of the last
    bit reorders the particles of the next sort), refracted rays and splats (a
    grazing ray, or two discs at one depth, take one branch or the other)."""
    if case["kind"] in ("batch", "refractive"):
        return None
    p, pos, vel = _scene(case, seed)
    if p.substeps != 1:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, v, rho, key = _exact_step(p, pos, vel, dev)
    if case["kind"] == "volumetric":
        return {"rgba": _exact_volumetric(case, p, x, key, dev)}
    one = torch.ones_like(x[:, :1])
    out = {"pos": torch.cat([x, one], 1), "vel": torch.cat([v, one], 1), "density": rho}
    if case["kind"] == "frame":
        out["rgba"] = out["depth"] = None
    return out
