"""The workloads this package's speed is measured on, each through its public entry points.

A case is a dict of plain values with a `kind`:

  frame     LBMEngine.step_and_extract_slice: a few substeps, forces, slice image, macro field
  run       a stretch of time steps of one tunnel, then the forces and the macro field (and, in the
            two FP64-arithmetic modes, the populations) read into the host's own pinned buffers
  batch     LBMBatch: a sweep of tunnels stepped together, then every tunnel's forces and macro field
  voxelize  a triangle mesh to flags, boundary list and link fractions
  diagnose  a few steps, then the Q-criterion and vorticity of the flow
  train     Adam iterations of the learned subgrid closure

Tunnels hold a seeded ellipsoid at an angle of attack with exact link fractions and restart from a
seeded field (a uniform stream with long waves of velocity and density), as a program does that
resumes a run.  Sizes are those of the package's own configurations (aerosim_b200/cases.py): the
64x32x32 sphere tunnel, the 128x64x64 interactive tunnel, the 256x128x128 benchmark and its 512x256x256
refinement, and the 128..190-cell sweep, with odd and ragged lattices between them.
"""
import ctypes as C
import math
import os

import numpy as np
import torch

import aerosim_b200
from aerosim_b200 import LBMBatch, LBMEngine, VoxelGridResult, sgs, voxelize_mesh_to_lattice
from aerosim_b200 import _native as N

DEV = "cuda"
# D3Q19: rest, 6 faces, 12 edges; directions 2k+1 and 2k+2 are opposite
VEL = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
       (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1),
       (0, -1, 1)]
OPP = [0] + [d + 1 if d % 2 else d - 1 for d in range(1, 19)]
W64 = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
W32 = [float(np.float32(w)) for w in W64]  # the collision's and the force integrator's weights
ELEM = {"f32": 4, "f32_mirror": 4, "f16s": 2, "bf16s": 2, "f16c": 2, "f64": 8}
CLOSURE = os.path.join(os.path.dirname(aerosim_b200.__file__), "data", "sgs_mlp_ellipsoid.npz")
CS, CHORD = 0.1, 0.2  # Smagorinsky constant; body semi-length in units of nx


def _flow(name, kind, nx, ny, nz, precision, steps, ground=False, closure=False):
    return {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": precision, "steps": steps,
            "ground": ground, "closure": closure}


def listed():
    return [
        # the interactive loop on the smallest tunnel: latency of a frame, its launches and readbacks
        _flow("frame_64x32x32_f32", "frame", 64, 32, 32, "f32", 4),
        # the headline workload, and its 16-bit storage
        _flow("run_256x128x128_f32", "run", 256, 128, 128, "f32", 40),
        _flow("run_256x128x128_f16s", "run", 256, 128, 128, "f16s", 40),
        # an odd, ragged lattice with the no-slip ground of the vehicle presets, BF16 storage
        _flow("run_191x95x97_bf16s_ground", "run", 191, 95, 97, "bf16s", 40, ground=True),
        # the fine run behind the closure's training data: the largest lattice in use
        _flow("run_512x256x256_f32", "run", 512, 256, 256, "f32", 30),
        # the coarse run with the learned closure
        _flow("run_256x128x128_closure", "run", 256, 128, 128, "f32", 30, closure=True),
        # the bit-parity mode, as a regression run compares it: populations read back
        _flow("run_128x64x64_mirror", "run", 128, 64, 64, "f32_mirror", 20),
        # an angle-of-attack sweep on growing lattices
        {"name": "batch_12_f16s", "kind": "batch", "count": 12, "nx": 128, "grow": 4, "precision": "f16s", "steps": 50},
        # a body set up for the benchmark lattice, and the interactive tunnel's nose cone
        {"name": "voxelize_256x128x128_ellipsoid", "kind": "voxelize", "nx": 256, "ny": 128, "nz": 128,
         "body": "ellipsoid", "rings": 80, "segments": 128, "engine": True},
        {"name": "voxelize_128x64x64_ogive", "kind": "voxelize", "nx": 128, "ny": 64, "nz": 64, "body": "ogive",
         "rings": 62, "segments": 72, "engine": False},
        # vortex cores of a running flow
        _flow("diagnose_192x96x96_f32", "diagnose", 192, 96, 96, "f32", 4),
        # a stretch of the closure's training
        {"name": "train_400k_b16384", "kind": "train", "rows": 400_000, "batch": 16384, "iters": 40},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run"] * 9 + ["frame"] * 3 + ["batch"] * 2 + ["voxelize"] * 3 + ["diagnose"] * 2 + ["train"] * 2)
    if kind == "train":
        return {"kind": kind, "rows": _log(rng, 20_000, 400_000), "batch": _log(rng, 512, 16384), "iters": rng.randint(5, 40)}
    if kind == "voxelize":
        nx = _log(rng, 48, 256)
        return {"kind": kind, "nx": nx, "ny": max(24, nx // 2 + rng.randint(-7, 7)),
                "nz": max(24, nx // 2 + rng.randint(-7, 7)), "body": rng.choice(["ellipsoid", "ogive"]),
                "rings": rng.randint(20, 80), "segments": rng.randint(24, 128), "engine": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 12), "nx": rng.randint(64, 130), "grow": rng.choice([1, 2, 3, 4]),
                "precision": rng.choice(["f32", "f16s", "bf16s", "f16c"]), "steps": rng.randint(5, 50)}
    prec = rng.choice(["f32", "f32", "f32", "f16s", "f16s", "bf16s", "f16c", "f32_mirror", "f64"]) if kind == "run" else "f32"
    nx = _log(rng, 40, 160 if prec in ("f32_mirror", "f64") else 200 if kind == "diagnose" else 400)
    ny, nz = (max(16, nx // 2 + rng.randint(-9, 9)) for _ in range(2))
    steps = rng.randint(4, 40) if kind == "run" else rng.randint(1, 8)
    closure = prec == "f32" and kind == "run" and rng.random() < 0.25
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": prec, "steps": steps,
            "ground": rng.random() < 0.3, "closure": closure}


# ---- inputs ---------------------------------------------------------------------------


def _grid(nx, ny, nz, seed):
    """A voxel grid (lattice unit 1 m) of an ellipsoid at an angle of attack, its shape, place and
    angle from the seed: the closed-form counterpart of a voxelized mesh."""
    r = np.random.default_rng(seed)
    scale = nx / 256.0
    axes = np.array([40.0, 16.0, 12.0]) * scale * r.uniform(0.9, 1.1, 3)
    axes = np.minimum(np.maximum(axes, 2.6), np.array([0.4 * nx, 0.35 * ny, 0.35 * nz]))
    angle = math.radians(r.uniform(-8.0, 12.0))
    centre = np.array([nx / 4, ny / 2, nz / 2]) + r.uniform(-0.5, 0.5, 3)  # in cells
    c, s = math.cos(angle), math.sin(angle)
    rot = torch.tensor([[c, -s, 0.0], [s, c, 0.0], [0.0, 0.0, 1.0]], dtype=torch.float64, device=DEV)
    inv = torch.tensor(1.0 / axes, device=DEV)

    def local(p):  # cell-centre coordinates to the unit sphere's
        return ((p - torch.tensor(centre, device=DEV)) @ rot.T) * inv

    z, y, x = torch.meshgrid(*(torch.arange(n, device=DEV, dtype=torch.float64) + 0.5 for n in (nz, ny, nx)), indexing="ij")
    solid = torch.zeros(nz, ny, nx, dtype=torch.bool, device=DEV)
    for k in range(nz):  # a plane at a time: the largest lattice needs no 64-bit copy of itself
        solid[k] = (local(torch.stack([x[k], y[k], z[k]], -1)) ** 2).sum(-1) <= 1.0
    del x, y, z
    link = torch.zeros(18, *solid.shape, dtype=torch.bool, device=DEV)
    for d in range(1, 19):
        link[d - 1] = _shifted(solid, VEL[d], False) & ~solid
    flags = solid.to(torch.uint8)
    flags[link.any(0)] = 2
    cells = torch.nonzero(flags.reshape(-1) == 2).reshape(-1)
    q = torch.full((cells.numel(), 18), -1.0, dtype=torch.float64, device=DEV)
    at = torch.stack([cells % nx, cells // nx % ny, cells // (nx * ny)], -1).double() + 0.5
    p = local(at)
    for d in range(1, 19):  # |p + t v| = 1
        v = (torch.tensor(VEL[d], dtype=torch.float64, device=DEV) @ rot.T) * inv
        a, b, cc = (v * v).sum(), (p * v).sum(-1), (p * p).sum(-1) - 1.0
        t = (-b - torch.sqrt(torch.clamp(b * b - a * cc, min=0.0))) / a
        has = link[d - 1].reshape(-1)[cells]
        q[:, d - 1] = torch.where(has, t.clamp(1e-4, 1.0), q[:, d - 1])
    q = q.float()
    bmap = torch.full((solid.numel(),), -1, dtype=torch.int32, device=DEV)
    bmap[cells] = torch.arange(cells.numel(), dtype=torch.int32, device=DEV)
    minq = torch.where(q > 0, q, torch.ones_like(q)).amin(1)
    n_solid = int(solid.sum())
    host = [t.reshape(-1).cpu().numpy() for t in (flags, bmap, cells.int(), q, minq)]
    return VoxelGridResult(nx, ny, nz, 1.0, 1.0, 1.0, -nx / 2, -ny / 2, -nz / 2, *host, n_solid, cells.numel(),
                           nx * ny * nz - n_solid - cells.numel(), 0.0)


def _shifted(a, v, outside):
    """b[z, y, x] = a[z + vz, y + vy, x + vx], `outside` beyond the lattice."""
    b = torch.full_like(a, outside)
    src, dst = [], []
    for n, c in zip(a.shape, (v[2], v[1], v[0])):
        src.append(slice(max(0, c), n + min(0, c)))
        dst.append(slice(max(0, -c), n + min(0, -c)))
    b[tuple(dst)] = a[tuple(src)]
    return b


def _config(case, seed, nx, ny, nz):
    u = 0.05 + 0.03 * float(np.random.default_rng(seed + 1).random())
    return {"uInletLattice": u, "nuLattice": u * 2 * CHORD * nx / 2e4, "smagorinskyCs": CS,
            "groundNoSlip": bool(case.get("ground", False)), "precision": case["precision"],
            "frontalAreaM2": math.pi * (0.06 * nx) * (0.047 * nx), "characteristicLengthM": 2 * CHORD * nx,
            "tunnel": {"length": float(nx), "width": float(nz), "height": float(ny)}}


def _equilibrium(rho, u):
    sq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    for (a, b, c), w in zip(VEL, W64):
        cu = 3.0 * (a * u[0] + b * u[1] + c * u[2])
        yield w * rho * (1.0 + cu + 0.5 * cu * cu - 1.5 * sq)


def _restart(grid, u0, seed):
    """Populations [19, nz, ny, nx] float32 on the GPU: the equilibrium of a stream u0 with long waves."""
    r = np.random.default_rng(seed + 2)
    nz, ny, nx = grid.nz, grid.ny, grid.nx
    ax = [torch.arange(n, device=DEV, dtype=torch.float32) / n for n in (nx, ny, nz)]
    fields = []
    for _ in range(4):
        acc = torch.zeros(nz, ny, nx, device=DEV)
        for _ in range(3):
            k, ph = r.integers(1, 5, 3), r.uniform(0, 2 * math.pi, 3)
            w = [torch.sin(2 * math.pi * int(k[i]) * ax[i] + float(ph[i])) for i in range(3)]
            acc += w[2][:, None, None] * w[1][None, :, None] * w[0][None, None, :]
        fields.append(acc)
    solid = torch.from_numpy(grid.cellFlags).to(DEV).reshape(nz, ny, nx) == 1
    open_ = (~solid).float()
    u = [(u0 * (i == 0) + 0.1 * u0 * fields[i]) * open_ for i in range(3)]
    rho = 1.0 + 5e-4 * fields[3] * open_
    f = torch.empty(19, nz, ny, nx, device=DEV)
    for d, e in enumerate(_equilibrium(rho, u)):
        f[d] = e
    return f


def _start(case, seed, nx, ny, nz):
    """(engine, grid, config): a tunnel ready to resume from a seeded field."""
    grid = _grid(nx, ny, nz, seed)
    cfg = _config(case, seed, nx, ny, nz)
    eng = LBMEngine(0)
    eng.set_voxel_grid(grid, cfg)
    if case.get("closure"):
        eng.set_sgs_mlp(np.load(CLOSURE)["params"])
    return eng, grid, cfg


def _pinned(n, dtype=torch.float32):
    return torch.empty(n, dtype=dtype, pin_memory=True)


def _ptr(t, c_type):
    return C.cast(t.data_ptr(), C.POINTER(c_type))


def _host_buffers(case, cells):
    """What a program that reads a tunnel's fields keeps on the host."""
    s = {"macro": [_pinned(cells) for _ in range(4)]}
    if case["precision"] in ("f32_mirror", "f64"):
        s["pops"] = _pinned(19 * cells, torch.float64 if case["precision"] == "f64" else torch.float32)
    return s


def _mesh(case, seed):
    """(positions, indices), a column-major world matrix and the tunnel of a body of revolution about x:
    closed, `rings` x `segments`, at an angle of attack; the ellipsoid with a long-wave dent."""
    r = np.random.default_rng(seed)
    nx, rings, seg = case["nx"], case["rings"], case["segments"]
    t = np.linspace(0.0, 1.0, rings + 1)[1:-1]
    if case["body"] == "ellipsoid":
        x, rad = -np.cos(math.pi * t), np.sin(math.pi * t)
        ends, size = (-1.0, 1.0), np.array([40.0, 16.0, 12.0])
    else:  # tangent ogive on a body tube, tip towards the inlet
        x = 2.0 * t - 1.0
        nose, rho = 1.4, (0.36 ** 2 + 1.4 ** 2) / (2 * 0.36)
        rad = np.where(x < -1.0 + nose, np.sqrt(np.maximum(rho ** 2 - (nose - (x + 1.0)) ** 2, 0.0)) + 0.36 - rho, 0.36)
        ends, size = (-1.0, 1.0), np.array([36.0, 36.0, 36.0])
    ang = 2 * math.pi * np.arange(seg) / seg
    p = np.stack([np.repeat(x[:, None], seg, 1), rad[:, None] * np.cos(ang), rad[:, None] * np.sin(ang)], -1).reshape(-1, 3)
    if case["body"] == "ellipsoid":
        k = r.standard_normal(3) * 0.04
        p = p * (1.0 + k[0] * p[:, :1] * p[:, 1:2] + k[1] * p[:, 1:2] * p[:, 2:] + k[2] * (p[:, :1] ** 2 - p[:, 2:] ** 2))
    p = np.concatenate([p, [[ends[0], 0.0, 0.0], [ends[1], 0.0, 0.0]]])
    n, (i, j) = len(x), np.meshgrid(np.arange(len(x) - 1), np.arange(seg), indexing="ij")
    a, b = i * seg + j, i * seg + (j + 1) % seg
    j0, j1 = np.arange(seg), (np.arange(seg) + 1) % seg
    tri = np.concatenate([np.stack([a, b, a + seg], -1).reshape(-1, 3), np.stack([b, b + seg, a + seg], -1).reshape(-1, 3),
                          np.stack([np.full(seg, n * seg), j1, j0], -1),
                          np.stack([np.full(seg, n * seg + 1), (n - 1) * seg + j0, (n - 1) * seg + j1], -1)])
    size = np.minimum(size * nx / 256.0, 0.38 * min(case["ny"], case["nz"]) / np.array([0.9, 1.0, 1.0])) * r.uniform(0.95, 1.05)
    th = math.radians(r.uniform(-10.0, 14.0))
    m = np.eye(4)
    m[:2, :2] = [[math.cos(th), -math.sin(th)], [math.sin(th), math.cos(th)]]
    m[:3, 3] = [-nx / 5.0, 0.3, -0.2]
    return ((p * size).astype(np.float32), tri.astype(np.int32)), m.T.reshape(-1).copy(), \
        {"length": float(nx), "width": float(case["nz"]), "height": float(case["ny"])}


def _rows(case, seed):
    """Closure samples: strain rates of a wake, density, wall distance; targets with the scatter of a
    filtered flow, clipped at zero as the training data are."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = case["rows"]
    amp = torch.exp(torch.randn(n, 1, device=DEV, generator=g) * 0.8 - 1.5)
    s = torch.randn(n, 6, device=DEV, generator=g) * amp
    s[:, 2] = -s[:, 0] - s[:, 1]
    rho = torch.randn(n, 1, device=DEV, generator=g) * 0.3
    wall = torch.randint(1, 32, (n, 1), device=DEV, generator=g) / 16.0
    mag = (s * s).sum(1).sqrt()
    y = (3.0 * mag * (1.0 - torch.exp(-wall[:, 0])) + torch.randn(n, device=DEV, generator=g) * 0.7).clamp(0.0, 50.0)
    return torch.cat([s, rho, wall], 1).cpu().numpy(), y.cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "voxelize":
        mesh, world, tunnel = _mesh(case, seed)
        grid = {"nx": case["nx"], "ny": case["ny"], "nz": case["nz"]}
        cells = case["nx"] * case["ny"] * case["nz"]
        room = _room(case)
        # the host's grid, its boundary lists with room for any body
        lists = [torch.zeros(room, dtype=torch.int32), torch.zeros(room * 18), torch.zeros(room)]
        if case["engine"]:
            lists = [t.pin_memory() for t in lists]
        return {"case": case, "mesh": mesh, "world": world, "tunnel": tunnel, "grid": grid, "lists": lists,
                "dense": [_pinned(cells, torch.uint8), _pinned(cells, torch.int32)] if case["engine"] else None,
                "eng": LBMEngine(0) if case["engine"] else None}
    if kind == "train":
        X, Y = _rows(case, seed)
        return {"case": case, "X": X, "Y": Y, "params": sgs.init_params(seed), "seed": seed}
    if kind == "batch":
        s = {"case": case, "eng": [], "host": []}
        fields = []
        for k, (nx, ny, nz) in enumerate(_sweep(case)):
            e, grid, cfg = _start(case, seed + 10 * k, nx, ny, nz)
            s["eng"].append(e)
            s["host"].append(_host_buffers(case, nx * ny * nz))
            fields.append(_restart(grid, cfg["uInletLattice"], seed + 10 * k).cpu().numpy())
        s["batch"] = LBMBatch(s["eng"])
        s["batch"].autotune(10)
        for e, f in zip(s["eng"], fields):
            e.write_populations(f)
        return s
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    eng, grid, cfg = _start(case, seed, nx, ny, nz)
    eng.write_populations(_restart(grid, cfg["uInletLattice"], seed).cpu().numpy())
    s = {"case": case, "eng": eng}
    if kind == "run":
        s["host"] = _host_buffers(case, nx * ny * nz)
    return s


def _room(case):
    """Boundary cells that a host's lists have room for."""
    return 4 * int((case["nx"] * case["ny"] * case["nz"]) ** (2 / 3))


def _sweep(case):
    return [(n, n // 2, n // 2) for n in (case["nx"] + case["grow"] * k for k in range(case["count"]))]


# ---- one pass --------------------------------------------------------------------------


def _forces(f, precision):
    """The momentum-exchange sums, in the precision of the populations they are taken from."""
    t = torch.tensor([f.fx, f.fy, f.fz, f.mx, f.my, f.mz], dtype=torch.float64)
    return t if precision in ("f64", "f32_mirror") else t.float()


def _read(eng, host, precision):
    """Macro field (and populations, where the host keeps a buffer for them) into the host's buffers."""
    lib, h = N.load(), eng._h.h
    N.check(lib.aerosim_read_macro(h, *(_ptr(t, C.c_float) for t in host["macro"])), h)
    out = dict(zip(("ux", "uy", "uz", "rho"), host["macro"]))
    if "pops" in host:
        kind = N.DTYPE_F64 if host["pops"].dtype == torch.float64 else N.DTYPE_F32
        N.check(lib.aerosim_read_populations(h, C.c_void_p(host["pops"].data_ptr()), kind), h)
        out["f"] = host["pops"]
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "frame":
        r = state["eng"].step_and_extract_slice(case["steps"], read_macro_field=True,
                                                slice={"axis": "z", "fraction": 0.5, "mode": "velocity"})
        return {"forces": _forces(r["forces"], case["precision"]), "rgba": r["rgba"], "macro": r["macroField"]}
    if kind == "run":
        r = state["eng"].step_and_extract_slice(case["steps"])
        return {"forces": _forces(r["forces"], case["precision"]), "macro": _read(state["eng"], state["host"], case["precision"])}
    if kind == "batch":
        state["batch"].step(case["steps"])
        return [{"forces": _forces(e.read_forces(), case["precision"]), "macro": _read(e, h, case["precision"])}
                for e, h in zip(state["eng"], state["host"])]
    if kind == "diagnose":
        state["eng"].step(case["steps"])
        return state["eng"].q_criterion()
    if kind == "train":
        p, curve = sgs.train(state["params"], state["X"], state["Y"], iters=case["iters"], batch=case["batch"],
                             lr=2e-3, seed=state["seed"])
        return {"params": p, "curve": curve}
    cells, q, least = state["lists"]
    if state["eng"] is not None:  # into an engine that goes on to step; the grid into the host's buffers
        eng, (flags, bmap) = state["eng"], state["dense"]
        n = eng.voxelize(state["mesh"], state["world"], state["tunnel"], state["grid"]).boundary_cell_count
        assert n <= cells.numel()
        N.check(N.load().aerosim_read_voxel_grid(eng._h.h, _ptr(flags, C.c_uint8), _ptr(bmap, C.c_int32), _ptr(cells, C.c_int32),
                                                 _ptr(q, C.c_float), _ptr(least, C.c_float)), eng._h.h)
    else:
        v = voxelize_mesh_to_lattice(state["mesh"], state["world"], state["tunnel"], state["grid"])
        n, flags, bmap = v.boundaryCellCount, v.cellFlags, v.boundaryIndexMap
        for t, a in ((cells, v.boundaryCellIndices), (q, v.boundaryQValues), (least, v.boundaryMinQ)):
            t.numpy()[:a.size] = a
    return {"flags": flags, "map": bmap, "count": int(n), "cells": cells, "q": q, "min_q": least}


def work(case):
    kind = case["kind"]
    if kind == "train":
        rows = case["iters"] * case["batch"]
        return {"bytes": 36.0 * rows, "flops": 6.0 * (8 * 32 + 32 * 32 + 32) * rows}
    if kind == "batch":
        cells = sum(a * b * c for a, b, c in _sweep(case))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "voxelize":
        tris = 2 * case["segments"] * (case["rings"] - 1)
        # the grid written (flags, map); an engine's flow is reset with it, populations and macro field
        return {"bytes": 5.0 * cells + 36.0 * tris + (19 * 4 + 16.0) * cells, "flops": 50.0 * tris}
    per_step = (38.0 * ELEM[case["precision"]], 280.0 + (6000.0 if case.get("closure") else 0.0))
    read = {"frame": 16, "run": 16, "batch": 16, "diagnose": 20 + 12}[kind]
    if kind == "run" and case["precision"] in ("f32_mirror", "f64"):
        read += 19 * ELEM[case["precision"]]
    return {"bytes": cells * (case["steps"] * per_step[0] + 2.0 * read), "flops": cells * case["steps"] * per_step[1]}


# ---- the same in 64 bits, in plain torch -------------------------------------------------


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _network(p, x):
    w1, b1, w2, b2, w3, b3 = torch.split(p, [256, 32, 1024, 32, 32, 1])
    h = _gelu(x @ w1.reshape(32, 8).T + b1)
    h = _gelu(h @ w2.reshape(32, 32).T + b2)
    return torch.nn.functional.softplus(h @ w3 + b3)


class _Flow:
    """D3Q19 regularized BGK with Smagorinsky (or the closure's) viscosity, Bouzidi walls, inlet, outlet,
    slip walls and the mean-density rescale, in 64 bits."""

    def __init__(self, grid, cfg, f, closure=None):
        self.n = (grid.nz, grid.ny, grid.nx)
        self.cfg, self.grid, self.step_index = cfg, grid, 0
        self.f = f.double()
        self.flags = torch.from_numpy(grid.cellFlags).to(DEV).reshape(self.n)
        self.solid = self.flags == 1
        self.closure = None if closure is None else torch.tensor(closure, dtype=torch.float64, device=DEV)
        nz, ny, nx = self.n
        q = torch.from_numpy(grid.boundaryQValues).to(DEV).reshape(-1, 18).double()
        bmap = torch.from_numpy(grid.boundaryIndexMap).to(DEV).long()
        self.links, near = {}, torch.zeros(self.n, dtype=torch.bool, device=DEV)
        flat = self.solid.reshape(-1)
        for d in range(1, 19):
            hit = self._pull(self.solid, VEL[d]) & ~self.solid
            near |= hit
            c = torch.nonzero(hit.reshape(-1)).reshape(-1)
            qq = torch.where(bmap[c] >= 0, q[bmap[c].clamp(min=0), OPP[d] - 1], torch.full_like(c, 0.5, dtype=torch.float64))
            qq = torch.where(qq > 0, qq, torch.full_like(qq, 0.5))
            x, y, z = c % nx, c // nx % ny, c // (nx * ny)
            ff = (x + VEL[d][0]).clamp(0, nx - 1) + nx * ((y + VEL[d][1]).clamp(0, ny - 1) + ny * (z + VEL[d][2]).clamp(0, nz - 1))
            self.links[d] = (c, ff, qq, flat[ff])
        self.near = near
        if self.closure is not None:
            self.wall = self._wall_distance()

    def _wall_distance(self):
        """Cells to the nearest solid cell centre, rounded, at most 31, as the closure's input holds it."""
        pts = torch.nonzero(self.solid & ~(self._pull(self.solid, (1, 0, 0)) & self._pull(self.solid, (-1, 0, 0))
                                           & self._pull(self.solid, (0, 1, 0)) & self._pull(self.solid, (0, -1, 0))
                                           & self._pull(self.solid, (0, 0, 1)) & self._pull(self.solid, (0, 0, -1)))).float()
        d2 = torch.full(self.n, 31.0 ** 2, device=DEV)
        lo = (pts.amin(0).long() - 32).clamp(min=0).tolist()
        hi = (pts.amax(0).long() + 33).tolist()
        box = tuple(slice(a, min(b, n)) for a, b, n in zip(lo, hi, self.n))
        cells = torch.stack(torch.meshgrid(*(torch.arange(s.start, s.stop, device=DEV).float() for s in box), indexing="ij"), -1)
        shape = cells.shape[:3]
        cells = cells.reshape(-1, 3)
        best = torch.cat([torch.cdist(part, pts, compute_mode="donot_use_mm_for_euclid_dist").amin(1) for part in cells.split(16384)])
        d2[box] = best.reshape(shape).clamp(max=31.0)
        d2[d2 > 31.0] = 31.0
        return torch.where(self.solid, torch.zeros_like(d2), torch.round(d2)).double()

    def _pull(self, a, v):
        """a at clamp(cell - v)."""
        for dim, c in ((2, v[0]), (1, v[1]), (0, v[2])):
            if c:
                n = a.shape[dim]
                i = (torch.arange(n, device=DEV) - c).clamp(0, n - 1)
                a = a.index_select(dim, i)
        return a

    def _relaxation(self, rho, pxx, pyy, pzz, pxy, pxz, pyz):
        tau0, pn = 3.0 * self.cfg["nuLattice"] + 0.5, torch.sqrt(pxx ** 2 + pyy ** 2 + pzz ** 2 + 2 * (pxy ** 2 + pxz ** 2 + pyz ** 2))
        tau = 0.5 * (tau0 + torch.sqrt(tau0 ** 2 + 18.0 * math.sqrt(2.0) * self.cfg["smagorinskyCs"] ** 2 * pn / rho))
        if self.closure is not None:  # near-wall cells keep Smagorinsky
            k = -150.0 / (rho * tau)
            x = torch.stack([k * p for p in (pxx, pyy, pzz, pxy, pxz, pyz)] + [100.0 * (rho - 1.0), self.wall / 16.0], -1)
            nu0 = (max(tau0, 0.5015) - 0.5) / 3.0
            ratio = torch.cat([_network(self.closure, part) for part in x.reshape(-1, 8).split(1 << 20)]).reshape(rho.shape)
            tau = torch.where(self.near, tau, 3.0 * nu0 * (1.0 + ratio) + 0.5)
        return 1.0 / tau.clamp(0.5015, 1.95)

    def step(self):
        nz, ny, nx = self.n
        v = torch.empty_like(self.f)
        src = self.f.reshape(19, -1)
        for d in range(19):
            v[d] = self._pull(self.f[d], VEL[d])
            if d:
                c, ff, q, blocked = self.links[d]
                w = src[OPP[d]]
                lin = torch.where(q < 0.5, 2 * q * w[c] + (1 - 2 * q) * w[ff], w[c] / (2 * q) + (1 - 1 / (2 * q)) * src[d][c])
                v[d].reshape(-1)[c] = torch.where(blocked, w[c], lin)
        mom = [sum(VEL[d][a] * v[d] for d in range(19) if VEL[d][a]) for a in range(3)]
        rho = v.sum(0).clamp(0.5, 1.8)
        u = [m / rho for m in mom]
        sp = torch.sqrt(u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        lim = torch.where(sp > 0.22, 0.22 / sp.clamp(min=1e-30), torch.ones_like(sp))
        u = [a * lim for a in u]
        sq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        p = {k: 0.0 for k in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))}
        for d in range(19):
            cu = 3.0 * sum(VEL[d][a] * u[a] for a in range(3))
            eq = W32[d] * rho * (1.0 + cu + 0.5 * cu * cu - 1.5 * sq)
            fn = v[d] - eq
            for a, b in p:
                if VEL[d][a] * VEL[d][b]:
                    p[a, b] = p[a, b] + VEL[d][a] * VEL[d][b] * fn
            v[d] = eq
        om = self._relaxation(rho, *(p[k] for k in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))))
        tr = (p[0, 0] + p[1, 1] + p[2, 2]) / 3.0
        for d in range(19):
            cpc = sum((1 if a == b else 2) * VEL[d][a] * VEL[d][b] * t for (a, b), t in p.items() if VEL[d][a] * VEL[d][b])
            v[d] += (1.0 - om) * 4.5 * W32[d] * (cpc - tr)
        self._boundaries(v, rho, u)
        mean = rho[~self.solid].mean()
        if abs(float(mean) - 1.0) > 1e-4:
            open_ = ~self.solid
            rho = torch.where(open_, rho / mean, rho)
            v = torch.where(open_, v / mean, v)
        keep = self.solid
        for d in range(19):
            v[d][keep] = self.f[d][keep]
        for a in u:
            a[keep] = 0.0
        rho[keep] = 1.0
        self.f, self.u, self.rho = v, u, rho
        self.step_index += 1

    def _boundaries(self, v, rho, u):
        nz, ny, nx = self.n
        u_in, ground = self.cfg["uInletLattice"], self.cfg["groundNoSlip"]
        y = torch.arange(ny, device=DEV, dtype=torch.float64)
        ux = torch.full_like(y, u_in)
        if ground:
            ux = u_in * torch.clamp(0.35 + 0.8 * ((y + 0.5) / ny) ** 0.3, max=1.15)
        uy = torch.zeros_like(y)
        if self.step_index < 120:
            uy = 0.015 * u_in * torch.sin(self.step_index * 0.15 + y / ny * math.pi * 2.0)
        ux, uy = ux.expand(nz, ny), uy.expand(nz, ny)
        at1 = torch.where(self.solid[..., 1], torch.ones_like(ux), rho[..., 1])
        s2 = self.solid[..., nx - 2]
        at2 = [torch.where(s2, torch.full_like(ux, fill), t[..., nx - 2]) for t, fill in ((rho, 1.0), (u[0], 0.0), (u[1], 0.0), (u[2], 0.0))]
        ins, outs = ~self.solid[..., 0], ~self.solid[..., nx - 1]
        r_in, r_out = 0.85 * at1 + 0.15, 0.85 * at2[0] + 0.15
        zero = torch.zeros_like(ux)
        for d, (e, o) in enumerate(zip(_equilibrium(r_in, [ux, uy, zero]), _equilibrium(r_out, at2[1:]))):
            prev = torch.where(s2, self.f[d][..., nx - 2], v[d][..., nx - 2])
            v[d][..., 0] = torch.where(ins, e, v[d][..., 0])
            v[d][..., nx - 1] = torch.where(outs, 0.75 * prev + 0.25 * o, v[d][..., nx - 1])
        for t, a, b in ((rho, r_in, r_out), (u[0], ux, at2[1]), (u[1], uy, at2[2]), (u[2], zero, at2[3])):
            t[..., 0], t[..., nx - 1] = torch.where(ins, a, t[..., 0]), torch.where(outs, b, t[..., nx - 1])
        walls = [((slice(None), 0), (0, 1, 2) if ground else (1,)), ((slice(None), ny - 1), (1,))]
        if nz > 4:
            walls += [((0,), (2,)), ((nz - 1,), (2,))]
        for where, still in walls:
            sel = where + (Ellipsis, slice(1, nx - 1))
            free = self.flags[sel] == 0
            for a in still:
                u[a][sel] = torch.where(free, torch.zeros_like(u[a][sel]), u[a][sel])
            for d, e in enumerate(_equilibrium(rho[sel], [a[sel] for a in u])):
                v[d][sel] = torch.where(free, e, v[d][sel])

    def forces(self):
        nz, ny, nx = self.n
        g, f = self.grid, self.f.reshape(19, -1)
        c = torch.from_numpy(g.boundaryCellIndices).to(DEV).long()
        q = torch.from_numpy(g.boundaryQValues).to(DEV).reshape(-1, 18).double()
        x = torch.stack([c % nx, c // nx % ny, c // (nx * ny)], -1)
        total, flat = torch.zeros(c.numel(), 3, dtype=torch.float64, device=DEV), self.solid.reshape(-1)
        for d in range(1, 19):
            a, b, e = VEL[OPP[d]]
            ff = (x[:, 0] + a).clamp(0, nx - 1) + nx * ((x[:, 1] + b).clamp(0, ny - 1) + ny * (x[:, 2] + e).clamp(0, nz - 1))
            qq = q[:, d - 1]
            fo, s = f[d][c], qq.clamp(min=1e-4)
            fi = torch.where(qq < 0.5, 2 * s * fo + (1 - 2 * s) * f[d][ff], fo / (2 * s) + (1 - 1 / (2 * s)) * f[OPP[d]][c])
            m = fo + torch.where(flat[ff], fo, fi) - 2.0 * W32[d]
            total += torch.where(qq > 0, m, torch.zeros_like(m))[:, None] * torch.tensor(VEL[d], dtype=torch.float64, device=DEV)
        arm = x.double() + 0.5 - 0.5 * torch.tensor([nx, ny, nz], dtype=torch.float64, device=DEV)
        return torch.cat([total.sum(0), torch.linalg.cross(arm, total).sum(0)]).cpu()


def _exact_flow(case, seed, nx, ny, nz):
    grid = _grid(nx, ny, nz, seed)
    cfg = _config(case, seed, nx, ny, nz)
    f = _restart(grid, cfg["uInletLattice"], seed)
    flow = _Flow(grid, cfg, f, np.load(CLOSURE)["params"] if case.get("closure") else None)
    del f
    for _ in range(case["steps"]):
        flow.step()
    return flow


def _exact_fields(flow, populations):
    out = dict(zip(("ux", "uy", "uz", "rho"), (t.reshape(-1) for t in (*flow.u, flow.rho))))
    if populations:
        out["f"] = flow.f.reshape(-1)
    return out


def _exact_vortices(flow):
    solid = flow.solid

    def slope(a, dim):
        n = a.shape[dim]
        i = torch.arange(n, device=DEV)
        lo, hi = (i - 1).clamp(min=0), (i + 1).clamp(max=n - 1)
        shape = [1, 1, 1]
        shape[dim] = n
        return (a.index_select(dim, hi) - a.index_select(dim, lo)) / (hi - lo).double().reshape(shape)

    g = [[slope(a, 2 - k) for k in range(3)] for a in flow.u]
    sym = sum((0.5 * (g[a][b] + g[b][a])) ** 2 for a in range(3) for b in range(3))
    asym = sum((0.5 * (g[a][b] - g[b][a])) ** 2 for a in range(3) for b in range(3))
    w = torch.stack([g[2][1] - g[1][2], g[0][2] - g[2][0], g[1][0] - g[0][1]], -1)
    q, m = 0.5 * (asym - sym), w.norm(dim=-1)
    q, m, w = (torch.where(solid.reshape(solid.shape + (1,) * (t.dim() - 3)), torch.zeros_like(t), t) for t in (q, m, w))
    return {"qValues": q.reshape(-1), "omegaMag": m.reshape(-1), "omegaVec": w.reshape(-1), "maxQ": max(1e-6, float(q.max())),
            "maxOmega": max(1e-6, float(m.max()))}


def _exact_training(case, seed):
    X, Y = (torch.tensor(a, dtype=torch.float64, device=DEV) for a in _rows(case, seed))
    p = torch.tensor(sgs.init_params(seed), dtype=torch.float64, device=DEV, requires_grad=True)
    opt = torch.optim.Adam([p], lr=float(np.float32(2e-3)), betas=(0.9, 0.999), eps=1e-8)
    curve = []
    for it in range(case["iters"]):
        with np.errstate(over="ignore"):  # the mini-batch's rows: a splitmix64 hash
            i = np.arange(case["batch"], dtype=np.uint64) + np.uint64(it * 1000003 + 1)
            z = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * i
            z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
            z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
            z ^= z >> np.uint64(31)
        rows = torch.from_numpy((z % np.uint64(case["rows"])).astype(np.int64)).to(DEV)
        loss = ((_network(p, X[rows]) - Y[rows]) ** 2).mean()
        opt.zero_grad()
        loss.backward()
        opt.step()
        curve.append(loss.detach())
    return {"params": p.detach(), "curve": torch.stack(curve)}


def _exact_links(case, seed):
    """Link fractions of the mesh by testing every triangle."""
    (pos, idx), world, _ = _mesh(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    m = torch.tensor(world.reshape(4, 4).T, device=DEV)
    p = torch.tensor(pos.astype(np.float64), device=DEV)
    p = p @ m[:3, :3].T + m[:3, 3]
    tri = p[torch.tensor(idx.astype(np.int64), device=DEV)]
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    axis = [torch.arange(n, device=DEV, dtype=torch.float64) + 0.5 - 0.5 * n for n in (nx, ny, nz)]
    solid = torch.zeros(nz, ny, nx, dtype=torch.bool, device=DEV)
    det = -e1[:, 1] * e2[:, 2] + e1[:, 2] * e2[:, 1]
    ok = det.abs() >= 1e-13
    for k in range(nz):  # scanlines along x, a hair off the cell centres
        ty, tz = axis[1][:, None] + 1.37e-8 - a[:, 1], axis[2][k] + 2.93e-8 - a[:, 2]
        u = (-ty * e2[:, 2] + tz * e2[:, 1]) / det
        v = (ty * e1[:, 2] - tz * e1[:, 1]) / det
        hit = ok & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1)
        if not bool(hit.any()):
            continue
        x = a[:, 0] + u * e1[:, 0] + v * e2[:, 0]
        if bool((hit.sum(1) % 2).any()):
            return None
        for j in torch.nonzero(hit.any(1)).reshape(-1).tolist():
            cross = x[j][hit[j]].sort().values
            solid[k, j] = (torch.searchsorted(cross, axis[0]) % 2) == 1
    flags = solid.to(torch.uint8)
    link = torch.stack([_shifted(solid, VEL[d], False) & ~solid for d in range(1, 19)])
    cells = torch.nonzero(link.any(0).reshape(-1)).reshape(-1)
    q = torch.full((cells.numel(), 18), -1.0, dtype=torch.float64, device=DEV)
    at = torch.stack([axis[0][cells % nx], axis[1][cells // nx % ny], axis[2][cells // (nx * ny)]], -1)
    for d in range(1, 19):
        has = torch.nonzero(link[d - 1].reshape(-1)[cells]).reshape(-1)
        v = torch.tensor(VEL[d], dtype=torch.float64, device=DEV)
        pv = torch.linalg.cross(v.expand_as(e2), e2)
        dt = (e1 * pv).sum(-1)
        good = dt.abs() >= 1e-13
        for part in has.split(2000):
            t0 = at[part][:, None] - a
            uu = (t0 * pv).sum(-1) / dt
            qv = torch.linalg.cross(t0, e1.expand_as(t0))
            vv = (qv @ v) / dt
            t = (qv * e2).sum(-1) / dt
            hit = good & (uu >= -1e-7) & (uu <= 1 + 1e-7) & (vv >= -1e-7) & (uu + vv <= 1 + 1e-7) & (t > 1e-7) & (t <= 1 + 1e-7)
            t = torch.where(hit, t, torch.full_like(t, math.inf)).amin(1)
            q[part, d - 1] = torch.where(torch.isinf(t), torch.full_like(t, 0.5), t.clamp(1e-4, 1.0))
    least = torch.where(q > 0, q, torch.ones_like(q)).amin(1)
    room = _room(case)
    return {"flags": None, "map": None, "count": None, "cells": None,
            "q": torch.nn.functional.pad(q.reshape(-1), (0, 18 * room - q.numel())),
            "min_q": torch.nn.functional.pad(least, (0, room - least.numel()))}


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_training(case, seed)
    if kind == "voxelize":
        return _exact_links(case, seed)
    if kind == "batch":
        out = []
        for k, (nx, ny, nz) in enumerate(_sweep(case)):
            flow = _exact_flow(case, seed + 10 * k, nx, ny, nz)
            out.append({"forces": flow.forces(), "macro": {n: t.cpu() for n, t in _exact_fields(flow, False).items()}})
        return out
    flow = _exact_flow(case, seed, case["nx"], case["ny"], case["nz"])
    if kind == "diagnose":
        return _exact_vortices(flow)
    fields = _exact_fields(flow, kind == "run" and case["precision"] in ("f32_mirror", "f64"))
    return {"forces": flow.forces(), **({"rgba": None} if kind == "frame" else {}), "macro": fields}
