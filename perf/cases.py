"""Performance cases of the framework, through its public entry points.

Every case is a dict of plain values; `prepare` makes what a program holds
before the call, `run` makes one pass, `work` states what the pass cannot do
without and `exact` gives the 64-bit result where there is one.

Kinds:
  step    the coupled SPH + height-field step: the host owns the state, so a
          pass uploads every scene's particle records and height fields from
          page-locked memory, advances `steps` steps and hands on the sim's
          device buffers.
  passes  grid, density and force of one state, one pass at a time.
  wave    the wave module stepped alone (cwa_wave_advance).
  frame   one rendered frame into host memory.
  sph2d   the 2D solver family: upload, `frames` frames, read back.
  pbd     position-based boxes: upload, `frames` frames, read back.
  points  the stand-alone uniform-grid build on device buffers.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from coupledwateranimation_gb300 import Sim, _abi, scenes
from coupledwateranimation_gb300._abi import PARTICLE_DTYPE, PBD_BOX_DTYPE, PREC_COMPENSATED, PREC_FP32, PREC_FP64
from coupledwateranimation_gb300.pbd import PbdSim, make_boxes, pbd_defaults
from coupledwateranimation_gb300.sim import render_defaults
from coupledwateranimation_gb300.sim2d import Sim2D, defaults2d


def _dam(name, lattice, spacing, wave, steps, zsub, precision=PREC_COMPENSATED, kind="step", box_x=1.0):
    return {"name": name, "kind": kind, "nx": lattice[0], "ny": lattice[1], "nz": lattice[2], "spacing": spacing,
            "wave_x": wave[0], "wave_z": wave[1], "steps": steps, "zsub": zsub, "precision": precision,
            "box_x": box_x}


def listed():
    return [
        # the reference app's own scene, a few display frames' worth of steps: small launches, latency counts
        {"name": "step_reference_20k", "kind": "reference", "wave_x": 64, "wave_z": 64, "steps": 16},
        # the small dam break (32^3 particles, 256^2 field)
        _dam("step_dam_32k", (32, 32, 32), 0.02, (256, 256), 16, 1),
        # the benchmark's scene: 1,048,576 particles, 1024^2 field, sort cells h x h x h/4
        _dam("step_dam_1m", (128, 64, 128), 0.0075, (1024, 1024), 10, 4),
        # the largest single scene (4,194,304 particles, 2048^2 field), plain float sums
        _dam("step_dam_4m_fp32", (256, 128, 128), 0.004, (2048, 2048), 4, 4, PREC_FP32, box_x=1.024),
        # many independent scenes of mixed sizes in one sim
        {"name": "step_batch_64", "kind": "batch", "scenes": 64, "n_lo": 2048, "n_hi": 65536, "steps": 8, "zsub": 4},
        # density and force in double on a ragged lattice with moving particles
        _dam("passes_fp64_67k", (41, 37, 45), 0.015, (333, 217), 1, 2, PREC_FP64, "passes"),
        # the wave module alone on a large field, and on a small field of odd width
        {"name": "wave_4096", "kind": "wave", "wave_x": 4096, "wave_z": 4096, "steps": 32},
        {"name": "wave_773x1021", "kind": "wave", "wave_x": 773, "wave_z": 1021, "steps": 29},
        # a full-HD frame of the 1M-particle scene
        {"name": "frame_1080p_1m", "kind": "frame", "nx": 128, "ny": 64, "nz": 128, "spacing": 0.0075,
         "wave_x": 1024, "wave_z": 1024, "width": 1920, "height": 1080},
        # the 2D app's scene and the box demo's scene, several frames between host accesses
        {"name": "sph2d_4096", "kind": "sph2d", "particles": 4096, "wave_kind": 0, "frames": 16},
        {"name": "pbd_4096", "kind": "pbd", "boxes": 4096, "cells": 16, "frames": 8},
        # the uniform grid of a million scattered points
        {"name": "points_1m", "kind": "points", "points": 1000003, "cells_x": 63, "cells_y": 64, "cells_z": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lattice(rng, n_lo, n_hi):
    """A lattice of roughly log-uniform size with uneven sides, and a spacing that fits it into the unit box."""
    n = math.exp(rng.uniform(math.log(n_lo), math.log(n_hi)))
    a, b = rng.uniform(0.5, 1.0), rng.uniform(0.6, 1.0)
    side = (n / (a * b)) ** (1.0 / 3.0)
    dims = [max(4, int(side)), max(4, int(a * side)), max(4, int(b * side))]
    return dims, rng.uniform(0.6, 0.98) / max(dims)


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "reference", "batch", "passes", "passes", "wave", "wave",
                       "frame", "sph2d", "pbd", "points"])
    if kind in ("step", "passes"):
        dims, s = _lattice(rng, 20000, 2000000 if kind == "step" else 90000)
        w = (_log_int(rng, 64, 1536), _log_int(rng, 64, 1536))
        if rng.random() < 0.6:
            w = (w[0] & ~3, w[1] & ~3)
        c = _dam("", dims, s, w, rng.randint(2, 10) if kind == "step" else 1, rng.choice([1, 2, 4]),
                 rng.choice([PREC_FP32, PREC_COMPENSATED, PREC_COMPENSATED] + [PREC_FP64] * (kind == "passes")), kind)
        del c["name"]
        return c
    if kind == "reference":
        return {"kind": kind, "wave_x": _log_int(rng, 32, 512), "wave_z": _log_int(rng, 32, 512),
                "steps": rng.randint(4, 24)}
    if kind == "batch":
        lo = _log_int(rng, 1024, 8192)
        return {"kind": kind, "scenes": rng.randint(8, 96), "n_lo": lo, "n_hi": lo * rng.randint(2, 8),
                "steps": rng.randint(4, 10), "zsub": rng.choice([1, 4])}
    if kind == "wave":
        w = _log_int(rng, 128, 4096)
        return {"kind": kind, "wave_x": w & ~3 if rng.random() < 0.5 else w, "wave_z": _log_int(rng, 128, 4096),
                "steps": rng.randint(9, 32)}
    if kind == "frame":
        dims, s = _lattice(rng, 20000, 700000)
        return {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "spacing": s, "wave_x": 256,
                "wave_z": _log_int(rng, 64, 512), "width": rng.randint(320, 1920), "height": rng.randint(240, 1080)}
    if kind == "sph2d":
        return {"kind": kind, "particles": 128 * rng.randint(12, 36), "wave_kind": rng.randint(0, 1),
                "frames": rng.randint(4, 24)}
    if kind == "pbd":
        n = _log_int(rng, 500, 20000)  # about as crowded as the demo's 4096 boxes in 16^3 cells
        return {"kind": kind, "boxes": n, "cells": round(16 * (n / 4096) ** (1 / 3) * rng.uniform(0.95, 1.3)),
                "frames": rng.randint(2, 12)}
    return {"kind": kind, "points": _log_int(rng, 10000, 2000000), "cells_x": rng.randint(8, 100),
            "cells_y": rng.randint(8, 100), "cells_z": rng.randint(8, 100)}


class _Device:
    """Device memory of the library as __cuda_array_interface__; it keeps the sim that owns the memory alive for as
    long as a tensor over it lives."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3,
                                         "strides": None}


def _views(state, scene):
    """The scene's live device buffers as tensors (made once per buffer, as the pointers alternate)."""
    sim, made = state["sim"], state["views"]
    v = sim.device_view(scene)
    n, out = v.n_particles, {}
    want = [("u_n", v.wave_u_n, (v.wave_nz, v.wave_nx), "<f4"), ("u_nm1", v.wave_u_nm1, (v.wave_nz, v.wave_nx), "<f4")]
    if n:
        want += [("pos", v.pos, (n, 4), "<f4"), ("vel", v.vel, (n, 4), "<f4"), ("force", v.force, (n, 4), "<f4"),
                 ("rho_p", v.rho_p, (n, 2), "<f4"), ("id", v.particle_id, (n,), "<i4")]
    for name, ptr, shape, kind in want:
        key = (ptr, shape)
        if key not in made:
            made[key] = torch.as_tensor(_Device(sim, ptr, shape, kind), device="cuda")
        out[name] = made[key]
    return out


def _pinned(array):
    """A page-locked copy of a host array, and its numpy view of the same type."""
    t = torch.empty(array.nbytes, dtype=torch.uint8, pin_memory=True)
    v = t.numpy().view(array.dtype).reshape(array.shape)
    v[...] = array
    return t, v


def _dam_scene(case, seed):
    return scenes.dam_break((case["nx"], case["ny"], case["nz"]), case["spacing"], (case["wave_x"], case["wave_z"]),
                            box_hi=(case.get("box_x", 1.0), 1.0, 1.0), seed=seed, zsub=case.get("zsub", 1))


def _moving(scene, seed):
    """The scene's particles with velocities, as in a flow."""
    rng = np.random.default_rng(seed)
    scene.particles["vel"][:, :3] = rng.uniform(-0.5, 0.5, (len(scene.particles), 3)).astype(np.float32)
    return scene


def _batch_sizes(case, seed):
    rng = np.random.default_rng(case["scenes"])  # the sizes belong to the case, the jitter and waves to the seed
    out = []
    for k in range(case["scenes"]):
        target = float(np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"]))))
        aspect, fill = float(rng.uniform(0.5, 2.0)), float(rng.uniform(0.2, 0.5))
        w = int((64, 128, 256, 512)[rng.integers(4)])
        block = np.array([aspect, 1.0, 1.0]) * fill ** (1.0 / 3.0)
        s = float((np.prod(block) / target) ** (1.0 / 3.0))
        dims = tuple(int(x) for x in np.maximum(1, np.round(block / s)).astype(int))
        out.append((dims, s, w, aspect))
    return out


def _scenes(case, seed):
    if case["kind"] == "reference":
        s = scenes.reference()
        scenes.set_wave_grid(s.desc, case["wave_x"], case["wave_z"])
        rng = np.random.default_rng(seed)
        s.particles["pos"][:, :3] += rng.uniform(-5e-4, 5e-4, (len(s.particles), 3)).astype(np.float32)
        z, x = np.mgrid[0:case["wave_z"], 0:case["wave_x"]].astype(np.float32)
        c = rng.uniform(0.2, 0.8, 2)
        s.wave = (0.5 * np.exp(-((x / case["wave_x"] - c[0]) ** 2 + (z / case["wave_z"] - c[1]) ** 2) / 0.01)).astype(
            np.float32)
        return [s]
    if case["kind"] == "batch":
        return [scenes.dam_break(d, s, (w, w), box_hi=(a, 1.0, 1.0), seed=seed + k, zsub=case["zsub"])
                for k, (d, s, w, a) in enumerate(_batch_sizes(case, seed))]
    return [_dam_scene(case, seed)]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "reference", "batch"):
        made = _scenes(case, seed)
        sim = Sim([s.desc for s in made], precision=case.get("precision", PREC_COMPENSATED))
        host = [(_pinned(s.particles), _pinned(s.wave)) for s in made]
        return {"kind": "step", "sim": sim, "host": host, "steps": case["steps"], "views": {},
                "stream": torch.cuda.ExternalStream(sim.device_view(0).stream)}
    if kind == "passes":
        s = _moving(_dam_scene(case, seed), seed)
        sim = Sim(s.desc, precision=case["precision"])
        sim.upload_particles(0, s.particles)
        sim.upload_wave(0, s.wave)
        return {"kind": kind, "sim": sim, "views": {}}
    if kind == "wave":
        d = scenes.defaults(_abi.PRESET_MULLER, 0.05)
        scenes.set_wave_grid(d, case["wave_x"], case["wave_z"])
        d.n_particles = 0
        u = _wave_field(case, seed)
        sim = Sim(d)
        sim.upload_wave(0, u)
        return {"kind": kind, "sim": sim, "steps": case["steps"], "views": {}}
    if kind == "frame":
        s = _dam_scene(case, seed)
        sim = Sim(s.desc)
        sim.upload_particles(0, s.particles)
        sim.upload_wave(0, s.wave)
        sim.step(2)
        sim.synchronize()
        cam, prm = render_defaults(case["width"], case["height"])
        image = _pinned(np.zeros((case["height"], case["width"], 4), np.uint8))
        return {"kind": kind, "sim": sim, "cam": cam, "prm": prm, "image": image}
    if kind == "sph2d":
        p = defaults2d(case["wave_kind"])
        p.n_particles = case["particles"]
        sim = Sim2D(p)
        parts = sim.download_particles()
        rng = np.random.default_rng(seed)
        parts["pos"][:, :2] += rng.uniform(-0.005, 0.005, (len(parts), 2)).astype(np.float32)
        parts["vel"][:, :2] = rng.uniform(-0.1, 0.1, (len(parts), 2)).astype(np.float32)
        return {"kind": kind, "sim": sim, "parts": parts, "wave": sim.download_wave(), "frames": case["frames"]}
    if kind == "pbd":
        p = pbd_defaults()
        p.n_boxes = case["boxes"]
        for a in range(3):
            p.grid_cells[a] = case["cells"]
        return {"kind": kind, "sim": PbdSim(p), "boxes": make_boxes(p, seed), "frames": case["frames"]}
    n, dims = case["points"], (case["cells_x"], case["cells_y"], case["cells_z"])
    nc = dims[0] * dims[1] * dims[2]
    lib = _abi.load()
    size = lib.cwa_grid_workspace_bytes(n, nc)
    return {"kind": kind, "n": n, "cell": _cell_edge(case), "lo": (C.c_float * 3)(0.0, 0.0, 0.0),
            "dims": (C.c_int32 * 3)(*dims), "pos": _points(case, seed), "workspace": torch.empty(
                size, dtype=torch.uint8, device="cuda"), "start": torch.empty(nc + 1, dtype=torch.int32, device="cuda"),
            "index": torch.empty(n, dtype=torch.int32, device="cuda"),
            "cell_of": torch.empty(n, dtype=torch.int32, device="cuda")}


def _wave_field(case, seed):
    rng = np.random.default_rng(seed)
    x = np.linspace(0.0, 1.0, case["wave_x"], dtype=np.float32)
    z = np.linspace(0.0, 1.0, case["wave_z"], dtype=np.float32)
    a, s = rng.uniform(0.01, 0.05, 8).astype(np.float32), rng.uniform(0.02, 0.1, 8).astype(np.float32)
    cx, cz = rng.uniform(size=8).astype(np.float32), rng.uniform(size=8).astype(np.float32)
    along_x = a[:, None] * np.exp(-((x - cx[:, None]) / s[:, None]) ** 2)
    return np.ascontiguousarray(np.exp(-((z - cz[:, None]) / s[:, None]) ** 2).T @ along_x)  # eight bumps


def _cell_edge(case):
    return 1.0 / max(case["cells_x"], case["cells_y"], case["cells_z"])


def _points(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    p = torch.rand(case["points"], 4, generator=g, device="cuda")
    edge = _cell_edge(case)
    return p * torch.tensor([case["cells_x"] * edge, case["cells_y"] * edge, case["cells_z"] * edge, 1.0],
                            device="cuda") * 1.02 - 0.01


def run(state):
    kind = state["kind"]
    if kind == "step":
        sim = state["sim"]
        for k, ((_, records), (_, field)) in enumerate(state["host"]):
            sim.upload_particles(k, records)
            sim.upload_wave(k, field)
        sim.step(state["steps"])
        if len(state["host"]) == 1:
            return _views(state, 0)
        # every scene's result in one tensor of each kind
        every = [_views(state, k) for k in range(len(state["host"]))]
        mine = torch.cuda.current_stream()
        mine.wait_stream(state["stream"])
        out = {name: torch.cat([v[name].reshape(-1) for v in every]) for name in ("pos", "vel", "id", "u_n")}
        state["stream"].wait_stream(mine)  # the next pass writes those buffers again
        return out
    if kind == "passes":
        sim = state["sim"]
        sim.grid()
        sim.rho_pres()
        sim.force()
        v = _views(state, 0)
        return {"pos": v["pos"], "rho_p": v["rho_p"], "force": v["force"], "id": v["id"]}
    if kind == "wave":
        state["sim"].wave_advance(state["steps"])
        return _views(state, 0)
    if kind == "frame":
        sim, image = state["sim"], state["image"][1]
        _abi.check(_abi.load().cwa_render(sim.handle, 0, C.byref(state["cam"]), C.byref(state["prm"]),
                                          image.ctypes.data), "cwa_render")
        return image
    if kind == "sph2d":
        sim = state["sim"]
        sim.upload_particles(state["parts"])
        sim.upload_wave(state["wave"])
        sim.step(state["frames"])
        parts = sim.download_particles()
        return {"pos": parts["pos"], "vel": parts["vel"], "acc": parts["acc"], "wave": sim.download_wave()}
    if kind == "pbd":
        sim = state["sim"]
        sim.upload(state["boxes"])
        sim.step(state["frames"])
        out = sim.download()
        return out.view(np.float32).reshape(len(out), PBD_BOX_DTYPE.itemsize // 4)
    _abi.check(_abi.load().cwa_grid_build(
        _abi.ptr(state["pos"]), state["n"], state["lo"], state["cell"], state["dims"], _abi.ptr(state["start"]),
        _abi.ptr(state["index"]), _abi.ptr(state["cell_of"]), _abi.ptr(state["workspace"]), state["workspace"].numel(),
        C.c_void_p(torch.cuda.current_stream().cuda_stream)), "cwa_grid_build")
    return {"start": state["start"], "index": state["index"], "cell_of": state["cell_of"]}


_NEIGHBOURS = 33  # lattice points within h = 2 s of a particle
_STEP_BYTES = 96  # pos, vel, id read; pos, vel, force, (rho, p), id written
_STEP_FLOPS = _NEIGHBOURS * 50 + 60


def work(case):
    kind = case["kind"]
    if kind in ("step", "reference", "batch"):
        if kind == "step":
            n, w = case["nx"] * case["ny"] * case["nz"], case["wave_x"] * case["wave_z"]
        elif kind == "reference":
            n, w = 20480, case["wave_x"] * case["wave_z"]
        else:
            sizes = _batch_sizes(case, 0)
            n, w = sum(int(np.prod(d)) for d, _, _, _ in sizes), sum(x * x for _, _, x, _ in sizes)
        return {"bytes": n * PARTICLE_DTYPE.itemsize + 4 * w + case["steps"] * (_STEP_BYTES * n + 12 * w),
                "flops": case["steps"] * (_STEP_FLOPS * n + 8 * w)}
    if kind == "passes":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": n * (36 + 24 + 36), "flops": n * _NEIGHBOURS * 50}
    if kind == "wave":
        w = case["wave_x"] * case["wave_z"]
        return {"bytes": 16 * w, "flops": 8 * w * case["steps"]}
    if kind == "frame":
        n, pixels = case["nx"] * case["ny"] * case["nz"], case["width"] * case["height"]
        return {"bytes": 20 * n + 4 * case["wave_x"] * case["wave_z"] + 4 * pixels, "flops": n * 45 * 100}
    if kind == "sph2d":
        n = case["particles"]
        return {"bytes": 96 * n * (1 + 2 * case["frames"]), "flops": n * 2 * case["frames"] * 50 * 40}
    if kind == "pbd":
        n = case["boxes"]
        return {"bytes": 2 * 128 * n * (1 + case["frames"]), "flops": n * case["frames"] * 12 * 80}
    nc = case["cells_x"] * case["cells_y"] * case["cells_z"]
    return {"bytes": (16 + 4 + 4) * case["points"] + 4 * (nc + 1), "flops": 0}


def _sorted_ids(pos, d):
    """Upload indexes in cell order: the float32 cell hash, then a stable sort."""
    dims = (C.c_int32 * 3)()
    _abi.check(_abi.load().cwa_grid_dims(C.byref(d), dims), "cwa_grid_dims")
    edge = (d.cell_size, d.cell_size, d.cell_size_z if d.cell_size_z > 0 else d.cell_size)
    key = torch.zeros(len(pos), dtype=torch.int64, device=pos.device)
    for a in range(3):
        t = (pos[:, a] - torch.tensor(d.box_lo[a], device=pos.device)) / torch.tensor(edge[a], device=pos.device)
        key = key * dims[a] + torch.clamp(torch.floor(t), 0, dims[a] - 1).to(torch.int64)
    return torch.sort(key, stable=True).indices


def _exact_passes(case, seed):
    s = _moving(_dam_scene(case, seed), seed)
    d = s.desc
    pos32 = torch.from_numpy(np.ascontiguousarray(s.particles["pos"])).cuda()
    vel32 = torch.from_numpy(np.ascontiguousarray(s.particles["vel"])).cuda()
    order = _sorted_ids(pos32, d)
    pos32, vel32 = pos32[order], vel32[order]
    x, v = pos32[:, :3].double(), vel32[:, :3].double()
    n, h, m = len(x), float(d.smoothing_length), float(d.mass)
    rho = torch.empty(n, dtype=torch.float64, device="cuda")
    block = max(1, 40_000_000 // n)

    def pairs(b):
        r2 = torch.zeros(len(x[b:b + block]), n, dtype=torch.float64, device="cuda")
        for a in range(3):
            r2 += (x[b:b + block, a, None] - x[None, :, a]) ** 2
        return r2

    for b in range(0, n, block):
        rho[b:b + block] = torch.clamp(h * h - pairs(b), min=0.0).pow(3).sum(1)
    rho *= m * 315.0 / (64.0 * math.pi * h ** 9)
    p = float(d.gas_const) * (rho - float(d.rest_rho))
    force = torch.zeros(n, 4, dtype=torch.float64, device="cuda")
    grad = 45.0 / (math.pi * h ** 6) * m
    for b in range(0, n, block):
        r = torch.sqrt(pairs(b))
        hr = torch.clamp(h - r, min=0.0)
        near = torch.where(r > 0, 1.0 / r, torch.zeros_like(r)) * hr * hr / rho
        press, visc = 0.5 * grad * near * (p[b:b + block, None] + p[None, :]), grad * float(d.visc) * hr / rho
        for a in range(3):
            f = press.sum(1) * x[b:b + block, a] - press @ x[:, a]
            f += visc @ v[:, a] - visc.sum(1) * v[b:b + block, a]
            force[b:b + block, a] = f + rho[b:b + block] * float(d.gravity[a])
    return {"pos": None, "rho_p": torch.stack([rho, p], 1), "force": force, "id": None}


def _exact_wave(case, seed):
    d = scenes.defaults(_abi.PRESET_MULLER, 0.05)
    scenes.set_wave_grid(d, case["wave_x"], case["wave_z"])
    u = torch.from_numpy(_wave_field(case, seed)).cuda().double()
    prev, lam, beta, atten = u.clone(), float(d.wave_lambda), float(d.wave_beta), float(d.wave_atten)
    for _ in range(case["steps"]):
        q = torch.nn.functional.pad(u[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
        ring = q[2:, 1:-1] + q[:-2, 1:-1] + q[1:-1, 2:] + q[1:-1, :-2]
        u, prev = atten * ((2.0 - 4.0 * lam - beta) * u + lam * ring - (1.0 - beta) * prev), u
    return {"u_n": u, "u_nm1": prev}


def exact(case, seed):
    if case["kind"] == "passes":
        return _exact_passes(case, seed)
    if case["kind"] == "wave":
        return _exact_wave(case, seed)
    return None
