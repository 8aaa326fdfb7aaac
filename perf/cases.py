"""The workloads this framework is timed on, through its public entry points.

Each case is one thing a cloth application has the library do: advance a garment by a frame (a small sheet, the 10k and
60k tubes, a garment too large for the on-chip solve, a garment with the learned preconditioner), drape for a few frames
on the device, advance a batch of uneven garments, bake a body's collision field, multiply by a Newton matrix, solve a
Newton system without allocating, and take a training gradient of the preconditioner's network. Sizes span the
workloads of the tests and the benchmark (1,600 to 60,060 particles, batches of 2k-40k) and go beyond them to both sides.

A frame case evolves its state as an application does: every pass is the next frame. Garments start sewn shut around the
body, 1 mm above its contact distance, with seeded jitter, and settle under gravity, so contact, friction, stretch and
bending all act from the first frames on.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "drape-2_b200") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "drape-2_b200"))

from drape_b200 import bake as bake_api  # noqa: E402
from drape_b200 import batch as batch_api  # noqa: E402
from drape_b200 import cuda as cuda_api  # noqa: E402
from drape_b200 import learned as learned_api  # noqa: E402
from drape_b200 import meshes, scenes  # noqa: E402
from drape_b200.scene import SETTLING, Field, Settings, drape_drape_options  # noqa: E402

DEV = "cuda"


# ---------------------------------------------------------------------------------------------------------------
# The cases.

def listed():
    return [
        # The interactive editor's smallest garment: the 40 x 40 sheet on the sphere, one substep a frame. Latency of
        # launches and grid exchanges, nothing else.
        {"name": "frame_sheet_1600", "kind": "frame", "shape": "sheet", "particles": 1600, "substeps": 1,
         "learned": False},
        # The default quality: the 10k tube, two substeps a frame (the defaults of Solver::step).
        {"name": "frame_tube_10k", "kind": "frame", "shape": "tube", "particles": 10080, "substeps": 2,
         "learned": False},
        # High quality: the 60k tube, the drape runner's frames (one substep, device-side statistics, replayed graphs).
        # Its seams start closed, so the pass holds the change from Assembling to Settling that every drape has.
        {"name": "drape_tube_60k", "kind": "drape", "shape": "tube", "particles": 60060, "frames": 6},
        # A long garment (a gown, a curtain) beyond what the chip's shared memory holds.
        {"name": "frame_tube_150k", "kind": "frame", "shape": "tube", "particles": 150000, "substeps": 1,
         "learned": False},
        # The learned preconditioner in the solver: network inference and learned PCG in every Newton iteration.
        {"name": "frame_tube_10k_learned", "kind": "frame", "shape": "tube", "particles": 10080, "substeps": 1,
         "learned": True},
        # A few frames of the hanging sheet (two pins, no body), the runner on a small garment.
        {"name": "drape_hanging_2601", "kind": "drape", "shape": "hanging", "particles": 2601, "frames": 10},
        # A size set: uneven garments advanced together, 2k-40k particles each.
        {"name": "batch_16_tubes", "kind": "batch", "garments": 16, "smallest": 2000, "largest": 40000},
        # A body's collision field at the default 4 mm cells (the five-component test body).
        {"name": "bake_body_4mm", "kind": "bake", "body": "test_body", "cell_mm": 4.0},
        # Products with a Newton matrix: one garment's, and one larger than the L2.
        {"name": "spmv_10k", "kind": "spmv", "rows": 10080},
        {"name": "spmv_700k", "kind": "spmv", "rows": 720000},
        # A frame-paced host that may not allocate: a solve on device buffers near the entry point's size limit.
        {"name": "pcg_noalloc_8k", "kind": "pcg", "rows": 8000, "tolerance": 1e-5},
        # Training the preconditioner: loss and gradient on one 10k Newton system.
        {"name": "train_grad_10k", "kind": "train", "particles": 10080},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame", "frame", "frame", "drape", "batch", "bake", "spmv", "spmv", "pcg", "train"])
    if kind == "frame":
        learned = rng.random() < 0.25
        return {"kind": "frame", "shape": rng.choice(["tube", "tube", "sheet"]),
                "particles": log(400, 40000 if learned else 150000), "substeps": rng.choice([1, 2]),
                "learned": learned}
    if kind == "drape":
        return {"kind": "drape", "shape": rng.choice(["tube", "hanging"]), "particles": log(400, 60060),
                "frames": rng.randint(2, 10)}
    if kind == "batch":
        low = log(500, 5000)
        return {"kind": "batch", "garments": rng.randint(2, 16), "smallest": low, "largest": low * rng.randint(1, 8)}
    if kind == "bake":
        return {"kind": "bake", "body": rng.choice(["test_body", "capsules", "sphere"]),
                "cell_mm": round(rng.uniform(4.0, 12.0), 5)}
    if kind == "spmv":
        return {"kind": "spmv", "rows": log(300, 720000)}
    if kind == "pcg":
        return {"kind": "pcg", "rows": log(200, 8190), "tolerance": rng.choice([1e-4, 1e-5])}
    return {"kind": "train", "particles": log(1000, 12000)}


# ---------------------------------------------------------------------------------------------------------------
# Scenes. The mesh and the body's field do not depend on the seed and are kept; the start positions do.

def _panel_grid(particles):
    """Vertices of one 0.55 x 0.7 m panel (of two): the 10k and 60k tubes' own grids at their sizes."""
    per = particles / 2
    nx = max(4, int(round(math.sqrt(per * 0.55 / 0.7))))
    return nx, max(4, int(round(per / nx)))


def _capsule(p, a, b, r):
    a, b = (torch.tensor(v, dtype=torch.float64, device=DEV) for v in (a, b))
    ab = b - a
    t = (((p - a) @ ab) / (ab @ ab)).clamp(0, 1)
    return (p - a - t[..., None] * ab).norm(dim=-1) - r


@functools.lru_cache(maxsize=24)
def _capsule_field(n, torso=0.15, arm=0.05):
    """The lying capsule-union body of the tube workloads sampled on n^3 points over 0.762 m."""
    cell, band = 0.762 / (n - 1), 0.02
    origin = np.array([-0.381, 0.16 - 0.762, -0.381])
    i = torch.arange(n, dtype=torch.float64, device=DEV) * cell
    out = np.empty((n, n, n), np.float32)
    s = 0.45 * math.sqrt(0.5)
    for k0 in range(0, n, 32):
        z, y, x = torch.meshgrid(i[k0:k0 + 32] + origin[2], i + origin[1], i + origin[0], indexing="ij")
        p = torch.stack([x, y, z], -1)
        d = _capsule(p, (0.0, 0.0, -0.3), (0.0, 0.0, 0.3), torso)
        for g in (1.0, -1.0):
            d = torch.minimum(d, _capsule(p, (0.0, 0.0, 0.3 * g), (0.0, -s, (0.3 + s) * g), arm))
        out[k0:k0 + 32] = d.clamp(-band, band).float().cpu().numpy()
    return Field(origin, cell, (n, n, n), band, out)


@functools.lru_cache(maxsize=1)
def _sphere_field():
    return scenes.sphere_field()


@functools.lru_cache(maxsize=64)
def _scene(shape, particles):
    if shape == "sheet":
        n = max(4, int(round(math.sqrt(particles))))
        return scenes.sheet_on_sphere(n=n, height=0.1545, jitter=0.0, cg_tolerance=1e-2, max_cg=50,
                                      field=_sphere_field())
    if shape == "hanging":
        n = max(4, int(round(math.sqrt(particles))))
        g = scenes.piece_garment("sheet", 0.5, 0.5, n, n, scenes.jersey_fabric())
        g.initial_positions = np.stack([g.rest[:, 0], 0.5 + g.rest[:, 1], np.zeros(g.vertex_count)], axis=1)
        scene = scenes.Scene([g])
        for v in ((n - 1) * n, n * n - 1):
            scene.pins.append((v, tuple(g.initial_positions[v])))
        return scene
    nx, ny = _panel_grid(particles)
    return _tube(nx, ny, _capsule_field(256 if particles > 40000 else 128), 0.15, "tube")


def _tube(nx, ny, field, torso, gid):
    """Two panels sewn shut around the torso, hanging 1 mm above contact along its top line."""
    radius = 0.55 / math.pi
    sc = scenes.seamed_tube(nx, ny, radius=radius, field=field, settings=Settings(), gid=gid)
    g = sc.garments[0]
    g.initial_positions = g.initial_positions + np.array([0.0, torso + 0.0043 - radius, 0.0])
    return sc


def _jittered(scene, rng, amount):
    """The scene with every start coordinate moved by a seeded uniform amount (pinned particles keep theirs)."""
    g = scene.garments[0]
    x = g.initial_positions + rng.uniform(-amount, amount, g.initial_positions.shape)
    for p, pos in scene.pins:
        x[p] = pos
    moved = scenes.Garment(g.id, g.rest, g.vertex_piece, g.vertex_area, g.triangles, g.triangle_piece, g.piece_grain,
                           g.piece_fabric, g.seam_pairs, x, g.boundary)
    return scenes.Scene([moved], scene.body, pins=scene.pins, forces=scene.forces, settings=scene.settings)


def _batch_sizes(case):
    k = np.arange(case["garments"])
    t = (k * 0.6180339887 % 1.0)
    return np.round(case["smallest"] * (case["largest"] / case["smallest"]) ** t).astype(int)


# ---------------------------------------------------------------------------------------------------------------
# Newton-like block systems on the GPU: a seeded SPD matrix on the stencil of a cloth grid (two rows in each direction).

_OFFSETS = [(0, 1), (1, -1), (1, 0), (1, 1), (0, 2), (2, 0)]  # (rows, columns) to each later neighbour


def _system(rows, seed):
    w = max(3, int(round(math.sqrt(rows * 0.8))))
    n = rows
    gen = torch.Generator(device=DEV).manual_seed(seed)
    i = torch.arange(n, device=DEV)
    r, c = i // w, i % w
    entries = []
    diag = torch.zeros((n, 3, 3), dtype=torch.float32, device=DEV)
    eye = torch.eye(3, device=DEV)
    for dr, dc in _OFFSETS:
        j = i + dr * w + dc
        ok = (c + dc >= 0) & (c + dc < w) & (j < n)
        a, b = i[ok], j[ok]
        d = torch.nn.functional.normalize(torch.randn((len(a), 3), generator=gen, device=DEV), dim=1)
        k = 0.2 + 0.8 * torch.rand((len(a), 1, 1), generator=gen, device=DEV)
        block = k * (d[:, :, None] * d[:, None, :] + 0.05 * eye)
        diag.index_add_(0, a, block)
        diag.index_add_(0, b, block)
        entries += [(a, b, -block), (b, a, -block)]
    diag += (0.02 + 0.02 * torch.rand((n, 1, 1), generator=gen, device=DEV)) * eye
    row = torch.cat([i] + [e[0] for e in entries])
    col = torch.cat([i] + [e[1] for e in entries])
    blocks = torch.cat([diag] + [e[2] for e in entries])
    order = torch.argsort(row * n + col)
    row, col, blocks = row[order], col[order], blocks[order]
    slots = len(col)
    padded = (slots + 31) // 32 * 32
    planes = torch.zeros((9, padded), device=DEV)
    planes[:, :slots] = blocks.reshape(slots, 9).T
    start = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    start[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    pinned = (torch.rand(n, generator=gen, device=DEV) < 0.002).to(torch.uint8)
    return {"n": n, "slots": slots, "padded": padded, "row_start": start.to(torch.int32),
            "col_index": col.to(torch.int32), "planes": planes, "pinned": pinned, "gen": gen}


def _vec4(gen, n, scale=1.0):
    v = torch.zeros((n, 4), device=DEV)
    v[:, :3] = scale * torch.randn((n, 3), generator=gen, device=DEV)
    return v


def _product64(s, x):
    """A x in 64 bits over unpinned rows and columns; x is (n, 3)."""
    n, B = s["n"], s["slots"]
    live = (s["pinned"] == 0).double()[:, None]
    col = s["col_index"].long()
    row = torch.repeat_interleave(torch.arange(n, device=DEV), (s["row_start"][1:] - s["row_start"][:-1]).long())
    out = torch.zeros((n, 3), dtype=torch.float64, device=DEV)
    a = s["planes"][:, :B].double().T.reshape(B, 3, 3)
    return out.index_add_(0, row, torch.einsum("sij,sj->si", a, (x * live)[col])) * live


# ---------------------------------------------------------------------------------------------------------------
# prepare / run.

def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    state = {"case": case}
    if kind in ("frame", "drape"):
        scene = _jittered(_scene(case["shape"], case["particles"]), rng, 3e-5)
        s = cuda_api.CudaSolver(0)
        s.build(scene)
        if kind == "frame":
            s.set_phase(scene.garments[0].id, SETTLING)
            if case["learned"]:
                net = learned_api.LearnedPreconditioner(0, learned_api.load_weights("tube"))
                s.set_precond(net)
                net.close()
        else:
            o = drape_drape_options(substeps=1, iterations=2, frame_dt=1.0 / 60.0, max_assembly_seconds=3.0,
                                    seam_gap_done=0.001, settle_rms_speed=0.002, settle_hold_frames=60,
                                    max_sim_seconds=case["frames"] / 60.0, snapshot_every=30, max_retries=3,
                                    energy_rise_frames=60, frames_per_wait=10)
            state.update(options=o, garment=scene.garments[0].id)
        state["solver"] = s
    elif kind == "batch":
        b = batch_api.BatchSolver(0)
        for k, n in enumerate(_batch_sizes(case)):
            torso = 0.15 * (1.0 + 0.04 * math.sin(2.4 * k))
            nx, ny = _panel_grid(int(n))
            b.add(_jittered(_batch_scene(nx, ny, 48 if n < 8000 else 96, round(torso, 4)), rng, 3e-5))
        b.build()
        for k in range(case["garments"]):
            b.set_phase(k, SETTLING)
        state["batch"] = b
    elif kind == "bake":
        parts = {"test_body": meshes.test_body, "capsules": meshes.capsule_union_body,
                 "sphere": lambda: [meshes.icosphere((0.0, 0.0, 0.0), 0.15, 3)]}[case["body"]]()
        # A body of another size on a grid that grows with it, so the sample counts stay the case's own.
        scale = rng.uniform(0.97, 1.03)
        state["parts"] = [meshes.TriangleMesh(scale * m.vertices, m.triangles) for m in parts]
        state["options"] = bake_api.options(scale * case["cell_mm"] / 1000.0, scale * 0.0507, scale * 0.02)
    elif kind == "spmv":
        state.update(_system(case["rows"], seed))
        state["x"] = _vec4(state["gen"], state["n"])
        state["y"] = torch.zeros_like(state["x"])
        state["lib"] = cuda_api.load()
    elif kind == "pcg":
        state.update(_system(case["rows"], seed))
        n, gen = state["n"], state["gen"]
        state["grad"] = _vec4(gen, n, 1e-3) * (state["pinned"] == 0).float()[:, None]
        state["active"] = (torch.rand(n, generator=gen, device=DEV) < 0.2).to(torch.uint8)
        state["normals"] = torch.nn.functional.normalize(_vec4(gen, n), dim=1)
        state["step"], state["resid"] = (torch.zeros((n, 4), device=DEV) for _ in range(2))
        state["iterations"] = torch.zeros(1, dtype=torch.int32, device=DEV)
        state["lib"] = cuda_api.load()
    else:
        scene = _jittered(_scene("tube", case["particles"]), rng, 3e-5)
        s = cuda_api.CudaSolver(0)
        s.build(scene)
        s.set_phase(scene.garments[0].id, SETTLING)
        sysm = s.capture_system(1.0 / 60.0)
        s.close()
        n = len(sysm["diag_slot"])
        net = learned_api.LearnedPreconditioner(0, learned_api.load_weights("tube"))
        net.add_sample(sysm["row_start"], sysm["col_index"], sysm["blocks"], np.zeros(n, np.uint8), sysm["active"],
                       rng.standard_normal((1, n, 3)))
        state["net"] = net
    return state


@functools.lru_cache(maxsize=64)
def _batch_scene(nx, ny, field_n, torso):
    return _tube(nx, ny, _capsule_field(field_n, torso), torso, "tube")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "frame":
        s = state["solver"]
        s.step(1.0 / 60.0, case["substeps"], 2)
        return {"positions": s.positions(), "velocities": s.velocities()}
    if kind == "drape":
        s = state["solver"]
        res = s.drape_to_rest([state["garment"]], state["options"])
        return {"positions": s.positions(), "velocities": s.velocities(), "frames": int(res.frames_run)}
    if kind == "batch":
        b = state["batch"]
        b.step(1.0 / 60.0, 1, 2)
        return [b.positions(k) for k in range(case["garments"])]
    if kind == "bake":
        return bake_api.bake_field(state["parts"], state["options"]).values
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if kind == "spmv":
        code = state["lib"].drape_cuda_spmv_device(
            state["n"], state["row_start"].data_ptr(), state["col_index"].data_ptr(), state["planes"].data_ptr(),
            state["padded"], state["pinned"].data_ptr(), state["x"].data_ptr(), state["y"].data_ptr(), stream)
        if code != 0:
            raise RuntimeError(state["lib"].drape_cuda_last_error(None))
        return state["y"]
    if kind == "pcg":
        code = state["lib"].drape_cuda_pcg_noalloc(
            state["n"], state["slots"], state["row_start"].data_ptr(), state["col_index"].data_ptr(),
            state["planes"].data_ptr(), state["padded"], state["pinned"].data_ptr(), state["active"].data_ptr(),
            state["normals"].data_ptr(), state["grad"].data_ptr(), 400, case["tolerance"], state["step"].data_ptr(),
            state["resid"].data_ptr(), state["iterations"].data_ptr(), stream)
        if code != 0:
            raise RuntimeError(state["lib"].drape_cuda_last_error(None))
        return {"step": state["step"], "resid": state["resid"], "iterations": state["iterations"]}
    loss, grad = state["net"].loss_grad(0, 0)
    return {"loss": loss, "gradient": grad}


# ---------------------------------------------------------------------------------------------------------------
# The work no implementation can do without.

SLOTS = 13.5  # block slots a row of a cloth grid has (its own, six edges, six and a half hinge partners)


def _newton_work(n, iterations, pcg):
    """`iterations` Newton iterations of `pcg` PCG iterations each: terms and state in, state out; the products."""
    bytes_ = n * (2 * 48 + 3 * 32 + 5 * 16) * 1.0
    flops = iterations * n * (pcg * (18 * SLOTS + 60) + 4000.0)
    return bytes_, flops


def work(case):
    kind = case["kind"]
    if kind in ("frame", "drape"):
        steps = case["substeps"] if kind == "frame" else case["frames"]
        b, f = _newton_work(case["particles"], 2 * steps, 50)
        return {"bytes": steps * b, "flops": f}
    if kind == "batch":
        b, f = _newton_work(float(_batch_sizes(case).sum()), 2, 50)
        return {"bytes": b, "flops": f}
    if kind == "bake":
        parts = {"test_body": (0.85, 0.99, 0.30), "capsules": (0.40, 0.63, 1.37), "sphere": (0.4, 0.4, 0.4)}
        x, y, z = parts[case["body"]]
        cells = x * y * z / (case["cell_mm"] / 1000.0) ** 3
        return {"bytes": 4.0 * cells, "flops": 100.0 * cells}
    if kind in ("spmv", "pcg"):
        n = case["rows"]
        products = 1 if kind == "spmv" else 120
        return {"bytes": n * (40.0 * 12.6 + 40.0), "flops": products * n * (18 * 12.6 + (0 if kind == "spmv" else 60))}
    n = case["particles"]
    per_slot = 2.0 * (64 * 16 + 4 * 64 * 128 + 16 * 192)
    return {"bytes": n * SLOTS * 40.0, "flops": 3 * n * (SLOTS * per_slot + 2.0 * (64 * 16 + 4 * 64 * 128))}


# ---------------------------------------------------------------------------------------------------------------
# 64-bit values, where plain torch gives them in a few seconds. A whole Newton step and the network's gradient (BF16
# activations by design) have none here.

def exact(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        s = prepare(case, seed)
        y = torch.zeros((s["n"], 4), dtype=torch.float64, device=DEV)
        y[:, :3] = _product64(s, s["x"][:, :3].double())
        return y
    if kind == "pcg":
        return {"step": _solve64(prepare(case, seed)), "resid": None, "iterations": None}
    if kind == "bake" and case["cell_mm"] >= 4.0:
        return _field64(prepare(case, seed))
    return None


def _solve64(s):
    """The contact-filtered system's solution by conjugate gradients in 64 bits."""
    n = s["n"]
    live = (s["pinned"] == 0).double()[:, None]
    nrm = torch.nn.functional.normalize(s["normals"][:, :3].double(), dim=1) * s["active"].double()[:, None]

    def filtered(v):
        v = v * live
        return v - nrm * (nrm * v).sum(1, keepdim=True)

    b = filtered(-s["grad"][:, :3].double())
    x = torch.zeros_like(b)
    r = b.clone()
    p = r.clone()
    rr = (r * r).sum()
    first = rr
    for _ in range(4000):
        ap = filtered(_product64(s, filtered(p)))
        alpha = rr / (p * ap).sum()
        x += alpha * p
        r -= alpha * ap
        new = (r * r).sum()
        if new <= 1e-20 * first:
            break
        p = r + (new / rr) * p
        rr = new
    out = torch.zeros((n, 4), dtype=torch.float64, device=DEV)
    out[:, :3] = x
    return out


def _field64(s):
    """The union's signed distance, clamped to the band: unsigned distance over all triangles of a component, its sign
    from the winding number, components by minimum."""
    o = s["options"]
    cell, pad, band = o.cell_size, o.padding, o.band
    v = np.concatenate([m.vertices for m in s["parts"]])
    lo = v.min(0) - pad
    dims = [int(math.ceil((e + 2 * pad) / cell)) + 1 for e in v.max(0) - v.min(0)]
    axis = [torch.tensor(lo[a] + cell * np.arange(dims[a]), device=DEV) for a in range(3)]
    out = torch.full((dims[2], dims[1], dims[0]), band, dtype=torch.float64, device=DEV)
    for m in s["parts"]:
        tri = torch.tensor(m.vertices[m.triangles.astype(np.int64)], device=DEV)  # (T, 3, 3)
        sel = [torch.nonzero((axis[a] >= m.vertices[:, a].min() - band) & (axis[a] <= m.vertices[:, a].max() + band))
               .flatten() for a in range(3)]
        z, y, x = torch.meshgrid(axis[2][sel[2]], axis[1][sel[1]], axis[0][sel[0]], indexing="ij")
        p = torch.stack([x, y, z], -1).reshape(-1, 3)
        d = torch.empty(len(p), dtype=torch.float64, device=DEV)
        step = max(1, 24_000_000 // len(tri))
        for k in range(0, len(p), step):
            d[k:k + step] = _signed64(p[k:k + step], tri)
        d = d.clamp(-band, band).reshape(len(sel[2]), len(sel[1]), len(sel[0]))
        part = out[sel[2][0]:sel[2][-1] + 1, sel[1][0]:sel[1][-1] + 1, sel[0][0]:sel[0][-1] + 1]
        part.copy_(torch.minimum(part, d))
    return out


def _signed64(p, tri):
    q = tri[None] - p[:, None, None, :]  # (P, T, 3 corners, 3)
    best = None
    for a, b in ((0, 1), (1, 2), (2, 0)):
        e = (tri[:, b] - tri[:, a])[None]
        t = (-(q[:, :, a] * e).sum(-1) / (e * e).sum(-1)).clamp(0, 1)
        d2 = ((q[:, :, a] + t[..., None] * e) ** 2).sum(-1)
        best = d2 if best is None else torch.minimum(best, d2)
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    nn = (nrm * nrm).sum(-1)
    w = -q[:, :, 0]
    b2 = (torch.linalg.cross(e1[None].expand_as(w), w) * nrm).sum(-1) / nn
    b1 = (torch.linalg.cross(w, e2[None].expand_as(w)) * nrm).sum(-1) / nn
    inside = (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1)
    plane = (w * nrm).sum(-1) ** 2 / nn
    best = torch.where(inside, torch.minimum(best, plane), best).amin(1).sqrt()
    a, b, c = q[:, :, 0], q[:, :, 1], q[:, :, 2]
    la, lb, lc = a.norm(dim=-1), b.norm(dim=-1), c.norm(dim=-1)
    num = (a * torch.linalg.cross(b, c)).sum(-1)
    den = la * lb * lc + (a * b).sum(-1) * lc + (b * c).sum(-1) * la + (c * a).sum(-1) * lb
    wind = (2 * torch.atan2(num, den)).sum(1) / (4 * math.pi)
    return torch.where(wind > 0.5, -best, best)
