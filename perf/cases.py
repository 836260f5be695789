"""Workloads of the particle engine as its users run them: what is timed, on which inputs, and what the results are in 64 bits.

Every case hands the engine a state that is on the GPU, runs one call of a simulation loop (one step, one tick of
substeps, one frame, one training run) through the public handles of `gpe`, and takes the results in device buffers.
Particles are laid out and disturbed on the GPU from the seed: lattice blocks with the spacing, jitter and physics of
the engine's own workloads (gpe.scenes), moving with a smooth swirl, part of them a splash in random directions.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "gpu-physics-engine_gb300"))
import gpe  # noqa: E402
from gpe import scenes  # noqa: E402

DEV = "cuda"
F32, F64 = torch.float32, torch.float64
SPACING = 0.01  # lattice spacing of the PBF workloads, half the smoothing radius


def listed() -> list[dict]:
    return [
        # a small interactive scene: the 16,384-particle dam break, where launches and latency count
        {"name": "pbf_dam_16k", "kind": "pbf", "n": 16384, "aspect": 1.0, "iters": 4, "dt": 1 / 480, "splash": 0.0,
         "vort": 0.0, "scorr": 0.0},
        # an ordinary scene of odd size with every force switched on: vorticity confinement, artificial pressure
        {"name": "pbf_vorticity_100k", "kind": "pbf", "n": 100003, "aspect": 1.7, "iters": 3, "dt": 1 / 480,
         "splash": 0.1, "vort": 0.5, "scorr": 1e-14},
        # the headline workload: a deep block and a splash, 1,048,576 particles
        {"name": "pbf_million", "kind": "pbf", "n": 1048576, "aspect": 0.94, "iters": 4, "dt": 1 / 2000,
         "splash": 0.0625, "vort": 0.0, "scorr": 0.0},
        # many independent scenes in one engine, 2,048 to 65,536 particles each: the largest PBF work
        {"name": "pbf_batched_256", "kind": "pbf_batch", "scenes": 256, "lo": 2048, "hi": 65536, "iters": 4,
         "dt": 1 / 480},
        # one 32 ms tick of the engine this one drops in for: its constants, 20 substeps, 16,384 atoms
        {"name": "pbf_reference_tick", "kind": "pbf_tick", "n": 16384, "steps": 20},
        # the learned warm start on the headline workload: the memory-starting step and seven network steps
        {"name": "pbf_learned_million", "kind": "pbf_learned", "n": 1048576, "iters": 2, "steps": 8},
        # training the warm-start network: one epoch over half a million pairs
        {"name": "mlp_train_epoch", "kind": "train", "pairs": 524288, "batch": 8192, "epochs": 1},
        # a small elastic scene (two colliding squares), one re-sort interval of steps
        {"name": "mpm_elastic_64k", "kind": "mpm", "n": 65536, "grid": 128, "what": "elastic", "steps": 16},
        # a tick of the drop-in MLS-MPM path: water, particles never re-sorted, 20 substeps
        {"name": "mpm_fluid_tick", "kind": "mpm", "n": 262147, "grid": 0, "what": "fluid", "steps": 20},
        # the large mixed-material scene (water, snow, jelly), one re-sort interval of steps
        {"name": "mpm_mixed_4m", "kind": "mpm", "n": 4194304, "grid": 1024, "what": "mixed", "steps": 32},
        # 32 mixed-material scenes of 64k to 512k particles in one engine
        {"name": "mpm_batched_32", "kind": "mpm_batch", "scenes": 32, "lo": 65536, "hi": 524288, "steps": 32},
        # a rendered frame: a million particles published to chunks and drawn at 2048 x 2048
        {"name": "render_million", "kind": "render", "n": 1048576, "width": 2048, "height": 2048},
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["pbf", "pbf", "pbf", "pbf_batch", "pbf_tick", "pbf_learned", "train", "mpm", "mpm", "mpm",
                       "mpm_batch", "render"])
    if kind == "pbf":
        n = _log(rng, 4096, 1048576)
        return {"kind": kind, "n": n, "aspect": round(math.exp(rng.uniform(-1.0, 1.0)), 3),
                "iters": rng.choice([2, 3, 4, 6]), "dt": 1 / 2000 if n > 262144 else 1 / 480,
                "splash": rng.choice([0.0, 0.0625, 0.2]), "vort": rng.choice([0.0, 0.0, 0.5]),
                "scorr": rng.choice([0.0, 0.0, 1e-14])}
    if kind == "pbf_batch":
        return {"kind": kind, "scenes": _log(rng, 2, 200), "lo": 2048, "hi": _log(rng, 4096, 65536),
                "iters": rng.choice([2, 4]), "dt": 1 / 480}
    if kind == "pbf_tick":
        return {"kind": kind, "n": _log(rng, 4096, 524288), "steps": rng.randint(5, 20)}
    if kind == "pbf_learned":
        return {"kind": kind, "n": _log(rng, 32768, 1048576), "iters": rng.choice([1, 2, 3]),
                "steps": rng.randint(4, 8)}
    if kind == "train":
        return {"kind": kind, "pairs": _log(rng, 32768, 524288), "batch": _log(rng, 2000, 16384), "epochs": 1}
    if kind == "mpm":
        what = rng.choice(["elastic", "fluid", "mixed", "mixed", "library"])
        n = _log(rng, 16384, 262144 if what == "elastic" else 2097152)
        # particles in the squares (an eighth of the box, 16 to 32 a cell) and in the discs (about 13 a cell)
        per = rng.uniform(16.0, 32.0) * 0.125 if what == "elastic" else 13.3 * 0.3
        grid = 0 if what == "fluid" else max(64, int(math.sqrt(n / per) / 8) * 8)
        return {"kind": kind, "n": n, "grid": grid, "what": what, "steps": rng.randint(8, 32)}
    if kind == "mpm_batch":
        return {"kind": kind, "scenes": _log(rng, 2, 24), "lo": 32768, "hi": _log(rng, 65536, 524288),
                "steps": rng.randint(8, 32)}
    return {"kind": "render", "n": _log(rng, 16384, 1048576), "width": rng.randint(640, 2048),
            "height": rng.randint(480, 2048)}


# ----- inputs --------------------------------------------------------------------------------------------------
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _rand(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=F64) * (hi - lo) + lo


def _lattice(n: int, aspect: float, origin=(0.0, 0.0), spacing: float = SPACING):
    """n points of a square lattice, row by row, width / height about `aspect`; its columns and rows."""
    nx = max(1, int(round(math.sqrt(n * aspect))))
    i = torch.arange(n, device=DEV)
    p = torch.stack([(i % nx + 0.5) * spacing + origin[0], (i // nx + 0.5) * spacing + origin[1]], 1).to(F64)
    return p, nx, -(-n // nx)


def _swirl(p, amp: float, wave: float):
    k = 2 * math.pi / wave
    return torch.stack([amp * torch.sin(k * p[:, 1]), amp * torch.sin(k * p[:, 0])], 1)


def _dam(n: int, aspect: float, splash: float, g):
    """The fluid block in the lower-left corner of a box of twice its size (swirling), with a share of the
    particles as a splash block above it, in random directions at up to 2 units per second."""
    ns = int(n * splash)
    p, nx, ny = _lattice(n - ns, aspect)
    w, h = 2.0 * nx * SPACING, 2.0 * ny * SPACING
    v = _swirl(p, 0.2, 0.4 * max(w, h))
    if ns:
        q, sx, sy = _lattice(ns, 1.0)
        h += sy * SPACING
        w = max(w, (sx + 4) * SPACING)
        q = q + torch.tensor([(w - sx * SPACING) / 2, h - sy * SPACING - 2 * SPACING], device=DEV, dtype=F64)
        a, s = _rand(g, 0, 2 * math.pi, ns), _rand(g, 0, 2, ns)
        p, v = torch.cat([p, q]), torch.cat([v, torch.stack([s * torch.cos(a), s * torch.sin(a)], 1)])
    p = p + _rand(g, -0.0002, 0.0002, n, 2)
    v = v + _rand(g, -0.01, 0.01, n, 2)
    return p.to(F32), v.to(F32), (0.0, 0.0, w, h)


def _pbf_params(c: dict):
    p = scenes.dam_params(iters=c["iters"])
    p.dt = c.get("dt", scenes.MILLION_DT)
    p.vort_eps = c.get("vort", 0.0)
    p.scorr_k = c.get("scorr", 0.0)  # beside mass times multiplier, about 1e-14 in these scenes
    return p


def _counts(c: dict) -> np.ndarray:
    """Particles of each scene of a batch: log-uniform, the same for every seed (a user's plan)."""
    r = np.random.default_rng(c["scenes"])
    return np.exp(r.uniform(math.log(c["lo"]), math.log(c["hi"]), c["scenes"])).astype(np.int64)


def _batch(c: dict, g):
    """Dam breaks side by side, box aspect 0.5 to 2."""
    pos, vel, dom, boxes, x0 = [], [], [], [], 0.0
    aspect = np.random.default_rng(c["scenes"] + 1).uniform(0.5, 2.0, c["scenes"])
    for s, n in enumerate(_counts(c)):
        p, nx, ny = _lattice(int(n), float(aspect[s]), (x0, 0.0))
        pos.append(p)
        dom.append(torch.full((int(n),), s, dtype=torch.int32, device=DEV))
        boxes.append((x0, 0.0, 2 * nx * SPACING, 2 * ny * SPACING))
        x0 += 2 * nx * SPACING + 1.0
    pos, dom = torch.cat(pos), torch.cat(dom)
    vel = _swirl(pos, 0.2, 1.0) + _rand(g, -0.01, 0.01, len(pos), 2)
    pos = pos + _rand(g, -0.0002, 0.0002, len(pos), 2)
    return pos.to(F32), vel.to(F32), dom, boxes


def _tick(n: int, g):
    """Atoms on a lattice of spacing 1.05 in a walled world of whole 32 x 32 chunks, twice the block's size."""
    p, nx, ny = _lattice(n, 1.5, (32.0, 32.0), 1.05)
    box = (0.0, 0.0, 32.0 * math.ceil(1.05 * nx / 16 + 1), 32.0 * math.ceil(1.05 * ny / 16 + 1))
    p = p + _rand(g, -0.05, 0.05, n, 2)
    return p.to(F32), _rand(g, -0.05, 0.05, n, 2).to(F32), box


# standardisation of the 12 features in these scenes, in the network's order, and of its target
_FEAT_MU = np.array([12, 0, 0, 0.01, 0.01, 0, 0, 10, 1e8, 0, 3, 0], np.float32)
_FEAT_SD = np.array([2, 1e-10, 0.02, 0.02, 0.01, 10, 10, 10, 3e7, 1e-10, 1, 1e-10], np.float32)


def _network(seed: int) -> np.ndarray:
    """Parameters of a network that has learned the first multiplier (r = cold lambda - lambda_prev) plus 1% of
    whatever else: a step with it is as stable as the plain step."""
    r = np.random.default_rng(seed)
    w1, b1 = r.normal(0, 0.4, (64, 12)), np.zeros(64)
    w2, b2 = r.normal(0, 0.15, (64, 64)), np.zeros(64)
    w3 = r.normal(0, 0.001, 64)
    w1[:4], w2[:4], w2[:, :4] = 0, 0, 0
    for u, (f, s) in enumerate([(9, 1), (9, -1), (1, 1), (1, -1)]):
        w1[u, f] = s
        w2[u, u] = 1
        w3[u] = s if f == 9 else -s
    flat = np.concatenate([w1.ravel(), b1, w2.ravel(), b2, w3, [0.0], _FEAT_MU, _FEAT_SD, [0.0, 1e-10]])
    return flat.astype(np.float32)


def _pairs(n: int, g):
    """Feature vectors as the solver's, and the multiplier changes they go with, up to 10% of noise."""
    z = torch.randn(n, 12, generator=g, device=DEV, dtype=F64)
    t = z[:, 9] - z[:, 1] + 0.3 * torch.tanh(z[:, 2] * z[:, 5]) + 0.1 * torch.randn(n, generator=g, device=DEV, dtype=F64)
    mu, sd = (torch.from_numpy(a).to(DEV, F64) for a in (_FEAT_MU, _FEAT_SD))
    return (z * sd + mu).to(F32).cpu().numpy(), (t * 1e-10).to(F32).cpu().numpy()


def _by_cell(pos, mat, grid: int):
    cell = (pos[:, 1] * grid).floor().long() * grid + (pos[:, 0] * grid).floor().long()
    order = torch.argsort(cell, stable=True)
    return pos[order], mat[order]


def _discs(n: int, grid: int, materials, g, seed: int):
    """n particles in discs of equal radius (three per material, 0.3 of the unit box), cell by cell."""
    k = 3 * len(materials)
    r = math.sqrt(0.3 / (k * math.pi))
    centre = torch.from_numpy(np.random.default_rng(seed).uniform(0.15 + r, 0.85 - r, (k, 2))).to(DEV)
    d = torch.arange(n, device=DEV) * k // n
    rad, th = r * torch.sqrt(_rand(g, 0, 1, n)), _rand(g, 0, 2 * math.pi, n)
    pos = centre[d] + torch.stack([rad * torch.cos(th), rad * torch.sin(th)], 1)
    mat = torch.tensor(materials, device=DEV, dtype=torch.int32)[d // 3]
    return _by_cell(pos, mat, grid)


_MIXED = (gpe.MPM_MAT_FLUID, gpe.MPM_MAT_SNOW, gpe.MPM_MAT_COROTATED)
_LIBRARY = _MIXED + (gpe.MPM_MAT_NEOHOOKEAN, gpe.MPM_MAT_SAND)


def _mpm(c: dict, seed: int):
    """(params, scene table or None, pos, vel, material or None, scene ids or None)"""
    g = _gen(seed)
    if c["kind"] == "mpm_batch":
        counts = _counts(c)
        p = scenes.mixed_params(4194304)
        table, pos, mat, sid = [], [], [], []
        for q, n in enumerate(counts):
            side = int(math.ceil(1024.0 * math.sqrt(n / 4194304) / 8.0)) * 8
            size = side * p.dx
            x, m = _discs(int(n), side, _MIXED, g, seed * 64 + q)
            table.append((side, side, (2 * p.dx, 2 * p.dx), (size - 3 * p.dx, size - 3 * p.dx)))
            pos.append(x * size)
            mat.append(m)
            sid.append(torch.full((int(n),), q, dtype=torch.int32, device=DEV))
        pos, mat, sid = torch.cat(pos), torch.cat(mat), torch.cat(sid)
        return p, table, pos.to(F32), (_swirl(pos, 0.3, 0.5)).to(F32), mat, sid
    n = c["n"]
    if c["what"] == "fluid":
        # the drop-in constants: a lattice of spacing 1.1 (rest volume 1.2 a particle), stored as emitted
        p = scenes.reference_mpm_params()
        x, nx, ny = _lattice(n, 1.5, (16.0, 16.0), 1.1)
        size = (math.ceil(1.1 * nx / 16) * 32.0, math.ceil(1.1 * ny / 16) * 32.0)
        p.nx, p.ny = int(size[0]) // 2 + 4, int(size[1]) // 2 + 4
        p.clamp_hi[0], p.clamp_hi[1] = size
        x = x + _rand(g, -0.1, 0.1, n, 2)
        return p, None, x.to(F32), (_swirl(x, 20.0, 100.0) + _rand(g, -1, 1, n, 2)).to(F32), None, None
    if c["what"] == "elastic":
        p = scenes.elastic_params(n, c["grid"])
        p.mass = 1.0 / n
        p.sort_interval = 16
        x = _rand(g, 0.0, 0.25, n, 2)
        left = torch.arange(n, device=DEV) < n // 2
        x = x + torch.where(left[:, None], torch.tensor([0.2, 0.2], device=DEV, dtype=F64),
                            torch.tensor([0.55, 0.45], device=DEV, dtype=F64))
        v = _swirl(x, 0.2, 0.25)
        v[:, 0] += torch.where(left, 0.5, -0.5)
        return p, None, x.to(F32), v.to(F32), None, None
    p = scenes.mixed_params(n, c["grid"])
    x, m = _discs(n, c["grid"], _LIBRARY if c["what"] == "library" else _MIXED, g, seed)
    return p, None, x.to(F32), _swirl(x, 0.3, 0.5).to(F32), m, None


# ----- the cases ---------------------------------------------------------------------------------------------
class _State:
    pass


def _pbf_state(params, boxes, pos, vel, dom=None) -> _State:
    s = _State()
    s.pos, s.vel, s.dom = pos, vel, dom
    s.eng = gpe.Pbf(params, boxes, capacity=len(pos))
    s.out = [torch.empty_like(pos), torch.empty_like(vel)]
    s.steps = 1
    return s


def prepare(case: dict, seed: int):
    kind, g = case["kind"], _gen(seed)
    if kind == "pbf":
        pos, vel, box = _dam(case["n"], case["aspect"], case["splash"], g)
        s = _pbf_state(_pbf_params(case), [box], pos, vel)
    elif kind == "pbf_batch":
        pos, vel, dom, boxes = _batch(case, g)
        s = _pbf_state(_pbf_params(case), boxes, pos, vel, dom)
    elif kind == "pbf_tick":
        pos, vel, box = _tick(case["n"], g)
        s = _pbf_state(scenes.reference_pbf_params(2), [box], pos, vel)
        s.steps = case["steps"]
    elif kind == "pbf_learned":
        pos, vel, box = _dam(case["n"], 0.94, 0.0625, g)
        s = _pbf_state(_pbf_params(case), [box], pos, vel)
        s.net = gpe.Mlp(seed=1)
        s.net.set_blob(_network(seed))
        s.eng.set_warm_start(gpe.WARM_MLP, s.net)
        s.steps = case["steps"]
    elif kind == "train":
        s = _State()
        s.net = gpe.Mlp(max_pairs=case["pairs"], seed=1)
        s.net.set_pairs(*_pairs(case["pairs"], g))
        s.blob = _network(seed)
        s.tp = gpe.make_train_params(epochs=case["epochs"], batch=case["batch"], lr=2e-3, seed=seed, lr_schedule=1)
    elif kind in ("mpm", "mpm_batch"):
        s = _State()
        p, table, s.pos, s.vel, s.mat, s.sid = _mpm(case, seed)
        s.eng = gpe.Mpm(p, capacity=len(s.pos), scenes=[gpe.make_mpm_scene(*t) for t in table] if table else None)
        s.steps, n = case["steps"], len(s.pos)
        s.out = [torch.empty(n, w, dtype=F32, device=DEV) for w in (2, 2, 4, 4)] + [torch.empty(n, dtype=F32, device=DEV)]
    else:
        n, w, h = case["n"], case["width"], case["height"]
        pos, vel, box = _dam(n, 1.0, 0.0625, g)
        s = _pbf_state(_pbf_params({"iters": 4}), [box], pos, vel)
        s.eng.set_state(pos, vel)
        # chunks of an eighth of the box; the fullest holds its share of the block
        dim = max(box[2], box[3]) / 8
        cap = int(1.3 * (dim / SPACING + 2) ** 2) + 64
        s.view_pos = torch.empty(64 * cap, 2, dtype=F32, device=DEV)
        s.view_vel = torch.empty_like(s.view_pos)
        s.view_n = torch.zeros(64, dtype=torch.int32, device=DEV)
        s.view = gpe.View(s.view_pos.data_ptr(), s.view_vel.data_ptr(), s.view_n.data_ptr(), 8, 8, dim, cap)
        s.img = torch.zeros(h, 4 * w, dtype=torch.uint8, device=DEV)
        s.cover = torch.zeros(h, w, dtype=torch.int32, device=DEV)
        s.raster = gpe.Raster(s.img.data_ptr(), 4 * w, w, h, min(w / box[2], h / box[3]), dim, s.cover.data_ptr())
    s.kind = kind
    return s


def run(s):
    if s.kind == "train":
        s.net.set_blob(s.blob)
        train_loss, val_loss = s.net.train(s.tp)
        blob = s.net.blob()
        return {"weights": blob[:gpe.MLP_NUM_WEIGHTS], "norm": blob[gpe.MLP_NUM_WEIGHTS:], "train_loss": train_loss,
                "val_loss": val_loss}
    if s.kind == "render":
        s.eng.publish(s.view)
        gpe.render_frame(s.raster, s.view)
        return [s.img, s.view_n]
    if s.kind in ("mpm", "mpm_batch"):
        s.eng.set_state(s.pos, s.vel, material=s.mat, scene_id=s.sid)
        s.eng.step(s.steps)
        s.eng.get_state_device(*s.out)
        return s.out
    s.eng.set_state(s.pos, s.vel, s.dom)
    s.eng.step(s.steps)
    s.eng.get_state(*s.out)
    return s.out


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("pbf", "pbf_batch", "pbf_tick", "pbf_learned"):
        n = int(_counts(case).sum()) if kind == "pbf_batch" else case["n"]
        # per step: position and velocity in and out; per pass and neighbour (12 on the lattice) about 20 operations
        passes = [2 * case["iters"] + 1 + (1 if case.get("vort") else 0)] if kind in ("pbf", "pbf_batch") else (
            [5] * case["steps"] if kind == "pbf_tick" else [41] + [2 * case["iters"] + 1] * (case["steps"] - 1))
        flops = 240.0 * n * sum(passes)
        if kind == "pbf_learned":
            flops += 2.0 * (12 * 64 + 64 * 64 + 64) * n * (case["steps"] - 1)
        return {"bytes": 32.0 * n * len(passes), "flops": flops}
    if kind == "train":
        n = case["pairs"] * case["epochs"]
        return {"bytes": 52.0 * n, "flops": 6.0 * (12 * 64 + 64 * 64 + 64) * n}
    if kind in ("mpm", "mpm_batch"):
        n = int(_counts(case).sum()) if kind == "mpm_batch" else case["n"]
        # per step: x and F or J in and out (v and C only pass between the halves of a step); 27 sums and 9
        # gathers a particle
        per = {"elastic": 48, "fluid": 56}.get(case.get("what"), 60)
        return {"bytes": float(per) * n * case["steps"] + 52.0 * n, "flops": 450.0 * n * case["steps"]}
    px = case["width"] * case["height"]
    return {"bytes": 32.0 * case["n"] + 4.0 * px, "flops": 10.0 * px}


# ----- the results in 64 bits ------------------------------------------------------------------------------------
def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "pbf":
        pos, vel, box = _dam(case["n"], case["aspect"], case["splash"], _gen(seed))
        return _pbf_exact(_pbf_params(case), [box], pos, vel, torch.zeros(len(pos), dtype=torch.long, device=DEV))
    if kind == "pbf_batch":
        pos, vel, dom, boxes = _batch(case, _gen(seed))
        return _pbf_exact(_pbf_params(case), boxes, pos, vel, dom.long())
    if kind in ("mpm", "mpm_batch"):
        return _mpm_exact(*_mpm(case, seed), case["steps"])
    if kind == "train":
        return _train_exact(case, seed)
    # several PBF steps: a particle that rounding puts into another cell moves to another place of the sorted
    # output, so there is no value to compare place by place; images are bytes
    return None


def _pbf_exact(p, boxes, pos, vel, dom):
    """One PBF step (Macklin & Mueller 2013, as gpe.h states it). The prediction, the cells and the order of the
    particles are FP32 by definition; everything after them is in 64 bits."""
    f = np.float32
    cell, h = f(p.h), float(p.h)
    inv = float(f(1) / cell)
    b = torch.tensor(boxes, dtype=F32, device=DEV)
    org, ext = b[:, :2], b[:, 2:]
    nc = torch.ceil((ext / float(cell)).double()).long().clamp(min=1)
    off = torch.cumsum(nc[:, 0] * nc[:, 1], 0) - nc[:, 0] * nc[:, 1]
    cells = int((nc[:, 0] * nc[:, 1]).sum())
    lo, hi = org.double(), ((org + ext) - float(f(p.wall_margin))).double()
    dt = float(p.dt)
    g2 = torch.tensor([float(f(p.dt) * f(p.dt) * f(g)) for g in p.gravity], dtype=F32, device=DEV)
    xs = (pos.double() + dt * vel.double()).float() + g2

    def cell_of(x, d):
        return torch.minimum(((x - org[d]) * inv).floor().long().clamp(min=0), nc[d] - 1)

    at = cell_of(xs, dom)
    key, order = torch.sort(off[dom] + at[:, 1] * nc[dom, 0] + at[:, 0], stable=True)
    start = torch.zeros(cells + 1, dtype=torch.long, device=DEV)
    start[1:] = torch.cumsum(torch.bincount(key, minlength=cells), 0)
    x, dom = pos[order].double(), dom[order]
    d = xs[order].double() - x
    n = len(x)
    me = torch.arange(n, device=DEV)

    def scan(body):
        """body(j, r, r2, near) for the slots of the 3 x 3 cells around every particle's present cell"""
        c = cell_of((x.float() + d.float()), dom)
        w = nc[dom, 0]
        for row in (-1, 0, 1):
            y = c[:, 1] + row
            ok = (y >= 0) & (y < nc[dom, 1])
            base = off[dom] + y.clamp(min=0) * w
            base = torch.where(ok, base, off[dom])
            s = start[base + (c[:, 0] - 1).clamp(min=0)]
            e = start[base + torch.minimum(c[:, 0] + 1, w - 1) + 1]
            e = torch.where(ok, e, s)
            for t in range(int((e - s).max())):
                j = (s + t).clamp(max=n - 1)
                r = (x - x[j]) + (d - d[j])
                r2 = (r * r).sum(1)
                near = (s + t < e) & (r2 <= h * h) & (j != me)
                body(j, r, r2, near)

    c6 = 4.0 / (math.pi * h ** 8)
    cs = 30.0 / (math.pi * h ** 5)
    m, rho0 = float(p.mass), float(p.rho0)
    w_dq = c6 * (h * h - float(p.scorr_dq) ** 2) ** 3

    def spiky(r2, near):
        """(h - r)^2 / r, 0 for coincident pairs"""
        far = near & (r2 > 1e-12)
        rr = torch.sqrt(torch.where(far, r2, torch.ones_like(r2)))
        return torch.where(far, (h - rr) ** 2 / rr, torch.zeros_like(r2)), torch.where(far, (h - rr) ** 2, torch.zeros_like(r2))

    for _ in range(p.iters):
        s6 = torch.full((n,), h ** 6, dtype=F64, device=DEV)
        s4, sg = torch.zeros(n, dtype=F64, device=DEV), torch.zeros(n, 2, dtype=F64, device=DEV)

        def lam_body(j, r, r2, near):
            s6.add_(torch.where(near, h * h - r2, torch.zeros_like(r2)) ** 3)
            a, q = spiky(r2, near)
            s4.add_(q * q)
            sg.add_(a[:, None] * r)

        scan(lam_body)
        rho = m * c6 * s6
        grad = ((cs * m) ** 2 / m) * ((sg * sg).sum(1) + s4) / rho0 ** 2
        lam = -(rho / rho0 - 1).clamp(min=float(p.c_min)) / (grad + float(p.eps))
        sd = torch.zeros(n, 2, dtype=F64, device=DEV)

        def dp_body(j, r, r2, near):
            a, _ = spiky(r2, near)
            l = m * (lam + lam[j])
            if p.scorr_k:
                l = l - float(p.scorr_k) * (c6 * torch.where(near, h * h - r2, torch.zeros_like(r2)) ** 3 / w_dq) ** 4
            sd.add_((a * l)[:, None] * r)

        scan(dp_body)
        d = d - (cs * float(p.omega) / (m * rho0)) * sd
        d = torch.minimum(torch.maximum(x + d, lo[dom]), hi[dom]) - x
    v = d / dt
    dv, om = torch.zeros_like(v), torch.zeros(n, dtype=F64, device=DEV)

    def xsph_body(j, r, r2, near):
        u = v[j] - v
        dv.add_(torch.where(near, h * h - r2, torch.zeros_like(r2))[:, None] ** 3 * u)
        if p.vort_eps:
            a, _ = spiky(r2, near)
            om.add_(a * (u[:, 0] * r[:, 1] - u[:, 1] * r[:, 0]))

    scan(xsph_body)
    out = v + float(p.xsph_c) * c6 * dv
    if p.vort_eps:
        om = cs * om
        eta = torch.zeros_like(v)

        def vort_body(j, r, r2, near):
            a, _ = spiky(r2, near)
            eta.sub_(((om[j].abs() - om.abs()) * a)[:, None] * r)

        scan(vort_body)
        e2 = (eta * eta).sum(1)
        unit = torch.where((e2 > 1e-40)[:, None], eta / torch.sqrt(e2.clamp(min=1e-300))[:, None], torch.zeros_like(eta))
        out = out + (dt * float(p.vort_eps)) * torch.stack([unit[:, 1] * om, -unit[:, 0] * om], 1)
    return [x + d, out]


def _polar(F):
    c, s = F[:, 0] + F[:, 3], F[:, 2] - F[:, 1]
    n = torch.sqrt(c * c + s * s).clamp(min=1e-150)
    c, s = c / n, s / n
    return torch.stack([c, -s, s, c], 1)


def _mul(A, B):
    return torch.stack([A[:, 0] * B[:, 0] + A[:, 1] * B[:, 2], A[:, 0] * B[:, 1] + A[:, 1] * B[:, 3],
                        A[:, 2] * B[:, 0] + A[:, 3] * B[:, 2], A[:, 2] * B[:, 1] + A[:, 3] * B[:, 3]], 1)


def _t(A):
    return A[:, [0, 2, 1, 3]]


def _svd(F):
    """F = U diag(s) V^T with rotations U and V (the signs follow the polar rotation)"""
    R = _polar(F)
    S = _mul(_t(R), F)
    th = 0.5 * torch.atan2(2 * S[:, 1], S[:, 0] - S[:, 3])
    c, s = torch.cos(th), torch.sin(th)
    V = torch.stack([c, -s, s, c], 1)
    D = _mul(_t(V), _mul(S, V))
    return _mul(R, V), D[:, [0, 3]], V


def _usv(U, s, V):
    z = torch.zeros_like(s[:, 0])
    return _mul(U, _mul(torch.stack([s[:, 0], z, z, s[:, 1]], 1), _t(V)))


def _mpm_exact(p, table, pos, vel, mat, sid, steps):
    """MLS-MPM (quadratic B-splines, APIC) as gpe.h states it, every operation in 64 bits."""
    n = len(pos)
    x, v = pos.double(), vel.double()
    C = torch.zeros(n, 4, dtype=F64, device=DEV)
    eye = torch.tensor([1.0, 0, 0, 1.0], dtype=F64, device=DEV)
    F = eye.repeat(n, 1)
    J = torch.ones(n, dtype=F64, device=DEV)
    mat = torch.full((n,), p.material, device=DEV) if mat is None else mat.long()
    table = table or [(p.nx, p.ny, tuple(p.clamp_lo), tuple(p.clamp_hi))]
    sid = torch.zeros(n, dtype=torch.long, device=DEV) if sid is None else sid.long()
    f32 = lambda v: [float(np.float32(q)) for q in v]  # noqa: E731
    nx = torch.tensor([t[0] for t in table], device=DEV)
    sizes = nx * torch.tensor([t[1] for t in table], device=DEV)
    goff = torch.cumsum(sizes, 0) - sizes
    lo = torch.tensor([f32(t[2]) for t in table], dtype=F64, device=DEV)[sid]
    hi = torch.tensor([f32(t[3]) for t in table], dtype=F64, device=DEV)[sid]
    nodes, width = int(sizes.sum()), p.bc_width
    wall = []
    for a, b, _, _ in table:
        ix, iy = torch.arange(a, device=DEV).repeat(b), torch.arange(b, device=DEV).repeat_interleave(a)
        wall.append(torch.stack([ix <= width, ix >= a - 1 - width, iy <= width, iy >= b - 1 - width], 1))
    wall = torch.cat(wall)
    dx, dt, m, vol0 = float(p.dx), float(p.dt), float(p.mass), float(p.vol0)
    E, nu = float(p.E), float(p.nu)
    mu0, la0 = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
    is_ = {k: (mat == k)[:, None] for k in range(5)}
    has = {k: bool(is_[k].any()) for k in range(5)}
    for _ in range(steps):
        gx = x / dx + float(p.grid_offset)
        base = (gx - 0.5).floor()
        fx = gx - base
        w = [0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2]
        node = goff[sid] + base[:, 1].long() * nx[sid] + base[:, 0].long()
        # Kirchhoff stress times the particle's volume
        tau = torch.zeros_like(F)
        det = F[:, 0] * F[:, 3] - F[:, 1] * F[:, 2]
        if has[0]:
            pr = (float(p.k_bulk) * (J ** -float(p.gamma) - 1)).clamp(float(p.p_min), float(p.p_max))
            tau = torch.where(is_[0], (-pr * J)[:, None] * eye, tau)
        if has[1] or has[2]:
            hard = torch.where(mat == 2, torch.exp(float(p.hardening) * (1 - J)), torch.ones_like(J))
            t = (2 * mu0 * hard)[:, None] * _mul(F - _polar(F), _t(F)) + (la0 * hard * (det - 1) * det)[:, None] * eye
            tau = torch.where(is_[1] | is_[2], t, tau)
        if has[3]:
            t = mu0 * (_mul(F, _t(F)) - eye) + (la0 * torch.log(det.clamp(min=1e-6)))[:, None] * eye
            tau = torch.where(is_[3], t, tau)
        if has[4]:
            U, s, V = _svd(F)
            e = torch.log(s.clamp(min=1e-6))
            tau = torch.where(is_[4], _usv(U, 2 * mu0 * e + la0 * e.sum(1, keepdim=True), U), tau)
        Q = m * C - (dt * vol0 * 4 / dx ** 2) * tau
        grid = torch.zeros(nodes, 3, dtype=F64, device=DEV)
        for i in range(3):
            for j in range(3):
                ww = w[i][:, 0] * w[j][:, 1]
                ox, oy = (i - fx[:, 0]) * dx, (j - fx[:, 1]) * dx
                mom = torch.stack([m * v[:, 0] + Q[:, 0] * ox + Q[:, 1] * oy, m * v[:, 1] + Q[:, 2] * ox + Q[:, 3] * oy,
                                   torch.full_like(ox, m)], 1)
                grid.index_add_(0, node + j * nx[sid] + i, ww[:, None] * mom)
        full = grid[:, 2] > 0
        nv = torch.where(full[:, None], grid[:, :2] / torch.where(full, grid[:, 2], torch.ones_like(grid[:, 2]))[:, None]
                         + dt * torch.tensor(list(p.gravity), dtype=F64, device=DEV), torch.zeros_like(grid[:, :2]))
        if p.bc_type == gpe.MPM_BC_STICKY:
            nv = torch.where(wall.any(1)[:, None], torch.zeros_like(nv), nv)
        else:
            for a in range(2):
                u = nv[:, a]
                stop = (wall[:, 2 * a] & (u < 0)) | (~wall[:, 2 * a] & wall[:, 2 * a + 1] & (u > 0))
                nv[:, a] = torch.where(stop, torch.zeros_like(u), u)
        v, B = torch.zeros_like(v), torch.zeros_like(C)
        for i in range(3):
            for j in range(3):
                ww = (w[i][:, 0] * w[j][:, 1])[:, None]
                u = nv[node + j * nx[sid] + i]
                o = torch.stack([(i - fx[:, 0]) * dx, (j - fx[:, 1]) * dx], 1)
                v = v + ww * u
                B = B + ww * torch.stack([u[:, 0] * o[:, 0], u[:, 0] * o[:, 1], u[:, 1] * o[:, 0], u[:, 1] * o[:, 1]], 1)
        x, C = x + dt * v, (4 / dx ** 2) * B
        v = torch.where(x < lo, v.clamp(min=0), torch.where(x > hi, v.clamp(max=0), v))
        x = torch.minimum(torch.maximum(x, lo), hi)
        A = eye + dt * C
        keep = (mat != 0)[:, None] if not p.flags & gpe.MPM_FLAG_FLUID_F else torch.ones_like(is_[0])
        F = torch.where(keep, _mul(A, F), F)
        if has[0]:
            J = torch.where(mat == 0, (J * (A[:, 0] * A[:, 3] - A[:, 1] * A[:, 2])).clamp(float(p.J_min), float(p.J_max)), J)
        if has[2]:
            U, s, V = _svd(F)
            c = s.clamp(1 - float(p.theta_c), 1 + float(p.theta_s))
            J = torch.where(mat == 2, J * (s[:, 0] * s[:, 1]) / (c[:, 0] * c[:, 1]), J)
            F = torch.where(is_[2], _usv(U, c, V), F)
        if has[4]:
            # Drucker-Prager return mapping (Klar et al. 2016), friction angle 35 + (9 q - 10) exp(-0.2 q) degrees
            U, s, V = _svd(F)
            e = torch.log(s.clamp(min=1e-6))
            tr = e.sum(1)
            dev = e - 0.5 * tr[:, None]
            nrm = torch.sqrt((dev * dev).sum(1))
            q = J - 1
            sp = torch.sin((35 + (9 * q - 10) * torch.exp(-0.2 * q)) * (math.pi / 180))
            alpha = math.sqrt(2 / 3) * 2 * sp / (3 - sp)
            dg = nrm + (2 * la0 + 2 * mu0) / (2 * mu0) * tr * alpha
            tip, cone = tr >= 0, (tr < 0) & (dg > 0)
            e1 = torch.where(tip[:, None], torch.zeros_like(e),
                             e - (dg / nrm.clamp(min=1e-300))[:, None] * dev)
            moved = (mat == 4) & (tip | cone)
            J = torch.where(moved, J + torch.where(tip, torch.sqrt((e * e).sum(1)), dg), J)
            F = torch.where(moved[:, None], _usv(U, torch.exp(e1), V), F)
    return [x, v, C, F, J]


def _shuffled(n: int, seed: int, epochs: int):
    """The epochs' orders of the training pairs: Fisher-Yates driven by SplitMix64, each epoch from the identity."""
    mask = (1 << 64) - 1
    s = (seed ^ 0xBB67AE8584CAA73B) & mask
    for _ in range(epochs):
        o = list(range(n))
        for q in range(n - 1, 0, -1):
            s = (s + 0x9E3779B97F4A7C15) & mask
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (q + 1)
            o[q], o[j] = o[j], o[q]
        yield torch.tensor(o, device=DEV)


def _train_exact(case, seed):
    """The training run in 64 bits (no BF16 operands): standardisation, shuffles, AdamW with a cosine schedule."""
    X, T = (torch.from_numpy(a).to(DEV).double() for a in _pairs(case["pairs"], _gen(seed)))
    n = len(T) - int(len(T) * float(np.float32(0.1)))
    mu, sd = X[:n].mean(0), X[:n].std(0, unbiased=False)
    ymu, ysd = T[:n].mean(), T[:n].std(unbiased=False)
    Z, Y = (X - mu) / sd, (T - ymu) / ysd
    flat = torch.from_numpy(_network(seed)).to(DEV).double()
    shapes = [(64, 12), (64,), (64, 64), (64,), (1, 64), (1,)]
    W, at = [], 0
    for sh in shapes:
        k = math.prod(sh)
        W.append(flat[at:at + k].reshape(sh).clone().requires_grad_())
        at += k

    def net(z):
        a = torch.relu(z @ W[0].T + W[1])
        return (torch.relu(a @ W[2].T + W[3]) @ W[4].T + W[5])[:, 0]

    B, t, loss = case["batch"], 0, 0.0
    mom = [(torch.zeros_like(w), torch.zeros_like(w)) for w in W]
    total = case["epochs"] * -(-n // B)
    for order in _shuffled(n, seed, case["epochs"]):
        loss = 0.0
        for b in range(0, n, B):
            idx = order[b:b + B]
            sq = ((net(Z[idx]) - Y[idx]) ** 2)
            loss += float(sq.detach().sum())
            grads = torch.autograd.grad(sq.mean(), W)
            lr = 0.5 * float(np.float32(2e-3)) * (1 + math.cos(math.pi * t / total))
            t += 1
            with torch.no_grad():
                for k, (w, g, (a, v)) in enumerate(zip(W, grads, mom)):
                    a.mul_(0.9).add_(0.1 * g)
                    v.mul_(0.999).add_(0.001 * g * g)
                    decay = 1e-4 if k in (0, 2, 4) else 0.0
                    w -= lr * ((a / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8) + decay * w)
    with torch.no_grad():
        val = float(((net(Z[n:]) - Y[n:]) ** 2).mean())
    return {"weights": torch.cat([w.detach().reshape(-1) for w in W]), "norm": torch.cat([mu, sd, ymu[None], ysd[None]]),
            "train_loss": loss / n, "val_loss": val}
