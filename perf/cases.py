"""The work a user has this library do, as timed cases over its public entry points.

Kinds:
  diffuse   a diffusion tick on the caller's device buffers (marl_diffuse_device, or its
            allocation-free form), as a program whose field lives in torch tensors calls it
  seam      the same tick on host arrays (diffuse_tick_with_cells, the reference's plugin seam)
  seeded    a new run: Engine from seeding, stepped with host fate, state read back
  steps     a segment of a run that goes on: a kept Engine, stepped with host fate,
            state read back
  device    a run with fate on the device from a kept Context: state up, ticks, state back
  ensemble  a segment of a kept Batch of runs of unequal grids, every run read back
  infer     surrogate inference on standardised rows in device memory
  train     surrogate training steps on prepared pairs, weights and losses read back
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "marl-ochre_b200"))

import marl_cuda as marl  # noqa: E402

S = 12  # external species
ENSEMBLE = ((64, 64, 32), (96, 96, 48), (128, 128, 64), (128, 128, 96))  # the configured ensemble's grids
NOALLOC_VOXELS, NOALLOC_MASK = 1 << 18, 1 << 20  # limits of the allocation-free diffusion
HID, IN_PAD, OUT = 256, 128, 16


def listed() -> list[dict]:
    return [
        # A small odd grid (the tests' ragged one) in a loop that may not allocate: launches and latency.
        {"name": "diffuse_37x21x13", "kind": "diffuse", "x": 37, "y": 21, "z": 13, "substeps": 10, "noalloc": True},
        # The ensemble's small grid.
        {"name": "diffuse_64x64x32", "kind": "diffuse", "x": 64, "y": 64, "z": 32, "substeps": 10, "noalloc": False},
        # The default run's grid: both buffers together stay in L2.
        {"name": "diffuse_128x128x64", "kind": "diffuse", "x": 128, "y": 128, "z": 64, "substeps": 10,
         "noalloc": False},
        # The field microbenchmark's grid: the buffers exceed L2.
        {"name": "diffuse_256x256x128", "kind": "diffuse", "x": 256, "y": 256, "z": 128, "substeps": 10,
         "noalloc": False},
        # The drop-in for the reference's GPU diffuser, whose field stays on the host.
        {"name": "seam_128x128x64", "kind": "seam", "x": 128, "y": 128, "z": 64},
        # The default run from seeding, its first ticks (few cells).
        {"name": "seeded_128x128x64", "kind": "seeded", "x": 128, "y": 128, "z": 64, "ticks": 500},
        # The default run from tick 1000 on (about 38,000 cells).
        {"name": "steps_128x128x64", "kind": "steps", "x": 128, "y": 128, "z": 64, "at": 1000, "ticks": 100},
        # A small odd grid run for many ticks with fate on the device: one call, no host round trips.
        {"name": "device_60x52x30", "kind": "device", "x": 60, "y": 52, "z": 30, "seeds": 30, "at": 300, "ticks": 300},
        # A large grid with a dense seeding, fate on the device.
        {"name": "device_192x160x96", "kind": "device", "x": 192, "y": 160, "z": 96, "seeds": 1000, "at": 200,
         "ticks": 150},
        # Two runs of each of the configured ensemble's grids.
        {"name": "ensemble_8_runs", "kind": "ensemble", "runs": 8, "scale": 1.0, "at": 200, "ticks": 100},
        # The inference figure's row count for a dense default grid.
        {"name": "infer_300000", "kind": "infer", "rows": 300_000},
        # Training at the default batch.
        {"name": "train_b8192", "kind": "train", "batch": 8192, "pairs": 100_000, "steps": 16},
    ]


def _log_uniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _dims(rng, lo: float, hi: float, least=(1, 1, 1)) -> tuple[int, int, int]:
    """A grid of lo..hi voxels (over the logarithm) of an aspect near the default grid's 2:2:1."""
    while True:
        v = _log_uniform(rng, lo, hi)
        x = round((v * 2) ** (1 / 3) * rng.uniform(0.7, 1.4))
        y = round((v * 2) ** (1 / 3) * rng.uniform(0.7, 1.4))
        z = round(v / max(1, x * y))
        if x >= least[0] and y >= least[1] and z >= least[2] and x * y * z <= hi:
            return x, y, z


def draw(rng) -> dict:
    kind = rng.choice(["diffuse"] * 5 + ["seam", "seeded", "steps"] + ["device"] * 2 + ["ensemble"] + ["infer"] * 2 +
                      ["train"])
    if kind == "infer":
        return {"kind": kind, "rows": int(_log_uniform(rng, 100, 300_000))}
    if kind == "train":
        return {"kind": kind, "batch": 128 * int(_log_uniform(rng, 4, 64.9)), "pairs": rng.randrange(20_000, 100_000),
                "steps": 16}
    if kind == "ensemble":
        return {"kind": kind, "runs": rng.randrange(2, 9), "scale": round(rng.uniform(0.5, 1.0), 3),
                "at": rng.randrange(50, 201), "ticks": rng.randrange(40, 101)}
    if kind == "diffuse":
        x, y, z = _dims(rng, 2_000, 256 * 256 * 128)
        fits = x * y * z <= NOALLOC_VOXELS and z * y * ((x + 15) // 16 * 16) <= NOALLOC_MASK
        return {"kind": kind, "x": x, "y": y, "z": z, "substeps": rng.choice([1, 4, 10, 10]),
                "noalloc": fits and rng.random() < 0.3}
    least = (16, 16, 12)
    if kind == "seam":
        x, y, z = _dims(rng, 10_000, 128 * 128 * 64, least)
        return {"kind": kind, "x": x, "y": y, "z": z}
    if kind == "seeded":
        x, y, z = _dims(rng, 30_000, 128 * 128 * 64, least)
        return {"kind": kind, "x": x, "y": y, "z": z, "ticks": rng.randrange(100, 501)}
    if kind == "steps":
        x, y, z = _dims(rng, 60_000, 128 * 128 * 64, least)
        return {"kind": kind, "x": x, "y": y, "z": z, "at": rng.randrange(200, 1001), "ticks": rng.randrange(40, 101)}
    x, y, z = _dims(rng, 30_000, 192 * 160 * 96, least)
    return {"kind": kind, "x": x, "y": y, "z": z, "seeds": max(20, min(1000, x * y * z // 3000)), "at": rng.randrange(100, 301),
            "ticks": rng.randrange(80, 151)}


# ------------------------------------------------------------------ inputs ----
def _grid(case) -> tuple[int, int, int]:
    return case["x"], case["y"], case["z"]


def _capacity(dims) -> int:
    """The cell table of a run: half the grid's voxels, as the ensemble's."""
    return max(1024, math.prod(dims) // 2)


def _snapshot(dims) -> np.ndarray:
    """The caller's buffer for a run's cells, kept between read-backs."""
    return np.zeros(_capacity(dims) if math.prod(dims) <= 1 << 18 else math.prod(dims) // 8, marl.CELL_DTYPE)


def _ensemble(case, seed: int) -> list[tuple]:
    dims = [tuple(max(16, int(d * case["scale"])) for d in ENSEMBLE[r % len(ENSEMBLE)]) for r in range(case["runs"])]
    return [(d, seed * 64 + r, 30, _capacity(d)) for r, d in enumerate(dims)]


def _field(dims, seed: int) -> torch.Tensor:
    """Concentrations of 0..0.5 with more of the boundary species near their boundary, deposits in patches."""
    x, y, z = dims
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = torch.rand((z, y, x, S), generator=g, device="cuda") * 0.5
    depth = torch.linspace(0.0, 1.0, z, device="cuda").view(z, 1, 1)
    f[..., 1] *= 1.0 - depth
    f[..., 2] *= depth
    f[..., 7] *= (torch.rand((z, y, x), generator=g, device="cuda") < 0.2) * 4.0
    return f


def _occupancy(dims, seed: int, frac: float = 0.04) -> torch.Tensor:
    """About the share of occupied voxels of the default run at tick 1000."""
    x, y, z = dims
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    return (torch.rand((z, y, x), generator=g, device="cuda") < frac).to(torch.uint8)


def _mlp_params(seed: int) -> np.ndarray:
    r = np.random.default_rng(seed)
    w1 = np.zeros((HID, IN_PAD), np.float32)
    w1[:, : marl.SURR_FEATURES] = r.normal(0, 0.1, (HID, marl.SURR_FEATURES))
    parts = [w1, r.normal(0, 0.1, HID), r.normal(0, 0.06, (HID, HID)), r.normal(0, 0.1, HID),
             r.normal(0, 0.06, (OUT, HID)), r.normal(0, 0.1, OUT)]
    return np.concatenate([np.asarray(p, np.float32).ravel() for p in parts])


def _mlp_norm(seed: int) -> np.ndarray:
    r = np.random.default_rng(seed + 7)
    n = marl.SURR_FEATURES
    return np.concatenate([r.normal(0, 1, n), r.uniform(0.5, 2, n), r.normal(0, 0.1, OUT),
                           r.uniform(0.01, 0.2, OUT)]).astype(np.float32)


def _pairs(n: int, seed: int) -> np.ndarray:
    """Raw rows as the cell loop captures them: state, environment, light and kinetics, then the reactions' deltas."""
    r = np.random.default_rng(seed)
    rows = np.zeros((n, marl.SURR_RAW_STRIDE), np.float32)
    rows[:, :29] = r.random((n, 29), dtype=np.float32)
    k = rows[:, 29:93].reshape(n, 16, 4)
    k[:, :, 0] = 0.01 + 0.99 * r.random((n, 16), dtype=np.float32)
    k[:, :, 1] = np.exp(r.standard_normal((n, 16), dtype=np.float32))
    k[:, :, 2] = 0.01 + 0.99 * r.random((n, 16), dtype=np.float32)
    k[:, :, 3] = r.random((n, 16)) < 0.25
    x = rows[:, :16]
    flux = k[:, :, 1] * x / (k[:, :, 0] + x) * np.roll(x, 1, axis=1) * 0.2
    rows[:, 93:109] = np.minimum(np.roll(flux, 3, axis=1), 1.0) - np.minimum(flux, x)
    return rows


def prepare(case: dict, seed: int):
    kind = case["kind"]
    st = {"kind": kind, "case": case, "seed": seed}
    if kind in ("diffuse", "seam"):
        dims = _grid(case)
        st["dims"], st["params"] = dims, marl.default_params()
        st["field"], st["occ"] = _field(dims, seed), _occupancy(dims, seed)
        if kind == "seam":
            st["field"], st["occ"] = st["field"].cpu().numpy(), st["occ"].cpu().numpy()
            st["ctx"] = marl.Context(dims, st["params"], cell_capacity=1024)
        else:
            st["scratch"] = torch.empty_like(st["field"])
        return st
    if kind in ("seeded", "steps", "device"):
        dims = _grid(case)
        st["out"] = _snapshot(dims)
        if kind == "seeded":
            return st
        e = marl.Engine(dims, rng_seed=seed, seed_count=case.get("seeds", 30), cell_capacity=_capacity(dims))
        e.step(case["at"])
        if kind == "steps":
            st["engine"] = e
            return st
        st["field"], st["cells"] = e.field(), e.cells()
        e.close()
        st["ctx"] = marl.Context(dims, cell_capacity=_capacity(dims))
        return st
    if kind == "ensemble":
        runs = _ensemble(case, seed)
        st["batch"], st["out"] = marl.Batch(runs), [_snapshot(r[0]) for r in runs]
        st["batch"].step(case["at"])
        return st
    if kind == "infer":
        s = marl.Surrogate(max_pairs=128, batch=128)
        s.set_stream(torch.cuda.current_stream().cuda_stream)
        s.set_weights(_mlp_params(seed), _mlp_norm(seed))
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn((case["rows"], IN_PAD), generator=g, device="cuda").to(torch.bfloat16)
        x[:, marl.SURR_FEATURES:] = 0
        st["s"], st["x"], st["y"] = s, x, torch.empty((OUT, case["rows"]), device="cuda")
    if kind == "train":
        s = marl.Surrogate(max_pairs=case["pairs"], batch=case["batch"], seed=seed)
        s.upload_pairs(_pairs(case["pairs"], seed))
        s.set_weights(_mlp_params(seed))
        s.prepare(case["pairs"])
        st["s"] = s
    return st


# --------------------------------------------------------------------- run ----
def _cells(read, handle, out: np.ndarray) -> dict:
    """The cells read back into the caller's buffer: the whole records, as plain arrays (views)."""
    got = ctypes.c_uint32()
    status = read(*handle, out.ctypes.data, len(out), ctypes.byref(got))
    if status:
        raise marl.MarlError(status, "read the cells back")
    return _arrays(out)


def _arrays(cells: np.ndarray) -> dict:
    n, at = len(cells), marl.CELL_DTYPE.fields["ruleset"][1]
    ruleset = np.ndarray((n, marl.RULESET_DTYPE.itemsize), np.uint8, cells, at, (marl.CELL_DTYPE.itemsize, 1))
    return {"pos": cells["pos"].view("<i2"), "internal": cells["internal"], "ruleset": ruleset,
            "lineage": cells["lineage_id"].view("<i8"), "age": cells["age"].view("<i4"),
            "prep": cells["prep_remaining"].view("<i2"), "kind": cells["starter_type"], "quiescent": cells["quiescent"]}


def run(st):
    case, kind = st["case"], st["kind"]
    if kind == "diffuse":
        stream = torch.cuda.current_stream().cuda_stream
        if case["noalloc"]:
            marl.diffuse_device_noalloc(st["field"].data_ptr(), st["occ"].data_ptr(), st["dims"], st["params"],
                                        case["substeps"], stream)
        else:
            marl.diffuse_device(st["field"].data_ptr(), st["scratch"].data_ptr(), st["occ"].data_ptr(), st["dims"],
                                st["params"], case["substeps"], stream)
        return st["field"]
    if kind == "seam":
        st["ctx"].diffuse_tick_with_cells(st["field"], st["occ"])
        return st["field"]
    if kind in ("seeded", "steps"):
        dims = _grid(case)
        e = st.get("engine") or marl.Engine(dims, rng_seed=st["seed"], cell_capacity=_capacity(dims))
        e.step(case["ticks"])
        out = {"field": e.field(), "light": e.light(), "cells": _cells(e.lib.marl_engine_get_cells, (e.h,), st["out"])}
        if kind == "seeded":
            e.close()
        return out
    if kind == "device":
        ctx = st["ctx"]
        ctx.upload_field(st["field"])
        ctx.upload_cells(st["cells"])
        ctx.fate_init(st["seed"], case["at"])
        ctx.run_ticks(case["ticks"])
        return {"field": ctx.download_field(), "light": ctx.download_light(),
                "cells": _cells(ctx.lib.marl_download_cells, (ctx.h,), st["out"])}
    if kind == "ensemble":
        b = st["batch"]
        b.step(case["ticks"])
        out = []
        for r, buf in enumerate(st["out"]):
            c = _cells(b.lib.marl_batch_get_cells, (b.h, r), buf)
            out.append([b.field(r), b.light(r)] + [c[k] for k in ("pos", "internal", "ruleset", "lineage", "age")])
        return out
    if kind == "infer":
        n = case["rows"]
        st["s"].infer_device(st["x"].data_ptr(), n, st["y"].data_ptr(), n)
        return st["y"]
    loss = st["s"].train(case["steps"])
    return {"loss": loss, "params": st["s"].get_weights()[0]}


# ------------------------------------------------------------------- exact ----
def _exact_diffusion(field: torch.Tensor, occ: torch.Tensor, p, substeps: int) -> torch.Tensor:
    """Masked 7-point diffusion with decay; a wall or an occupied neighbour reads as the centre voxel."""
    f, wall = field.double(), occ.bool()
    d = torch.tensor([float(v) for v in p.d_voxel], dtype=torch.float64, device=f.device)
    lam = torch.tensor([float(v) for v in p.lambda_decay], dtype=torch.float64, device=f.device)
    dt = float(p.dt) / int(p.diffusion_substeps)
    for _ in range(substeps):
        niche = 1.0 - p.alpha_eps * f[..., 7] / (p.k_eps + f[..., 7])
        lap = torch.zeros_like(f)
        for axis in range(3):
            n = f.shape[axis]
            for step in (-1, 1):
                at = torch.arange(n, device=f.device) + step
                off = (at < 0) | (at >= n)
                at = at.clamp(0, n - 1)
                view = [1, 1, 1]
                view[axis] = n
                blocked = wall.index_select(axis, at) | off.view(view)
                lap += torch.where(blocked.unsqueeze(-1), f, f.index_select(axis, at)) - f
        new = (f + dt * (d * niche.unsqueeze(-1) * lap - lam * f)).clamp_min(0.0)
        f = torch.where(wall.unsqueeze(-1), f, new)
    return f


def _split(params: torch.Tensor):
    sizes = [HID * IN_PAD, HID, HID * HID, HID, OUT * HID, OUT]
    w1, b1, w2, b2, w3, b3 = torch.split(params, sizes)
    return w1.view(HID, IN_PAD), b1, w2.view(HID, HID), b2, w3.view(OUT, HID), b3


def _forward(params: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    w1, b1, w2, b2, w3, b3 = _split(params)
    h = torch.nn.functional.gelu(x @ w1.T + b1, approximate="tanh")
    h = torch.nn.functional.gelu(h @ w2.T + b2, approximate="tanh")
    return h @ w3.T + b3


def _mix64(z: np.ndarray) -> np.ndarray:
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _exact_train(case, seed: int) -> dict:
    """The same steps in 64 bits: standardised pairs, the library's batch draws, MSE, Adam."""
    rows = _pairs(case["pairs"], seed).astype(np.float64)
    feats = rows[:, :93].copy()
    logs = [29 + 4 * r + i for r in range(16) for i in range(3)]
    feats[:, logs] = np.log(np.abs(feats[:, logs]) + 1e-3)
    cols = np.concatenate([feats, rows[:, 93:109]], axis=1)
    sd = cols.std(axis=0)
    cols = (cols - cols.mean(axis=0)) / np.where(sd > 1e-6, sd, 1.0)
    x = torch.zeros((len(rows), IN_PAD), dtype=torch.float64, device="cuda")
    x[:, :93] = torch.from_numpy(cols[:, :93]).cuda()
    t = torch.from_numpy(cols[:, 93:]).cuda()
    p = torch.from_numpy(_mlp_params(seed)).double().cuda().requires_grad_()
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    lr, b1, b2, eps = 1e-3, 0.9, 0.999, 1e-8
    r = np.arange(case["batch"], dtype=np.uint64)
    with np.errstate(over="ignore"):
        for i in range(case["steps"]):
            at = _mix64(np.uint64(seed) ^ _mix64(np.uint64(i) * np.uint64(0x100000001B3) + r)) % np.uint64(len(rows))
            at = torch.from_numpy(at.astype(np.int64)).cuda()
            loss = ((_forward(p, x[at]) - t[at]) ** 2).mean()
            (g,) = torch.autograd.grad(loss, p)
            losses.append(float(loss.detach()))
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            with torch.no_grad():
                p -= lr * (m / (1 - b1 ** (i + 1))) / ((v / (1 - b2 ** (i + 1))).sqrt() + eps)
    return {"loss": np.array(losses), "params": p.detach()}


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("diffuse", "seam"):
        dims, p = _grid(case), marl.default_params()
        return _exact_diffusion(_field(dims, seed), _occupancy(dims, seed), p,
                                case.get("substeps", int(p.diffusion_substeps)))
    if kind == "infer":
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn((case["rows"], IN_PAD), generator=g, device="cuda").to(torch.bfloat16)
        x[:, marl.SURR_FEATURES:] = 0
        norm = torch.from_numpy(_mlp_norm(seed)).double().cuda()
        y = _forward(torch.from_numpy(_mlp_params(seed)).double().cuda(), x.double())
        return (y * norm[-OUT:] + norm[-2 * OUT:-OUT]).T.contiguous()
    if kind == "train":
        return _exact_train(case, seed)
    return None  # hundreds of ticks of the sequential cell loop: far over 20 seconds in 64 bits


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "infer":
        n = case["rows"]
        return {"bytes": n * (2 * IN_PAD + 4 * OUT) + 2 * marl.SURR_PARAMS,
                "flops": 2.0 * n * (93 * HID + HID * HID + HID * OUT)}
    if kind == "train":
        n = case["batch"] * case["steps"]
        return {"bytes": n * (2 * IN_PAD + 4 * OUT) + 2 * 4 * marl.SURR_PARAMS,
                "flops": 6.0 * n * (93 * HID + HID * HID + HID * OUT)}
    if kind == "ensemble":
        v = sum(math.prod(r[0]) for r in _ensemble(case, 0))
    else:
        v = case["x"] * case["y"] * case["z"]
    ticks = case.get("ticks", 1)
    substeps = case.get("substeps", 10)
    # Field in and out once (and the mask, or the light out); 18 operations per species, voxel and substep.
    return {"bytes": v * (2 * 4 * S + (1 if kind in ("diffuse", "seam") else 4)),
            "flops": 18.0 * S * v * substeps * ticks}
