"""The work that users of this framework have it do, as measurable cases.

Five kinds, each through the package's public entry points:

  search  the neighbour-search building blocks on their own: the stable radix
          sort of cell keys and the cell start/end finder (the reference's
          RadixSort and NeighbourCellFinder)
  step    one scene: upload a state, advance it some substeps, read it back
  batch   many independent scenes in one handle, the same round trip
  train   forward and backward of whole substeps through the autograd
          function: final state, loss gradients of the initial state and of
          the scalar parameters
  splat   the depth and thickness images of a particle set

Sizes are those of the repository's scenes (16,384, 32,768, 65,536 and
2,097,152 particles, batches of 256 and 64 scenes), the tests' odd sizes and
lattices with odd sides.
"""
from __future__ import annotations

import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import pbf_gb300 as pg
from pbf_gb300 import _capi, autograd, scenes, splat

SPACING = scenes.SPACING


def listed():
    return [
        # one small scene's neighbour search, where launches and waits count
        {"name": "search_16k", "kind": "search", "n": 16384, "grid_x": 64, "grid_y": 64,
         "grid_z": 64},
        # a large cloud's neighbour search, an odd number of particles
        {"name": "search_4m", "kind": "search", "n": 4194301, "grid_x": 257, "grid_y": 129,
         "grid_z": 257},
        # the small plain dam break: a handful of substeps from its start
        step_case("dam_16k", (32, 16, 32), (64, 64, 64), 3, 0.01, 4),
        # the same run well into its collapse (piles of coincident particles),
        # where most of its 200 substeps' time goes
        step_case("dam_16k_late", (32, 16, 32), (64, 64, 64), 3, 0.01, 4, start=96),
        # the reference application's own scene and defaults (support of two
        # cells, five iterations, no vorticity confinement)
        {"name": "two_blocks_65k", "kind": "step", "scene": "two_blocks", "substeps": 8},
        # a mid-size scene with odd lattice sides, the stable relaxation and
        # moving particles
        step_case("dam_250k", (63, 65, 61), (101, 67, 97), 4, 5.0, 8, vel=0.25),
        # the large dam break: the benchmark's window of 20 substeps
        step_case("dam_2m", (128, 128, 128), (256, 128, 256), 4, 0.01, 20),
        # the 256-scene batch of uneven scenes (9.3 million particles)
        batch_case("batch_256", 256, 4096, 65536, 32, 96, 4, 0.01, 4),
        # one training step of the differentiable scene: two checkpoint segments
        train_case("train_32k", 1, 32768, 32768, 64, 64, 4, 16, 8),
        # one training step of the batched parameter recovery
        train_case("train_64_scenes", 64, 8192, 32768, 48, 80, 4, 16, 8),
        # the reference application's two particle passes over its own scene
        {"name": "splat_65k", "kind": "splat", "lattice_x": 64, "lattice_y": 32, "lattice_z": 32,
         "spacing": 0.94, "width": 1280, "height": 720, "thick_width": 512, "thick_height": 512},
        # the same passes over a million particles, full-HD images
        {"name": "splat_1m", "kind": "splat", "lattice_x": 128, "lattice_y": 61,
         "lattice_z": 134, "spacing": 0.5, "width": 1920, "height": 1080, "thick_width": 960,
         "thick_height": 540},
    ]


def step_case(name, lattice, box, iterations, epsilon, substeps, vel=0.0, start=0, vorticity=True):
    c = {"kind": "step", "scene": "block", "lattice_x": lattice[0], "lattice_y": lattice[1],
         "lattice_z": lattice[2], "box_x": box[0], "box_y": box[1], "box_z": box[2],
         "iterations": iterations, "epsilon": epsilon, "substeps": substeps, "vel": vel,
         "start": start, "vorticity": vorticity}
    return {"name": name, **c} if name else c


def batch_case(name, num, nmin, nmax, box_min, box_max, iterations, epsilon, substeps, spec=7):
    c = {"kind": "batch", "scenes": num, "nmin": nmin, "nmax": nmax, "box_min": box_min,
         "box_max": box_max, "iterations": iterations, "epsilon": epsilon, "substeps": substeps,
         "spec": spec}
    return {"name": name, **c} if name else c


def train_case(name, num, nmin, nmax, box_min, box_max, iterations, substeps, every, spec=11):
    c = batch_case(name, num, nmin, nmax, box_min, box_max, iterations, 5.0, substeps, spec)
    return {**c, "kind": "train", "every": every}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "step", "step", "step", "batch", "train", "splat"])
    if kind == "search":
        n = _log(rng, 1000, 6_000_000)
        side = max(4, int(round((2.0 * n) ** (1 / 3))))
        return {"kind": kind, "n": n, "grid_x": side + rng.randrange(7),
                "grid_y": max(2, side // 2 + rng.randrange(5)), "grid_z": side + rng.randrange(9)}
    if kind == "step":
        n = _log(rng, 2000, 1_500_000)
        lat = [max(4, int(round(n ** (1 / 3) * rng.uniform(0.7, 1.4)))) for _ in range(3)]
        box = [int(math.ceil(SPACING * l)) + rng.randrange(3, 4 + l) for l in lat]
        total, eps = lat[0] * lat[1] * lat[2], rng.choice([0.01, 5.0])
        late = rng.choice([0, 40, 100]) if total < 20_000 and eps < 1.0 else 0
        return step_case(None, lat, box, rng.randrange(2, 6), eps,
                         rng.randrange(1, 9) if total < 400_000 else rng.randrange(1, 5),
                         vel=rng.choice([0.0, 0.25]), start=late, vorticity=rng.random() < 0.8)
    if kind == "batch":
        lo = _log(rng, 500, 8000)
        return batch_case(None, rng.randrange(3, 100), lo, lo * rng.randrange(2, 7), 24,
                          rng.randrange(40, 97), rng.randrange(2, 5), rng.choice([0.01, 5.0]),
                          rng.randrange(1, 5), rng.randrange(1000))
    if kind == "train":
        if rng.random() < 0.5:
            n = _log(rng, 2000, 80_000)
            return train_case(None, 1, n, n, 40, rng.randrange(60, 90), rng.randrange(2, 5),
                              rng.randrange(3, 13), rng.randrange(2, 9), rng.randrange(1000))
        lo = _log(rng, 1000, 8000)
        return train_case(None, rng.randrange(2, 33), lo, lo * 3, 40, 80, rng.randrange(2, 5),
                          rng.randrange(3, 9), rng.randrange(2, 5), rng.randrange(1000))
    n = _log(rng, 4000, 1_000_000)
    lat = [max(3, int(round(n ** (1 / 3) * rng.uniform(0.6, 1.5)))) for _ in range(3)]
    return {"kind": "splat", "lattice_x": lat[0], "lattice_y": lat[1], "lattice_z": lat[2],
            "spacing": rng.choice([0.5, 0.94]), "width": rng.randrange(320, 1921),
            "height": rng.randrange(240, 1081), "thick_width": rng.randrange(256, 1025),
            "thick_height": rng.randrange(256, 1025)}


# ---- inputs -----------------------------------------------------------------

def _block(gen, lattice, spacing=SPACING, jitter=0.01, vel=0.0, origin=None):
    """A jittered lattice block (id order x outermost, then z, then y) and
    uniform velocities, as float4 tensors on the GPU."""
    dev = gen.device
    ii, kk, jj = torch.meshgrid(*(torch.arange(lattice[a], device=dev) for a in (0, 2, 1)),
                                indexing="ij")
    idx = torch.stack([ii.reshape(-1), jj.reshape(-1), kk.reshape(-1)], 1).double()
    at = torch.tensor(origin or (0.5 * spacing,) * 3, device=dev, dtype=torch.float64)
    n = idx.shape[0]
    jit = (torch.rand((n, 3), generator=gen, device=dev, dtype=torch.float64) * 2 - 1) * jitter
    x = torch.zeros((n, 4), device=dev)
    x[:, :3] = (at + idx * spacing + jit).float()
    v = torch.zeros((n, 4), device=dev)
    if vel:
        v[:, :3] = (torch.rand((n, 3), generator=gen, device=dev) * 2 - 1) * vel
    return x, v


def _two_blocks(gen):
    """The reference application's start: two 32^3 blocks of spacing 0.94 in
    opposite corners (scenes.reference_two_blocks, jitter from this seed)."""
    a, _ = _block(gen, (32, 32, 32), 0.94, 0.005, origin=(32.5, 0.5, 32.5))
    b, _ = _block(gen, (32, 32, 32), 0.94, 0.005, origin=(95.5, 0.5, 95.5))
    for axis in (0, 2):
        b[:, axis] = 2 * 95.5 - b[:, axis]
    x = torch.cat([a, b])
    return x, torch.zeros_like(x)


def _params(case):
    if case.get("scene") == "two_blocks":
        p = pg.default_params((128, 64, 128))
        p.h = 2.0
        p.tensile_instability_scale = float(np.float32(1.0 / scenes.wpoly6(0.2, 2.0)))
        return p
    return scenes.dam_params([case["box_x"], case["box_y"], case["box_z"]], case["iterations"],
                             epsilon=case["epsilon"], vorticity=case["vorticity"])


def _state(case, gen):
    if case.get("scene") == "two_blocks":
        return _two_blocks(gen)
    return _block(gen, [case["lattice_x"], case["lattice_y"], case["lattice_z"]],
                  vel=case["vel"])


def _scene_specs(case):
    specs = scenes.batch_scene_specs(case["scenes"], case["spec"], case["nmin"], case["nmax"],
                                     case["box_min"], case["box_max"])
    params = [scenes.dam_params(s["box"], case["iterations"], epsilon=case["epsilon"])
              for s in specs]
    counts = [s["lattice"][0] * s["lattice"][1] * s["lattice"][2] for s in specs]
    return specs, params, counts


def _scene_states(specs, gen, vel):
    xs, vs = zip(*(_block(gen, s["lattice"], vel=vel) for s in specs))
    return torch.cat(xs), torch.cat(vs)


def _handle(params, counts):
    if len(params) == 1:
        return pg.SPH(counts[0], tuple(params[0].grid), params[0])
    return pg.SPHBatch(params, counts)


def _advance(sim, x, v, substeps, xo, vo):
    sim.set_state_device(x.data_ptr(), v.data_ptr())
    sim.step(substeps)
    sim.get_state_into(xo.data_ptr(), vo.data_ptr(), pg.PBF_DEVICE)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    if kind == "search":
        # particles anywhere in the lower left of the grid, ids in no spatial order
        g = [case["grid_x"], case["grid_y"], case["grid_z"]]
        r = torch.rand((case["n"], 3), generator=gen, device="cuda")
        c = (r * torch.tensor([0.6 * s for s in g], device="cuda")).to(torch.int64)
        keys = (c[:, 0] + c[:, 1] * (g[0] * g[2]) + c[:, 2] * g[0]).to(torch.int32)
        cells = g[0] * g[1] * g[2]
        new = lambda k: torch.empty(k, dtype=torch.int32, device="cuda")  # noqa: E731
        return {"kind": kind, "lib": pg.load(), "n": case["n"], "cells": cells, "keys": keys,
                "bits": int(cells - 1).bit_length(), "sorted": new(case["n"]),
                "perm": new(case["n"]), "start": new(cells), "end": new(cells)}
    if kind == "splat":
        x, _ = _block(gen, [case["lattice_x"], case["lattice_y"], case["lattice_z"]],
                      case["spacing"], origin=(32.5, 0.5, 32.5))
        return {"kind": kind, "x": x, "view": splat.reference_view(case["width"], case["height"]),
                "depth": (case["width"], case["height"]),
                "thick": (case["thick_width"], case["thick_height"])}
    if kind == "step":
        x, v = _state(case, gen)
        params, counts = [_params(case)], [x.shape[0]]
    else:
        specs, params, counts = _scene_specs(case)
        x, v = _scene_states(specs, gen, 0.5 if kind == "batch" else 0.25)
    sim = _handle(params, counts)
    torch.cuda.synchronize()
    if kind == "train":
        # the target: the final positions of the same start with other velocities
        _, vb = _scene_states(specs, gen, 0.25)
        target = torch.empty_like(x)
        _advance(sim, x, vb, case["substeps"], target, vb)
        return {"kind": kind, "sim": sim, "x": x.requires_grad_(True), "v": v.requires_grad_(True),
                "theta": autograd.theta_of(sim).requires_grad_(True), "target": target,
                "substeps": case["substeps"], "every": case["every"]}
    if case.get("start"):  # a state from later in the run
        _advance(sim, x, v, case["start"], x, v)
    return {"kind": kind, "sim": sim, "x": x, "v": v, "substeps": case["substeps"],
            "xo": torch.empty_like(x), "vo": torch.empty_like(v)}


def run(state):
    kind = state["kind"]
    if kind == "search":
        s, lib = state, state["lib"]
        st = torch.cuda.current_stream().cuda_stream or None
        _capi.check(lib.pbf_radix_sort(s["keys"].data_ptr(), s["sorted"].data_ptr(),
                                       s["perm"].data_ptr(), s["n"], s["bits"], st))
        _capi.check(lib.pbf_find_cells(s["sorted"].data_ptr(), s["n"], s["cells"],
                                       s["start"].data_ptr(), s["end"].data_ptr(), st))
        return {k: s[k] for k in ("sorted", "perm", "start", "end")}
    if kind == "splat":
        return {"depth": splat.splat(splat.DEPTH, state["x"], state["view"], *state["depth"]),
                "thickness": splat.splat(splat.THICKNESS, state["x"], state["view"],
                                         *state["thick"])}
    if kind == "train":
        s = state
        x, v = autograd.run(s["sim"], s["x"], s["v"], s["theta"], s["substeps"], s["every"])
        loss = ((x - s["target"])[:, :3] ** 2).sum(1).mean()
        gx, gv, gt = torch.autograd.grad(loss, (s["x"], s["v"], s["theta"]))
        return {"x": x.detach(), "v": v.detach(), "loss": loss.detach(), "grad_x": gx,
                "grad_v": gv, "grad_theta": gt}
    _advance(state["sim"], state["x"], state["v"], state["substeps"], state["xo"], state["vo"])
    return {"x": state["xo"], "v": state["vo"]}


# ---- what a pass cannot do without -------------------------------------------

# FP32 operations of one in-range neighbour pair, an fma counted as two:
# density and constraint gradient; position correction; XSPH and vorticity;
# confinement
PAIR_FLOPS = {"lambda": 37, "delta_p": 38, "vort_a": 46, "vort_b": 26}


def _pairs_per_particle(h, spacing):
    m = int(h / spacing) + 1
    r = range(-m, m + 1)
    return sum(1 for a in r for b in r for c in r
               if 0 < (a * a + b * b + c * c) * spacing * spacing <= h * h)


def work(case):
    kind = case["kind"]
    if kind == "search":
        cells = case["grid_x"] * case["grid_y"] * case["grid_z"]
        return {"bytes": 12 * case["n"] + 8 * cells, "flops": 0}
    if kind == "splat":
        n = case["lattice_x"] * case["lattice_y"] * case["lattice_z"]
        px = case["width"] * case["height"] + case["thick_width"] * case["thick_height"]
        return {"bytes": 2 * 16 * n + 4 * px, "flops": 2 * 150 * n}
    if kind == "step" and case["scene"] == "two_blocks":
        n, iters, vort, pairs = 65536, 5, False, _pairs_per_particle(2.0, 0.94)
    else:
        pairs = _pairs_per_particle(1.0, SPACING)
        iters, vort = case["iterations"], case.get("vorticity", True)
        if kind == "step":
            n = case["lattice_x"] * case["lattice_y"] * case["lattice_z"]
        else:
            n = sum(_scene_specs(case)[2])
    f = PAIR_FLOPS
    per_pair = iters * (f["lambda"] + f["delta_p"])
    if vort:
        per_pair += f["vort_a"] + f["vort_b"]
    flops = float(n) * case["substeps"] * pairs * per_pair
    if kind == "train":  # the reverse of each pair term costs about twice the term
        return {"bytes": 5 * 32 * n, "flops": 3 * flops}
    return {"bytes": 64 * n, "flops": flops}


# ---- the same substeps in 64 bits ----------------------------------------------

def _substep64(p, theta, x, v):
    """One substep of the scene with parameters p in float64 torch operations:
    x, v (n, 3) in id order, theta = (epsilon, s_corr k, XSPH c, vorticity
    epsilon); differentiable with the sort and the candidates held fixed."""
    h, dt, oorho = p.h, p.timestep, p.one_over_rho_0
    grid = [int(g) for g in p.grid]
    k6 = 1.56668147106 / h ** 9
    kg = -3.0 * 4.774648292756860 / h ** 6
    lo = torch.tensor(list(p.wall_lo), device=x.device, dtype=torch.float64)
    hi = torch.tensor(list(p.wall_hi), device=x.device, dtype=torch.float64)
    fall = torch.tensor([0.0, p.gravity * dt, 0.0], device=x.device, dtype=torch.float64)
    xs = x + dt * (v - fall)
    with torch.no_grad():
        # candidates: the 3x3x3 cells around each predicted position, row by row
        cell = torch.stack([xs[:, a].clamp(0, grid[a] - 1).floor() for a in range(3)], 1).long()
        key = cell[:, 0] + cell[:, 1] * (grid[0] * grid[2]) + cell[:, 2] * grid[0]
        skey, order = torch.sort(key, stable=True)
        centre = xs.detach().trunc().long()
        me = torch.arange(x.shape[0], device=x.device)
        cand = []
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                cy, cz = centre[:, 1] + dy, centre[:, 2] + dz
                x0, x1 = (centre[:, 0] - 1).clamp(min=0), (centre[:, 0] + 1).clamp(max=grid[0] - 1)
                ok = (cy >= 0) & (cy < grid[1]) & (cz >= 0) & (cz < grid[2]) & (x1 >= x0)
                base = cy * (grid[0] * grid[2]) + cz * grid[0]
                b = torch.searchsorted(skey, base + x0)
                cnt = (torch.searchsorted(skey, base + x1, right=True) - b).clamp(min=0) * ok
                i = torch.repeat_interleave(me, cnt)
                first = torch.repeat_interleave(b - (torch.cumsum(cnt, 0) - cnt), cnt)
                j = order[first + torch.arange(i.shape[0], device=x.device)]
                cand.append((i, j))

    def pairs(q):
        with torch.no_grad():
            kept = []
            for i, j in cand:
                r2 = ((q[i] - q[j]) ** 2).sum(1)
                keep = (r2 <= h * h) & (i != j)
                kept.append((i[keep], j[keep]))
            i, j = torch.cat([a for a, _ in kept]), torch.cat([b for _, b in kept])
        d = q[i] - q[j]
        r2 = (d * d).sum(1)
        away = r2 > 0
        r = torch.sqrt(torch.where(away, r2, torch.ones_like(r2))) * away
        w = k6 * (h * h - r2) ** 3
        s = torch.where(away, kg * (h - r) ** 2 / torch.where(away, r, torch.ones_like(r)),
                        torch.zeros_like(r))
        return i, j, w, s[:, None] * d

    def total(i, t):
        return torch.zeros((x.shape[0],) + t.shape[1:], device=x.device,
                           dtype=torch.float64).index_add(0, i, t)

    def length(t):
        n2 = (t * t).sum(1)
        some = n2 > 0
        return torch.sqrt(torch.where(some, n2, torch.ones_like(n2))) * some

    q = xs
    for _ in range(int(p.num_solver_iterations)):
        i, j, w, g = pairs(q)
        c = total(i, w) * oorho - 1.0
        gi = total(i, g) * oorho
        lam = -c / (total(i, ((g * oorho) ** 2).sum(1)) + (gi * gi).sum(1) + theta[0])
        s = -theta[1] * (p.tensile_instability_scale * w) ** 4
        dp = total(i, (lam[i] + lam[j] + s)[:, None] * g)
        q = torch.minimum(torch.maximum(q + oorho * dp, lo), hi)
    v1 = (q - x) / dt
    if not p.vorticity_confinement:
        return q, v1
    i, j, w, g = pairs(q)
    vij = v1[j] - v1[i]
    vx = v1 + theta[2] * total(i, w[:, None] * vij)
    om = total(i, torch.linalg.cross(vij, g))
    eta = total(i, length(om)[j][:, None] * g)
    le = length(eta)
    unit = eta / torch.where(le > 0, le, torch.ones_like(le))[:, None]
    return q, vx + dt * theta[3] * torch.linalg.cross(unit, om)


def _run64(p, theta, x, v, substeps, grads):
    for _ in range(substeps):
        if grads:
            x, v = checkpoint(_substep64, p, theta, x, v, use_reentrant=False)
        else:
            x, v = _substep64(p, theta, x, v)
    return x, v


def _four(t):
    return torch.cat([t, torch.zeros_like(t[:, :1])], 1)


def exact(case, seed):
    """run()'s outputs in 64 bits: the sort and the cells as plain integer
    operations, the substeps and their gradients as float64 torch operations.

    None for the images (which pixels a sprite covers is decided by the
    rounding rules, so the images have no value apart from them), for the runs
    with epsilon = 0.01 (unstable: 32-bit and 64-bit trajectories part within
    three substeps) and for batches too large to redo scene by scene."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    if kind == "search":
        s = prepare(case, seed)
        keys, order = torch.sort(s["keys"], stable=True)
        cells = torch.arange(s["cells"], device="cuda", dtype=torch.int32)
        b = torch.searchsorted(keys, cells).int()
        e = torch.searchsorted(keys, cells, right=True).int()
        none = b == e
        return {"sorted": keys, "perm": order.int(), "start": torch.where(none, -1, b),
                "end": torch.where(none, -1, e)}
    if kind == "splat":
        return None
    if kind == "step":
        if case["scene"] == "block" and case["epsilon"] < 1.0:
            return None
        x, v = _state(case, gen)
        params, counts = [_params(case)], [x.shape[0]]
    else:
        specs, params, counts = _scene_specs(case)
        if case["epsilon"] < 1.0 or len(counts) > 8:
            return None
        x, v = _scene_states(specs, gen, 0.5 if kind == "batch" else 0.25)
    train = kind == "train"
    if train:
        target = prepare(case, seed)["target"].double()  # an input: any positions would do
    theta = torch.tensor([[getattr(p, nm) for nm in autograd.PARAMS] for p in params],
                         device="cuda", dtype=torch.float64, requires_grad=train)
    x64 = x[:, :3].double().requires_grad_(train)
    v64 = v[:, :3].double().requires_grad_(train)
    outs, at = [], 0
    for k, (p, n) in enumerate(zip(params, counts)):
        outs.append(_run64(p, theta[k], x64[at:at + n], v64[at:at + n], case["substeps"], train))
        at += n
    xe, ve = (torch.cat([o[a] for o in outs]) for a in (0, 1))
    if not train:
        return {"x": _four(xe), "v": _four(ve)}
    loss = ((xe - target[:, :3]) ** 2).sum(1).mean()
    gx, gv, gt = torch.autograd.grad(loss, (x64, v64, theta))
    return {"x": _four(xe.detach()), "v": _four(ve.detach()), "loss": loss.detach(),
            "grad_x": _four(gx), "grad_v": _four(gv), "grad_theta": gt.cpu()}
