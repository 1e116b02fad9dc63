"""The work that programs built on gvdb2 have it do, as cases that can be
prepared, run and checked one by one.

Each case is one pass of a user's loop through gvdb2.VolumeGVDB: a dynamic
step (rebuild, splat, apron, gather), a few frames of the incremental state
machine, a step of differentiable splatting, many clouds in one volume, a
large sparse scene with its adjoint, a fluid's level set, the reference's
density path, and the NanoVDB-form export of a volume.  Inputs are made on
the GPU from a seed; `exact` restates every pass in 64 bits with torch alone.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gvdb-voxels_b200"))

import gvdb2  # noqa: E402

RADIUS = 2.0   # activation radius of every rebuild, in voxels
APRON = 1
BOX = 2 + 4    # an activation box reaches RADIUS below a point's voxel and 2 * RADIUS above it
SUBCELL = 4    # subcell edge of the level-set and density gathers
FRAME_SHIFT = (3.0, -1.5, 2.0)  # voxels a block moves per frame, besides its points' own velocities
DT = 0.1
TAPS = {"tent": 2, "cubic": 4}


def listed():
    return [
        # the smallest step anyone runs: a preview or a unit of a larger program, all launches and waits
        {"name": "step_20k", "kind": "step", "cloud": "shell", "n": 20_000, "kernel": "tent", "channels": 1,
         "brick": 3, "deterministic": False},
        # a density field of a million surface points
        {"name": "step_1m", "kind": "step", "cloud": "shell", "n": 1_000_000, "kernel": "tent", "channels": 1,
         "brick": 3, "deterministic": False},
        # the dynamic step of a large particle simulation: mass and momentum out, velocity back
        {"name": "step_16m", "kind": "step", "cloud": "block", "nx": 256, "ny": 256, "nz": 256, "dy": 0.5,
         "kernel": "cubic", "channels": 4, "brick": 3, "deterministic": False},
        # a smaller simulation that lets the topology follow its points, a rebuilt frame and two incremental ones
        {"name": "frames_4m", "kind": "frames", "nx": 256, "ny": 64, "nz": 256, "dy": 2.0, "kernel": "cubic",
         "channels": 4, "frames": 3},
        # an optimiser's iteration: splat, loss against a target, adjoints; the topology stays
        {"name": "diff_1m", "kind": "diff", "cloud": "shell", "n": 1_000_000, "kernel": "tent", "channels": 1,
         "brick": 3, "deterministic": False},
        # the same with weighted vector attributes, bit-reproducible, on a cloud with a dense middle
        {"name": "diff_300k", "kind": "diff", "cloud": "blob", "n": 300_007, "sigma": 24.0, "kernel": "cubic",
         "channels": 3, "brick": 3, "deterministic": True},
        # a training batch: clouds of very different sizes in one volume, forward and adjoint
        {"name": "batch_24", "kind": "batch", "clouds": 24, "smallest": 10_000, "largest": 1_000_000,
         "kernel": "cubic"},
        # a large sparse scene in 32^3 bricks, forward and adjoint over 8 channels
        {"name": "sparse_16m", "kind": "sparse", "n": 16_777_216, "blobs": 8, "space": 2048, "brick": 5},
        # the surface of a fluid of 1.5 million particles
        {"name": "surface_1m5", "kind": "surface", "nx": 128, "ny": 96, "nz": 122, "dy": 1.0, "fp16": False},
        # a small fluid with 16-bit lists
        {"name": "surface_200k", "kind": "surface", "nx": 61, "ny": 55, "nz": 61, "dy": 1.0, "fp16": True},
        # the reference's own density path over a dense block
        {"name": "density_4m", "kind": "density", "nx": 256, "ny": 64, "nz": 256, "dy": 2.0},
        # a velocity volume handed to a renderer or written out
        {"name": "export_4m", "kind": "export", "nx": 256, "ny": 64, "nz": 256, "dy": 2.0, "channels": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_block(rng, most):
    n = _log(rng, 40_000, most)
    dy = rng.choice([0.5, 1.0, 2.0])
    nx, nz = (max(24, min(256, round(n ** (1 / 3) * rng.uniform(0.7, 1.4)))) for _ in range(2))
    return {"nx": nx, "ny": max(8, min(256, round(n / nx / nz))), "nz": nz, "dy": dy}


def draw(rng):
    kind = rng.choice(["step", "step", "frames", "diff", "batch", "sparse", "surface", "density", "export"])
    c = {"kind": kind}
    if kind in ("step", "diff"):
        cloud = rng.choice(["shell", "blob", "block"] if kind == "step" else ["shell", "blob"])
        c["cloud"] = cloud
        if cloud == "block":
            c.update(_draw_block(rng, 12_000_000))
        else:
            c["n"] = _log(rng, 5_000, 4_000_000)
            if cloud == "blob":
                c["sigma"] = round(rng.uniform(8.0, 64.0), 2)
        c.update(kernel=rng.choice(["tent", "cubic"]), channels=rng.choice([1, 4] if kind == "step" else [1, 2, 3]),
                 brick=rng.choice([3, 3, 3, 4, 5]), deterministic=rng.random() < 0.25)
    elif kind == "batch":
        c.update(clouds=rng.randint(3, 24), smallest=_log(rng, 3_000, 30_000), largest=_log(rng, 50_000, 1_000_000),
                 kernel=rng.choice(["tent", "cubic"]))
    elif kind == "sparse":
        c.update(n=_log(rng, 500_000, 12_000_000), blobs=rng.randint(2, 8), space=2048, brick=rng.choice([4, 5]))
    else:
        c.update(_draw_block(rng, 4_000_000))
        if kind == "frames":
            c.update(kernel=rng.choice(["tent", "cubic"]), channels=rng.choice([1, 4]), frames=rng.randint(2, 4))
        elif kind == "surface":
            c["fp16"] = rng.random() < 0.5
        elif kind == "export":
            c["channels"] = rng.choice([1, 3])
    return c


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def _rng(seed):
    return torch.Generator("cuda").manual_seed(int(seed))


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda")


def _shell(g, n, r_in=96.0, r_out=100.0, center=128.0):
    u = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    r = (r_in ** 3 + u * (r_out ** 3 - r_in ** 3)) ** (1.0 / 3.0)
    d = _normal(g, n, 3).double()
    return (center + d / d.norm(dim=1, keepdim=True) * r[:, None]).float()


def _block(g, c):
    """Jittered lattice points, x fastest, at spacing (1, dy, 1) from (64, 64, 64)."""
    z, y, x = torch.meshgrid(*(torch.arange(c[k], device="cuda", dtype=torch.float32) for k in ("nz", "ny", "nx")),
                             indexing="ij")
    p = torch.stack([x.reshape(-1) + 0.5, (y.reshape(-1) + 0.5) * c["dy"], z.reshape(-1) + 0.5], 1) + 64.0
    return p + (torch.rand(p.shape, generator=g, device="cuda") * 0.2 - 0.1)


def _blob(g, n, sigma, center=512.0, space=1024.0):
    return (_normal(g, n, 3) * sigma + center).clamp_(0.0, space - 1.0)


def _points(g, c):
    if c.get("cloud") == "shell":
        return _shell(g, c["n"])
    if c.get("cloud") == "blob":
        return _blob(g, c["n"], c["sigma"])
    return _block(g, c)


def _batch_shapes(c):
    """(points, sigma) of each cloud: sizes evenly spread on a log scale, widths in another order."""
    k = c["clouds"]
    t = [i / max(1, k - 1) for i in range(k)]
    return [(int(c["smallest"] * (c["largest"] / c["smallest"]) ** t[i]), 8.0 + 56.0 * t[i * 7 % k]) for i in range(k)]


def _mixture(g, c):
    """Equal Gaussian blobs of widths 8 to 64 with random centres, in random order."""
    k = torch.randint(0, c["blobs"], (c["n"],), generator=g, device="cuda")
    mean = torch.rand((c["blobs"], 3), generator=g, device="cuda") * (c["space"] - 800.0) + 400.0
    sigma = torch.linspace(8.0, 64.0, c["blobs"], device="cuda")
    return (mean[k] + _normal(g, c["n"], 3) * sigma[k][:, None]).clamp_(8.0, c["space"] - 8.0)


def _in_voxels(g, p):
    """Points at new places in the voxels of p."""
    return p.floor() + (torch.rand(p.shape, generator=g, device="cuda") * 0.998 + 0.001)


def _inputs(c, seed):
    """The input tensors of a case, from the seed.  Which voxels hold points is the case's own, so that its bricks, and
    with them the shapes of its results, are the same for every seed; the seed gives the places in them and the values."""
    g, where = _rng(seed), _rng(1)
    kind = c["kind"]
    if kind == "batch":
        return {"clouds": [_in_voxels(g, _blob(where, n, s)) for n, s in _batch_shapes(c)]}
    if kind == "sparse":
        pos = _in_voxels(g, _mixture(where, c))
    elif "cloud" in c and c["cloud"] != "block":
        pos = _in_voxels(g, _points(where, c))
    else:
        pos = _block(g, c)
    n = pos.shape[0]
    d = {"pos": pos}
    if kind in ("step", "frames", "export") and c["channels"] > 1 or kind == "sparse":
        d["vel"] = _normal(g, n, 3) * (2.0 if kind == "sparse" else 1.0)
    if kind == "frames":
        v = torch.tensor(FRAME_SHIFT, device="cuda") + DT * _normal(where, n, 3)
        d["frames"] = [pos] + [_in_voxels(g, _block(where, c) + k * v) for k in range(1, c["frames"])]
    if kind == "diff":
        # a wider, sparser version of the cloud is the target
        if c["cloud"] == "shell":
            d["target"] = _shell(g, n, 90.0, 104.0)
        else:
            d["target"] = _blob(g, n, 1.2 * c["sigma"])
        d["weight"] = torch.rand(n, generator=g, device="cuda") + 0.5
        d["attr"] = _normal(g, n, c["channels"])
        d["target_attr"] = _normal(g, n, c["channels"])
        d["grad_out"] = _normal(g, n, c["channels"])
    if kind == "sparse":
        d["grad_out"] = _normal(g, n, 3)
    return d


def _volume(c):
    v = gvdb2.VolumeGVDB(0)
    kind = c["kind"]
    channels = {"diff": 3 * c.get("channels", 1), "batch": 2, "sparse": 8, "surface": 1, "density": 2}.get(kind)
    if kind == "surface":
        v.Configure(3, 3, 3, 3, 5)  # gFluidSurface's 32^3 bricks
    else:
        v.Configure(3, 3, 3, {3: 3, 4: 4, 5: 4}[c.get("brick", 3)], c.get("brick", 3))
    for k in range(channels or c["channels"]):
        v.AddChannel(k, gvdb2.T_FLOAT, APRON)
    if c.get("deterministic"):
        v.SetDeterministic(True)
    return v


def _kernel(c):
    return gvdb2.KERNEL_TENT1 if c.get("kernel") == "tent" else gvdb2.KERNEL_CUBIC2


def _momentum(vel):
    """Attributes of a mass-and-momentum splat: the weight, then the weight times each velocity component."""
    return [None, (vel, 0), (vel, 1), (vel, 2)]


def _step(v, c, s, pos, full):
    """One dynamic step; returns the gathered velocities (or densities)."""
    n, ch = pos.shape[0], c["channels"]
    v.SetPoints(pos)
    if full:
        v.RequestFullRebuild(True)
    v.RebuildTopology(n, RADIUS)
    v.UpdateAtlas()
    v.ScatterKernel(_kernel(c), n, list(range(ch)), weight=1.0, attrs=_momentum(s["vel"]) if ch == 4 else None)
    v.UpdateApron(-1, 0.0)
    back = [1, 2, 3] if ch == 4 else [0]
    return v.GatherKernel(_kernel(c), n, back, out=s["out"])


def prepare(case, seed):
    c = dict(case)
    s = _inputs(c, seed)
    s["case"] = c
    v = s["v"] = _volume(c)
    kind = c["kind"]

    def empty(*shape):
        return torch.empty(shape, device="cuda")
    if kind in ("step", "frames"):
        s["out"] = empty(s["pos"].shape[0], 3 if c["channels"] == 4 else 1)
    if kind == "frames":  # the state machine's first two rebuilds are full ones
        for _ in range(2):
            v.SetPoints(s["frames"][0])
            v.RebuildTopology(s["frames"][0].shape[0], RADIUS)
    elif kind == "diff":
        n, ch = s["pos"].shape[0], c["channels"]
        v.SetPoints(s["pos"])
        v.RebuildTopology(n, RADIUS)
        v.UpdateAtlas()
        for k in range(3 * ch):
            v.ClearChannel(k)
        v.SetPoints(s["target"])
        v.ScatterKernel(_kernel(c), n, list(range(ch, 2 * ch)), attrs=[s["target_attr"][:, k] for k in range(ch)])
        s["rho"] = _atlases(v, range(ch))
        s["rho_t"] = [v.atlas_tensor(ch + k) for k in range(ch)]
        s["grad"] = [v.atlas_tensor(2 * ch + k) for k in range(ch)]
        s["out"] = empty(n, ch)
        s["grad_pos"], s["grad_pos_s"], s["grad_weight"], s["grad_attr"] = empty(n, 3), empty(n, 3), empty(n), empty(n, ch)
    elif kind in ("batch", "sparse"):
        n = sum(len(p) for p in s["clouds"]) if kind == "batch" else s["pos"].shape[0]
        back, wide = (1, 1) if kind == "batch" else (3, 4)
        s["n"], s["out"] = n, empty(n, back)
        s["grad_pos"], s["grad_pos_s"], s["grad_weight"], s["grad_attr"] = empty(n, 3), empty(n, 3), empty(n), empty(n, wide)
    elif kind == "export":
        n, ch = s["pos"].shape[0], c["channels"]
        v.SetPoints(s["pos"])
        v.RebuildTopology(n, RADIUS)
        v.UpdateAtlas()
        v.SetDeterministic(True)
        v.ScatterKernel(gvdb2.KERNEL_CUBIC2, n, list(range(ch)), weight=1.0,
                        attrs=_momentum(s["vel"])[1:] if ch == 3 else None)
        v.UpdateApron(-1, 0.0)
    return s


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------
def run(s):
    return {"step": _run_step, "frames": _run_frames, "diff": _run_diff, "batch": _run_batch, "sparse": _run_sparse,
            "surface": _run_surface, "density": _run_density, "export": _run_export}[s["case"]["kind"]](s)


def _atlas(v, channel):
    """A channel's tiles; the view keeps its volume, which owns the memory."""
    t = v.atlas_tensor(channel)
    t.volume = v
    return t


def _atlases(v, channels):
    return [_atlas(v, k) for k in channels]


def _run_step(s):
    c, v = s["case"], s["v"]
    out = _step(v, c, s, s["pos"], True)
    return {"gathered": out, "atlas": _atlases(v, range(c["channels"]))}


def _run_frames(s):
    c, v = s["case"], s["v"]
    for k, pos in enumerate(s["frames"]):
        out = _step(v, c, s, pos, k == 0)
    return {"gathered": out, "atlas": _atlases(v, range(c["channels"]))}


def _run_diff(s):
    c, v = s["case"], s["v"]
    K, n, ch = _kernel(c), s["pos"].shape[0], c["channels"]
    field, grads = list(range(ch)), list(range(2 * ch, 3 * ch))
    attrs = [s["attr"][:, k] for k in range(ch)]
    v.SetPoints(s["pos"])  # an optimiser moved them in place
    v.ScatterKernel(K, n, field, weight=s["weight"], attrs=attrs)
    v.GatherKernel(K, n, field, out=s["out"])
    v.GatherDensityBackward(K, n, field, s["grad_out"], grad_chans=grads, grad_pos=s["grad_pos"])
    for g, rho, rho_t in zip(s["grad"], s["rho"], s["rho_t"]):  # d/drho of sum (rho - rho_t)^2
        g.add_(rho, alpha=2.0).sub_(rho_t, alpha=2.0)
    v.ScatterDensityBackward(K, n, grads, weight=s["weight"], attrs=attrs, grad_pos=s["grad_pos_s"],
                             grad_weight=s["grad_weight"], grad_attr=s["grad_attr"])
    return {"rho": s["rho"], "gathered": s["out"], "grad_pos_gather": s["grad_pos"], "grad_pos": s["grad_pos_s"],
            "grad_weight": s["grad_weight"], "grad_attr": s["grad_attr"]}


def _run_batch(s):
    c, v, n = s["case"], s["v"], s["n"]
    K = _kernel(c)
    v.BatchPoints(s["clouds"], 10)
    v.RequestFullRebuild(True)
    v.RebuildTopology(n, RADIUS)
    v.UpdateAtlas()
    v.ScatterKernel(K, n, [0], weight=1.0)
    v.UpdateApron(0, 0.0)
    out = v.GatherKernel(K, n, [0], out=s["out"])
    v.GatherDensityBackward(K, n, [0], out, grad_chans=[1], grad_pos=s["grad_pos"])
    v.ScatterDensityBackward(K, n, [1], weight=1.0, grad_pos=s["grad_pos_s"], grad_weight=s["grad_weight"],
                             grad_attr=s["grad_attr"])
    return {"atlas": _atlas(v, 0), "gathered": out, "grad_pos_gather": s["grad_pos"], "grad_pos": s["grad_pos_s"],
            "grad_weight": s["grad_weight"]}


def _run_sparse(s):
    v, n, K = s["v"], s["n"], gvdb2.KERNEL_CUBIC2
    attrs = _momentum(s["vel"])
    v.SetPoints(s["pos"])
    v.RequestFullRebuild(True)
    v.RebuildTopology(n, RADIUS)
    v.UpdateAtlas()
    v.ScatterKernel(K, n, [0, 1, 2, 3], weight=1.0, attrs=attrs)
    for k in range(4):
        v.UpdateApron(k, 0.0)
    v.GatherKernel(K, n, [1, 2, 3], out=s["out"])
    v.GatherDensityBackward(K, n, [1, 2, 3], s["grad_out"], grad_chans=[5, 6, 7], grad_pos=s["grad_pos"])
    torch.mul(v.atlas_tensor(0), 2.0, out=v.atlas_tensor(4))  # d/drho of sum rho^2
    v.ScatterDensityBackward(K, n, [4, 5, 6, 7], weight=1.0, attrs=attrs, grad_pos=s["grad_pos_s"],
                             grad_weight=s["grad_weight"], grad_attr=s["grad_attr"])
    return {"atlas": _atlases(v, range(4)), "gathered": s["out"], "grad_pos_gather": s["grad_pos"],
            "grad_pos": s["grad_pos_s"], "grad_weight": s["grad_weight"], "grad_attr": s["grad_attr"]}


def _run_surface(s):
    c, v, n = s["case"], s["v"], s["pos"].shape[0]
    v.SetPoints(s["pos"])
    v.RequestFullRebuild(True)
    v.RebuildTopology(n, RADIUS)
    v.FinishTopology(False, True)
    v.UpdateAtlas()
    if c["fp16"]:
        ln = v.InsertPointsSubcell_FP16(SUBCELL, n, RADIUS)
        v.GatherLevelSet_FP16(SUBCELL, n, 1.0, (0, 0, 0), ln, 0)
    else:
        ln = v.InsertPointsSubcell(SUBCELL, n, RADIUS)
        v.GatherLevelSet(SUBCELL, n, 1.0, (0, 0, 0), ln, 0)
    v.UpdateApron(0, 3.0)
    return {"entries": ln, "atlas": _atlas(v, 0)}


def _run_density(s):
    v, n = s["v"], s["pos"].shape[0]
    v.SetPoints(s["pos"])
    v.RequestFullRebuild(True)
    v.RebuildTopology(n, RADIUS)
    v.UpdateAtlas()
    v.ClearChannel(0)
    v.InsertPoints(n)
    v.ScatterDensity(n, 1.0, 1.0, (0, 0, 0), True)
    ln = v.InsertPointsSubcell(SUBCELL, n, RADIUS)
    v.GatherDensity(SUBCELL, n, 1.0, (0, 0, 0), ln, 1)
    v.UpdateApron(-1, 0.0)
    return {"entries": ln, "atlas": _atlases(v, range(2))}


def _run_export(s):
    return s["v"].ExportToNanoVDB(list(range(s["case"]["channels"])), 0.0, "velocity", 0)


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------
def _blob_bricks(n, sigma, res):
    """Expected active bricks of a Gaussian cloud: a brick is active when the box it is reached from holds a point."""
    vol, total, dr = (res + BOX) ** 3, 0.0, sigma / 64.0
    for k in range(6 * 64):
        r = (k + 0.5) * dr
        rho = n * math.exp(-0.5 * (r / sigma) ** 2) / (2.0 * math.pi * sigma * sigma) ** 1.5
        total += 4.0 * math.pi * r * r * dr * -math.expm1(-rho * vol)
    return max(1.0, total / res ** 3)


def _bricks(c):
    res = {"surface": 32}.get(c["kind"], 1 << c.get("brick", 3))
    if c["kind"] == "batch":
        return sum(_blob_bricks(n, s, res) for n, s in _batch_shapes(c)), res
    if c["kind"] == "sparse":
        k = c["blobs"]
        return sum(_blob_bricks(c["n"] / k, 8.0 + 56.0 * i / max(1, k - 1), res) for i in range(k)), res
    if c.get("cloud") == "blob":
        return _blob_bricks(c["n"], c["sigma"], res), res
    if c.get("cloud") == "shell":  # bricks whose box crosses the shell, fewer when the points don't reach them all
        w = res + BOX
        full = 4.0 * math.pi * 98.0 ** 2 * (4.0 + w) / res ** 3
        return full * -math.expm1(-c["n"] * w ** 3 / (4.0 * math.pi * 98.0 ** 2 * (4.0 + w))), res
    return math.prod((e + BOX) // res + 1 for e in (c["nx"], int(c["ny"] * c["dy"]), c["nz"])), res


def _count(c):
    if c["kind"] == "batch":
        return sum(n for n, _ in _batch_shapes(c))
    return c["n"] if "n" in c else c["nx"] * c["ny"] * c["nz"]


def work(case):
    """Positions, attributes and results once each, every active brick's tile of each channel once, a node and a
    neighbour row a brick; the multiplies and adds of every point's stencil."""
    c, n = case, _count(case)
    bricks, res = _bricks(c)
    tile = 4.0 * (res + 2 * APRON) ** 3 * bricks
    topo = bricks * (64.0 + 27 * 4.0 + 8.0)
    kind, ch, taps = c["kind"], c.get("channels", 1), TAPS[c.get("kernel", "cubic")] ** 3
    if kind in ("step", "frames"):
        back = 3 if ch == 4 else 1
        attr = 12.0 * n if ch == 4 else 0.0
        f = c.get("frames", 1)
        return {"bytes": f * (12.0 * n + attr + topo + tile * ch + 4.0 * n * back),
                "flops": f * n * taps * 2.0 * (ch + back + 1)}
    if kind == "diff":
        return {"bytes": n * (12.0 + 4.0 + 8.0 * ch) + tile * 2 * ch + n * (24.0 + 4.0 + 8.0 * ch),
                "flops": n * taps * 2.0 * (2 * ch + ch + 3 * ch + 4 * ch + 6)}
    if kind == "batch":
        return {"bytes": 12.0 * n + topo + 2 * tile + n * (4.0 + 24.0 + 8.0), "flops": n * taps * 2.0 * (1 + 1 + 1 + 3 + 4 + 6)}
    if kind == "sparse":
        return {"bytes": n * (12.0 + 12.0 + 12.0) + topo + 8 * tile + n * (12.0 + 24.0 + 4.0 + 16.0),
                "flops": n * taps * 2.0 * (4 + 3 + 3 + 9 + 16 + 6)}
    entries = n * ((1.0 + 2 * RADIUS) / SUBCELL + 1.0) ** 3
    if kind == "surface":
        return {"bytes": 12.0 * n + topo + tile, "flops": entries * SUBCELL ** 3 * 6.0}
    if kind == "density":
        return {"bytes": 12.0 * n + topo + 2 * tile, "flops": entries * SUBCELL ** 3 * 6.0 + n * 7 * 12.0}
    return {"bytes": tile * ch + 4.0 * res ** 3 * bricks * ch + topo, "flops": 0.0}


# ----------------------------------------------------------------------------
# the same in 64 bits
# ----------------------------------------------------------------------------
CHUNK = 1 << 21


def _unique_keys(bricks):
    """Sorted keys of integer brick coordinates, ordered by x, then y, then z."""
    return torch.unique((bricks[:, 0] << 32) | (bricks[:, 1] << 16) | bricks[:, 2])


class _Field:
    """The active bricks of a full rebuild, in atlas order, and channel values on them in 64 bits."""

    def __init__(self, pos, log2, origin=None):
        self.log2, self.res = log2, 1 << log2
        self.t = self.res + 2 * APRON
        iw = pos.int()
        o = 0 if origin is None else origin
        base = _unique_keys((iw + o).long() >> log2)
        lo = ((iw.float() - RADIUS).int().clamp_(min=0) + o).long() >> log2
        hi = ((iw.float() + 2.0 * RADIUS).int() + o).long() >> log2
        found = []
        for k in range(8):  # an activation box is narrower than a brick: its corners name all its bricks
            pick = torch.tensor([k >> 2 & 1, k >> 1 & 1, k & 1], device="cuda", dtype=torch.bool)
            found.append(_unique_keys(torch.where(pick, hi, lo)))
        box = torch.unique(torch.cat(found))
        extra = box[~torch.isin(box, base)]
        keys = torch.cat([base, extra])  # pool order: the points' own bricks, then the boxes'
        self.corner = torch.stack([keys >> 32, keys >> 16 & 0xFFFF, keys & 0xFFFF], 1)
        self.first = self.corner.min(0).values - 1
        self.dims = self.corner.max(0).values + 2 - self.first
        self.first_l, self.dims_l = self.first.tolist(), self.dims.tolist()
        b = self.corner - self.first
        self.map = torch.full((math.prod(self.dims_l),), -1, dtype=torch.int32, device="cuda")
        self.map[(b[:, 0] * self.dims_l[1] + b[:, 1]) * self.dims_l[2] + b[:, 2]] = \
            torch.arange(len(keys), dtype=torch.int32, device="cuda")
        self.slots = len(keys)

    def zeros(self, channels):
        """(voxels + 1, channels): the last row stands for every voxel outside the active bricks."""
        return torch.zeros((self.slots * self.t ** 3 + 1, channels), dtype=torch.float64, device="cuda")

    def index(self, x, y, z):
        """Row of voxel (x, y, z); voxels outside the active bricks take the last row."""
        m = self.res - 1
        b = [(q >> self.log2) - f for q, f in zip((x, y, z), self.first_l)]
        inside = (b[0] >= 0) & (b[0] < self.dims_l[0]) & (b[1] >= 0) & (b[1] < self.dims_l[1]) & (b[2] >= 0) & (b[2] < self.dims_l[2])
        slot = self.map[torch.where(inside, (b[0] * self.dims_l[1] + b[1]) * self.dims_l[2] + b[2], 0)].long()
        at = slot * self.t ** 3 + (((z & m) + APRON) * self.t + (y & m) + APRON) * self.t + (x & m) + APRON
        return torch.where(inside & (slot >= 0), at, self.slots * self.t ** 3)

    def tiles(self, values, c):
        return values[:-1, c].reshape(self.slots, self.t, self.t, self.t)

    def with_apron(self, values, outside=0.0):
        """Every tile voxel's value as its owner holds it; `outside` where no active brick does."""
        values[-1] = outside
        out = torch.empty_like(values)
        a = torch.arange(self.t, device="cuda") - APRON
        z, y, x = (q.reshape(1, -1) for q in torch.meshgrid(a, a, a, indexing="ij"))
        per = max(1, (1 << 24) // self.t ** 3)
        for s in range(0, self.slots, per):
            w = self.corner[s:s + per] * self.res
            at = self.index(w[:, 0:1] + x, w[:, 1:2] + y, w[:, 2:3] + z).reshape(-1)
            out[s * self.t ** 3:s * self.t ** 3 + len(at)] = values[at]
        return out


def _weights(kernel, x):
    """First tap, weights and derivatives along one axis, for voxel centres at i + 0.5."""
    u = x - 0.5
    b = u.floor()
    t = u - b
    if kernel == "tent":
        one = torch.ones_like(t)
        return b.long(), [1.0 - t, t], [-one, one]

    def spline(d, inner):  # the cubic B-spline and its derivative at distance d >= 0
        if inner:
            return 2.0 / 3.0 - d * d + 0.5 * d ** 3, -2.0 * d + 1.5 * d * d
        return (2.0 - d) ** 3 / 6.0, -0.5 * (2.0 - d) ** 2
    (w0, d0), (w1, d1), (w2, d2), (w3, d3) = spline(1.0 + t, False), spline(t, True), spline(1.0 - t, True), spline(2.0 - t, False)
    return b.long() - 1, [w0, w1, w2, w3], [d0, d1, -d2, -d3]


def _taps(field, kernel, pos, origin):
    """For chunks of points: their slice and a generator of (row, weight, derivative along each axis) per tap."""
    n = pos.shape[0]
    for first in range(0, n, CHUNK):
        part = slice(first, min(n, first + CHUNK))
        p = pos[part].double()
        ax = [_weights(kernel, p[:, a]) for a in range(3)]
        o = [0, 0, 0] if origin is None else [origin[part, a].long() for a in range(3)]

        def each(ax=ax, o=o):
            (fx, wx, dx), (fy, wy, dy), (fz, wz, dz) = ax
            for k in range(len(wz)):
                for j in range(len(wy)):
                    for i in range(len(wx)):
                        at = field.index(fx + i + o[0], fy + j + o[1], fz + k + o[2])
                        yield at, wx[i] * wy[j] * wz[k], (dx[i] * wy[j] * wz[k], wx[i] * dy[j] * wz[k], wx[i] * wy[j] * dz[k])
        yield part, each()


def _scatter(field, kernel, pos, amounts, origin=None):
    values = field.zeros(amounts.shape[1])
    for part, taps in _taps(field, kernel, pos, origin):
        a = amounts[part].double()
        for at, w, _ in taps:
            values.index_add_(0, at, a * w[:, None])
    values[-1] = 0.0
    return values


def _gather(field, kernel, pos, values, origin=None, slopes=False):
    """Sums of values over each point's stencil and, with slopes, their derivatives (n, channels, 3)."""
    n, ch = pos.shape[0], values.shape[1]
    out = torch.empty((n, ch), dtype=torch.float64, device="cuda")
    grad = torch.empty((n, ch, 3), dtype=torch.float64, device="cuda") if slopes else None
    for part, taps in _taps(field, kernel, pos, origin):
        s = torch.zeros((len(pos[part]), ch), dtype=torch.float64, device="cuda")
        d = torch.zeros((len(pos[part]), ch, 3), dtype=torch.float64, device="cuda") if slopes else None
        for at, w, dw in taps:
            g = values[at]
            s += g * w[:, None]
            if slopes:
                for a in range(3):
                    d[:, :, a] += g * dw[a][:, None]
        out[part] = s
        if slopes:
            grad[part] = d
    return out, grad


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "export":
        return None  # bytes
    if c.get("fp16"):
        return None  # the lists' 16-bit positions are the result's own rounding
    return {"step": _exact_step, "frames": _exact_frames, "diff": _exact_diff, "batch": _exact_batch,
            "sparse": _exact_sparse, "surface": _exact_surface, "density": _exact_density}[kind](c, _inputs(c, seed))


def _momentum_amounts(d, channels):
    one = torch.ones((d["pos"].shape[0], 1), device="cuda")
    return torch.cat([one, d["vel"]], 1) if channels == 4 else one


def _exact_step(c, d):
    f = _Field(d["pos"], c["brick"])
    v = _scatter(f, c["kernel"], d["pos"], _momentum_amounts(d, c["channels"]))
    out, _ = _gather(f, c["kernel"], d["pos"], v[:, 1:] if c["channels"] == 4 else v)
    v = f.with_apron(v)
    return {"gathered": out, "atlas": [f.tiles(v, k) for k in range(c["channels"])]}


def _exact_frames(c, d):
    pos = d["frames"][-1]
    f = _Field(pos, 3)  # holds every voxel the last frame's stencils reach
    v = _scatter(f, c["kernel"], pos, _momentum_amounts(d, c["channels"]))
    out, _ = _gather(f, c["kernel"], pos, v[:, 1:] if c["channels"] == 4 else v)
    return {"gathered": out, "atlas": [None] * c["channels"]}  # atlas order follows the pool's history


def _exact_diff(c, d):
    ch, K, pos = c["channels"], c["kernel"], d["pos"]
    f = _Field(pos, c["brick"])
    w, a = d["weight"].double(), d["attr"].double()
    rho = _scatter(f, K, pos, w[:, None] * a)
    target = _scatter(f, K, d["target"], d["target_attr"])
    out, slope = _gather(f, K, pos, rho, slopes=True)
    go = d["grad_out"].double()
    grad = _scatter(f, K, pos, go) + 2.0 * (rho - target)
    s, ds = _gather(f, K, pos, grad, slopes=True)
    return {"rho": [f.tiles(rho, k) for k in range(ch)], "gathered": out,
            "grad_pos_gather": (go[:, :, None] * slope).sum(1), "grad_pos": ((w[:, None] * a)[:, :, None] * ds).sum(1),
            "grad_weight": (a * s).sum(1), "grad_attr": w[:, None] * s}


def _exact_batch(c, d):
    sizes, K = [len(p) for p in d["clouds"]], c["kernel"]
    k = next(k for k in range(1, 99) if k ** 3 >= len(sizes))
    cloud = torch.arange(len(sizes), device="cuda").repeat_interleave(torch.tensor(sizes, device="cuda"))
    origin = torch.stack([cloud % k, cloud // k % k, cloud // (k * k)], 1).int() << 11  # blocks of twice 2^10 voxels
    pos = torch.cat(d["clouds"])
    f = _Field(pos, 3, origin)
    rho = _scatter(f, K, pos, torch.ones((len(pos), 1), device="cuda"), origin)
    out, slope = _gather(f, K, pos, rho, origin, slopes=True)
    grad = _scatter(f, K, pos, out, origin)
    s, ds = _gather(f, K, pos, grad, origin, slopes=True)
    return {"atlas": f.tiles(f.with_apron(rho), 0), "gathered": out, "grad_pos_gather": out * slope[:, 0],
            "grad_pos": ds[:, 0], "grad_weight": s[:, 0]}


def _exact_sparse(c, d):
    pos, go, vel = d["pos"], d["grad_out"].double(), d["vel"].double()
    f = _Field(pos, c["brick"])
    v = _scatter(f, "cubic", pos, _momentum_amounts(d, 4))
    out, slope = _gather(f, "cubic", pos, v[:, 1:].contiguous(), slopes=True)
    grad_gather = (go[:, :, None] * slope).sum(1)
    del slope
    grad = torch.cat([2.0 * v[:, :1], _scatter(f, "cubic", pos, go)], 1)
    s, ds = _gather(f, "cubic", pos, grad, slopes=True)
    del grad
    v = f.with_apron(v)
    a = torch.cat([torch.ones((len(pos), 1), device="cuda", dtype=torch.float64), vel], 1)
    s_attr = s.clone()
    s_attr[:, 0] = 0.0  # the weight alone has no attribute
    return {"atlas": [f.tiles(v, k) for k in range(4)], "gathered": out, "grad_pos_gather": grad_gather,
            "grad_pos": (a[:, :, None] * ds).sum(1), "grad_weight": (a * s).sum(1), "grad_attr": s_attr}


def _nearest(f, pos):
    """Each voxel corner's squared distance to the nearest point listed in its subcell, and the list entries."""
    best = torch.full((f.slots * f.t ** 3 + 1,), math.inf, dtype=torch.float64, device="cuda")
    entries = 0
    for first in range(0, len(pos), CHUNK):
        p = pos[first:first + CHUNK]
        lo = (p - RADIUS).int() // SUBCELL
        hi = (p + 1 + RADIUS).int() // SUBCELL
        most = int((hi - lo).max()) + 1
        q = p.double()
        for k in range(most ** 3):
            cell = lo + torch.tensor([k // most ** 2, k // most % most, k % most], device="cuda", dtype=torch.int32)
            on = (cell <= hi).all(1)
            v = cell[on].long() * SUBCELL
            entries += int((f.index(v[:, 0], v[:, 1], v[:, 2]) < len(best) - 1).sum())
            x = q[on]
            for j in range(SUBCELL ** 3):
                w = v + torch.tensor([j % 4, j // 4 % 4, j // 16], device="cuda")
                best.scatter_reduce_(0, f.index(w[:, 0], w[:, 1], w[:, 2]), (x - w).square().sum(1), "amin")
    return best[:, None].sqrt(), entries


def _exact_surface(c, d):
    f = _Field(d["pos"], 5)
    dist, entries = _nearest(f, d["pos"])
    return {"entries": entries, "atlas": f.tiles(f.with_apron((dist - 1.0).clamp_(max=3.0), 3.0), 0)}


def _exact_density(c, d):
    pos = d["pos"]
    f = _Field(pos, 3)
    dist, entries = _nearest(f, pos)
    near = f.with_apron((1.0 - dist).clamp_(min=0.0))
    splat = f.zeros(1)
    iw, p = pos.long(), pos.double()
    for step in ((0, 0, 0), (-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1)):
        q = iw + torch.tensor(step, device="cuda")
        on = ((q >> 3) == (iw >> 3)).all(1)  # a point adds to its own brick
        r2 = (p - q).square().sum(1)
        w = 1.0 + r2 * (-3.0 + r2 * (3.0 - r2))
        splat.index_add_(0, f.index(q[on, 0], q[on, 1], q[on, 2]), w[on][:, None])
    splat = f.with_apron(splat)
    return {"entries": entries, "atlas": [f.tiles(splat, 0), f.tiles(near, 0)]}
