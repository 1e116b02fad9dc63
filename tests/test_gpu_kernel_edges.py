"""GPU parity at the sizes where single kernels can go wrong: the ends of
their tiles, remainders, the smallest and the largest of their range."""
import numpy as np
import pytest

from _helpers import REL_TOL, interior, make_oracle, rel_err
from test_gpu_topology import compare_topology, gpu_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [0.4, 2.0, 9.5])
@pytest.mark.parametrize("sc,cfg", [(2, (3, 3, 3, 3, 3)), (8, (3, 3, 3, 3, 3)), (4, (3, 3, 3, 3, 5)), (16, (3, 3, 3, 3, 5))])
def test_subcell_table(gvdb2_mod, oracle_mod, sc, cfg, radius):
    """Every subcell's node, corner and list length, for 1, 8, 64 and 512 subcells a brick and boxes over one brick to
    four, against the oracle (exact)."""
    rng = np.random.default_rng(20)
    pts = rng.uniform(70.0, 170.0, (3001, 3)).astype(np.float32)
    o = make_oracle(oracle_mod, cfg)
    assert o.rebuild_topology(pts, 2.0) == 0
    ln = o.insert_points_subcell(sc, pts, radius)
    cnt, nid, pos = o.subcells()
    v = gpu_volume(gvdb2_mod, pts, cfg)
    v.RebuildTopology(len(pts), 2.0)
    assert v.InsertPointsSubcell(sc, len(pts), radius) == ln
    g = v.subcells(len(cnt))
    for a, b in zip(g, (cnt, nid, pos)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("lo,hi", [
    ((70.0, 70.0, 70.0), (73.0, 73.0, 73.0)),       # a grid of less than one 32-bit word
    ((68.0, 70.0, 66.0), (69.0, 71.0, 320.0)),      # one brick thick, several parents long
    ((61.0, 3.0, 509.0), (67.0, 260.0, 900.0)),     # parents that start inside the grid, two levels of them
])
@pytest.mark.parametrize("radius", [2.0, 45.0])
def test_parent_levels(gvdb2_mod, oracle_mod, lo, hi, radius):
    """Node pools and child lists of small and thin brick grids, with activation boxes of one brick and of 18 (runs over
    word ends, boxes cut at the root), against the oracle (exact)."""
    rng = np.random.default_rng(21)
    pts = rng.uniform(lo, hi, (400, 3)).astype(np.float32)
    o = make_oracle(oracle_mod)
    assert o.rebuild_topology(pts, radius) == 0
    v = gpu_volume(gvdb2_mod, pts)
    v.RebuildTopology(len(pts), radius)
    compare_topology(v, o)


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("nch", [1, 2, 3, 4])
@pytest.mark.parametrize("per_cell", [1, 32, 33, 96, 97, 129, 193, 767, 768, 2048, 2049])
def test_scatter_cell_classes(gvdb2_mod, oracle_mod, kernel, nch, per_cell):
    """One cell of per_cell points among empty ones, at a cell corner of a 16^3 brick so that neighbours in and beyond
    the brick get them: the ends of a 32-source step, of a source list, and of each class of cells (light, neighbour of
    a heavy one, owner-computes, fixed point, rows); against the FP64 oracle within 1e-5 of the largest value."""
    import torch
    rng = np.random.default_rng(22)
    pts = np.concatenate([rng.uniform(80.0, 87.999 if per_cell > 128 else 80.4, (per_cell, 3)), [[100.0, 100.0, 100.0]]]).astype(np.float32)
    vel = rng.normal(size=(len(pts), 4)).astype(np.float32)
    chans = list(range(nch))
    cfg = (3, 3, 3, 3, 4)
    o = make_oracle(oracle_mod, cfg, chans)
    assert o.rebuild_topology(pts, 2.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts, cfg, chans)
    v.RebuildTopology(len(pts), 2.0)
    v.UpdateAtlas()
    tv = torch.from_numpy(vel).cuda()
    v.ScatterKernel(kernel, len(pts), chans, attrs=[(tv, c) for c in chans])
    o.scatter_kernel(kernel, pts, chans, attrs=[vel[:, c] for c in chans])
    for c in chans:
        assert rel_err(interior(v.atlas(c), 1), interior(o.atlas(c), 1)) < REL_TOL


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("nch", [1, 3])
@pytest.mark.parametrize("per_cell", [32, 33])
def test_gather_at_brick_corner(gvdb2_mod, oracle_mod, kernel, nch, per_cell):
    """Stencils over a corner where eight 8^3 bricks meet and some are missing (radius 0), for the most points of a
    light cell and one more; gather and position gradient against the FP64 oracle within 1e-5 of the largest value."""
    import torch
    rng = np.random.default_rng(23)
    pts = rng.uniform(80.001, 82.5, (per_cell, 3))
    # two of the seven neighbours exist
    pts = np.concatenate([pts, [[79.2, 80.5, 80.5], [79.5, 79.5, 80.5], [100.0, 100.0, 100.0]]]).astype(np.float32)
    n, chans = len(pts), list(range(nch))
    vel = rng.normal(size=(n, nch)).astype(np.float32)
    go = rng.normal(size=(n, nch)).astype(np.float32)
    o = make_oracle(oracle_mod, chans=chans)
    assert o.rebuild_topology(pts, 0.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts, chans=chans)
    v.RebuildTopology(n, 0.0)
    v.UpdateAtlas()
    tv = torch.from_numpy(vel).cuda()
    v.ScatterKernel(kernel, n, chans, attrs=[(tv, c) for c in chans])
    o.scatter_kernel(kernel, pts, chans, attrs=[vel[:, c] for c in chans])
    assert rel_err(v.GatherKernel(kernel, n, chans).cpu().numpy(), o.gather_kernel(kernel, pts, chans)) < REL_TOL
    gp = v.GatherDensityBackward(kernel, n, chans, torch.from_numpy(go).cuda()).cpu().numpy()
    assert rel_err(gp, o.gather_kernel_backward(kernel, pts, chans, go)) < REL_TOL


@pytest.mark.parametrize("nch,cfg,apron", [(1, (3, 3, 3, 3, 3), 1), (2, (3, 3, 3, 3, 4), 2), (3, (3, 3, 3, 3, 2), 1),
                                           (5, (3, 3, 3, 3, 3), 2)])
def test_apron_channels(gvdb2_mod, nch, cfg, apron):
    """Every channel's apron in one call, in groups of 4 and a remainder, for bricks of 4^3 to 16^3: copies of the
    owners' interior values and the boundary value, exactly, and interiors left alone."""
    import torch
    rng = np.random.default_rng(24)
    pts = rng.uniform(70.0, 110.0, (200, 3)).astype(np.float32)
    chans = list(range(nch))
    v = gpu_volume(gvdb2_mod, pts, cfg, chans, apron)
    v.RebuildTopology(len(pts), 2.0)
    v.UpdateAtlas()
    tiles = []
    for c in chans:
        t = rng.integers(0, 1 << 20, v.atlas(c).shape).astype(np.float32)
        v.atlas_tensor(c).copy_(torch.from_numpy(t).cuda())
        tiles.append(t)
    v.UpdateApron(-1, -7.0)
    pos = v.atlas_map()["mPos"][:len(tiles[0])]
    where = {tuple(p): s for s, p in enumerate(pos.tolist())}
    res, t = 1 << cfg[4], tiles[0].shape[1]
    for c in chans:
        got = v.atlas(c)
        for s in range(0, len(pos), max(1, len(pos) // 40)):
            for z, y, x in ((0, 0, 0), (0, t - 1, apron), (apron, apron, t - 1), (t - 1, apron, 0), (apron, 0, t - 1)):
                w = np.array((x, y, z)) - apron + pos[s]
                own = where.get(tuple((w // res * res).tolist()))
                lx, ly, lz = w % res + apron
                assert got[s, z, y, x] == (-7.0 if own is None else tiles[c][own, lz, ly, lx])
            assert np.array_equal(interior(got, apron)[s], interior(tiles[c], apron)[s])


@pytest.mark.parametrize("levelset", [False, True])
@pytest.mark.parametrize("per_list", [1, 2, 63, 64, 65, 129])
def test_voxel_gathers_list_ends(gvdb2_mod, oracle_mod, levelset, per_list):
    """4^3 subcells with lists of one point, of odd and even lengths and around the 64 points staged at a time; against
    the FP64 oracle within 1e-5 of the largest value."""
    rng = np.random.default_rng(25)
    pts = np.concatenate([rng.uniform(82.0, 82.9, (per_list, 3)), [[100.0, 100.0, 100.0]]]).astype(np.float32)
    o = make_oracle(oracle_mod)
    assert o.rebuild_topology(pts, 2.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts)
    v.RebuildTopology(len(pts), 2.0)
    v.UpdateAtlas()
    ln = v.InsertPointsSubcell(4, len(pts), 0.5)
    assert o.insert_points_subcell(4, pts, 0.5) == ln
    if levelset:
        v.GatherLevelSet(4, len(pts), 1.5, (0, 0, 0), ln, 0)
        o.gather_level_set(4, 1.5, 0)
    else:
        v.GatherDensity(4, len(pts), 1.5, (0, 0, 0), ln, 0)
        o.gather_density(4, 1.5, 0)
    assert rel_err(interior(v.atlas(0), 1), interior(o.atlas(0), 1)) < REL_TOL


@pytest.mark.parametrize("outside", [0, 1, 300])
def test_points_outside_the_bricks(gvdb2_mod, outside):
    """Gathers and gradients of points outside every brick are zero whatever the buffers held, and the others are those
    of a call without them (deterministic mode, exactly)."""
    import torch
    rng = np.random.default_rng(26)
    inside = rng.uniform(70.0, 90.0, (1000, 3)).astype(np.float32)
    pts = np.concatenate([inside, rng.uniform(300.0, 400.0, (outside, 3)).astype(np.float32)])
    n, res = len(pts), []
    for p in (inside, pts):
        v = gpu_volume(gvdb2_mod, inside, chans=[0])
        v.SetDeterministic(True)
        v.RebuildTopology(len(inside), 2.0)
        v.UpdateAtlas()
        t = torch.from_numpy(p).cuda()
        v.SetPoints(t)
        v.ScatterKernel(2, len(p), [0])
        out = [torch.full(s, float("nan"), device="cuda") for s in ((len(p), 1), (len(p), 3), (len(p),), (len(p), 1), (len(p), 3))]
        v.GatherKernel(2, len(p), [0], out=out[0])
        v.ScatterDensityBackward(2, len(p), [0], attrs=[torch.ones(len(p), device="cuda")], grad_pos=out[1],
                                 grad_weight=out[2], grad_attr=out[3])
        v.GatherDensityBackward(2, len(p), [0], torch.ones((len(p), 1), device="cuda"), grad_pos=out[4])
        res.append([o.cpu().numpy() for o in out])
    for a, b in zip(*res):
        assert np.array_equal(b[:1000], a)
        assert not b[1000:n].any()


@pytest.mark.parametrize("per_cell", [1024, 1025, 2048, 2049, 4097])
def test_gather_huge_cells(gvdb2_mod, oracle_mod, per_cell):
    """A cell at the ends of the heavy class and of the gather's items of 2,048 points: gather and both adjoints against
    the FP64 oracle within 1e-5 of the largest value, every point served."""
    import torch
    rng = np.random.default_rng(27)
    pts = np.concatenate([rng.uniform(80.0, 87.99, (per_cell, 3)), [[100.0, 100.0, 100.0]]]).astype(np.float32)
    n = len(pts)
    o = make_oracle(oracle_mod, chans=[0])
    assert o.rebuild_topology(pts, 2.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts, chans=[0])
    v.RebuildTopology(n, 2.0)
    v.UpdateAtlas()
    assert v.info().splat_cells == -1
    v.ScatterKernel(2, n, [0])
    o.scatter_kernel(2, pts, [0])
    assert v.info().splat_cells == 2
    out = torch.full((n, 1), float("nan"), device="cuda")
    assert rel_err(v.GatherKernel(2, n, [0], out=out).cpu().numpy(), o.gather_kernel(2, pts, [0])) < REL_TOL
    go = rng.normal(size=(n, 1)).astype(np.float32)
    gp = v.GatherDensityBackward(2, n, [0], torch.from_numpy(go).cuda()).cpu().numpy()
    assert rel_err(gp, o.gather_kernel_backward(2, pts, [0], go)) < REL_TOL
