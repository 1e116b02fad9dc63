"""GPU parity of the cubic splat's cells of 768 to 2,048 points, whose sums are taken in float registers, where those sums
can go wrong: however many of a cell's points share a stencil."""
import numpy as np
import pytest

from _helpers import interior, make_oracle
from test_gpu_topology import gpu_volume

pytestmark = pytest.mark.gpu

U = 2.0 ** -24
# Roundings on the way to a voxel, each at most U of the sum of the |contributions|: three weights of at most 4 each, two
# products, 32 terms of a window column (8 a first column, 4 of them), 8 sums in a plane's column, 8 partials merged
ROWS_TOL = (3 * 4 + 2 + 32 + 8 + 8) * U


def cell_points(kind, n, rng):
    """n points in the cell [80, 88)^3."""
    if kind == "uniform":
        return rng.uniform(80.0, 87.99, (n, 3))
    if kind == "voxel":
        return rng.uniform(83.51, 84.49, (n, 3))
    if kind == "coincident":
        return np.tile((84.7, 83.3, 83.9), (n, 1))
    q = rng.uniform(80.0, 87.99, (n, 3))
    q[:, 1:] = (83.3, 84.9)
    return q  # a line along x


@pytest.mark.parametrize("amounts", ["equal", "positive", "signed"])
@pytest.mark.parametrize("kind", ["uniform", "voxel", "coincident", "line"])
@pytest.mark.parametrize("n", [768, 1031, 2048])
@pytest.mark.parametrize("nch", [1, 4])
def test_sums_of_points_that_share_a_stencil(gvdb2_mod, oracle_mod, amounts, kind, n, nch):
    import torch
    rng = np.random.default_rng(32)
    pts = np.concatenate([cell_points(kind, n, rng), [[100.0, 100.0, 100.0]]]).astype(np.float32)
    a = {"equal": np.full((n + 1, nch), 1.1), "positive": rng.uniform(0.5, 1.5, (n + 1, nch)),
         "signed": rng.normal(size=(n + 1, nch))}[amounts].astype(np.float32)
    chans, grads = list(range(nch)), list(range(nch, 2 * nch))
    o = make_oracle(oracle_mod, chans=chans + grads)
    assert o.rebuild_topology(pts, 2.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts, chans=chans)
    v.RebuildTopology(len(pts), 2.0)
    v.UpdateAtlas()
    ta = torch.from_numpy(a).cuda()
    v.ScatterKernel(2, len(pts), chans, attrs=[(ta, c) for c in chans])
    o.scatter_kernel(2, pts, chans, attrs=[a[:, c] for c in chans])
    o.scatter_kernel(2, pts, grads, attrs=[np.abs(a[:, c]) for c in chans])
    for c in chans:
        err = np.abs(interior(v.atlas(c), 1).astype(np.float64) - interior(o.atlas(c), 1)).max()
        assert err <= ROWS_TOL * interior(o.atlas(grads[c]), 1).max()


def test_bit_reproducible_whatever_the_binning(gvdb2_mod):
    """Bins are filled through atomics, so the order of a cell's points changes from binning to binning: the sums of
    cells of 768 to 2,048 points do not (all of the points here, 64 cells of some 1,500)."""
    import torch
    rng = np.random.default_rng(33)
    pts = rng.uniform(80.0, 111.99, (96_000, 3)).astype(np.float32)
    n = len(pts)
    v = gpu_volume(gvdb2_mod, pts, chans=[0, 1])
    a = torch.from_numpy(rng.normal(size=n).astype(np.float32)).cuda()
    want = None
    for _ in range(8):
        v.RebuildTopology(n, 2.0)
        v.UpdateAtlas()
        v.ScatterKernel(2, n, [0, 1], attrs=[None, a])
        got = [interior(v.atlas(c), 1) for c in (0, 1)]
        want = want or got
        for g, w in zip(got, want):
            assert np.array_equal(g, w)


@pytest.mark.parametrize("nch", [1, 3])
@pytest.mark.parametrize("n", [768, 2048])
def test_amounts_that_are_not_finite(gvdb2_mod, oracle_mod, nch, n):
    """Infinite and NaN amounts reach the voxels of their own stencils and no others; the rest of the cell and the
    channels whose amounts are finite are those of the FP64 oracle, to the bound above."""
    import torch
    rng = np.random.default_rng(34)
    pts = np.concatenate([rng.uniform(80.0, 87.99, (n, 3)), [[100.0, 100.0, 100.0]]]).astype(np.float32)
    pts[:4] = [[81.3, 81.4, 81.2], [86.8, 81.7, 86.6], [81.7, 86.7, 82.4], [81.9, 86.2, 82.3]]
    a = rng.uniform(0.5, 1.5, (n + 1, nch)).astype(np.float32)
    a[:4, nch - 1] = (np.inf, np.nan, -np.inf, np.inf)
    chans = list(range(nch))
    o = make_oracle(oracle_mod, chans=chans)
    assert o.rebuild_topology(pts, 2.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts, chans=chans)
    v.RebuildTopology(len(pts), 2.0)
    v.UpdateAtlas()
    ta = torch.from_numpy(a).cuda()
    v.ScatterKernel(2, len(pts), chans, attrs=[(ta, c) for c in chans])
    o.scatter_kernel(2, pts, chans, attrs=[a[:, c] for c in chans])
    for c in chans:
        g, w = interior(v.atlas(c), 1).astype(np.float64), interior(o.atlas(c), 1)
        assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(np.isinf(g), np.isinf(w))
        ok = np.isfinite(w)
        assert np.array_equal(g[np.isinf(w)], w[np.isinf(w)])
        assert np.abs(g[ok] - w[ok]).max() <= ROWS_TOL * np.abs(w[ok]).max()
    assert np.isnan(w).any() and np.isinf(w).any()


@pytest.mark.parametrize("nch", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("slice_", [512, 4096])
@pytest.mark.parametrize("side", [8, 10, 11])
def test_few_and_many_row_cells(gvdb2_mod, oracle_mod, nch, slice_, side):
    """512, 1,000 and 1,331 cells of some 800 points, fewer than, between and more than the counts at which 2 to 4
    channels take the row sums; slices of a cell and whole cells; a group of channels and its remainder: against the
    FP64 oracle, to the bound above (all of a voxel's contributions positive)."""
    import torch
    rng = np.random.default_rng(38)
    n = 800 * side ** 3
    pts = rng.uniform(80.0, 80.0 + 8 * side - 0.01, (n, 3)).astype(np.float32)
    a = rng.uniform(0.5, 1.5, (n, nch)).astype(np.float32)
    w = rng.uniform(0.5, 1.5, n).astype(np.float32)
    chans = list(range(nch))
    o = make_oracle(oracle_mod, chans=chans)
    assert o.rebuild_topology(pts, 2.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts, chans=chans)
    v.SetTuning(512, slice_, 32)
    v.RebuildTopology(n, 2.0)
    v.UpdateAtlas()
    ta, tw = torch.from_numpy(a).cuda(), torch.from_numpy(w).cuda()
    v.ScatterKernel(2, n, chans, weight=tw, attrs=[(ta, c) for c in chans])
    o.scatter_kernel(2, pts, chans, weight=w, attrs=[a[:, c] for c in chans])
    for c in chans:
        g, want = interior(v.atlas(c), 1).astype(np.float64), interior(o.atlas(c), 1)
        assert np.abs(g - want).max() <= (ROWS_TOL + U) * want.max()  # and the product of weight and attribute


def row_cells(rng, sizes, kinds, side=9):
    """side^3 cells, cell i with sizes[i] points of kinds[i] (cyclic), in random order."""
    out = []
    for i in range(side ** 3):
        q = cell_points(kinds[i % len(kinds)], sizes[i % len(sizes)], rng)
        out.append(q + 8.0 * np.array((i % side, i // side % side, i // side ** 2)))
    p = np.concatenate(out).astype(np.float32)
    return p[rng.permutation(len(p))]


@pytest.mark.parametrize("amounts", ["equal", "signed"])
def test_many_cells_of_points_that_share_a_stencil(gvdb2_mod, oracle_mod, amounts):
    """729 cells, enough for the row sums of 4 channels, of 768 to 2,048 points that share stencils as above; one amount
    in some cells infinite or NaN: against the FP64 oracle, to the bound above."""
    import torch
    rng = np.random.default_rng(40)
    pts = row_cells(rng, (768, 1031, 2048, 1300, 800), ("uniform", "voxel", "coincident", "line"))
    n, chans, grads = len(pts), [0, 1, 2, 3], [4]
    a = (np.full((n, 4), 1.1) if amounts == "equal" else rng.normal(size=(n, 4))).astype(np.float32)
    a[rng.choice(n, 6, replace=False), 2] = (np.inf, np.nan, -np.inf, np.inf, np.nan, np.inf)
    o = make_oracle(oracle_mod, chans=chans + grads)
    assert o.rebuild_topology(pts, 2.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts, chans=chans)
    v.RebuildTopology(n, 2.0)
    v.UpdateAtlas()
    ta = torch.from_numpy(a).cuda()
    v.ScatterKernel(2, n, chans, attrs=[(ta, c) for c in chans])
    o.scatter_kernel(2, pts, chans, attrs=[a[:, c] for c in chans])
    for c in chans:
        o.scatter_kernel(2, pts, grads, attrs=[np.abs(np.where(np.isfinite(a[:, c]), a[:, c], 0)).astype(np.float32)])
        g, w = interior(v.atlas(c), 1).astype(np.float64), interior(o.atlas(c), 1)
        assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(np.isinf(g), np.isinf(w))
        ok = np.isfinite(w)
        assert np.abs(g[ok] - w[ok]).max() <= ROWS_TOL * interior(o.atlas(4), 1).max()


def test_many_cells_bit_reproducible_whatever_the_binning(gvdb2_mod):
    """The row sums of 729 cells after bins filled in another order each time: the same bits."""
    import torch
    rng = np.random.default_rng(41)
    pts = row_cells(rng, (800, 1500), ("uniform", "voxel"))
    n, chans = len(pts), [0, 1, 2, 3]
    v = gpu_volume(gvdb2_mod, pts, chans=chans)
    a = torch.from_numpy(rng.normal(size=(n, 4)).astype(np.float32)).cuda()
    want = None
    for _ in range(5):
        v.RebuildTopology(n, 2.0)
        v.UpdateAtlas()
        v.ScatterKernel(2, n, chans, attrs=[(a, c) for c in chans])
        got = [v.atlas_tensor(c).clone() for c in chans]
        want = want or got
        for g, w in zip(got, want):
            assert torch.equal(g, w)


def test_batched_row_cells(gvdb2_mod, oracle_mod):
    """Two clouds of row cells in one volume, default mode: each cloud's grid is that of the FP64 oracle on its own
    points, to the bound above."""
    import torch
    rng = np.random.default_rng(42)
    clouds = [row_cells(rng, (800, 1100), ("uniform",), 7), row_cells(rng, (900,), ("uniform", "line"), 7) + np.float32(24.0)]
    n, chans = sum(map(len, clouds)), [0, 1, 2, 3]
    a = rng.uniform(0.5, 1.5, (n, 4)).astype(np.float32)
    v = gvdb2_mod.VolumeGVDB(0)
    v.Configure(3, 3, 3, 3, 3)
    for c in chans:
        v.AddChannel(c, gvdb2_mod.T_FLOAT, 1)
    dev = [torch.from_numpy(p).cuda() for p in clouds]
    first = v.BatchPoints(dev, 10)
    v.RebuildTopology(n, 2.0)
    v.UpdateAtlas()
    ta = torch.from_numpy(a).cuda()
    v.ScatterKernel(2, n, chans, attrs=[(ta, c) for c in chans])
    pos = v.atlas_map()["mPos"][:int(v.info().atlas_slots)]
    for k, p in enumerate(clouds):
        o = make_oracle(oracle_mod, chans=chans)
        assert o.rebuild_topology(p, 2.0) == 0
        o.update_atlas()
        o.scatter_kernel(2, p, chans, attrs=[a[first[k]:first[k + 1], c] for c in chans])
        where = {tuple(q): s for s, q in enumerate((pos - np.array(v.BatchOrigin(k))).tolist())}
        slots = [where[tuple(q)] for q in o.atlas_map()["mPos"][:o.atlas_slots()].tolist()]
        for c in chans:
            w = interior(o.atlas(c), 1)
            assert np.abs(interior(v.atlas(c), 1)[slots].astype(np.float64) - w).max() <= ROWS_TOL * w.max()
