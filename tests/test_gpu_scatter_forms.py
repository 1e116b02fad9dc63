"""GPU tests of the owner-computes scatter's forms: a warp's registers or a tile in shared memory by a cell's estimate of
sources, and the lists that the cells are taken from, in volumes of few and of many cells."""
import numpy as np
import pytest

from _helpers import REL_TOL, interior, make_oracle, rel_err
from test_gpu_topology import gpu_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("nch", [1, 2, 3, 4])
@pytest.mark.parametrize("own", [1, 5, 8])
def test_forms_give_the_same_bits(gvdb2_mod, kernel, nch, own):
    """A cell of a few points alone in its 16^3 brick, and with 400 points in the middle of the brick's opposite cell,
    which raise the brick's estimate and reach no voxel of the first: the first cell's sums, bit for bit (deterministic
    mode, points in index order)."""
    import torch
    rng = np.random.default_rng(35)
    a = rng.uniform(80.0, 87.99, (own, 3))
    got = []
    for extra in (0, 400):
        # the other brick keeps the volume's layout the same; the extra points come last
        pts = np.concatenate([a, [[130.0, 130.0, 130.0]], rng.uniform(90.1, 93.9, (extra, 3))]).astype(np.float32)
        attr = np.random.default_rng(36).normal(size=(own + 401, nch)).astype(np.float32)[:len(pts)].copy()
        v = gpu_volume(gvdb2_mod, pts, (3, 3, 3, 3, 4), list(range(nch)))
        v.SetDeterministic(True)
        v.RebuildTopology(len(pts), 2.0)
        v.UpdateAtlas()
        t = torch.from_numpy(attr).cuda()
        v.ScatterKernel(kernel, len(pts), list(range(nch)), attrs=[(t, c) for c in range(nch)])
        pos = v.atlas_map()["mPos"][:int(v.info().atlas_slots)]
        slot = int(np.nonzero((pos == (80, 80, 80)).all(1))[0][0])
        got.append([interior(v.atlas(c), 1)[slot, :8, :8, :8] for c in range(nch)])
    for x, y in zip(*got):
        assert np.array_equal(x, y) and x.any()


@pytest.mark.parametrize("kernel,nch,brick,even", [(1, 1, 3, True), (2, 3, 3, True), (1, 3, 4, False), (2, 1, 4, True),
                                                   (2, 4, 5, False), (1, 2, 6, True)])
def test_many_cells(gvdb2_mod, oracle_mod, kernel, nch, brick, even):
    """More than 65,536 cells of every class of sources, most of them with points or most without: against the FP64
    oracle within 1e-5 of the largest value, every voxel written."""
    import torch
    rng = np.random.default_rng(37)
    n, cfg = 90_000, (3, 3, 3, 3, brick)
    if even:
        p = rng.uniform(64.0, 64.0 + 8 * 41, (n, 3))
        p[:9_000] = rng.uniform(200.0, 216.0, (9_000, 3))  # 8 cells of more than 1,000
        p[9_000:40_000] = rng.uniform(80.0, 144.0, (31_000, 3))  # 512 cells of some 60
    else:
        p = np.concatenate([rng.normal(c, s, (n // 3, 3)) for c, s in ((300.0, 60.0), (500.0, 6.0), (700.0, 25.0))])
    p = np.clip(p, 8.0, 900.0).astype(np.float32)
    a = rng.normal(size=(n, nch)).astype(np.float32)
    chans = list(range(nch))
    o = make_oracle(oracle_mod, cfg, chans)
    radius = 2.0 if even else 12.0
    assert o.rebuild_topology(p, radius) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, p, cfg, chans)
    v.RebuildTopology(n, radius)
    v.UpdateAtlas()
    slots = int(v.info().atlas_slots)
    assert slots * (1 << (brick - 3)) ** 3 > 65_536
    for c in chans:
        v.atlas_tensor(c).fill_(float("nan"))
    t = torch.from_numpy(a).cuda()
    v.ScatterKernel(kernel, n, chans, attrs=[(t, c) for c in chans])
    o.scatter_kernel(kernel, p, chans, attrs=[a[:, c] for c in chans])
    for c in chans:
        assert rel_err(interior(v.atlas(c), 1)[:slots], interior(o.atlas(c), 1)) < REL_TOL
