"""GPU test of the apron copies where a tile's apron takes several blocks and a call several groups of channels."""
import numpy as np
import pytest

from test_gpu_topology import gpu_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nch", [1, 4, 6, 9])
@pytest.mark.parametrize("brick,apron", [(3, 1), (4, 2), (5, 1), (5, 3), (6, 1)])
def test_every_apron_voxel(gvdb2_mod, nch, brick, apron):
    """Every apron voxel of every channel is the owner's interior value or the boundary value, exactly, and interiors
    stay as they were."""
    import torch
    rng = np.random.default_rng(43)
    pts = rng.uniform(100.0, 180.0, (300, 3)).astype(np.float32)
    pts = np.concatenate([pts, [[300.0, 300.0, 300.0]]]).astype(np.float32)
    chans = list(range(nch))
    v = gpu_volume(gvdb2_mod, pts, (3, 3, 3, 3, brick), chans, apron)
    v.RebuildTopology(len(pts), 2.0)
    v.UpdateAtlas()
    slots, res, a = int(v.info().atlas_slots), 1 << brick, apron
    pos = v.atlas_map()["mPos"][:slots]
    lo = pos.min(0) - a
    size = pos.max(0) + res + a - lo
    for c in chans:
        t = v.atlas_tensor(c)
        t.copy_(torch.from_numpy(rng.integers(0, 1 << 20, tuple(t.shape)).astype(np.float32)).cuda())
    before = [v.atlas(c)[:slots].copy() for c in chans]
    v.UpdateApron(-1, -7.0)
    for c in chans:
        grid = np.full(tuple(size[::-1]), -7.0, np.float32)  # z, y, x
        for s, p in enumerate(pos - lo):
            grid[p[2]:p[2] + res, p[1]:p[1] + res, p[0]:p[0] + res] = before[c][s, a:a + res, a:a + res, a:a + res]
        got = v.atlas(c)
        for s, p in enumerate(pos - lo):
            z, y, x = (slice(p[k] - a, p[k] + res + a) for k in (2, 1, 0))
            assert np.array_equal(got[s], grid[z, y, x])
