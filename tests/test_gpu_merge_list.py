"""GPU parity of the merge of dense cells' partials where the list of cells is longer than the merge's grid."""
import numpy as np
import pytest

from _helpers import REL_TOL, interior, make_oracle, rel_err
from test_gpu_topology import gpu_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("nch", [1, 4])
@pytest.mark.parametrize("dense", [0, 1, 2, 5])
def test_list_longer_than_the_grid(gvdb2_mod, oracle_mod, kernel, nch, dense):
    """None to five cells of 512 points far apart, so that each lists all of its 27 neighbours, between cells of a few
    points: every voxel written, within 1e-5 of the largest value of the FP64 oracle's."""
    import torch
    rng = np.random.default_rng(41)
    base = 80.0 + 32.0 * np.arange(max(dense, 1))
    p = [np.stack([rng.uniform(b, b + 7.99, 512) for b in (x, 80.0, 80.0)], 1) for x in base[:dense]]
    p = np.concatenate(p + [np.stack([rng.uniform(x - 8.0, x + 15.99, 40) for x in (b, 80.0, 80.0)], 1) for b in base])
    p = p.astype(np.float32)
    a = rng.normal(size=(len(p), nch)).astype(np.float32)
    cfg, chans = (3, 3, 3, 3, 3), list(range(nch))
    o = make_oracle(oracle_mod, cfg, chans)
    assert o.rebuild_topology(p, 8.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, p, cfg, chans)
    v.RebuildTopology(len(p), 8.0)
    v.UpdateAtlas()
    slots = int(v.info().atlas_slots)
    for c in chans:
        v.atlas_tensor(c).fill_(float("nan"))
    t = torch.from_numpy(a).cuda()
    v.ScatterKernel(kernel, len(p), chans, attrs=[(t, c) for c in chans])
    o.scatter_kernel(kernel, p, chans, attrs=[a[:, c] for c in chans])
    for c in chans:
        assert rel_err(interior(v.atlas(c), 1)[:slots], interior(o.atlas(c), 1)) <= REL_TOL
