"""GPU parity of the owner-computes scatter where some amounts are infinite or NaN."""
import numpy as np
import pytest

from _helpers import REL_TOL, interior, make_oracle
from test_gpu_topology import gpu_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own,many,kernel,nch", [(own, False, k, c) for own in (6, 60, 300) for k in (1, 2) for c in (1, 3)] +
                         [(300, True, 1, 1), (300, True, 2, 2)])
def test_not_finite_amounts_reach_their_own_stencils(gvdb2_mod, oracle_mod, own, many, kernel, nch):
    """Cells of few and of many points, in volumes of few cells and of more than 65,536: the NaN and infinite voxels, and
    all others, of the FP64 oracle within 1e-5 of the largest value; then the same call with finite amounts."""
    import torch
    rng = np.random.default_rng(46)
    pts = np.concatenate([rng.uniform(880.0, 887.99, (own, 3)), rng.uniform(888.0, 895.99, (4, 3)), [[900.0, 900.0, 900.0]]])
    if many:  # activation boxes of 69,000 cells
        pts = np.concatenate([pts, [[200.0, 200.0, 200.0], [200.0, 600.0, 200.0], [600.0, 200.0, 200.0]]])
    pts = pts.astype(np.float32)
    pts[:2] = [[881.3, 881.4, 881.2], [886.8, 882.7, 886.6]]
    n, chans = len(pts), list(range(nch))
    radius = 76.0 if many else 2.0
    o = make_oracle(oracle_mod, chans=chans)
    assert o.rebuild_topology(pts, radius) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts, chans=chans)
    v.RebuildTopology(n, radius)
    v.UpdateAtlas()
    assert (int(v.info().atlas_slots) > 65_536) == many
    for special in ((np.inf, np.nan), (1.0, 2.0), (-np.inf, 1.0))[:1 if many else 3]:
        a = rng.uniform(0.5, 1.5, (n, nch)).astype(np.float32)
        a[:2, nch - 1] = special
        t = torch.from_numpy(a).cuda()
        v.ScatterKernel(kernel, n, chans, attrs=[(t, c) for c in chans])
        o.scatter_kernel(kernel, pts, chans, attrs=[a[:, c] for c in chans])
        for c in chans:
            g, w = interior(v.atlas(c), 1).astype(np.float64), interior(o.atlas(c), 1)
            assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(np.isinf(g), np.isinf(w))
            ok = np.isfinite(w)
            assert np.abs(g[ok] - w[ok]).max() <= REL_TOL * np.abs(w[ok]).max()
