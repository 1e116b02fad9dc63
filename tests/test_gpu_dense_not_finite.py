"""GPU parity of the dense cells' fixed-point sums where some amounts are infinite or NaN."""
import numpy as np
import pytest

from _helpers import REL_TOL, interior, make_oracle
from test_gpu_topology import gpu_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("nch", [1, 2, 4])
@pytest.mark.parametrize("n", [512, 4096, 9001])
def test_not_finite_amounts_in_fixed_point(gvdb2_mod, oracle_mod, kernel, nch, n):
    """Cells of one slice of points and of several: infinite and NaN amounts reach the voxels of their own stencils, and
    the other voxels and channels are those of the FP64 oracle within 1e-5 of the largest value."""
    import torch
    rng = np.random.default_rng(39)
    pts = np.concatenate([rng.uniform(80.0, 87.99, (n, 3)), [[100.0, 100.0, 100.0]]]).astype(np.float32)
    pts[n - 4:n] = [[81.3, 81.4, 81.2], [86.8, 81.7, 86.6], [81.7, 86.7, 82.4], [81.9, 86.2, 82.3]]
    a = rng.uniform(0.5, 1.5, (n + 1, nch)).astype(np.float32)
    a[n - 4:n, nch - 1] = (np.inf, np.nan, -np.inf, np.inf)
    chans = list(range(nch))
    o = make_oracle(oracle_mod, chans=chans)
    assert o.rebuild_topology(pts, 2.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts, chans=chans)
    v.SetDeterministic(True)
    v.RebuildTopology(len(pts), 2.0)
    v.UpdateAtlas()
    t = torch.from_numpy(a).cuda()
    v.ScatterKernel(kernel, len(pts), chans, attrs=[(t, c) for c in chans])
    o.scatter_kernel(kernel, pts, chans, attrs=[a[:, c] for c in chans])
    for c in chans:
        g, w = interior(v.atlas(c), 1).astype(np.float64), interior(o.atlas(c), 1)
        assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(np.isinf(g), np.isinf(w))
        ok = np.isfinite(w)
        assert np.array_equal(g[np.isinf(w)], w[np.isinf(w)])
        assert np.abs(g[ok] - w[ok]).max() <= REL_TOL * np.abs(w[ok]).max()
    assert np.isnan(w).any() and np.isinf(w).any()
