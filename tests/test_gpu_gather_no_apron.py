"""GPU parity of the gathers without an apron: stencils that start in the brick below, so that only their upper taps lie
in the atlas."""
import numpy as np
import pytest

from _helpers import REL_TOL, interior, make_oracle, rel_err
from test_gpu_topology import gpu_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("apron", [0, 1])
@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("nch", [1, 3])
@pytest.mark.parametrize("per_cell", [1, 32, 33])
def test_gather_at_the_first_slots_low_corner(gvdb2_mod, oracle_mod, apron, kernel, nch, per_cell):
    """Points at the low corner of the first brick, with no brick below it: gather and both adjoints against the FP64
    oracle within 1e-5 of the largest value, for a light cell and one past it."""
    import torch
    rng = np.random.default_rng(31)
    pts = rng.uniform(80.001, 82.2, (per_cell, 3))
    pts = np.concatenate([pts, [[100.0, 100.0, 100.0]]]).astype(np.float32)
    n, chans, grads = len(pts), list(range(nch)), list(range(nch, 2 * nch))
    attr = rng.uniform(0.5, 1.5, (n, nch)).astype(np.float32)
    go = rng.normal(size=(n, nch)).astype(np.float32)
    o = make_oracle(oracle_mod, chans=chans + grads, apron=apron)
    assert o.rebuild_topology(pts, 0.0) == 0
    o.update_atlas()
    v = gpu_volume(gvdb2_mod, pts, chans=chans + grads, apron=apron)
    v.RebuildTopology(n, 0.0)
    v.UpdateAtlas()
    ta = torch.from_numpy(attr).cuda()
    for into in (chans, grads):
        v.ScatterKernel(kernel, n, into, attrs=[(ta, c) for c in range(nch)])
        o.scatter_kernel(kernel, pts, into, attrs=[attr[:, c] for c in range(nch)])
        for c in into:
            assert rel_err(interior(v.atlas(c), apron), interior(o.atlas(c), apron)) < REL_TOL
    assert rel_err(v.GatherKernel(kernel, n, chans).cpu().numpy(), o.gather_kernel(kernel, pts, chans)) < REL_TOL
    gp = v.GatherDensityBackward(kernel, n, chans, torch.from_numpy(go).cuda()).cpu().numpy()
    assert rel_err(gp, o.gather_kernel_backward(kernel, pts, chans, go)) < REL_TOL
    got = v.ScatterDensityBackward(kernel, n, grads, attrs=[(ta, c) for c in range(nch)])
    want = o.scatter_kernel_backward(kernel, pts, chans, grads, attrs=[attr[:, c] for c in range(nch)])
    for g, w in zip(got, want):
        assert rel_err(g.cpu().numpy(), np.asarray(w).reshape(tuple(g.shape))) < REL_TOL
