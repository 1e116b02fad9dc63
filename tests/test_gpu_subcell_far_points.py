"""GPU test of the subcell lists with points far outside the volume, up to the ends of float."""
import numpy as np
import pytest

from test_gpu_topology import gpu_volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sc", [2, 4, 8])
@pytest.mark.parametrize("fp16", [False, True])
def test_far_points_visit_nothing(gvdb2_mod, sc, fp16):
    """Coordinates of 1e9 to the largest float, infinite and negative ones: the lists are those of the other points."""
    import torch
    rng = np.random.default_rng(44)
    near = rng.uniform(70.0, 110.0, (2000, 3)).astype(np.float32)
    far = np.array([[x, 90.0, 90.0] for x in (1e9, 1.2e9, 2.1e9, 2147483520.0, 2147483648.0, 3e9, 3e38, np.inf, -1e9)] +
                   [[90.0, x, 90.0] for x in (1.1e9, 2147483520.0, np.inf)] +
                   [[x, x, x] for x in (1.5e9, 2147483520.0, 1e30, np.inf)], np.float32)
    got = []
    for pts in (near, np.concatenate([far, near, far])):
        v = gpu_volume(gvdb2_mod, near)
        v.RebuildTopology(len(near), 2.0)
        v.UpdateAtlas()
        t = torch.from_numpy(pts).cuda()
        v.SetPoints(t)
        ln = (v.InsertPointsSubcell_FP16 if fp16 else v.InsertPointsSubcell)(sc, len(pts), 1.5)
        got.append((ln,) + tuple(v.subcells(int(v.info().atlas_slots) * (8 // sc) ** 3)))
    assert got[0][0] == got[1][0] > 0
    for a, b in zip(got[0][1:], got[1][1:]):
        assert np.array_equal(a, b)
