"""GPU test of the autotuner's cache: settings timed with earlier kernels are left alone."""
import numpy as np
import pytest

from test_gpu_topology import gpu_volume

pytestmark = pytest.mark.gpu


def test_settings_of_earlier_kernels_are_not_taken(gvdb2_mod, tmp_path):
    """A cache file whose entry has the class of the call but not the kernels' generation, as files written before there
    was one: the call keeps the volume's setting; with the entry as written it takes it."""
    rng = np.random.default_rng(45)
    pts = rng.uniform(80.0, 112.0, (20_000, 3)).astype(np.float32)
    n, path = len(pts), tmp_path / "tune.txt"
    v = gpu_volume(gvdb2_mod, pts)
    v.SetTuneCache(str(path))
    v.RebuildTopology(n, 2.0)
    v.UpdateAtlas()
    v.AutotuneScatter(gvdb2_mod.KERNEL_CUBIC2, n, [0])
    key, rest = path.read_text().splitlines()[0].split("\t")
    cls = key.rsplit("|g", 1)[0]
    assert cls != key
    v.SetAutotune(True)
    for k, want in ((cls, (512, 4096)), (cls + "|g2", (512, 4096)), (key, (1024, 8192))):
        path.write_text(f"{k}\t1024 8192 32 0.5\n")
        v.SetTuning(512, 4096, 32)
        v.ScatterKernel(gvdb2_mod.KERNEL_CUBIC2, n, [0])
        assert v.GetTuning()[:2] == want
