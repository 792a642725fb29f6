"""Stage times of a build (SVO_FLAG_TIMINGS) name the work that they say."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(n, size, seed=9):
    import torch

    rng = np.random.default_rng(seed)
    v = np.clip(rng.uniform(0, 1, (n, 1, 3)) + rng.normal(size=(n, 3, 3)) * size, 0, 1).astype(np.float32)
    return torch.from_numpy(v.reshape(-1, 3)).cuda(), torch.arange(3 * n, dtype=torch.int32).reshape(-1, 3).cuda()


def test_no_scan_stage(gpu_ctx, svo_mod):
    r = gpu_ctx.build(*_mesh(100, 0.05), 64, svo_mod.FLAG_TIMINGS)
    t = r.timings()
    assert t["scan"] == 0.0
    assert all(t[k] > 0.0 for k in ("total", "bbox", "voxelize", "pyramid", "compact", "emit"))
    assert t["total"] >= t["bbox"] + t["voxelize"] + t["pyramid"]
