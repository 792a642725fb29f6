"""Stage times of a build (SVO_FLAG_TIMINGS) name the work that they say."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _best(ctx, mesh, res, flags, stage, n=5):
    """The stage's least time over some builds, in ms (device times plus the odd host hiccup)."""
    return min(ctx.build(*mesh, res, flags).timings()[stage] for _ in range(n + 2))


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


def test_compact_stage_has_the_keys(gpu_ctx, svo_mod):
    """Above res 256 the keys have a launch and a stream of their own.  Writing
    them takes at least their bytes over the path from the SMs to L2 (32 bytes a
    clock and SM, 148 SMs, 1.965 GHz)."""
    mesh = _mesh(300, 0.4)
    flags = svo_mod.FLAG_TIMINGS | svo_mod.FLAG_NO_VERT_EDGE
    n_keys = gpu_ctx.build(*mesh, 512, flags).num_keys
    assert n_keys > 8_000_000
    with_keys = _best(gpu_ctx, mesh, 512, flags, "compact")
    without = _best(gpu_ctx, mesh, 512, flags | svo_mod.FLAG_NO_KEYS, "compact")
    assert with_keys - without > n_keys * 8 / (148 * 32 * 1.965e9) * 1e3


def test_unique_stage_is_not_the_wait_for_the_dedup(gpu_ctx, svo_mod):
    """No duplicates: nothing to remove, however long the dedup's stream runs on."""
    mesh = _mesh(20000, 0.01)
    flags = svo_mod.FLAG_TIMINGS | svo_mod.FLAG_NO_VERT_EDGE | svo_mod.FLAG_DEDUP
    t = [gpu_ctx.build(*mesh, 256, flags).timings() for _ in range(7)]
    assert min(x["unique"] for x in t) < 0.25 * min(x["dedup"] for x in t)
