"""Voxel sets of triangles of every size and shape against the oracle: walked
by one thread (serial tier) or column by column (serial_max 0 sends every
triangle there), at grid edges, with degenerate and badly scaled triangles."""
import numpy as np
import pytest

from conftest import random_mesh

pytestmark = pytest.mark.gpu


def _mesh(kind):
    v, f = random_mesh(77, 48, kind if kind in ("blob", "grid", "sliver") else "blob")
    rng = np.random.default_rng(78)
    if kind == "degenerate":  # points, segments and collinear triples among ordinary triangles
        f[::4, 1] = f[::4, 0]
        f[1::8] = f[1::8, :1]
        v[f[2::8, 2]] = (v[f[2::8, 0]] + v[f[2::8, 1]]) / 2
    elif kind == "far":  # coordinates that absorb the voxel size
        v = v + np.float32(3e5)
    elif kind == "tiny":  # squared lengths underflow
        v = v * np.float32(1e-17)
    elif kind == "flat":  # one axis of the bbox is empty
        v[:, 1] = np.float32(0.25)
    elif kind == "small":  # a few voxels each, all over the grid
        c = rng.uniform(0, 1, size=(400, 1, 3))
        v = (c + rng.normal(size=(400, 3, 3)) * 0.004).reshape(-1, 3).astype(np.float32)
        f = np.arange(1200, dtype=np.int32).reshape(-1, 3)
    return np.ascontiguousarray(v, dtype=np.float32), f


@pytest.mark.parametrize("strict", [False, True])
@pytest.mark.parametrize("res", [4, 5, 37, 64, 200, (128, 33, 200), (3, 256, 17)])
@pytest.mark.parametrize("kind", ["blob", "grid", "sliver", "degenerate", "far", "tiny", "flat", "small"])
def test_voxels(gpu_ctx, oracle_mod, svo_mod, kind, res, strict):
    v, f = _mesh(kind)
    flags = svo_mod.FLAG_NO_VERT_EDGE | (svo_mod.FLAG_STRICT_FP if strict else 0)
    want = oracle_mod.build_svo(v, f, res, flags=flags).keys
    saved = gpu_ctx.tuning
    try:
        for tuning in (saved, (0, 256, 0, 32, 0), (0, 1, 0, 32, 0), (8, 64, 0, 32, 0), (1 << 16, 256, 0, 32, 0)):
            gpu_ctx.tuning = tuning
            got = gpu_ctx.build(v, f, res, flags).keys()
            assert np.array_equal(got, want), (tuning, got.size, want.size)
    finally:
        gpu_ctx.tuning = saved
