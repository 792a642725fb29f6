"""Voxelizer work splits that send triangles down other routes: none, some or
all of them walked by one thread, queue entries of one brick column to 64, the
queue filled past its first capacity so that the counting phase runs again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPLITS = [(sm, wm) for sm in (0, 1, 8, 128) for wm in (1, 16, 17, 1024)]


@pytest.fixture
def tuned(gpu_ctx):
    saved = gpu_ctx.tuning
    yield gpu_ctx
    gpu_ctx.tuning = saved


def test_splits_keep_results(tuned, svo_mod):
    from svo_b200 import meshgen

    meshes = meshgen.batch(6, seed=11)
    pts, tris, _ = meshgen.torus_slivers(20000)
    meshes += [(pts, tris, 128), (pts, tris, 512)]
    want = [tuned.build(*m, svo_mod.FLAG_NO_VERT_EDGE) for m in meshes]
    for sm, wm in SPLITS:
        tuned.tuning = (sm, wm)
        assert tuned.tuning[:2] == (sm, wm)
        for m, a in zip(meshes, want):
            b = tuned.build(*m, svo_mod.FLAG_NO_VERT_EDGE)
            assert a.nodes().tobytes() == b.nodes().tobytes() and a.keys().tobytes() == b.keys().tobytes(), (sm, wm)


def test_queue_past_its_capacity(tuned, svo_mod):
    """1,000 triangles half a 512^3 grid across: over 65,536 entries of one
    column, the queue's first capacity; the phase's kernels are launched again."""
    rng = np.random.default_rng(12)
    v = rng.uniform(0, 1, size=(3000, 3)).astype(np.float32)
    f = np.arange(3000, dtype=np.int32).reshape(-1, 3)

    def build():
        before = svo_mod.kernel_launches()
        r = tuned.build(v, f, 512, svo_mod.FLAG_NO_VERT_EDGE)
        return r.keys(), svo_mod.kernel_launches() - before

    tuned.tuning = (0, 1 << 20)  # one entry a triangle
    want, once = build()
    tuned.tuning = (0, 1)
    got, twice = build()
    assert twice > once
    assert np.array_equal(got, want)
