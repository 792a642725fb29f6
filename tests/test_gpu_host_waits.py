"""Host waits of a build: their number does not grow where one wait serves all
meshes of a batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _waits(fn):
    import torch
    from torch.profiler import ProfilerActivity, profile

    fn()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        out = fn()
    return out, sum(e.name == "cudaStreamSynchronize" for e in prof.events())


@pytest.mark.parametrize("n", [1, 12])
def test_waits_of_meshes_with_duplicates(gpu_ctx, n):
    """Meshes far from the origin, whose edges have consecutive duplicates:
    a wait for the counts, one for the emission, one for the duplicate counters
    of all meshes, one for each mesh's edges, one at the end."""
    import torch
    from svo_b200 import meshgen

    v, f = meshgen.jittered_icosphere(2, np.random.default_rng(3))
    mesh = ((torch.from_numpy(v).cuda() + 1e6).contiguous(), torch.from_numpy(f).cuda(), 64)
    (results, st, rc), waits = _waits(lambda: gpu_ctx.build_batch([mesh] * n))
    assert rc == 0
    assert all(r.num_edges < 12 * r.num_nodes and r.num_vertices == 8 * r.num_nodes for r in results)
    assert 0 < waits <= 4 + n


def test_waits_of_an_ordinary_batch(gpu_ctx):
    from svo_b200 import meshgen

    meshes = meshgen.batch(8, seed=6)
    (results, st, rc), waits = _waits(lambda: gpu_ctx.build_batch(meshes))
    assert rc == 0 and waits == 2
