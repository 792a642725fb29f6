"""Batches of very many small meshes (an asset import): every mesh gets the
octree of its own build, whatever their number."""
import numpy as np
import pytest

from conftest import random_mesh

pytestmark = pytest.mark.gpu


def _kinds():
    import torch

    out = []
    for seed, res in ((40, 2), (41, 4), (42, 8)):
        v, f = random_mesh(seed, 2)
        out.append((torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda(), res))
    return out


def test_more_meshes_than_a_grid_axis(gpu_ctx):
    """More than 65,535 meshes, the limit of a launch grid's y and z."""
    kinds = _kinds()
    n = 65540
    want = [gpu_ctx.build(*k) for k in kinds]
    results, st, rc = gpu_ctx.build_batch([kinds[i % 3] for i in range(n)])
    assert rc == 0 and st == [0] * n
    assert all(results[i].num_nodes == want[i % 3].num_nodes for i in range(n))
    for i in (0, 1, 2, 1183, 1184, 32768, 65534, 65535, 65536, n - 1):
        for name in ("nodes", "vertices", "edges", "keys"):
            assert getattr(results[i], name)().tobytes() == getattr(want[i % 3], name)().tobytes(), (i, name)


def test_many_meshes_do_not_wait_for_other_streams(gpu_ctx, svo_mod):
    """A batch whose report is over 1 MiB (5,243 meshes) returns while work of
    another stream is still running: nothing in it waits for the device."""
    import torch

    kinds = _kinds()
    meshes = [kinds[i % 3] for i in range(6000)]
    side, own = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):  # pools and kept blocks
        results, st, rc = gpu_ctx.build_batch(meshes, svo_mod.FLAG_NO_VERT_EDGE, own.cuda_stream)
        assert rc == 0
        del results
    done = torch.cuda.Event()
    with torch.cuda.stream(side):
        torch.cuda._sleep(4_000_000_000)  # about two seconds
        done.record()
    results, st, rc = gpu_ctx.build_batch(meshes, svo_mod.FLAG_NO_VERT_EDGE, own.cuda_stream)
    running = not done.query()
    torch.cuda.synchronize()
    assert rc == 0 and running
