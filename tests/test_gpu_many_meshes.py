"""Batches of very many small meshes (an asset import): every mesh gets the
octree of its own build, whatever their number."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT, random_mesh

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


FRESH_PAGES = """
import sys, resource
sys.path[:0] = [sys.argv[1] + "/gpu-svo_b200", sys.argv[1] + "/tests"]
import ctypes as C
import torch, svo_b200
from conftest import random_mesh
v, f = random_mesh(41, 2)
mesh = (torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda(), 4)
ctx, n = svo_b200.Context(0), 4000
descs, keep = svo_b200._descs([mesh] * n, svo_b200.FLAG_NO_VERT_EDGE)
outs, st = (C.c_void_p * n)(), (C.c_int * n)()
for _ in range(4):
    before = resource.getrusage(resource.RUSAGE_SELF).ru_minflt
    assert svo_b200.lib().svo_build_batch(ctx.handle, descs, n, None, outs, st) == 0
    faults = resource.getrusage(resource.RUSAGE_SELF).ru_minflt - before
    for o in outs:
        svo_b200.lib().svo_result_free(o)
print(faults * resource.getpagesize() / n)
"""


def test_tables_of_many_meshes_are_made_once(svo_mod):
    """Fresh host memory of a batch, by the pages it faults in (every block of
    128 KiB and more its own mapping).  The per-mesh records (two of the mesh,
    its compaction job and its emission parameters, 24 levels each) are 4.0 KB
    together; made once they stay below one and a half times that."""
    env = dict(os.environ, MALLOC_MMAP_THRESHOLD_="131072")
    p = subprocess.run([sys.executable, "-c", FRESH_PAGES, ROOT], env=env, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]
    assert float(p.stdout) < 6000
