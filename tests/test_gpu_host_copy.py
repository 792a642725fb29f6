"""Results copied to ordinary host memory (staged through pinned slots by
several threads above 4 MiB) equal the same arrays copied to pinned memory
(one transfer), whole and in order, alone and from several threads at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = {"nodes": 168, "vertices": 16, "edges": 28, "keys": 8}


def _pinned(svo_mod, r, name):
    import torch

    n = getattr(r, "num_" + name)
    buf = torch.zeros(max(1, n * NAMES[name]), dtype=torch.uint8, pin_memory=True)
    assert getattr(svo_mod.lib(), f"svo_result_copy_{name}")(r.handle, buf.data_ptr(), n) == svo_mod.OK
    return buf.numpy()[: n * NAMES[name]]


@pytest.mark.parametrize("res", [16, 40, 64, 90, 128, 200])
def test_pageable_equals_pinned(gpu_ctx, svo_mod, res):
    from svo_b200 import meshgen

    v, f = meshgen.jittered_icosphere(4, np.random.default_rng(res))
    r = gpu_ctx.build(v, f, res)
    for name in NAMES:
        got = getattr(r, name)()
        assert np.array_equal(got.view(np.uint8), _pinned(svo_mod, r, name)), name


def test_small_capacity_is_refused(gpu_ctx, svo_mod):
    from svo_b200 import meshgen

    v, f = meshgen.jittered_icosphere(4, np.random.default_rng(1))
    r = gpu_ctx.build(v, f, 128)
    out = np.zeros(r.num_nodes, dtype=svo_mod.NODE_DTYPE)
    assert svo_mod.lib().svo_result_copy_nodes(r.handle, out.ctypes.data, r.num_nodes - 1) == svo_mod.ERR_INVALID_ARGUMENT
    assert not out.view(np.uint8).any()


def test_several_threads(svo_mod):
    """Copies from several threads at once: one is staged, the others take the driver's path."""
    from svo_b200 import meshgen

    ctx = svo_mod.Context(0)
    v, f = meshgen.jittered_icosphere(4, np.random.default_rng(2))
    results = [ctx.build(v, f, res) for res in (100, 128, 150)]
    want = [_pinned(svo_mod, r, "edges").copy() for r in results]
    bad = []

    def work(i):
        for _ in range(4):
            if not np.array_equal(results[i].edges().view(np.uint8), want[i]):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for r in results:
        r.close()
    ctx.close()
