"""Result copies while another thread captures a graph: a thread that has set
its capture mode to relaxed may copy, whatever threads the copy is made with."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RELAXED = 2  # cudaStreamCaptureModeRelaxed


@pytest.mark.parametrize("res", [16, 128])  # one transfer; staged by several threads
def test_copy_in_relaxed_mode(gpu_ctx, res):
    import torch
    from svo_b200 import meshgen

    cudart = C.CDLL("libcudart.so.12")
    v, f = meshgen.jittered_icosphere(3, np.random.default_rng(res))
    r = gpu_ctx.build(v, f, res)
    want = r.edges()
    got = []

    def copy():
        mode = C.c_int(RELAXED)
        got.append(cudart.cudaThreadExchangeStreamCaptureMode(C.byref(mode)))
        try:
            got.append(np.array_equal(r.edges().view(np.uint8), want.view(np.uint8)))
        except Exception as e:
            got.append(repr(e))

    x = torch.zeros(16, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.Stream()):
        graph.capture_begin(capture_error_mode="global")
        x += 1
        t = threading.Thread(target=copy)
        t.start()
        t.join()
        if got == [0, True]:
            x += 1
            graph.capture_end()
    assert got == [0, True]
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 16
