"""A built graph's k-NN lists stay in device memory until they are copied or the
graph is released: both may happen while a CUDA graph is being captured, and neither
changes the calling thread's device."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_copy_and_release_during_a_capture():
    import torch
    from parallel_anns_b200 import native as N
    from parallel_anns_b200.graph import build_nsg
    x = np.random.default_rng(1).random((3000, 24), dtype=np.float32)
    _, want = build_nsg(x, R=16, knn_k=24, with_knn=True)
    lib = N.load()
    handles = []
    for _ in range(2):
        h = ctypes.c_void_p()
        N.check(lib.panns_build_nsg_ex(0, N.ptr(x), 3000, 24, 24, 16, 0, ctypes.byref(h)))
        handles.append(h)
    knn = np.zeros((3000, 24), dtype=np.uint32)
    t = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        t += 1
        N.check(lib.panns_graph_copy(handles[0], None, None, N.ptr(knn)))
        N.check(lib.panns_graph_free(handles[0]))
        t += 1
    assert np.array_equal(knn, want)
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    assert t.eq(4).all()
    knn[:] = 0
    N.check(lib.panns_graph_copy(handles[1], None, None, N.ptr(knn)))
    N.check(lib.panns_graph_free(handles[1]))
    assert np.array_equal(knn, want)
