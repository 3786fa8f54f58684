"""A handle after an evaluation that is refused half-way.  The refusal is the
host's: the handle's stream is one under capture, on which an evaluation
cannot be waited for."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _refused(bvlib, D, theta):
    """D's evaluation on a stream under capture, which the runtime refuses."""
    import torch
    s = torch.cuda.Stream()
    rt = ctypes.CDLL("libcudart.so.12")  # torch's
    graph = ctypes.c_void_p()
    stream = ctypes.c_void_p(s.cuda_stream)
    D.set_stream(s.cuda_stream)
    assert rt.cudaStreamBeginCapture(stream, 1) == 0  # thread-local
    try:
        with pytest.raises(bvlib.BvError):
            D(theta)
    finally:
        assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) != 0  # invalidated
        rt.cudaGetLastError()
        D.set_stream(0)


@pytest.mark.parametrize("use_graph", [True, False])
def test_evaluation_after_a_refused_one(bvlib, use_graph):
    """The refusal is not found again by the next call's checks."""
    x, y = bvlib.generate_xy(2000, 0)
    L = bvlib.build_layout(x, y, np.random.default_rng(0).standard_normal(2000), 100, 30)
    L.knn_idx = bvlib.knn(L)
    with bvlib.LlhData(L, use_graph=use_graph) as D:
        v = D((1.0, 0.1, 1.5))
        _refused(bvlib, D, (1.0, 0.2, 1.5))
        assert D((1.0, 0.1, 1.5)) == v
        _refused(bvlib, D, (1.0, 0.2, 1.5))
        assert np.array_equal(bvlib.knn(L), L.knn_idx)


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("read_before", [True, False])
def test_times_after_a_refused_evaluation(bvlib, use_graph, read_before):
    """bv_get_status keeps everything of the last evaluation that gave a
    value, its times included, read before the refused one or after it."""
    x, y = bvlib.generate_xy(2000, 0)
    L = bvlib.build_layout(x, y, np.random.default_rng(0).standard_normal(2000), 100, 30)
    L.knn_idx = bvlib.knn(L)
    with bvlib.LlhData(L, use_graph=use_graph) as D:
        v = D((1.0, 0.1, 1.5))
        before = D.status() if read_before else None
        _refused(bvlib, D, (1.0, 0.2, 1.5))
        st = D.status()
        assert st["llk"] == v
        assert st["device_ms"] >= st["kernel_ms"] > 0.0
        if read_before:
            assert st == before
        assert D((1.0, 0.1, 1.5)) == v
        assert D.status()["device_ms"] > 0.0
