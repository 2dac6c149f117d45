"""GPU: a j push is refused on a stream that is being captured."""
import ctypes as C

import numpy as np
import pytest

import sapporo2_b200 as sp

pytestmark = pytest.mark.gpu


def _stage(s, addr, x):
    """Staged records (4th order: 16 doubles) of unit masses at rest in x."""
    stride = s.lib.sapb_j_stage_stride(s.dev)
    at = C.cast(s.lib.sapb_j_stage(s.dev, len(addr)), C.POINTER(C.c_double))
    buf = np.ctypeslib.as_array(at, (len(addr), stride))
    buf[:] = 0.0
    buf[:, 0] = np.stack([addr, addr], 1).astype(np.int32).copy().view(np.float64)[:, 0]
    buf[:, 2] = 1.0
    buf[:, 3:6] = x
    return len(addr)


def _positions(s, n):
    out = np.zeros((n, 24))
    assert s.lib.sapb_read_j(s.dev, 0, n, 0.0, 0, out) == 0
    return out[:, 0:3]


@pytest.mark.parametrize("n", [1, 512, 513])
def test_push_under_capture_is_refused(gpu, n):
    import torch
    rng = np.random.default_rng(n)
    x = rng.normal(size=(2, n, 3))
    with sp.Sapporo(order=sp.FOURTH, precision=sp.DOUBLESINGLE) as s:
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        assert s.lib.sapb_push_j(s.dev, _stage(s, np.arange(n), x[0])) == 0
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        one = torch.zeros(1, device="cuda")
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            one += 1
            assert s.lib.sapb_push_j(s.dev, _stage(s, np.arange(n), x[1])) != 0
        assert np.array_equal(_positions(s, n), x[0])
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(_positions(s, n), x[0])
        for k in (1, 0):  # and the pushes after it go through
            assert s.lib.sapb_push_j(s.dev, _stage(s, np.arange(n), x[k])) == 0
        assert np.array_equal(_positions(s, n), x[0])
        s.set_stream(0)
