"""GPU: small j pushes, which the scatter kernel reads from one pinned buffer:
that buffer is not rewritten while a push before it is still queued, and a push
is refused on a stream that is being captured."""
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


@pytest.mark.parametrize("n", [1, 511, 512, 513])
def test_pushes_behind_a_long_call(gpu, n):
    """Pushes queued behind a force call of some milliseconds, the staging
    overwritten after each: none of them has run when the next one comes."""
    import torch
    nj, ni = 65536, 65536
    rng = np.random.default_rng(n)
    with sp.Sapporo(order=sp.FOURTH, precision=sp.DOUBLE) as s:
        z = np.zeros((nj, 3))
        x = rng.normal(size=(nj, 3))
        s.set_j_particles(np.arange(nj), np.arange(nj), np.zeros(nj), np.ones(nj), x, z, z, z)
        s.force_prediction(nj)
        rec = sp.pack_i_records(sp.FOURTH, x[:ni], z[:ni], np.zeros(ni), np.arange(ni), None)
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        i = torch.from_numpy(rec).cuda()
        res = torch.zeros(ni, sp.RES_STRIDE, dtype=torch.float64, device="cuda")
        want = x[:8 * n].copy()
        torch.cuda.synchronize()
        assert s.lib.sapb_force_device(s.dev, nj, ni, i.data_ptr(), 1e-6, 0, res.data_ptr(),
                                       None, None) == 0
        before = torch.cuda.Event()
        before.record(stream)
        for k in range(6):
            addr = rng.permutation(8 * n)[:n]
            want[addr] = rng.normal(size=(n, 3))
            if k == 0 and n <= 512:
                assert not before.query()
            assert s.lib.sapb_push_j(s.dev, _stage(s, addr, want[addr])) == 0
        _stage(s, np.arange(n), np.full((n, 3), np.nan))  # not pushed
        assert np.array_equal(_positions(s, 8 * n), want)
        s.set_stream(0)


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
