"""GPU: the network's parameters travel on the handle's stream, in the order of
the calls, whatever the default stream is busy with."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 64, 256])
def test_parameters_do_not_wait_for_the_default_stream(gpu, n):
    import torch

    import sapporo2_b200 as sp
    from sapporo2_b200.learned_h2 import H2Net
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, M.IN)).astype(np.float32)
    t = rng.normal(size=n).astype(np.float32)
    with sp.Sapporo(order=sp.SIXTH) as s:
        net = H2Net(s, seed=3)
        start = [net.params()]
        start.append(start[0] * np.float32(0.5))
        want = []
        for p in start:  # also allocates the buffers
            net.set_params(p)
            net.train(x, t, epochs=2)
            want.append(net.params())
        assert not np.array_equal(want[0], want[1])
        torch.cuda.synchronize()
        torch.cuda._sleep(400_000_000)  # about 0.2 s of the default stream
        busy = torch.cuda.Event()
        busy.record()
        for k in range(8):
            net.set_params(start[k % 2])
            net.train(x, t, epochs=2)
            assert np.array_equal(net.params(), want[k % 2])
        assert not busy.query()  # nothing above went through the default stream
        torch.cuda.synchronize()
        net.close()


def test_parameters_under_capture_are_refused(gpu):
    import torch

    import sapporo2_b200 as sp
    from sapporo2_b200.learned_h2 import H2Net
    with sp.Sapporo(order=sp.SIXTH) as s:
        net = H2Net(s, seed=3)
        p = net.params()
        stream = torch.cuda.Stream()
        s.set_stream(stream.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        one = torch.zeros(1, device="cuda")
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            one += 1
            with pytest.raises(sp.SapporoError):
                net.set_params(p * 2)
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(net.params(), p)
        s.set_stream(0)
        net.close()
