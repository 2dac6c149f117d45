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
