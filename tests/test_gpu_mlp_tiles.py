"""GPU: the network's kernels at the edges of their 64-sample chunks and of
the backward kernel's grid (two blocks per SM), against the FP64 oracle.

Tolerance per parameter block, relative to its norm: FP32 dot products of 64
terms through three layers and back err by at most 6 * 64 * 2^-24 = 2.3e-5,
and a unit whose pre-activation is within that of zero may take the other
side of its ReLU, which moves a coherent gradient (targets offset from the
outputs) by about 1 / (8 n) per unit: 1e-4 covers both.
"""
import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 129, 18944, 18945, 20000])
def test_chunk_edges(gpu, n):
    import sapporo2_b200 as sp
    from sapporo2_b200.learned_h2 import H2Net
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, M.IN)).astype(np.float32)
    t = (rng.normal(size=n) + 3.0).astype(np.float32)
    with sp.Sapporo(order=sp.SIXTH) as s:
        net = H2Net(s, seed=17)
        p = net.params().astype(np.float64)
        y, yo = net.forward(x), M.forward(p, x)[0]
        assert np.max(np.abs(y - yo)) <= 1e-5 * max(1.0, np.max(np.abs(yo)))
        g, loss = net.gradient(x, t)
        again, _ = net.gradient(x, t)
        net.close()
    assert np.array_equal(g, again)  # fixed summation order
    assert abs(loss - M.loss(p, x, t)) <= 1e-5 * M.loss(p, x, t)
    got, want = M.unpack(g), M.unpack(M.gradient(p, x, t))
    for name in want:
        err = np.linalg.norm(got[name] - want[name])
        assert err <= 1e-4 * np.linalg.norm(want[name]), (name, err)
