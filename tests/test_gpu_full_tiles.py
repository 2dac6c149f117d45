"""GPU: 4th-order and GRAPE-5 mixed-precision calls on both sides of full j
tiles (256 records), which take a loop of their own: forces against FP64 sums.

Tolerance, in units of the sum of the terms' sizes: FP32 sums of at most
256 / tpi records per tile and about 20 roundings per term, half an ulp each,
and the conversion of the i and j data: (256 + 40) * 2^-24 at most."""
import numpy as np
import pytest

import sapporo2_b200 as sp

pytestmark = pytest.mark.gpu
TOL = (256 + 40) * 2.0 ** -24


@pytest.mark.parametrize("order", [sp.GRAPE5, sp.FOURTH])
@pytest.mark.parametrize("nj", [1, 255, 256, 257, 511, 512, 513, 1100])
def test_tile_edges(gpu, order, nj):
    import torch
    ni = 37
    rng = np.random.default_rng(nj)
    x, v, m = rng.normal(size=(nj, 3)), rng.normal(size=(nj, 3)), rng.uniform(0.5, 1.5, nj)
    xi, vi = rng.normal(size=(ni, 3)), rng.normal(size=(ni, 3))
    eps2, z = 1e-2, np.zeros((nj, 3))
    d = x[None] - xi[:, None]
    w = vi[:, None]
    dv = v[None] - w
    d2 = (d * d).sum(2)
    r3 = m * (d2 + eps2) ** -1.5
    s = -3 * (d * dv).sum(2) / (d2 + eps2)
    want = {"acc": (r3[..., None] * d).sum(1), "pot": -(m * (d2 + eps2) ** -0.5).sum(1),
            "jrk": (r3[..., None] * (dv + s[..., None] * d)).sum(1)}
    size_s = 3 * (np.abs(d) * np.abs(dv)).sum(2) / (d2 + eps2)
    size = {"acc": (r3[..., None] * np.abs(d)).sum(1), "pot": -want["pot"],
            "jrk": (r3[..., None] * (np.abs(dv) + size_s[..., None] * np.abs(d))).sum(1)}
    with sp.Sapporo(order=order, precision=sp.DOUBLESINGLE) as s_:
        s_.set_near(0.0)
        s_.set_j_particles(np.arange(nj), np.arange(nj), np.zeros(nj), m, x, v, z, z)
        s_.set_no_time()
        s_.force_prediction(nj)
        i = torch.from_numpy(sp.pack_i_records(order, xi, vi, np.zeros(ni), nj + np.arange(ni))).cuda()
        for shape in ((1, 2), (2, 2), (4, 2), (8, 2), (1, 4), (2, 4)):
            for slices in (1, 2):
                s_.set_launch(*shape, slices)
                res = torch.full((ni, sp.RES_STRIDE), float("nan"), dtype=torch.float64,
                                 device="cuda")
                torch.cuda.synchronize()
                assert s_.lib.sapb_force_device(s_.dev, nj, ni, i.data_ptr(), eps2, 0,
                                                res.data_ptr(), None, None) == 0
                torch.cuda.synchronize()
                r = res.cpu().numpy()
                got = {"acc": r[:, 0:3], "pot": r[:, 3], "jrk": r[:, 4:7]}
                for f in ("acc", "pot") + (("jrk",) if order == sp.FOURTH else ()):
                    err = np.abs(got[f] - want[f])
                    assert (err <= TOL * size[f]).all(), (shape, slices, f)
                if order == sp.FOURTH:
                    assert (r[:, 11] == d2.argmin(1)).all()
