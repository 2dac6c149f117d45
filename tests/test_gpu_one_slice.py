"""GPU: device-resident calls of one slice, which write their results without
the reduction, against the same call on the fixed scratch, which always takes
the reduction: the same bits."""
import numpy as np
import pytest

import sapporo2_b200 as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [sp.FOURTH, sp.SIXTH])
@pytest.mark.parametrize("precision", [sp.DOUBLESINGLE, sp.DOUBLE])
@pytest.mark.parametrize("nj", [1, 2, 257, 2047, 2100])
def test_with_and_without_the_reduction(gpu, order, precision, nj):
    import torch
    rng = np.random.default_rng(nj)
    # a lattice: several nearest neighbours at exactly the same distance
    x = rng.integers(0, 12, size=(nj, 3)) / 16.0
    z = np.zeros((nj, 3))
    ni = min(nj, 300)
    ids = rng.permutation(nj).astype(np.int32)
    shapes = [(8, 1), (8, 2), (16, 1), (32, 1), (4, 2), (1, 2)]
    with sp.Sapporo(order=order, precision=precision) as s:
        s.set_near(0.0)
        s.set_j_particles(np.arange(nj), ids, np.zeros(nj), np.ones(nj), x, z, z, z,
                          *([z, z] if order == sp.SIXTH else []))
        s.set_no_time()
        s.force_prediction(nj)
        rec = sp.pack_i_records(order, x[:ni], z[:ni], np.zeros(ni), ids[:ni],
                                z[:ni] if order == sp.SIXTH else None)
        i = torch.from_numpy(rec).cuda()
        for shape in shapes:
            s.set_launch(*shape, 1)
            out = []
            for call in (s.lib.sapb_force_device, s.lib.sapb_force_device_noalloc):
                res = torch.full((ni, sp.RES_STRIDE), float("nan"), dtype=torch.float64,
                                 device="cuda")
                torch.cuda.synchronize()
                assert call(s.dev, nj, ni, i.data_ptr(), 1e-2, 0, res.data_ptr(), None, None) == 0
                torch.cuda.synchronize()
                out.append(res.cpu().numpy())
            assert np.array_equal(out[0], out[1]), shape
