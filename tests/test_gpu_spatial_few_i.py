"""GPU: spatial mode asked for at every size is on at every size: planned shapes
are ones whose kernels evaluate tiles in it."""
import numpy as np
import pytest

import sapporo2_b200 as sp
from tests import cases as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("ni", [1, 255, 600, 1023, 1024])
def test_tiles_are_evaluated_in_spatial_mode(gpu, order, ni):
    case = T.build_case(order, 6000, seed=33)
    sel = np.random.default_rng(ni).permutation(6000)[:ni]
    got = T.run_library(case, sp.DOUBLESINGLE, sel=sel, spatial=(2, 0.0))
    want = T.oracle_force(case, sel=sel)
    far, tiles = got["far_tiles"]
    assert tiles >= 24 and 0 <= far <= tiles  # 24 tiles, each seen by a warp or more
    T.check_forces(got, want, order)
    T.check_nn(case, got["nnb"], want, sel=sel)
    T.check_neighbours(case, got["ngb_sets"], got["ngb_count"], want, sel=sel)


@pytest.mark.parametrize("ni,nj", [(1, 5000), (500, 1 << 20), (1000, 1 << 23), (5000, 70000)])
def test_planned_shapes_have_pairs_of_i(gpu, ni, nj):
    for order in (1, 2):
        with sp.Sapporo(order=order, precision=sp.DOUBLESINGLE) as s:
            s.set_spatial(2)
            assert s.plan(ni, nj)[1] % 2 == 0
