"""GPU: launch shapes that the planner picks for device-resident calls where
another family was measured slower."""
import pytest

import sapporo2_b200 as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,ni,nj,shapes", [
    (sp.SIXTH, 16384, 1 << 20, {(1, 4), (2, 4)}),  # (4, 2): 5-6 % slower
    (sp.FOURTH, 32768, 262144, {(1, 4), (2, 4)}),  # (4, 2): 7 % slower
    (sp.SIXTH, 59000, 200000, {(1, 4), (2, 4)}),
    (sp.SIXTH, 1000, 65536, {(16, 1)}),  # (32, 1): 27 % slower
])
def test_shapes(gpu, order, ni, nj, shapes):
    with sp.Sapporo(order=order, precision=sp.DOUBLESINGLE) as s:
        assert s.plan(ni, nj)[:2] in shapes


@pytest.mark.parametrize("ni,nj", [(65536, 65536), (262144, 262144), (1 << 20, 1 << 20)])
def test_large_fp64_calls(gpu, ni, nj):
    with sp.Sapporo(order=sp.SIXTH, precision=sp.DOUBLE) as s:
        assert s.plan(ni, nj)[:2] == (2, 2)  # (8, 2): 3 % slower at 262144 x 262144
