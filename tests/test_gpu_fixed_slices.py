"""GPU: slices fixed by the caller keep at least four j tiles each, and no plan
has more slices than the launch grid takes."""
import pytest

import sapporo2_b200 as sp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nj,asked,want", [
    (16384, 64, 16),  # 64 tiles
    (1000, 5, 1),
    (35937, 35, 29),  # 141 tiles: five each
    (1 << 25, 200000, 32768),
    (1 << 28, 200000, 61681),  # 2^20 tiles: 65535 slices of 17 at most
])
def test_fixed_slices(gpu, nj, asked, want):
    with sp.Sapporo(order=sp.FOURTH, precision=sp.DOUBLESINGLE) as s:
        s.set_launch(8, 2, asked)
        assert s.plan(64, nj) == (8, 2, want)


@pytest.mark.parametrize("precision", [sp.DOUBLESINGLE, sp.DOUBLE])
def test_planned_slices_fit_the_grid(gpu, precision):
    with sp.Sapporo(order=sp.SIXTH, precision=precision) as s:
        for ni in (1, 17, 1000):
            for nj in (1 << 20, 1 << 25, 1 << 28, 2 ** 30):
                assert 1 <= s.plan(ni, nj)[2] <= 65535
