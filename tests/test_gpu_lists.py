"""GPU: neighbour lists at the edges of the tiles and of the 32-record groups
whose hits the force kernels keep as one bit per record: j counts around 32
records per row and 256 per tile, every row count, dense lists (up to every j
a neighbour), radii of zero, below zero and NaN, both precisions and orders.

Sets must equal the FP64 ones except for pairs within 1e-6 (relative) of h2.
"""
import numpy as np
import pytest

import sapporo2_b200 as sp

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2, 1), (2, 2, 1), (4, 2, 2), (8, 2, 1), (8, 1, 1), (16, 1, 2), (32, 1, 1)]


def _check(nj, launch, precision, order, spatial=0):
    rng = np.random.default_rng(nj)
    x = rng.uniform(-1, 1, (nj, 3))
    z = np.zeros((nj, 3))
    ids = (rng.permutation(nj) + 7).astype(np.int32)
    ni = min(nj, 150)
    h2 = rng.uniform(0.0, 0.5, ni) * min(1.0, 600.0 / nj)
    h2[::11] = 100.0 if nj <= 250 else 0.0  # all j, or none
    h2[1::13] = -1.0
    h2[2::17] = np.nan
    with sp.Sapporo(order=order, precision=precision) as s:
        s.set_launch(*launch)
        s.set_spatial(spatial)
        six = (z, z) if order == sp.SIXTH else (None, None)
        s.set_j_particles(np.arange(nj), ids, np.zeros(nj), np.full(nj, 1.0 / nj), x, z, z, z, *six)
        s.set_no_time()
        s.start(nj, ids[:ni], x[:ni], z[:ni], z[:ni] if order == sp.SIXTH else None, 1e-6, h2)
        s.results(nj)
        assert not s.read_ngb_list()
        for i in range(ni):
            d2 = ((x - x[i]) ** 2).sum(1)
            d2[i] = np.inf
            with np.errstate(invalid="ignore"):
                want = set(ids[d2 < h2[i]])
                band = set(ids[np.abs(d2 - h2[i]) <= 1e-6 * h2[i]])
            ovf, count, got = s.get_ngb_list(i)
            assert not ovf and count == len(got) == len(set(got)), i
            assert (want ^ set(got)) <= band, (i, want ^ set(got))


@pytest.mark.parametrize("launch", SHAPES + [(1, 4, 1), (2, 4, 1)])
@pytest.mark.parametrize("nj", [1, 5, 31, 33, 64, 250, 257, 520, 1023, 2300])
def test_mixed(gpu, nj, launch):
    _check(nj, launch, sp.DOUBLESINGLE, sp.FOURTH)


@pytest.mark.parametrize("launch", SHAPES)
def test_fp64_and_6th_order(gpu, launch):
    _check(777, launch, sp.DOUBLE, sp.SIXTH)
    _check(777, launch, sp.DOUBLESINGLE, sp.SIXTH)


def test_spatial_mode(gpu):
    _check(5003, (2, 4, 3), sp.DOUBLESINGLE, sp.SIXTH, spatial=2)


def test_batch(gpu):
    """Clusters of ragged sizes in one launch, every j a neighbour."""
    n = [1, 33, 250, 100]
    first = np.concatenate([[0], np.cumsum(n)[:-1]])
    tot = int(np.sum(n))
    rng = np.random.default_rng(3)
    x, z = rng.uniform(-1, 1, (tot, 3)), np.zeros((tot, 3))
    with sp.Sapporo(order=sp.FOURTH) as s:
        s.set_j_particles(np.arange(tot), np.arange(tot), np.zeros(tot), np.ones(tot), x, z, z, z)
        s.force_prediction(tot)
        b = sp.Batch(s, len(n), tot)
        b.i_stage[:] = sp.pack_i_records(1, x, z, np.full(tot, 100.0), np.arange(tot))
        b.plan(first, n, n, np.zeros(len(n)), np.full(len(n), 1e-6))
        b.run(sp.F_NGB_LIST)
        b.results()
        cnt, lst = b.neighbours()
        b.close()
    for f, k in zip(first, n):
        for i in range(f, f + k):
            assert cnt[i] == k - 1
            assert sorted(lst[i, :cnt[i]]) == [j for j in range(f, f + k) if j != i]
