"""GPU: the nearest neighbour's id, looked up in the slice reduction.

A cubic lattice gives every inner particle six nearest neighbours at exactly
the same distance, spread over rows, tiles and slices by a random address
order: the exact-tie paths of the row combine and of the reduction.  One more
particle close to each of a few i makes unique neighbours beside them.
"""
import numpy as np
import pytest

import sapporo2_b200 as sp

pytestmark = pytest.mark.gpu

SIDE = 33  # 35937 j = 140.4 tiles of 256: up to 35 slices, a ragged last tile


def _lattice(seed):
    g = np.arange(SIDE, dtype=np.float64) / 32.0  # exact in float, as are all differences
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(seed)
    x = x[rng.permutation(len(x))]
    x[7] = x[11] + np.array([2.0 ** -9, 0.0, 0.0])  # unique neighbours of each other
    x[-1] = x[-2] + np.array([0.0, 2.0 ** -10, 0.0])  # in the ragged tile
    return x


@pytest.mark.parametrize("precision", [sp.DOUBLESINGLE, sp.DOUBLE])
@pytest.mark.parametrize("launch", [(1, 2, 1), (2, 2, 7), (4, 2, 35), (8, 2, 33), (16, 1, 35),
                                    (32, 1, 2)])
def test_lattice_ties(gpu, precision, launch):
    x = _lattice(5)
    n = len(x)
    ids = np.random.default_rng(6).permutation(n).astype(np.int32)
    at = np.empty(n, dtype=np.int64)
    at[ids] = np.arange(n)
    sel = np.r_[np.arange(0, 300), n - 2, n - 1]
    z = np.zeros((n, 3))
    with sp.Sapporo(order=sp.FOURTH, precision=precision) as s:
        s.set_launch(*launch)
        s.set_j_particles(np.arange(n), ids, np.zeros(n), np.full(n, 1.0 / n), x, z, z, z)
        s.set_no_time()
        s.start(n, ids[sel], x[sel], z[sel], None, 1e-6, np.zeros(len(sel)))
        r = s.results(n)
    for q, i in enumerate(sel):
        d2 = ((x - x[i]) ** 2).sum(1)
        d2[i] = np.inf
        assert r["ds2min"][q] == d2.min()
        assert d2[at[r["nnb"][q]]] == d2.min()
    assert r["nnb"][11] == ids[7] and r["nnb"][7] == ids[11]
    assert r["nnb"][-1] == ids[n - 2] and r["nnb"][-2] == ids[n - 1]
