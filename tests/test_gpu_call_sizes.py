"""GPU: host calls on both sides of the sizes where their path changes.

Pushes of up to 512 records and force calls of up to 16384 i take a path of
their own; neighbour lists in address order change theirs at 65536 j; the
slice reduction gives an i 8 or 32 lanes; spatial calls of few i take the
shapes of address order.  Pushed states must come back bit for bit, nearest
neighbours and lists must be those of FP64, forces within the rounding of a
FP64 sum (FP64 kernels) or the tolerances of the parity tests (mixed).
"""
import numpy as np
import pytest

import sapporo2_b200 as sp
from tests import cases as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 511, 512, 513, 1200])
def test_pushes_back_to_back(gpu, n):
    """Six pushes, with no call between them that waits for the GPU; each
    overwrites the half of the one before it."""
    rng = np.random.default_rng(n)
    nj = 2 * n
    x = np.full((nj, 3), np.nan)
    with sp.Sapporo(order=sp.FOURTH, precision=sp.DOUBLESINGLE) as s:
        z = np.zeros((nj, 3))
        s.set_j_particles(np.arange(nj), np.arange(nj), np.zeros(nj), np.ones(nj), z, z, z, z)
        s.set_no_time()
        s.start(nj, [nj], np.ones((1, 3)), z[:1], None, 1e-6, np.zeros(1))
        s.results(nj)
        for k in range(6):
            addr = rng.permutation(nj)[:n]
            x[addr] = rng.normal(size=(n, 3))
            s.set_j_particles(addr, addr, np.zeros(n), np.ones(n), x[addr], z[:n], z[:n], z[:n])
            s.start(nj, [nj], np.ones((1, 3)), z[:1], None, 1e-6, np.zeros(1))
        s.results(nj)
        for a in np.nonzero(np.isfinite(x[:, 0]))[0][:: max(1, n // 40)]:
            assert np.array_equal(s.retrieve_state(int(a))["pos"], x[a])


@pytest.mark.parametrize("ni", [16384, 16385])
def test_direct_calls(gpu, ni):
    nj = 700
    rng = np.random.default_rng(ni)
    x, v = rng.normal(size=(nj, 3)), rng.normal(size=(nj, 3))
    m = rng.uniform(0.5, 1.5, nj)
    xi, vi = rng.normal(size=(ni, 3)), rng.normal(size=(ni, 3))
    z = np.zeros((nj, 3))
    eps2, ids = 1e-2, np.arange(nj)
    with sp.Sapporo(order=sp.FOURTH, precision=sp.DOUBLE) as s:
        s.set_j_particles(ids, ids, np.zeros(nj), m, x, v, z, z)
        s.set_no_time()
        for _ in range(2):
            s.start(nj, np.arange(nj, nj + ni), xi, vi, None, eps2, np.full(ni, 0.01))
            r = s.results(nj)
        assert not s.read_ngb_list()
        sets = [s.get_ngb_list(i)[2] for i in (0, 1, ni // 2, ni - 2, ni - 1)]
    for i, got in zip((0, 1, ni // 2, ni - 2, ni - 1), sets):
        assert set(got) == set(ids[((x - xi[i]) ** 2).sum(1) < 0.01])
    for i in np.r_[0:40, ni - 300: ni]:
        dr, dv = x - xi[i], v - vi[i]
        d2 = (dr ** 2).sum(1)
        r3 = m * (d2 + eps2) ** -1.5
        # nj additions and about 20 roundings per term, half an ulp each, in
        # units of the sum of the terms' sizes
        tol = (nj + 20) * 2.0 ** -52
        assert r["nnb"][i] == d2.argmin()
        assert (np.abs(r["acc"][i] - r3 @ dr) <= tol * (r3 @ np.abs(dr))).all()
        jt = r3[:, None] * dv, (-3 * r3 * (dr * dv).sum(1) / (d2 + eps2))[:, None] * dr
        size = 3 * r3 * (np.abs(dr) * np.abs(dv)).sum(1) / (d2 + eps2)
        assert (np.abs(r["jrk"][i] - (jt[0] + jt[1]).sum(0))
                <= tol * (np.abs(jt[0]).sum(0) + size @ np.abs(dr))).all()


@pytest.mark.parametrize("nj", [65535, 65536])
def test_lists_on_many_j(gpu, nj):
    rng = np.random.default_rng(nj)
    x = rng.uniform(-1, 1, (nj, 3))
    z = np.zeros((nj, 3))
    sel = np.r_[0:100, nj - 100: nj]
    h2 = rng.uniform(0.0, 0.008, len(sel))
    with sp.Sapporo(order=sp.FOURTH, precision=sp.DOUBLESINGLE) as s:
        s.set_spatial(0)
        s.set_j_particles(np.arange(nj), np.arange(nj), np.zeros(nj), np.ones(nj), x, z, z, z)
        s.set_no_time()
        s.start(nj, sel, x[sel], z[sel], None, 1e-6, h2)
        s.results(nj)
        assert not s.read_ngb_list()
        for q, i in enumerate(sel):
            d2 = ((x - x[i]) ** 2).sum(1)
            d2[i] = np.inf
            got = s.get_ngb_list(q)[2]
            band = set(np.nonzero(np.abs(d2 - h2[q]) <= 1e-6 * h2[q])[0])
            assert len(set(got)) == len(got)
            assert (set(np.nonzero(d2 < h2[q])[0]) ^ set(got)) <= band


@pytest.mark.parametrize("precision", [sp.DOUBLESINGLE, sp.DOUBLE])
@pytest.mark.parametrize("ni", [9472, 9473])  # 64 i on each of 148 SMs
def test_reduction_lanes_on_a_lattice(gpu, precision, ni):
    """Exact ties between slices, read by 32 and by 8 lanes per i."""
    g = np.arange(22, dtype=np.float64) / 32.0
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    n = len(x)
    x = x[np.random.default_rng(3).permutation(n)]
    z = np.zeros((n, 3))
    sel = np.arange(ni)
    with sp.Sapporo(order=sp.FOURTH, precision=precision) as s:
        s.set_launch(4, 2, 11)
        s.set_j_particles(np.arange(n), np.arange(n), np.zeros(n), np.ones(n), x, z, z, z)
        s.set_no_time()
        s.start(n, sel, x[sel], z[sel], None, 1e-6, np.zeros(ni))
        r = s.results(n)
    d2 = ((x[r["nnb"]] - x[sel]) ** 2).sum(1)
    assert (r["nnb"] != sel).all()
    assert (d2 == 2.0 ** -10).all() and (r["ds2min"] == 2.0 ** -10).all()


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("ni", [1, 255, 600, 1023, 1024])
def test_spatial_calls_of_few_i(gpu, order, ni):
    """Spatial mode asked for at every size, planned shapes."""
    case = T.build_case(order, 6000, seed=31, binaries=0.1)
    sel = np.random.default_rng(ni).permutation(6000)[:ni]
    want = T.oracle_force(case, sel=sel)
    got = T.run_library(case, sp.DOUBLESINGLE, sel=sel, spatial=(2, 0.0))
    T.check_forces(got, want, order)
    T.check_nn(case, got["nnb"], want, sel=sel)
    T.check_neighbours(case, got["ngb_sets"], got["ngb_count"], want, sel=sel)


def test_prediction_times_by_address(gpu):
    """Calls that reach fewer j leave the others at the time they had."""
    n = 40
    z = np.zeros((n, 3))
    v = np.ones((n, 3))
    with sp.Sapporo(order=sp.FOURTH, precision=sp.DOUBLESINGLE) as s:
        s.set_j_particles(np.arange(n), np.arange(n), np.zeros(n), np.ones(n), z, v, z, z)
        for t, nj in ((1.0, 40), (2.0, 30), (3.0, 10), (4.0, 20)):
            s.set_time(t)
            s.start(nj, [n], np.ones((1, 3)), z[:1], None, 1e-6, np.zeros(1))
            s.results(nj)
        for addr, t in ((0, 4.0), (19, 4.0), (20, 2.0), (29, 2.0), (30, 1.0), (39, 1.0)):
            assert np.array_equal(s.retrieve_predicted(addr)["pos"], [t, t, t]), addr
