"""Performance cases: force calls, ensembles and the neighbour-radius network, each one pass
through the package's public entry points.

A case is a dict of plain values; `path` says which entry point it takes:

* ``class``     the `Sapporo` class on host arrays, as a block-step integrator calls it: the
                `sent` most recently corrected j go to the device again, then one force call on
                the `ni` active particles, then the results (and neighbour counts or lists);
* ``resident``  `sapb_predict` + `sapb_force_device` on tensors that stay on the GPU;
* ``ensemble``  `Batch`: many independent clusters in one launch;
* ``grape5``    the GRAPE-5 interface: new j and i on every call (a treecode's interaction list);
* ``learn``     `H2Net.train`, full-batch epochs from given weights;
* ``propose``   `H2Net.propose`.

Particles are Plummer spheres in Henon units (G = M = 1, E = -1/4), optionally with 10 % of the
particles in tight circular binaries (separations 1e-6 to 1e-4), softening 1e-6, each particle
at its own time within 7/1024 of the force call's.

The mixed-precision kernels sum FP32 terms, so what they return is kept here in single
precision; the FP64 kernels' results stay in double, ids and counts are integers.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import sapporo2_b200 as sp
from sapporo2_b200.learned_h2 import H2Net

EPS2 = 1e-6
TI = 1.0
PLUMMER_B = 3.0 * math.pi / 16.0
MLP_PARAMS = 8769  # W1[64][5] b1 W2[64][64] b2 W3[64][64] b3 W4[64] b4
PAIR_FLOPS = {0: 20, 1: 38, 2: 60}
EXACT_PAIRS = 1.5e10  # 64-bit sums beyond this take too long


# --------------------------------------------------------------------------- cases
def listed():
    return [
        # a deep block step of a small cluster through the class: few active particles, latency
        dict(name="step4_16k_48", path="class", order=1, fp64=False, n=16384, ni=48, sent=48,
             lists="none", binaries=False),
        # 6th order runs in FP64 by default; a regularising integrator reads its lists
        dict(name="step6_fp64_20k_57", path="class", order=2, fp64=True, n=20011, ni=57, sent=57,
             lists="ids", binaries=True),
        # an intermediate block step of a 10^5-body run, neighbour counts back for the radii
        dict(name="step6_100k_2001", path="class", order=2, fp64=False, n=100003, ni=2001,
             sent=2001, lists="counts", binaries=False),
        # a wide block step of 131072 bodies
        dict(name="step6_131k_12983", path="class", order=2, fp64=False, n=131072, ni=12983,
             sent=12983, lists="counts", binaries=False),
        # the plain 4th-order workload: all 16384 active
        dict(name="all4_16k", path="resident", order=1, fp64=False, n=16384, ni=16384,
             lists=False, binaries=False),
        # all-FP64 form, 6th order, all active
        dict(name="all6_fp64_50k", path="resident", order=2, fp64=True, n=50021, ni=50021,
             lists=False, binaries=False),
        # neighbour lists of a block of 8192, read on the device
        dict(name="lists6_131k_8192", path="resident", order=2, fp64=False, n=131072, ni=8192,
             lists=True, binaries=True),
        # precision form: all active, tight binaries; the largest
        dict(name="all6_500k", path="resident", order=2, fp64=False, n=500009, ni=500009,
             lists=False, binaries=True),
        # an ensemble of clusters of 256 to 16384 particles, uneven active sets
        dict(name="ensemble4_192", path="ensemble", order=1, fp64=False, clusters=192, nmin=256,
             nmax=16384),
        # a treecode's call: one interaction list for a group of particles
        dict(name="grape5_2k_9k", path="grape5", ni=2003, n=9001),
        # pretraining of the radius network on start-up counts
        dict(name="learn_65k", path="learn", n=65536, epochs=8),
        # radius proposals for a block of active particles
        dict(name="propose_20k", path="propose", n=20011),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["class"] * 4 + ["resident"] * 4 + ["ensemble", "grape5", "learn", "propose"])
    if path == "class":
        fp64, order = rng.random() < 0.35, rng.choice([1, 2])
        n = _log(rng, 512, 131072)
        ni = min(n, _log(rng, 1, 16384), int((5e8 if fp64 else 2e9) / n))
        lists = rng.choice(["none", "counts"] + (["ids"] if ni <= 128 else []))
        return dict(path=path, order=order, fp64=fp64, n=n, ni=ni, sent=ni, lists=lists,
                    binaries=rng.random() < 0.3)
    if path == "resident":
        fp64, order = rng.random() < 0.35, rng.choice([1, 2])
        n = _log(rng, 2048, 300000 if not fp64 else 65536)
        ni = n if rng.random() < 0.5 else min(n, _log(rng, 64, 65536))
        ni = min(ni, int((3e9 if fp64 else 7e10) / n))
        return dict(path=path, order=order, fp64=fp64, n=n, ni=ni,
                    lists=ni <= 8192 and rng.random() < 0.5, binaries=rng.random() < 0.5)
    if path == "ensemble":
        return dict(path=path, order=rng.choice([1, 1, 2]), fp64=False,
                    clusters=_log(rng, 4, 192), nmin=_log(rng, 64, 512),
                    nmax=_log(rng, 1024, 16384))
    if path == "grape5":
        return dict(path=path, ni=_log(rng, 16, 8192), n=_log(rng, 64, 65536))
    if path == "learn":
        return dict(path=path, n=_log(rng, 256, 65536), epochs=rng.randint(1, 8))
    return dict(path=path, n=_log(rng, 64, 131072))


# --------------------------------------------------------------------------- inputs
def _dirs(rng, n):
    u = rng.standard_normal((n, 3))
    return u / np.linalg.norm(u, axis=1)[:, None]


def _plummer(rng, n, binaries):
    """Positions, velocities, masses; derivatives to crackle from the Plummer field and each
    binary's companion."""
    cut = 10.0 / PLUMMER_B
    q = rng.random(n) * (cut * cut / (1 + cut * cut)) ** 1.5  # mass fraction within the cut
    r = 1.0 / np.sqrt(np.maximum(q, 1e-12) ** (-2.0 / 3.0) - 1.0)
    x = _dirs(rng, n) * (r * PLUMMER_B)[:, None]
    # speed fraction: g(w) ~ w^2 (1 - w^2)^3.5, so w^2 is Beta(3/2, 9/2)
    w = np.sqrt(rng.beta(1.5, 4.5, n))
    speed = w * math.sqrt(2.0 / PLUMMER_B) * (1.0 + r * r) ** -0.25
    v = _dirs(rng, n) * speed[:, None]
    m = np.full(n, 1.0 / n)
    pairs = None
    if binaries:
        k = n // 20
        idx = rng.permutation(n)[:2 * k].reshape(k, 2)
        sep = np.exp(rng.uniform(math.log(1e-6), math.log(1e-4), k))
        e1 = _dirs(rng, k)
        e2 = np.cross(e1, _dirs(rng, k))
        e2 /= np.linalg.norm(e2, axis=1)[:, None]
        dr, dv = sep[:, None] * e1, np.sqrt(2.0 / n / sep)[:, None] * e2
        xc, vc = x[idx[:, 0]].copy(), v[idx[:, 0]].copy()
        x[idx[:, 0]], x[idx[:, 1]] = xc - dr / 2, xc + dr / 2
        v[idx[:, 0]], v[idx[:, 1]] = vc - dv / 2, vc + dv / 2
        pairs = (idx, dr, dv)
    d2 = ((x * x).sum(1) + PLUMMER_B ** 2)[:, None]
    w2 = d2 ** -1.5
    xv, v2 = (x * v).sum(1)[:, None], (v * v).sum(1)[:, None]
    a = -w2 * x
    j = -w2 * (v - 3 * xv / d2 * x)
    s = -w2 * (a - 6 * xv / d2 * v + (15 * xv * xv / (d2 * d2) - 3 * (v2 + (x * a).sum(1)[:, None]) / d2) * x)
    c = -w2 * j
    if pairs is not None:
        idx, dr, dv = pairs
        p3 = ((dr * dr).sum(1) + EPS2)[:, None] ** -1.5 / n
        for col, sign in ((0, 1.0), (1, -1.0)):
            q = idx[:, col]
            a[q] += sign * p3 * dr
            j[q] += sign * p3 * dv
            s[q] -= sign * p3 * p3 * 2 * dr
            c[q] -= sign * p3 * p3 * 2 * dv
    return x, v, m, a, j, s, c


def _radius2(x, n):
    """Squared radius for about 32 neighbours at the local Plummer density, at most 0.3 of the
    distance to the centre in the halo."""
    r2 = (x * x).sum(1)
    rho = 3.0 / (4.0 * math.pi * PLUMMER_B ** 3) * (1.0 + r2 / PLUMMER_B ** 2) ** -2.5
    h2 = (32.0 / n / (4.0 / 3.0 * math.pi * rho)) ** (2.0 / 3.0)
    return np.minimum(h2, 0.09 * np.maximum(r2, PLUMMER_B ** 2))


def _predict(order, dt, x, v, a, j, s, c):
    dt = dt[:, None]
    if order < 2:
        return (x + dt * (v + dt / 2 * (a + dt / 3 * j)), v + dt * (a + dt / 2 * j), None)
    return (x + dt * (v + dt / 2 * (a + dt / 3 * (j + dt / 4 * (s + dt / 5 * c)))),
            v + dt * (a + dt / 2 * (j + dt / 3 * (s + dt / 4 * c))),
            a + dt * (j + dt / 2 * (s + dt / 3 * c)))


class State:
    """What a program holds between calls; closes its handles in the right order."""

    def __del__(self):
        for h in getattr(self, "handles", []):
            try:
                h.close()
            except Exception:
                pass


def _system(case, seed):
    rng = np.random.default_rng([seed, 11])
    n, order = case["n"], case["order"]
    x, v, m, a, j, s, c = _plummer(rng, n, case["binaries"])
    t0 = TI - rng.integers(0, 8, n) / 1024.0
    px, pv, pa = _predict(order, TI - t0, x, v, a, j, s, c)
    act = np.arange(n) if case["ni"] >= n else np.sort(rng.permutation(n)[:case["ni"]])
    return dict(n=n, x=x, v=v, m=m, a=a, j=j, s=s, c=c, t0=t0, px=px, pv=pv, pa=pa, act=act,
                h2=_radius2(px, n))


def _j_args(order, d, q):
    return [q, q.astype(np.int32), d["t0"][q], d["m"][q], d["x"][q], d["v"][q], d["a"][q],
            d["j"][q]] + ([d["s"][q], d["c"][q]] if order >= 2 else [])


def _prec(case):
    return sp.DOUBLE if case["fp64"] else sp.DOUBLESINGLE


def prepare(case, seed):
    st = State()
    st.case = case
    path = case["path"]
    if path in ("class", "resident"):
        d, order = _system(case, seed), case["order"]
        act = d["act"]
        st.sap = sp.Sapporo(order=order, precision=_prec(case))
        st.handles = [st.sap]
        st.sap.set_j_particles(*_j_args(order, d, np.arange(d["n"])))
        st.sap.set_time(TI)
        st.sap.force_prediction(d["n"])
        pa = d["pa"][act] if order >= 2 else None
        if path == "class":
            st.j = _j_args(order, d, act[:case["sent"]])
            st.i = (act.astype(np.int32), d["px"][act], d["pv"][act], pa, EPS2, d["h2"][act])
            return st
        rec = sp.pack_i_records(order, d["px"][act], d["pv"][act], d["h2"][act], act, pa)
        st.stream = torch.cuda.Stream()
        st.sap.set_stream(st.stream.cuda_stream)
        st.i = torch.from_numpy(rec).cuda()
        st.res = torch.zeros(len(act), sp.RES_STRIDE, dtype=torch.float64, device="cuda")
        st.count = st.ids = None
        if case["lists"]:
            st.count = torch.zeros(len(act), dtype=torch.int32, device="cuda")
            st.ids = torch.zeros(len(act), sp.NGB_PB, dtype=torch.int32, device="cuda")
            st.slot = torch.arange(sp.NGB_PB, device="cuda")[None, :]
        torch.cuda.synchronize()
        return st
    if path == "ensemble":
        d, order = _ensemble(case, seed), case["order"]
        st.sap = sp.Sapporo(order=order, precision=_prec(case))
        st.batch = sp.Batch(st.sap, case["clusters"], len(d["act"]))
        st.handles = [st.batch, st.sap]
        st.sap.set_j_particles(*_j_args(order, d, np.arange(len(d["m"]))))
        st.sap.force_prediction(len(d["m"]))
        act = d["act"]
        st.batch.i_stage[:] = sp.pack_i_records(order, d["px"][act], d["pv"][act], d["h2"][act], act,
                                                d["pa"][act] if order >= 2 else None)
        st.plan = (d["j_first"], d["j_count"], d["i_count"], d["t"], np.full(case["clusters"], EPS2))
        return st
    if path == "grape5":
        st.g5 = sp.G5()
        st.x, st.m, st.xi = _group(case, seed)
        return st
    st.sap = sp.Sapporo(order=2)
    st.net = H2Net(st.sap)
    st.handles = [st.net, st.sap]
    if path == "learn":
        st.params, st.x, st.t = _lesson(case, seed)
        return st
    st.net.set_params(_weights(np.random.default_rng([seed, 13])))
    st.net.mu, st.net.sd, st.prev = _history(case, seed)
    return st


def _ensemble(case, seed):
    """Clusters of log-uniform size, each with its own time and a log-uniform active share (sizes
    and shares belong to the case, the particles to the seed)."""
    shape = np.random.default_rng([case["clusters"], case["nmin"], case["nmax"]])
    size = np.exp(shape.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["clusters"])).astype(int)
    share = np.exp(-np.log(size) * shape.random(case["clusters"]))
    rng = np.random.default_rng([seed, 12])
    first = np.concatenate([[0], np.cumsum(size)[:-1]])
    parts, act, count = [], [], []
    times = TI + rng.integers(0, 64, case["clusters"]) / 64.0
    for n, j0, t, f in zip(size, first, times, share):
        x, v, m, a, j, s, c = _plummer(rng, n, False)
        t0 = t - rng.integers(0, 8, n) / 1024.0
        px, pv, pa = _predict(case["order"], t - t0, x, v, a, j, s, c)
        k = max(1, int(n * f))
        act.append(j0 + np.sort(rng.permutation(n)[:k]))
        count.append(k)
        parts.append(dict(x=x, v=v, m=m, a=a, j=j, s=s, c=c, t0=t0, px=px, pv=pv, h2=_radius2(px, n),
                          **({"pa": pa} if pa is not None else {})))
    d = {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
    return dict(d, j_first=first, j_count=size, i_count=np.array(count), t=times,
                act=np.concatenate(act))


def _group(case, seed):
    rng = np.random.default_rng([seed, 14])
    x, _, m, *_ = _plummer(rng, case["n"], False)
    xi = x[rng.integers(0, len(m), case["ni"])] + 1e-3 * rng.standard_normal((case["ni"], 3))
    return x, m, xi


def _weights(rng):
    p = np.zeros(MLP_PARAMS, dtype=np.float32)
    at = 0
    for rows, cols in ((64, 5), (64, 64), (64, 64), (1, 64)):
        p[at:at + rows * cols] = rng.uniform(-1, 1, rows * cols) * math.sqrt(6.0 / (cols + (rows == 1)))
        at += rows * cols + rows
    return p


def _lesson(case, seed):
    """Standardised features and clipped count corrections."""
    rng = np.random.default_rng([seed, 15])
    x = rng.standard_normal((case["n"], 5)).astype(np.float32)
    y = 0.3 * np.tanh(x[:, 0] - 0.5 * x[:, 3]) + 0.1 * rng.standard_normal(case["n"])
    return _weights(rng), x, np.clip(y, -1.0, 0.25).astype(np.float32)


def _history(case, seed):
    rng = np.random.default_rng([seed, 16])
    n = case["n"]
    x, _, m, a, j, *_ = _plummer(rng, n, False)
    count = rng.poisson(32, n).astype(np.float64)
    h2 = _radius2(x, 65536) * np.exp(0.1 * rng.standard_normal(n))
    lrho = np.log(32 / (4 / 3 * math.pi * h2 ** 1.5)) + 0.05 * rng.standard_normal(n)
    mu = np.array([lrho.mean(), 0.0, 0.0, 0.0, np.log(h2).mean()])
    return mu, np.array([2.0, 1.0, 1.0, 0.5, 1.0]), (count, h2, a, j, lrho)


# --------------------------------------------------------------------------- one pass
def run(st):
    return {"class": _run_class, "resident": _run_resident, "ensemble": _run_ensemble,
            "grape5": _run_grape5, "learn": _run_learn, "propose": _run_propose}[st.case["path"]](st)


def _run_class(st):
    case, s, n = st.case, st.sap, st.case["n"]
    if case["sent"]:
        s.set_j_particles(*st.j)
    s.set_time(TI)
    s.start(n, *st.i)
    r = s.results(n)
    real = np.float64 if case["fp64"] else np.float32
    out = {k: r[k].astype(real, copy=False) for k in ("acc", "jrk", "pot", "ds2min")}
    out["nnb"] = r["nnb"]
    if case["order"] >= 2:
        out["snp"] = r["snp"].astype(real, copy=False)
    if case["lists"] == "counts":
        out["count"] = s.neighbour_counts()
    elif case["lists"] == "ids":
        s.read_ngb_list()
        out["count"] = np.zeros(case["ni"], dtype=np.int32)
        out["ids"] = np.full((case["ni"], sp.NGB_PB), -1, dtype=np.int32)
        for k in range(case["ni"]):
            _, out["count"][k], ids = s.get_ngb_list(k)
            out["ids"][k, :len(ids)] = ids
    return out


def _run_resident(st):
    case, s = st.case, st.sap
    lib, flags = s.lib, sp.F_NGB_LIST if case["lists"] else 0
    with torch.cuda.stream(st.stream):
        rc = lib.sapb_predict(s.dev, case["n"], TI)
        rc |= lib.sapb_force_device(s.dev, case["n"], case["ni"], st.i.data_ptr(), EPS2, flags,
                                    st.res.data_ptr(), st.count.data_ptr() if flags else None,
                                    st.ids.data_ptr() if flags else None)
        if rc:
            raise RuntimeError("force call failed: %d" % rc)
        f = st.res[:, :11] if case["fp64"] else st.res[:, :11].float()
        out = _columns(f, case["order"])
        out["nnb"] = st.res[:, 11].to(torch.int32)
        if flags:
            out["count"] = st.count
            out["ids"] = torch.where(st.slot < st.count[:, None], st.ids, 1 << 30).sort(1)[0]
    return out


def _columns(f, order):
    """Result records by field: acc[3] pot jerk[3] snap[3] ds2min."""
    out = {"acc": f[:, 0:3], "pot": f[:, 3], "jrk": f[:, 4:7], "ds2min": f[:, 10]}
    if order >= 2:
        out["snp"] = f[:, 7:10]
    return out


def _run_ensemble(st):
    st.batch.plan(*st.plan)
    st.batch.run(sp.F_PREDICT)
    r = st.batch.results()
    out = _columns(r[:, :11].astype(np.float32), st.case["order"])
    out["nnb"] = r[:, 11].astype(np.int32)
    return out


def _run_grape5(st):
    st.g5.set_eps(math.sqrt(EPS2))
    st.g5.set_j(st.x, st.m)
    a, phi = st.g5.force(st.xi)
    return {"acc": a.astype(np.float32), "pot": phi.astype(np.float32)}


def _run_learn(st):
    st.net.set_params(st.params)
    loss = st.net.train(st.x, st.t, st.case["epochs"], 1e-3)
    return {"params": st.net.params(), "loss": np.float32(loss)}


def _run_propose(st):
    return st.net.propose(*st.prev).astype(np.float32)


# --------------------------------------------------------------------------- work
def work(case):
    path = case["path"]
    if path == "learn":
        n, e = case["n"], case["epochs"]
        return {"bytes": 24 * n + 8 * MLP_PARAMS + 4, "flops": 6 * 8576 * n * e}
    if path == "propose":
        return {"bytes": 40 * case["n"] + 4 * MLP_PARAMS, "flops": 2 * 8576 * case["n"]}
    if path == "grape5":
        return {"bytes": 32 * case["n"] + 24 * case["ni"] + 32 * case["ni"],
                "flops": PAIR_FLOPS[0] * case["n"] * case["ni"]}
    order = case["order"]
    jb, ib = (20 * 8 + 4, 12 * 8) if order >= 2 else (14 * 8 + 4, 8 * 8)
    if path == "ensemble":
        # expected sums over log-uniform sizes and active shares
        lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
        span = max(hi - lo, 1e-9)
        size = (math.exp(hi) - math.exp(lo)) / span
        grid = [math.exp(lo + (k + 0.5) / 64 * span) for k in range(64)]
        share = [(1 - 1 / g) / math.log(g) for g in grid]
        act = sum(g * s for g, s in zip(grid, share)) / 64
        pairs = sum(g * g * s for g, s in zip(grid, share)) / 64
        return {"bytes": case["clusters"] * (jb * size + (ib + 96) * act),
                "flops": case["clusters"] * PAIR_FLOPS[order] * pairs}
    n, ni = case["n"], case["ni"]
    sent = case.get("sent", 0) * (22 if order >= 2 else 16) * 8
    return {"bytes": jb * n + (ib + 96) * ni + sent, "flops": PAIR_FLOPS[order] * n * ni}


# --------------------------------------------------------------------------- 64-bit values
def _sum64(order, xi, vi, ai, own, xj, vj, aj, m):
    """acc, pot, jerk, snap and nearest ds2 of each i in 64 bits; `own`: the i's index among the
    j (its self pair is left out), None to keep every pair."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def put(q):
        return None if q is None else torch.from_numpy(np.ascontiguousarray(q)).to(dev)

    xi, vi, ai, own, xj, vj, aj, m = map(put, (xi, vi, ai, own, xj, vj, aj, m))
    n, out = len(m), []
    rows = max(1, int(1.6e7) // n)
    col = torch.arange(n, device=dev)[None, :]
    for i0 in range(0, len(xi), rows):
        sl = slice(i0, i0 + rows)
        d = [xj[None, :, k] - xi[sl, None, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        skip = None if own is None else own[sl, None] == col
        inv = (r2 + EPS2).rsqrt()
        mi = m[None, :] * inv
        if skip is not None:
            mi = mi.masked_fill(skip, 0.0)
            r2 = r2.masked_fill(skip, 1e11)
        i2 = inv * inv
        m3 = mi * i2
        f = [(m3 * q).sum(1) for q in d] + [-mi.sum(1)]
        if order >= 1:
            dv = [vj[None, :, k] - vi[sl, None, k] for k in range(3)]
            al = (d[0] * dv[0] + d[1] * dv[1] + d[2] * dv[2]) * i2
            jk = [m3 * (p - 3 * al * q) for p, q in zip(dv, d)]
            f += [q.sum(1) for q in jk]
            if order >= 2:
                da = [aj[None, :, k] - ai[sl, None, k] for k in range(3)]
                be = sum(p * p for p in dv) + sum(p * q for p, q in zip(d, da))
                be = be * i2 + al * al
                f += [(m3 * (p - 3 * be * q) - 6 * al * t).sum(1) for p, q, t in zip(da, d, jk)]
            else:
                f += [torch.zeros_like(f[0])] * 3
            f.append(r2.min(1)[0])
        out.append(torch.stack(f, 1))
    return torch.cat(out).cpu().numpy()


def _exact_fields(case, f):
    out = _columns(f, case["order"])
    out["nnb"] = None
    if case.get("lists") in (True, "counts", "ids"):
        out["count"] = None
    if case.get("lists") in (True, "ids"):
        out["ids"] = None
    return out


def exact(case, seed):
    path = case["path"]
    if path in ("class", "resident"):
        if float(case["n"]) * case["ni"] > EXACT_PAIRS:
            return None
        d = _system(case, seed)
        q = d["act"]
        return _exact_fields(case, _sum64(
            case["order"], d["px"][q], d["pv"][q], None if d["pa"] is None else d["pa"][q], q,
            d["px"], d["pv"], d["pa"], d["m"]))
    if path == "ensemble":
        d, out, i0 = _ensemble(case, seed), [], 0
        for j0, n, k in zip(d["j_first"], d["j_count"], d["i_count"]):
            j, q = slice(j0, j0 + n), d["act"][i0:i0 + k]
            pa = d.get("pa")
            out.append(_sum64(case["order"], d["px"][q], d["pv"][q], None if pa is None else pa[q],
                              q - j0, d["px"][j], d["pv"][j], None if pa is None else pa[j], d["m"][j]))
            i0 += k
        return _exact_fields(case, np.concatenate(out))
    if path == "grape5":
        x, m, xi = _group(case, seed)
        f = _sum64(0, xi, None, None, None, x, None, None, m)
        return {"acc": f[:, :3], "pot": f[:, 3]}
    if path == "learn":
        return _exact_learn(case, *_lesson(case, seed))
    mu, sd, (count, h2, a, j, lrho) = _history(case, seed)
    lr = np.log(count.clip(0.5)) - math.log(4 / 3 * math.pi) - 1.5 * np.log(h2)
    f = np.stack([lr, np.log(np.linalg.norm(a, axis=1)), np.log(np.linalg.norm(j, axis=1)), lrho - lr,
                  np.log(h2)], 1)
    p = torch.from_numpy(_weights(np.random.default_rng([seed, 13])).astype(np.float64))
    corr = _mlp64(p, torch.from_numpy((f - mu) / sd)).numpy().clip(-1.0, 0.25)
    return h2 * np.exp((2 / 3 * np.log(32 / count.clip(0.5)) + corr).clip(-4, 4))


def _mlp64(p, x):
    at = 0
    for rows, cols in ((64, 5), (64, 64), (64, 64), (1, 64)):
        w = p[at:at + rows * cols].view(rows, cols)
        at += rows * cols
        x = x @ w.T + p[at:at + rows]
        at += rows
        if rows > 1:
            x = x.relu()
    return x[:, 0]


def _exact_learn(case, params, x, t):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p, x, t = (torch.from_numpy(q.astype(np.float64)).to(dev) for q in (params, x, t))
    p.requires_grad_(True)
    m1, m2, loss = torch.zeros_like(p), torch.zeros_like(p), None
    for k in range(1, case["epochs"] + 1):
        loss = 0.5 * ((_mlp64(p, x) - t) ** 2).mean()
        g, = torch.autograd.grad(loss, p)
        with torch.no_grad():
            m1 = 0.9 * m1 + 0.1 * g
            m2 = 0.999 * m2 + 0.001 * g * g
            p -= 1e-3 * (m1 / (1 - 0.9 ** k)) / ((m2 / (1 - 0.999 ** k)).sqrt() + 1e-8)
    return {"params": p.detach().cpu().numpy(), "loss": float(loss.detach())}
