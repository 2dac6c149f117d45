"""CPU: which addresses a GRAPE-5 upload stages.  The reference hands the
particles to set_j_particle one after another (sapporoG5lib.cpp:111-115): each
address beyond the j memory lets it grow by 10 % once and is refused if that
is not enough (lib/src/sapporohostclass.cpp:453-466, 560-583).  The device side
is the stand-in of tests/host_fake."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import oracle as O

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "sapporo2_b200" / "csrc"

SOURCE = """
#include "sapb_cpu_fake.cpp"
#include "sapporoG5lib.cpp"
extern "C" int staged(int n, int *id, double *m, double *x) {
  grav5.send_j_particles_to_device();
  const sapb_dev *d = g_open[0];
  const int have = std::min(n, d->cap);
  for (int k = 0; k < have; k++) {
    id[k] = d->id[k];
    m[k] = d->m[k];
    for (int q = 0; q < 3; q++) x[3 * k + q] = d->x[3 * (size_t)k + q];
  }
  return d->cap;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    O.lib()  # builds oracle/liboracle.so when missing
    out = tmp_path_factory.mktemp("g5")
    (out / "g5.cpp").write_text(SOURCE)
    so = out / "libg5.so"
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-std=c++17", f"-I{ROOT / 'include'}",
                    f"-I{CSRC}", f"-I{ROOT / 'tests' / 'host_fake'}", str(out / "g5.cpp"),
                    str(CSRC / "sapporohostclass.cpp"), "-o", str(so), f"-L{ROOT / 'oracle'}",
                    "-loracle", f"-Wl,-rpath,{ROOT / 'oracle'}"], check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("addr,nj", [(0, 300), (16380, 10), (16384, 5), (18021, 4), (18022, 9),
                                     (18500, 12), (30000, 40), (-3, 9), (5, 0), (5, -1)])
def test_addresses_beyond_the_j_memory(lib, addr, nj):
    n = 40000
    rng = np.random.default_rng(1)
    x, m = rng.normal(size=(n, 3)), rng.uniform(1, 2, n)
    dp = C.POINTER(C.c_double)
    want, nj_max = {}, 16384
    for a in range(addr, addr + nj):
        if a < 0:
            continue
        if a >= nj_max:
            nj_max = int(nj_max * 1.1) + 1
        if a < nj_max:
            want[a] = a
    assert lib.g5_open_special(1, (C.c_int * 1)(0)) == 0
    try:
        # arrays indexed by address (three entries in front for the negative ones)
        xs, ms = np.concatenate([x[:3], x]), np.concatenate([m[:3], m])
        lib.g5_set_xmj(addr, nj, xs[3:].ctypes.data_as(dp), ms[3:].ctypes.data_as(dp))
        ids = np.full(n, -1, dtype=np.int32)
        gm, gx = np.zeros(n), np.zeros((n, 3))
        cap = lib.staged(n, ids.ctypes.data_as(C.POINTER(C.c_int)), gm.ctypes.data_as(dp),
                         gx.ctypes.data_as(dp))
    finally:
        lib.g5_close()
    assert cap == nj_max
    got = np.nonzero(ids >= 0)[0]
    assert list(got) == sorted(want) and (ids[got] == got).all()
    assert (gm[got] == m[got]).all() and (gx[got] == x[got]).all()
