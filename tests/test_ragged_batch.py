"""A batch of very many single atoms beside one large system: the energy reduction's work
follows the systems' sizes, and the large system's sums are the ones it gets alone.
"""
import ctypes as C

import numpy as np
import pytest
from conftest import ILP, TERSOFF

from lmff_gb300 import build, capi
from lmff_gb300 import structures as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def test_many_small_systems_beside_a_large_one():
    s = S.graphite_slab(2, 256, 257)          # 526,336 atoms
    small = 524_288
    x = np.ascontiguousarray(s.x)
    t = np.ascontiguousarray(s.type, dtype=np.int32)
    m = np.ascontiguousarray(s.mol, dtype=np.int64)
    lone = np.full((1, 3), 2.0)
    descs = (capi.SystemDesc * (small + 1))()
    d = np.frombuffer(descs, dtype=capi._DESC_DTYPE)
    d["natoms"], d["x"], d["type"], d["mol"], d["v"] = 1, lone.ctypes.data, t.ctypes.data, m.ctypes.data, 0
    d["lo"], d["hi"], d["periodic"] = 0.0, 4.0, 0
    k = 1000
    d["natoms"][k], d["x"][k] = s.n, x.ctypes.data
    d["lo"][k], d["hi"][k], d["periodic"][k] = s.box_lo, s.box_hi, np.asarray(s.periodic, bool)
    alone = capi.Engine(TERSOFF, ILP, elements=("C",), precision=capi.MIXED).compute_system(s)
    eng = capi.Engine(TERSOFF, ILP, elements=("C",), precision=capi.MIXED)
    lib = capi.load_library()
    eng._ck(lib.lmff_batch_set(eng._h, len(d), C.cast(descs, C.c_void_p)))
    res = (capi.Result * len(d))()
    f = np.empty((s.n + small, 3))
    eng._ck(lib.lmff_batch_compute(eng._h, f.ctypes.data_as(C.c_void_p), C.cast(res, C.c_void_p)))
    big = res[k].to_dict()
    for key in ("e_tersoff", "e_ilp"):
        assert big[key] == alone[key]
    for key in ("pvector", "virial_tersoff", "virial_ilp"):
        assert np.array_equal(big[key], alone[key])
    assert np.array_equal(f[k:k + s.n], alone["f"])
    assert not f[:k].any() and not f[k + s.n:].any()
    assert all(res[i].e_tersoff == 0.0 and res[i].e_ilp == 0.0 for i in range(0, len(d), 4099) if i != k)
