"""The allocation-free call where the pair list is built in one walk (equal shares of the
scratch) and where an atom's entries or the whole list do not fit that way, against the
resident device call.  The lists and kernels are the same, so the sums differ by a few
roundings at most: 1e-13 of the largest value in FP64, 1e-6 in the mixed mode.
"""
import numpy as np
import pytest
from conftest import ILP, TERSOFF

from lmff_gb300 import build, capi
from lmff_gb300 import structures as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


SYSTEMS = {
    "one_walk": lambda: S.graphite_slab(2, 12, 7),
    "long_lists": lambda: S.graphite_slab(6, 12, 7, mol_mode="unique"),
    "full": lambda: S.graphite_slab(8, 8, 7, mol_mode="unique"),
    "twisted": lambda: S.twisted_bilayer(11, 7, 3.0, top="hbn", spacing=3.3),
}


@pytest.mark.parametrize("which", [capi.TERSOFF, capi.ILP, capi.TERSOFF | capi.ILP])
@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_against_the_resident_call(name, precision, which):
    import torch
    s = S.displace(SYSTEMS[name](), 0.03, seed=4)
    assert s.n <= 2048
    x = torch.tensor(s.x, device="cuda")
    t = torch.tensor(s.type, dtype=torch.int32, device="cuda")
    m = torch.tensor(s.mol, dtype=torch.int64, device="cuda")
    eng = capi.Engine(TERSOFF, ILP, precision=precision)
    eng.set_box(s.box_lo, s.box_hi, s.periodic)
    ref = torch.zeros((s.n, 3), dtype=torch.float64, device="cuda")
    r = eng.compute_device(x, t, m, None, ref, which=which)
    tol = 1e-13 if precision == capi.FP64 else 1e-6
    for _ in range(2):
        f = torch.full((s.n, 3), float("nan"), dtype=torch.float64, device="cuda")
        g = eng.compute_device_noalloc(x, t, m, f, which=which)
        assert (f - ref).abs().max() <= tol * ref.abs().max()
        for k in ("virial_tersoff", "virial_ilp", "pvector"):
            assert np.abs(g[k] - r[k]).max() <= tol * np.abs(r[k]).max()
