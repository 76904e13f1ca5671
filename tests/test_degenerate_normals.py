"""Atoms whose two intralayer neighbours lie on one line have no normal: every evaluation
says so in either precision, with the interlayer style or with Tersoff alone, and the
engine serves the next call.
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


def _line():
    """A bilayer and, clear of it, three atoms on a line."""
    s = S.displace(S.flake_edges(5, 3), 0.03, seed=3)
    x = np.array([[0.0, 0.0, 0.0], [1.5, 0.0, 0.0], [3.0, 0.0, 0.0]]) + s.box_lo + np.array([4.0, 4.0, 40.0])
    n = s.n
    return (np.concatenate([s.x, x]), np.concatenate([s.type, [1, 1, 1]]), np.concatenate([s.mol, [7, 7, 7]]),
            np.arange(1, n + 4), s)


def _engine(s, precision):
    eng = capi.Engine(TERSOFF, ILP, precision=precision)
    eng.set_box(s.box_lo, s.box_hi + np.array([0.0, 0.0, 60.0]), s.periodic)
    return eng


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("which", [capi.TERSOFF, capi.ILP, capi.TERSOFF | capi.ILP])
@pytest.mark.parametrize("ev", [False, True])
def test_refused(which, precision, ev):
    x, t, m, g, s = _line()
    eng = _engine(s, precision)
    with pytest.raises(capi.LmffError, match="normal"):
        eng.compute(x, t, m, g, which=which, eflag=ev, vflag=ev)
    x[-1, 1] += 0.3
    eng.compute(x, t, m, g, which=which, eflag=ev, vflag=ev)


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("which", [capi.TERSOFF, capi.ILP, capi.TERSOFF | capi.ILP])
def test_refused_without_allocation(which, precision):
    import torch
    x, t, m, g, s = _line()
    eng = _engine(s, precision)
    f = torch.zeros(len(t), 3, dtype=torch.float64, device="cuda")
    args = [torch.tensor(a, device="cuda") for a in (t.astype(np.int32), m.astype(np.int64))]
    with pytest.raises(capi.LmffError, match="normal"):
        eng.compute_device_noalloc(torch.tensor(x, device="cuda"), *args, f, which=which)
    x[-1, 1] += 0.3
    eng.compute_device_noalloc(torch.tensor(x, device="cuda"), *args, f, which=which)


def test_per_atom_virial_leaves_no_error_behind():
    """Three atoms on a line whose cross product is zero in FP64 and a rounding in FP32: the
    mixed evaluation goes through, and so does the next one after the per-atom virial, which
    makes the normals in FP64."""
    x, t, m, g, s = _line()
    v = np.array([943718, 838861, 734003]) * 2.0 ** -20   # products exact in FP64, not in FP32
    x[-3:] = np.round(x[-2]) + np.array([-1.0, 0.0, 1.0])[:, None] * v
    eng = _engine(s, capi.MIXED)
    eng.compute(x, t, m, g)
    eng.set_precision(capi.FP64)
    eng.vatom(capi.ILP)
    x[-1, 1] += 0.3
    eng.compute(x, t, m, g, same_atoms=True)
