"""The FP64 mode's double-float interlayer kernel against the general FP64 one.

Option list_full keeps the general kernel (FP64 instructions throughout), so the two run on
the same system.  A pair's force is within ~3e-13 of its rms in either form (1/sqrt and 1/x
of the general one are a Newton step from an FP32 estimate); an atom sums some 1,500 such
errors of either sign against a net force of the same size or larger, so 1e-11 of the
largest force bounds the difference with an order of magnitude to spare.
"""
import numpy as np
import pytest
from conftest import ILP, TERSOFF

from lmff_gb300 import build, capi
from lmff_gb300 import structures as S

pytestmark = pytest.mark.gpu

TOL = 1e-11


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _pair(s, elements=("C", "B", "N"), tap=1, tpa=16, block=128, **kw):
    out = []
    for full in (0, 1):
        eng = capi.Engine(TERSOFF, ILP, elements=elements, tap_flag=tap)
        eng.set_option("tpa", tpa)
        eng.set_option("block", block)
        eng.set_option("list_full", full)
        out.append(eng.compute_system(s, which=capi.ILP, **kw))
    return out


def _close(a, b):
    assert np.abs(a["f"] - b["f"]).max() <= TOL * np.abs(b["f"]).max()


def _scalars(a, b):
    for k in ("pvector", "virial_ilp"):
        assert np.abs(a[k] - b[k]).max() <= TOL * np.abs(b[k]).max(), k


@pytest.mark.parametrize("tap", [0, 1])
@pytest.mark.parametrize("tpa,block", [(4, 64), (8, 128), (16, 256), (32, 32)])
def test_twisted_hbn_and_odd_sizes(tap, tpa, block):
    s = S.displace(S.twisted_bilayer(11, 7, 3.0, top="hbn", spacing=3.3), 0.05, seed=5)
    a, b = _pair(s, tap=tap, tpa=tpa, block=block, eatom=True)
    _close(a, b)
    _scalars(a, b)
    assert np.abs(a["eatom"] - b["eatom"]).max() <= TOL * np.abs(b["eatom"]).max()
    a, b = _pair(s, tap=tap, tpa=tpa, block=block, eflag=False, vflag=False)
    _close(a, b)


@pytest.mark.parametrize("n", [1, 2, 3])
def test_single_cells_with_many_images(n):
    """Boxes of one to three cells: several image shifts per dimension, every list entry
    an image, list lengths that leave single entries to the packed loop."""
    s = S.displace(S.graphite_slab(3, n, 1, mol_mode="unique"), 0.05, seed=n)
    for el in (("C",), ("C", "B", "N")):
        a, b = _pair(s, elements=el)
        _close(a, b)
        _scalars(a, b)


def test_far_from_the_origin_and_outside_the_box():
    """Boxes away from the origin (coarser position grids), and atoms far outside the box in
    its non-periodic dimension."""
    s = S.displace(S.graphite_slab(2, 6, 4), 0.03, seed=2)
    for off in (0.0, 500.0, -2000.0):
        t = s.copy()
        t.x = t.x + off
        t.box_lo, t.box_hi = t.box_lo + off, t.box_hi + off
        _close(*_pair(t))
    for dz in (300.0, 3.0e3, 2.0e4):
        t = s.copy()
        t.x[:, 2] += dz
        _close(*_pair(t))


def test_close_pairs_and_free_atoms():
    """Interlayer pairs down to 0.01 A (evaluated apart, in FP64) and free edges."""
    s = S.displace(S.flake_edges(6, 4), 0.03, seed=3)
    a, b = _pair(s)
    _close(a, b)
    _scalars(a, b)
    for r in (0.01, 0.3, 0.4999, 0.5001):
        t = S.displace(S.graphite_slab(2, 5, 3), 0.02, seed=4)
        j = t.n - 1
        t.x[j] = t.x[0] + r * np.array([0.6, 0.0, 0.8])
        a, b = _pair(t)
        _close(a, b)
        _scalars(a, b)
        rest = np.abs(b["f"]).max(axis=1) < 10.0   # atoms away from the close pair
        assert rest.sum() > 20
        assert np.abs(a["f"] - b["f"])[rest].max() <= 10.0 * TOL


def test_per_atom_virial():
    """The per-atom virial's double-float pass against the FP64 one: several elements and
    images, free edges with zero to three intralayer neighbours, a close pair."""
    t = S.displace(S.graphite_slab(2, 5, 3), 0.02, seed=4)
    t.x[-1] = t.x[0] + 0.3 * np.array([0.6, 0.0, 0.8])
    for s in (S.displace(S.twisted_bilayer(11, 7, 3.0, top="hbn", spacing=3.3), 0.05, seed=5),
              S.displace(S.graphite_slab(3, 1, 1, mol_mode="unique"), 0.05, seed=1),
              S.displace(S.flake_edges(6, 4), 0.03, seed=3), t):
        a, b = _pair(s, vatom=True)
        assert np.abs(a["vatom_ilp"] - b["vatom_ilp"]).max() <= TOL * np.abs(b["vatom_ilp"]).max()


@pytest.mark.parametrize("cut", [5.0, 7.0, 8.0, 16.0])
def test_per_atom_virial_near_and_far_pairs(cut):
    """Cutoffs below, at and above the distance that splits the pass's pairs, and a pair of
    layers about that distance apart."""
    for s in (S.displace(S.graphite_slab(4, 6, 4, mol_mode="unique"), 0.03, seed=9),
              S.displace(S.twisted_bilayer(11, 7, 3.0, top="hbn", spacing=7.0), 1e-6, seed=5)):
        r = []
        for full in (0, 1):
            eng = capi.Engine(TERSOFF, ILP, cut_global=cut)
            eng.set_option("list_full", full)
            r.append(eng.compute_system(s, which=capi.ILP, vatom=True)["vatom_ilp"])
        assert np.abs(r[0] - r[1]).max() <= TOL * np.abs(r[1]).max()


def test_per_atom_virial_after_a_change_of_precision():
    """The per-atom virial of a mixed evaluation asked for in FP64: an engine that has not
    evaluated in FP64 before."""
    s = S.displace(S.twisted_bilayer(11, 7, 3.0, top="hbn", spacing=3.3), 0.05, seed=5)
    eng = capi.Engine(TERSOFF, ILP, precision=capi.MIXED)
    eng.compute_system(s)
    eng.set_precision(capi.FP64)
    got = eng.vatom(capi.ILP)
    ref = capi.Engine(TERSOFF, ILP).compute_system(s, vatom=True)["vatom_ilp"]
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("ev", [False, True])
def test_subdomain_form(ev):
    s = S.displace(S.twisted_bilayer(14, 8, 2.0, top="hbn", spacing=3.3), 0.03, seed=7)
    L = s.box_hi - s.box_lo
    idx, gx = [np.arange(s.n)], [s.x]
    for sx in (-1, 0, 1):
        for sy in (-1, 0, 1):
            if sx or sy:
                idx.append(np.arange(s.n))
                gx.append(s.x + np.array([sx * L[0], sy * L[1], 0.0]))
    idx, x = np.concatenate(idx), np.concatenate(gx)
    r = []
    va = dict(vatom=ev)
    for full in (0, 1):
        eng = capi.Engine(TERSOFF, ILP)
        eng.set_option("list_full", full)
        r.append(eng.compute_ghost(s.n, x, s.type[idx], s.mol[idx], s.tag[idx], which=capi.ILP, eflag=ev, vflag=ev, **va))
    _close(*r)
    if ev:
        _scalars(*r)
        assert np.abs(r[0]["vatom_ilp"] - r[1]["vatom_ilp"]).max() <= TOL * np.abs(r[1]["vatom_ilp"]).max()
