"""The one-warp-per-atom list build against the 32-atoms-per-warp build (option
small_variants 0): the same entries in the same order, over boxes of one to several bins
per dimension, several images, atoms outside the box in non-periodic dimensions and far from
the origin, full and interlayer lists, several cutoffs.  Integers: no tolerance.
"""
import dataclasses

import numpy as np
import pytest
from conftest import ILP, TERSOFF

from lmff_gb300 import build, capi
from lmff_gb300 import structures as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _lists(s, full, cut=16.0, skin=2.0):
    out = []
    for sv in (1, 0):
        eng = capi.Engine(TERSOFF, ILP, cut_global=cut, skin=skin)
        eng.set_option("small_variants", sv)
        eng.set_option("list_full", full)
        r = eng.compute_system(s, eflag=False, vflag=False)
        out.append((eng.export_list(0), eng.export_list(1), r["f"]))
    return out


def _same(s, **kw):
    for full in (0, 1):
        a, b = _lists(s, full, **kw)
        for x, y in zip(a, b):
            assert np.array_equal(x, y)


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 1), (3, 3), (4, 2), (7, 5), (8, 4), (11, 7), (15, 9), (22, 13)])
@pytest.mark.parametrize("mode", ["unique", "alternate"])
def test_boxes_of_few_and_many_bins(nx, ny, mode):
    _same(S.displace(S.graphite_slab(3, nx, ny, mol_mode=mode), 0.05, seed=nx))


@pytest.mark.parametrize("cut,skin", [(16.0, 0.3), (6.0, 1.0), (3.5, 0.5), (11.0, 2.0)])
def test_cutoffs(cut, skin):
    _same(S.displace(S.twisted_bilayer(14, 8, 2.0, top="hbn", spacing=3.3), 0.05, seed=3), cut=cut, skin=skin)


@pytest.mark.parametrize("shift", [0.0, -700.0, 4000.0])
def test_atoms_outside_and_far_boxes(shift):
    s = S.displace(S.flake_edges(14, 8), 0.03, seed=3)
    s.x, s.box_lo, s.box_hi = s.x + shift, s.box_lo + shift, s.box_hi + shift
    rng = np.random.default_rng(1)
    for reach in (3.0, 25.0, 300.0):
        t = s.copy()
        t.x[:, 2] += np.where(t.mol == 2, reach, 0.0) + rng.uniform(-0.5, 0.5, t.n)
        t.x[:, 1] -= 0.5 * reach
        _same(t)


def test_more_layers_than_bins_and_a_stretched_box():
    s = S.displace(S.graphite_slab(12, 6, 4), 0.05, seed=2)
    _same(s)
    t = dataclasses.replace(s, box_hi=s.box_hi + np.array([9.7, 31.0, 50.0]), periodic=np.array([True, True, True]))
    _same(t)


def test_subdomain():
    s = S.displace(S.twisted_bilayer(14, 8, 2.0, top="hbn", spacing=3.3), 0.03, seed=7)
    L = s.box_hi - s.box_lo
    idx, gx = [np.arange(s.n)], [s.x]
    for sx in (-1, 0, 1):
        for sy in (-1, 0, 1):
            if sx or sy:
                idx.append(np.arange(s.n))
                gx.append(s.x + np.array([sx * L[0], sy * L[1], 0.0]))
    idx, x = np.concatenate(idx), np.concatenate(gx)
    f = []
    for sv in (1, 0):
        eng = capi.Engine(TERSOFF, ILP)
        eng.set_option("small_variants", sv)
        f.append(eng.compute_ghost(s.n, x, s.type[idx], s.mol[idx], s.tag[idx])["f"])
    assert np.array_equal(*f)


def test_batch_of_boxes():
    systems = [S.displace(S.graphite_slab(2, nx, ny), 0.05, seed=nx) for nx, ny in ((1, 1), (9, 3), (30, 20), (5, 12))]
    f = []
    for sv in (1, 0):
        eng = capi.Engine(TERSOFF, ILP, elements=("C",))
        eng.set_option("small_variants", sv)
        eng.batch_set(systems)
        f.append([r["f"] for r in eng.batch_compute()])
    for a, b in zip(*f):
        assert np.array_equal(a, b)
