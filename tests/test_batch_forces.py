"""A system's forces are the same to the bit alone and within a batch, whatever shares its
warps: systems of odd sizes, so that the atoms after them are grouped into warps otherwise
than alone, lists of very different lengths side by side, and cutoffs so short that pairs whose
normals' terms count stand at the lists' ends, over the lanes per atom.
Integers of bits: no tolerance.
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


def _piece(layers, nx, ny, n, seed):
    s = S.displace(S.graphite_slab(layers, nx, ny, mol_mode="unique"), 0.03, seed=seed)
    return dataclasses.replace(s, x=s.x[:n], type=s.type[:n], mol=s.mol[:n], tag=s.tag[:n], v=None)


SYSTEMS = [_piece(2, 2, 1, 13, 1), _piece(6, 9, 5, 1077, 2), S.displace(S.flake_edges(5, 3), 0.03, seed=3),
           _piece(3, 6, 4, 283, 4), _piece(2, 3, 2, 47, 5), _piece(8, 7, 4, 889, 6), _piece(2, 12, 7, 671, 7),
           _piece(5, 8, 5, 798, 8)]


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
@pytest.mark.parametrize("elements", [("C",), ("C", "B", "N")])
@pytest.mark.parametrize("cut,skin", [(16.0, 2.0), (6.0, 0.3), (4.5, 0.1)])
@pytest.mark.parametrize("tpa", [4, 8, 16])
def test_forces_alone_and_in_a_batch(tpa, cut, skin, elements, precision):
    kw = dict(elements=elements, precision=precision, cut_global=cut, skin=skin)
    eng = capi.Engine(TERSOFF, ILP, **kw)
    eng.set_option("tpa", tpa)
    eng.batch_set(SYSTEMS)
    out = eng.batch_compute()
    alone = capi.Engine(TERSOFF, ILP, **kw)
    alone.set_option("tpa", tpa)
    for s, b in zip(SYSTEMS, out):
        r = alone.compute_system(s)
        assert np.array_equal(b["f"], r["f"])
        for k in ("pvector", "virial_tersoff", "virial_ilp"):
            assert np.array_equal(b[k], r[k]), k
