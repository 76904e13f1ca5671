"""Energies of systems about and past the reduction's chunk of 2,048 atoms: the sum of the
per-atom energies, and the same to the bit alone and within a batch.

The kernel and numpy add the same numbers in another order, each sum within
log2(n) + n/2048 < 40 roundings of the magnitudes: 1e-14 of sum |e|.
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


def _slab(n):
    s = S.displace(S.graphite_slab(2, 16 * (1 + (n - 1) // 2048), 17), 0.02, seed=n)
    return dataclasses.replace(s, x=s.x[:n], type=s.type[:n], mol=s.mol[:n], tag=s.tag[:n], v=None)


def _check(r):
    e = r["eatom"]
    assert abs(e.sum() - (r["e_tersoff"] + r["e_ilp"])) <= 1e-14 * np.abs(e).sum()


@pytest.mark.parametrize("n", [1, 255, 2047, 2048, 2049, 4096, 6143])
def test_sum_of_the_atoms(n):
    """FP64 mode (the mixed mode forms per-atom energies and the total by different sums)."""
    eng = capi.Engine(TERSOFF, ILP, elements=("C",))
    _check(eng.compute_system(_slab(n), eatom=True))


@pytest.mark.parametrize("precision", [capi.FP64, capi.MIXED])
def test_batch_is_each_system_alone(precision):
    systems = [_slab(n) for n in (300, 2048, 2049, 6143, 4096, 2047)]
    eng = capi.Engine(TERSOFF, ILP, elements=("C",), precision=precision)
    eng.batch_set(systems)
    out = eng.batch_compute()
    for s, b in zip(systems, out):
        r = capi.Engine(TERSOFF, ILP, elements=("C",), precision=precision).compute_system(s)
        for k in ("e_tersoff", "e_ilp"):
            assert b[k] == r[k]
        for k in ("pvector", "virial_tersoff", "virial_ilp"):
            assert np.array_equal(b[k], r[k])


def test_one_engine_over_sizes():
    eng = capi.Engine(TERSOFF, ILP, elements=("C",))
    for n in (6143, 300, 4096, 2049, 6143):
        for _ in range(2):
            _check(eng.compute_system(_slab(n), eatom=True))
