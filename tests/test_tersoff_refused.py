"""FP64 Tersoff on systems whose atoms take the short form and the general one side by side:
the refused atoms are evaluated apart, in lanes or gathered into warps.  Sizes about the
limits of the forms' launches, disorder from a few refused atoms to most, and constants
for which an atom is refused only once b_ij's argument is known.

Tolerance as for the short form: about 50 roundings a bond, and g(theta)'s cancellation in the
oracle, 2e-14 of a force; disordered systems have bonds whose forces are ~10 x larger and
cancel, 1e-12 bounds them with room.
"""
import dataclasses
import os

import numpy as np
import pytest
from conftest import POT, TERSOFF, rel_max

from lmff_gb300 import build, capi
from lmff_gb300 import structures as S

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _check(s, file=TERSOFF, elements=("C", "B", "N")):
    from oracle import Oracle
    o = Oracle(file, None, elements=elements, nthreads=8)
    o.set_system(s)
    ref = o.forces(which=1, eatom=True)
    eng = capi.Engine(file, elements=elements)
    got = eng.compute_system(s, which=capi.TERSOFF, eatom=True)
    for k in ("f", "eatom", "virial"):
        assert rel_max(got[k], ref[k]) <= TOL, k
    got = eng.compute_system(s, which=capi.TERSOFF, eflag=False, vflag=False)
    assert rel_max(got["f"], ref["f"]) <= TOL


def _holes(s, share, seed):
    keep = np.random.default_rng(seed).random(s.n) > share
    return dataclasses.replace(s, x=s.x[keep], type=s.type[keep], mol=s.mol[keep], tag=s.tag[keep], v=None)


@pytest.mark.parametrize("sigma", [0.03, 0.09, 0.14])
@pytest.mark.parametrize("nx,ny", [(1, 1), (5, 3), (32, 31), (33, 31), (40, 31), (70, 70), (76, 70)])
def test_against_oracle(nx, ny, sigma):
    _check(_holes(S.displace(S.graphite_slab(2, nx, ny), sigma, seed=nx), 0.02, seed=ny), elements=("C",))


@pytest.mark.parametrize("nx,ny", [(5, 3), (40, 31)])
def test_refused_by_the_bond_order(nx, ny, tmp_path):
    """beta so small that b_ij's argument straddles the limit of its short form."""
    lines = []
    with open(os.path.join(POT, "C.opt.tersoff")) as f:
        for line in f:
            w = line.split("#")[0].split()
            if len(w) == 17:
                w[10] = "8.5e-16"
                line = " ".join(w) + "\n"
            lines.append(line)
    file = tmp_path / "C.tersoff"
    file.write_text("".join(lines))
    _check(S.displace(S.graphite_slab(2, nx, ny), 0.06, seed=1), file=str(file), elements=("C",))


def test_small_systems_use_the_lanes():
    """Forces alone on a small system: the refused atoms run one lane per bond, which shows in
    the last bits against the one-thread routine (option small_variants 0); the others take
    the same form on either route."""
    s = S.displace(S.graphite_slab(2, 16, 9), 0.14, seed=4)
    f = []
    for sv in (1, 0):
        eng = capi.Engine(TERSOFF, elements=("C",))
        eng.set_option("small_variants", sv)
        f.append(eng.compute_system(s, which=capi.TERSOFF, eflag=False, vflag=False)["f"])
    assert rel_max(f[0], f[1]) <= TOL
    assert not np.array_equal(f[0], f[1])
