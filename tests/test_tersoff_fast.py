"""The FP64 mode's short Tersoff form (two or three bonds inside R - D) and its rule against
the oracle: centres with none to four and more bonds, bonds on both sides of R - D, angles
over several elements, owned and ghost atoms.

Both sides evaluate a bond in some 50 roundings of terms no larger than ~10 x the largest
force; the oracle's g(theta) cancels two terms of c^2/d^2 ~ 8e7, 1e-12 of g and, through
b_ij's weak dependence on it, ~2e-14 of a force.  1e-12 bounds the difference.
"""
import numpy as np
import pytest
from conftest import TERSOFF, rel_max

from lmff_gb300 import build, capi
from lmff_gb300 import structures as S

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _interstitial():
    s = S.displace(S.graphite_slab(2, 6, 4), 0.03, seed=6)
    s.x[5] = s.x[0] + np.array([0.9, 0.9, 0.05])   # more than three bonds around it
    return s


def _reference(s):
    from oracle import Oracle
    o = Oracle(TERSOFF, None, nthreads=4)
    o.set_system(s)
    return o.forces(which=1, eatom=True)


SYSTEMS = {
    "intact": lambda: S.displace(S.twisted_bilayer(11, 7, 3.0, top="hbn", spacing=3.3), 0.03, seed=5),
    "around_R-D": lambda: S.displace(S.twisted_bilayer(11, 7, 3.0, top="hbn", spacing=3.3), 0.14, seed=8),
    "edges": lambda: S.displace(S.flake_edges(6, 4), 0.03, seed=3),
    "interstitial": _interstitial,
    "one_cell": lambda: S.displace(S.graphite_slab(3, 1, 1, mol_mode="unique"), 0.05, seed=1),
}


@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_against_oracle(name):
    s = SYSTEMS[name]()
    ref = _reference(s)
    got = capi.Engine(TERSOFF).compute_system(s, which=capi.TERSOFF, eatom=True)
    for k in ("f", "eatom", "virial"):
        assert rel_max(got[k], ref[k]) <= TOL, k
    assert abs(got["e_tersoff"] - ref["e_tersoff"]) <= TOL * abs(ref["e_tersoff"])
    got = capi.Engine(TERSOFF).compute_system(s, which=capi.TERSOFF, eflag=False, vflag=False)
    assert rel_max(got["f"], ref["f"]) <= TOL


@pytest.mark.parametrize("ev", [False, True])
def test_subdomain_form(ev):
    """Owned atoms with their images as ghosts: the ghosts' forces folded back."""
    s = S.displace(S.twisted_bilayer(14, 8, 2.0, top="hbn", spacing=3.3), 0.1, seed=7)
    L = s.box_hi - s.box_lo
    idx, gx = [np.arange(s.n)], [s.x]
    for sx in (-1, 0, 1):
        for sy in (-1, 0, 1):
            if sx or sy:
                idx.append(np.arange(s.n))
                gx.append(s.x + np.array([sx * L[0], sy * L[1], 0.0]))
    idx, x = np.concatenate(idx), np.concatenate(gx)
    got = capi.Engine(TERSOFF).compute_ghost(s.n, x, s.type[idx], s.mol[idx], s.tag[idx], which=capi.TERSOFF,
                                                  eflag=ev, vflag=ev)
    ref = _reference(s)
    f = np.zeros((s.n, 3))
    np.add.at(f, idx, got["f"])
    assert rel_max(f, ref["f"]) <= TOL
    if ev:
        assert abs(got["e_tersoff"] - ref["e_tersoff"]) <= TOL * abs(ref["e_tersoff"])


@pytest.mark.parametrize("name", sorted(SYSTEMS))
def test_per_atom_virial(name):
    from oracle import Oracle
    s = SYSTEMS[name]()
    o = Oracle(TERSOFF, None, nthreads=4)
    o.set_system(s)
    ref = o.forces(which=1, vatom=True)["vatom_tersoff"]
    got = capi.Engine(TERSOFF).compute_system(s, which=capi.TERSOFF, vatom=True)["vatom_tersoff"]
    assert rel_max(got, ref) <= TOL
