"""The FP64 Tersoff virial against extended precision: no rounding that every bond shares.

Scaling all positions leaves the angles and so, with bonds inside R - D and lambda3 = 0, every
b_ij as it is, and the virial's trace is sum over bonds of r/2 (A lambda1 e^(-lambda1 r) -
b_ij B lambda2 e^(-lambda2 r)): two large sums that nearly cancel.  Roundings that differ from bond
to bond average out over 4,000 atoms (about 10 of 1e-16 a bond, times the cancellation's ~27,
over the root of the bonds: below 3e-16).  One that all bonds share, A lambda1 or B lambda2
rounded beforehand (8e-17 for carbon), comes out 27 times as large, 2e-15.  1e-15 lies between.
"""
import dataclasses

import numpy as np
import pytest
from conftest import TERSOFF

from lmff_gb300 import build, capi
from lmff_gb300 import structures as S

pytestmark = pytest.mark.gpu
LD = np.longdouble


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _parameters(name):
    with open(TERSOFF) as f:
        for line in f:
            w = line.split("#")[0].split()
            if len(w) == 17 and w[:3] == [name] * 3:
                return dict(zip(("m", "gamma", "lam3", "c", "d", "h", "n", "beta", "lam2", "B", "R", "D", "lam1", "A"),
                                (LD(float(v)) for v in w[3:])))
    raise AssertionError(name)


def _trace(x, p):
    """x[n, 3] of one flat sheet without images."""
    near = np.abs(x[:, None, 0] - x[None, :, 0]) < 2.0
    near &= np.abs(x[:, None, 1] - x[None, :, 1]) < 2.0
    i, j = np.nonzero(near)
    d = x[j].astype(LD) - x[i].astype(LD)
    r = np.sqrt((d * d).sum(axis=1))
    keep = (r > 0) & (r < p["R"] + p["D"])
    i, j, d, r = i[keep], j[keep], d[keep], r[keep]
    assert (r < p["R"] - p["D"]).all()
    zeta = np.zeros(len(i), LD)
    first = np.searchsorted(i, np.arange(len(x)))
    count = np.bincount(i, minlength=len(x))
    c2, d2 = p["c"] ** 2, p["d"] ** 2
    for k in range(count.max()):   # the k-th bond of each bond's centre
        b = first[i] + k
        ok = (k < count[i]) & (b != np.arange(len(i)))
        b = np.where(ok, b, 0)
        cos = (d * d[b]).sum(axis=1) / (r * r[b])
        u2 = (p["h"] - cos) ** 2
        zeta += np.where(ok, p["gamma"] * (1 + c2 * u2 / (d2 * (d2 + u2))), LD(0))
    bij = (1 + (p["beta"] * zeta) ** p["n"]) ** (-1 / (2 * p["n"]))
    return (r / 2 * (p["A"] * p["lam1"] * np.exp(-p["lam1"] * r) - bij * p["B"] * p["lam2"] * np.exp(-p["lam2"] * r))).sum()


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_trace_of_the_virial(seed):
    if np.finfo(LD).eps > 1e-18:
        pytest.skip("long double is no wider than double")
    s = S.displace(S.graphite_slab(1, 40, 25), 0.03, seed=seed)
    s = dataclasses.replace(s, box_lo=s.box_lo - 5.0, box_hi=s.box_hi + 5.0, periodic=np.zeros(3, bool), v=None)
    ref = _trace(s.x, _parameters("C"))
    r = capi.Engine(TERSOFF, elements=("C",)).compute_system(s, which=capi.TERSOFF)
    v = r["virial_tersoff"].astype(LD)
    assert abs((v[0] + v[1] + v[2] - ref) / ref) <= 1e-15
