"""Pairs at the interlayer cutoff to the last bits of r^2: the FP64 mode's double-float
kernels take the ones that FP64 takes, as the general kernels (option list_full) do.  Without
the taper a pair's force ends in a step there, so its presence shows.  A sum of three squares
near 256 is within two roundings of the exact one however its products are fused, so pairs
within two last places (of numbers just below 256) of the cutoff's square may go either way.
"""
import numpy as np
import pytest
from conftest import ILP, TERSOFF

from lmff_gb300 import build, capi

pytestmark = pytest.mark.gpu
CUT = 16.0


@pytest.fixture(scope="module", autouse=True)
def _built():
    build.build()


def _rsq(d):
    return (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]


def _pairs(seed):
    """Lone pairs 50 A apart, each within a few last places of z of the cutoff."""
    rng = np.random.default_rng(seed)
    x, rsq = [], []
    for k in range(216):
        a = 50.0 * np.array([k % 6, k // 6 % 6, k // 36]) + rng.uniform(0.0, 1.0, 3)
        u = rng.normal(size=3)
        u[2] = abs(u[2]) + 0.5
        b = a + CUT * u / np.linalg.norm(u)
        while _rsq(a - b) < CUT * CUT:
            b[2] = np.nextafter(b[2], np.inf)
        while _rsq(a - b) >= CUT * CUT:
            b[2] = np.nextafter(b[2], -np.inf)
        for _ in range(rng.integers(0, 6)):
            b[2] = np.nextafter(b[2], np.inf if k % 2 else -np.inf)
        x += [a, b]
        rsq.append(_rsq(a - b))
    return np.array(x), np.array(rsq)


def _taken(f):
    return (np.abs(f.reshape(-1, 2, f.shape[1])).max(axis=2) > 0.0).all(axis=1)


@pytest.mark.parametrize("elements,types", [(("C",), 1), (("C", "B", "N"), 3)])
@pytest.mark.parametrize("ev", [False, True])
def test_pairs_at_the_cutoff(elements, types, ev):
    for seed in (1, 2):
        x, rsq = _pairs(seed)
        assert 40 < (rsq < CUT * CUT).sum() < len(rsq) - 40
        n = len(x)
        t = 1 + np.arange(n) % types
        m, g = 1 + np.arange(n) % 2, np.arange(1, n + 1)
        sure = np.abs(rsq - CUT * CUT) > 2.0 * 2.0 ** -45
        assert 100 < sure.sum()
        for full in (0, 1):
            eng = capi.Engine(TERSOFF, ILP, elements=elements, cut_global=CUT, tap_flag=0)
            eng.set_option("list_full", full)
            eng.set_box([-5.0] * 3, [330.0] * 3, [0, 0, 0])
            kw = dict(which=capi.ILP, eflag=ev, vflag=ev, vatom=True)
            for r in (eng.compute(x, t, m, g, **kw), eng.compute_ghost(n, x, t, m, g, **kw)):
                for k in ("f", "vatom_ilp"):
                    assert np.array_equal(_taken(r[k])[sure], (rsq < CUT * CUT)[sure]), (full, k)
