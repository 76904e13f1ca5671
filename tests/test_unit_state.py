"""The force units keep no host state of their own: an engine's constants reach its device
from the engine and from the call's storage, so threads that upload different potentials to
several devices at the same time do not meet.  Checked on the built objects' symbols: no
static local of a host function, and no namespace variable but the host names of the
device's (c_..., g_...).
"""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest
from conftest import ILP, TERSOFF

from lmff_gb300 import build


def test_no_process_wide_host_state():
    build.build()
    nm = shutil.which("nm")
    if nm is None:
        pytest.skip("nm not found")
    left = []
    for unit in ("forces64.cu.o", "forces32.cu.o"):
        out = subprocess.run([nm, os.path.join(build.BUILD, unit)], capture_output=True, text=True, check=True).stdout
        names = [w[-1] for w in (line.split() for line in out.splitlines()) if len(w) == 3 and w[1] in "bdBD"]
        left += [n for n in names if re.match(r"_ZZN4lmff3f(32|64)", n)]
        left += [n for n in names if re.match(r"_ZN4lmff3f(32|64)L?\d+(?!\d|[cg]_)", n)]
    assert not left


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_two_potentials_in_turn(precision):
    """Engines of two potentials on one device, called in turn and from two threads: each
    gets what it gets alone."""
    import threading

    from lmff_gb300 import capi
    from lmff_gb300 import structures as S
    s = S.displace(S.twisted_bilayer(11, 7, 3.0, top="hbn", spacing=3.3), 0.05, seed=5)
    kinds = [dict(cut_global=16.0), dict(cut_global=9.0, tap_flag=0)]
    alone = [capi.Engine(TERSOFF, ILP, precision=precision, **k).compute_system(s)["f"] for k in kinds]
    engines = [capi.Engine(TERSOFF, ILP, precision=precision, **k) for k in kinds]
    for _ in range(3):
        for e, f in zip(engines, alone):
            assert np.array_equal(e.compute_system(s)["f"], f)
    bad = []

    def work(k):
        for _ in range(10):
            if not np.array_equal(engines[k].compute_system(s)["f"], alone[k]):
                bad.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
