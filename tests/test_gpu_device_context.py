"""An engine whose device context is not the one that earlier engines of the
process ran in.  A kernel's opted-in shared memory and cluster size belong to a
context, and every device has its own, so nothing that one engine set up may be
taken for granted by the next.  On one device a new context stands for another
device's: the first engine ends, cudaDeviceReset ends its context, and the same
calls give the same results.  In a process of its own, as the reset ends every
context user in it."""
import os
import subprocess
import sys

import pytest

from conftest import PKG

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import ctypes
import numpy as np
import lvb200, lvgen

def graph(n, seed):
    n, s, d, w = lvgen.planted_powerlaw(n=n, target_edges=3 * n, max_deg=n // 10, comm_min=8,
                                        comm_max=n // 10, seed=seed, unit=False)
    return lvb200.Graph.from_edges(n, s, d, w)

def calls(rule, gain):
    out = []
    with lvb200.Engine(rule=rule, gain=gain) as e:
        for g in (graph(1200, 1), graph(30000, 2)):  # from the start, and once contracted
            r = e.run(g, 1e-6)
            out += [r.assignment, r.modularity]
            e.load(g)
            while e.phase_move(1e-6)[0]:
                e.phase_aggregate()
            out += [e.assignment()]
    return out

FORMS = [("py", "fp32"), ("cuda", "fp32"), ("py", "fp64"), ("cuda", "fp64")]
first = [calls(*f) for f in FORMS]
lvb200.lib()
assert ctypes.CDLL("libcudart.so.12").cudaDeviceReset() == 0
again = [calls(*f) for f in FORMS]
for a, b in zip(first, again):
    assert len(a) == len(b) and all(np.allclose(x, y, rtol=0, atol=1e-12) for x, y in zip(a, b))
print("same")
"""


def test_engine_in_a_new_context():
    env = dict(os.environ, PYTHONPATH=os.path.join(PKG, "python"))
    r = subprocess.run([sys.executable, "-c", SCRIPT], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]
