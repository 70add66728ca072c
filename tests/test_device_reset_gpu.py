"""Contexts made after a reset of their device (cudaDeviceReset, in a process of
its own) do not take over the streams of contexts closed before it, whose
handles may name other streams by then."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes
import numpy as np
from costuum_b200.tmatrix import Context

def run():
    cs = [Context(0) for _ in range(3)]
    out = []
    for c in cs:
        res = c.tmatrix_batch([1e-7, 2e-7], 1e-6, 1.5 + 0.1j, 0.8)
        out.append((res.q, np.array(c.observables([0.3]))))
        c.close()
    return out

first = run()
path = [l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l][0]
rt = ctypes.CDLL(path)
for _ in range(2):
    assert rt.cudaDeviceReset() == 0 and rt.cudaSetDevice(0) == 0
    # the handles of the streams made next may be those of the old ones
    streams = [ctypes.c_void_p() for _ in range(64)]
    for s in streams:
        assert rt.cudaStreamCreate(ctypes.byref(s)) == 0
    for _ in range(2):
        for a, b in zip(first, run()):
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
print("same")
"""


def test_contexts_after_a_reset():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, stdout=subprocess.PIPE,
                       stderr=subprocess.STDOUT, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("same"), r.stdout
