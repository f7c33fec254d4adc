"""A host program that resets the device between its uses of the library (cudaDeviceReset, as a C program
may between jobs): contexts made afterwards must find what the library keeps per device -- the Boys
tables, the pool of side streams, the kernels' shared-memory limits -- as new.  In a process of its own;
every context is destroyed before the reset."""
import subprocess
import sys

import pytest

from conftest import ROOT

CODE = r"""
import ctypes, importlib.util, os, sys
import numpy as np
sys.path.insert(0, os.path.join(%(root)r, "tests"))
from conftest import golden, golden_basis, load_sqb200
sqb = load_sqb200()
sqb.load_library()
rt = ctypes.CDLL("libcudart.so.12")
res = []
for run in range(3):
    out = []
    for case in ("h2co_631gs", "oh_qzp_uhf"):
        g = golden(case)
        r = bool(g["restricted"])
        eng = sqb.JKEngine(golden_basis(g))
        for _ in range(30):                    # past the builds that make a replay graph
            J = eng.build(g["PA"], None if r else g["PB"], restricted=r, scf_cutoff=1e-10)
        out += [x.copy() for x in J] + [np.float64(eng.stats()["quartets"])]
        if case == "h2co_631gs":
            xyz = list(dict.fromkeys(map(tuple, golden_basis(g).center)))
            out.append(eng.gradient(np.ones(len(xyz)), xyz, g["PA"], g["PA"], g["PA"]))
        eng.close()
    res.append(out)
    assert rt.cudaDeviceReset() == 0
for out in res[1:]:
    for x, y in zip(out, res[0]):
        assert np.abs(x - y).max() <= 1e-11 * max(1.0, np.abs(y).max())
print("ok")
"""


@pytest.mark.gpu
def test_contexts_after_a_device_reset():
    r = subprocess.run([sys.executable, "-c", CODE % {"root": ROOT}], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
