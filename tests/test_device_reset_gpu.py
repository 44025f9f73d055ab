"""A host program that resets the device between two runs: nothing that the library keeps between calls
may outlive the memory it was."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUN = r"""
import ctypes as C, os, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from ermod_openacc_b200 import Engine, _capi as A, slvfe
from ermod_openacc_b200 import systems as S

w = S.make_workload(2, small=True, maxins=64)
pos, cell = w.frame(0)

def run():
    eng = Engine(w.params, w.topo, w.hist)
    assert eng.engconst(1, pos, cell) >= 0
    a = eng.accum()                       # the correlation matrix passes through the pinned ring
    eng.close()
    n = 500
    e = np.linspace(-10, 10, n)
    rr = np.exp(-0.02 * e * e)
    rd = np.exp(-0.02 * (e + 1) ** 2)
    rr, rd = rr * 100 / rr.sum(), rd * 100 / rd.sum()
    mu = slvfe.delta_mu_gpu(rd, rr, np.diag(rr) + np.outer(rr, rr), e, np.ones(n, dtype=np.int32), 300.0, np.array([-1.0]))
    return a["edens"], a["ecorr"], mu[0]

first = run()
rt = C.CDLL(sys.argv[2])
lib = A.load_library()
for release in (False, True):
    assert rt.cudaDeviceReset() == 0
    if release:                           # what was lost is not given back a second time
        lib.ermod_staging_release()
        lib.ermod_slvfe_release()
    again = run()
    assert all(np.array_equal(x, y) for x, y in zip(first, again))
lib.ermod_staging_release()
lib.ermod_slvfe_release()
assert all(np.array_equal(x, y) for x, y in zip(first, run()))
print("ok")
"""


def test_runs_before_and_after_a_reset_agree(engine_lib):
    cudart = "/usr/local/cuda/lib64/libcudart.so.12"
    if not os.path.exists(cudart):
        pytest.skip("no shared CUDA runtime to reset the device with")
    r = subprocess.run([sys.executable, "-c", RUN, ROOT, cudart], capture_output=True, text=True, timeout=240)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stdout + r.stderr
