"""cudaDeviceReset between calls: streams and memory that the library keeps for
later belong to a context that is gone, and the next call works on the new one."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PACKAGE = Path(__file__).resolve().parent.parent / "parallelparticleswarms.jl_gb300"

PROGRAM = """
import ctypes
import numpy as np
import parallelparticleswarms as pps

def problem(D):
    return pps.OptimizationProblem(pps.REGISTRY["sphere"], np.zeros(D, np.float32), None,
                                   lb=np.full(D, -3, np.float32), ub=np.full(D, 4, np.float32))

def calls():
    out = [np.asarray(pps.solve(problem(3), pps.ParallelSyncPSOKernel(n), maxiters=9, seed=1).original)
           for n in (500, 20000)]
    with pps.Swarm(problem(4), 400, seed=2) as sw, pps.Swarm(problem(5), 300, seed=2) as other:
        out += [sw.init().positions_on_device().numpy(), other.init().positions()]
    return out

first = calls()
runtime = ctypes.CDLL("libcudart.so.13")
for _ in range(3):
    assert runtime.cudaDeviceReset() == 0
    for a, b in zip(first, calls()):
        assert np.array_equal(a, b)
print("equal")
"""


def test_calls_after_a_reset():
    env = dict(os.environ, PYTHONPATH=str(PACKAGE))
    r = subprocess.run([sys.executable, "-c", PROGRAM], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["equal"], (r.returncode, r.stdout, r.stderr)
