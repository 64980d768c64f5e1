"""Which form a call takes: short runs, batches of few iterations and mixed
batches are no slower than in another form of the same work that the library
has, and equal it bit for bit."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from test_gpu_sync_parity import assert_state_equal

pytestmark = pytest.mark.gpu

PACKAGE = Path(__file__).resolve().parent.parent / "parallelparticleswarms.jl_gb300"
GENERAL = dict(c1=1e-35, c2=1e-35)  # coefficients that only the general arithmetic takes


def _problem(pps, name, D, cons=False):
    f = pps.REGISTRY[name]
    rows = pps.quadratic_constraint(D, c=-6.25 * D, b=np.ones(D)) if cons else None
    return pps.OptimizationProblem(f, np.zeros(D, np.float32), list(f.default_params) or None,
                                   lb=np.full(D, -5.0, np.float32), ub=np.full(D, 5.0, np.float32), cons=rows)


@pytest.mark.parametrize("name,D,n,cons", [("sphere", 10, 140000, False), ("sphere", 10, 100000, True)])
def test_one_synchronous_iteration(pps, name, D, n, cons):
    with pps.Swarm(_problem(pps, name, D, cons), n, seed=1) as sw:
        sw.init()
        short = min(sw.sync_run(1) for _ in range(40))
        general = min(sw.sync_run(1, **GENERAL) for _ in range(40))
    assert short <= 1.12 * general


@pytest.mark.parametrize("D", [3, 5, 8])
def test_one_asynchronous_iteration(pps, D):
    with pps.Swarm(_problem(pps, "sphere", D), 1000000, seed=1) as sw:
        sw.init()
        short = min(sw.async_run(1) for _ in range(40))
        general = min(sw.async_run(1, **GENERAL) for _ in range(40))
    assert short <= 1.12 * general


@pytest.mark.parametrize("n", [1000, 160001])  # both sides of the grid's second round
@pytest.mark.parametrize("D", [4, 5, 8])
def test_asynchronous_runs_in_pieces(pps, orc, n, D):
    prob = _problem(pps, "rastrigin", D)
    ref = orc.OracleSwarm(orc.OracleProblem(2, D, prob.lb, prob.ub, params=[10.0]), n, 5).init()
    with pps.Swarm(prob, n, seed=5) as sw:
        sw.init()
        for k in (1, 3, 4, 11):
            sw.async_run(k)
            ref.async_run(k)
        assert_state_equal(sw, ref, "after the pieces")


@pytest.mark.parametrize("count,n", [(1, 1), (1, 511), (3, 512), (2, 513), (1, 20000), (4, 20000), (200, 1100), (320, 700)])
def test_batch_sampling(pps, count, n):
    def run(shape):
        with pps.Batch() as b:
            if shape:
                b.set_shape(*shape)
            for k in range(count):
                b.add(_problem(pps, ("sphere", "rosenbrock", "rastrigin", "ackley")[k % 4], 40), n, maxiters=0, seed=k)
            b.run()
            ms = min(b.run() for _ in range(9))
            return ms, [b.result(k) for k in range(count)], b.state(count - 1)
    ms, got, state = run(None)
    fixed, want, ref = run((256, 1))
    for a, b in zip(got, want):
        assert np.array_equal(a[0], b[0]) and a[1:] == b[1:]
    for f in ref:
        assert np.array_equal(state[f], ref[f])
    if count <= 4:
        assert ms <= 1.3 * fixed + 0.02


def _fit(pps, steps, seed=0):
    data = np.linspace(0.5, 1.5, 2 * (steps // 10 + 1), dtype=np.float32).reshape(-1, 2) * (1.0 + 0.01 * seed)
    return pps.ode.lv_problem(data.astype(np.float32), dt=0.01, nsteps=steps, save_every=10)


@pytest.mark.parametrize("count", [1, 19, 20, 34, 35])
@pytest.mark.parametrize("n", [4095, 4096, 8193])
def test_large_fits_beside_a_swarm(pps, count, n):
    with pps.Batch() as b:
        for k in range(count):
            b.add(_fit(pps, 40, k % 3), n, maxiters=2, seed=k % 3)
        b.add(_problem(pps, "sphere", 4), 100, maxiters=2, seed=1)
        b.run()
        for k in range(min(count, 3)):
            with pps.Swarm(_fit(pps, 40, k), n, seed=k) as sw:
                sw.init().sync_run(2)
                u, cost, idx = sw.gbest()
            for slot in range(k, count, 3):
                got = b.result(slot)
                assert np.array_equal(got[0], u) and got[1:] == (cost, idx)


@pytest.mark.parametrize("every", [1, 2, 3, 4, 5, 6, 7, 10, 15, 60])
@pytest.mark.parametrize("n", [300, 3000])
def test_steps_between_saves(pps, every, n):
    data = np.linspace(0.5, 1.5, 2 * (60 // every + 1), dtype=np.float32).reshape(-1, 2)
    fit = pps.ode.fhn_problem(data, dt=0.02, nsteps=60, save_every=every)
    with pps.Swarm(fit, n, seed=2) as sw, pps.Batch() as b:
        sw.init().sync_run(3)
        b.add(fit, n, maxiters=3, seed=2)
        b.add(_problem(pps, "sphere", 4), 100, maxiters=3, seed=1)
        b.run()
        x, got = sw.state(), b.state(0)
    for f in ("x", "pcost", "cost"):
        assert np.array_equal(x[f], got[f]), f


MIXED = """
import sys
import numpy as np
import parallelparticleswarms as pps
count, n, steps, every = map(int, sys.argv[1:])
data = np.linspace(0.5, 1.5, 2 * (steps // every + 1), dtype=np.float32).reshape(-1, 2)
fit = pps.ode.lv_problem(data, dt=0.01, nsteps=steps, save_every=every)
small = pps.OptimizationProblem(pps.REGISTRY["sphere"], np.zeros(4, np.float32), None,
                                lb=np.full(4, -3, np.float32), ub=np.full(4, 4, np.float32))
with pps.Batch() as b:
    b.set_shape(256, 1)
    for k in range(count):
        b.add(fit, n, maxiters=10, seed=k)
    b.add(small, 100, maxiters=10, seed=1)
    b.run()
    print(min(b.run() for _ in range(5)))
"""


@pytest.mark.parametrize("batch", [("24", "8192", "1000", "10"), ("1", "3000", "600", "1")])
def test_time_of_large_fits_beside_a_swarm(batch):
    def ms(**env):
        r = subprocess.run([sys.executable, "-c", MIXED, *batch], env=dict(os.environ, PYTHONPATH=str(PACKAGE), **env),
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        return float(r.stdout)
    assert ms() <= 1.1 * ms(PPS_ODE_THREADS="512")
