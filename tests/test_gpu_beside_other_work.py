"""Runs that need every SM beside work that holds some of them for long: a late
block of the grid is waited for, it is no failure, however short the limit of
an exchange between running blocks is (PPS_WAIT_POLLS).  Every result equals
the same solve alone, and the other work's its own."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(pps, name, D):
    f = pps.REGISTRY[name]
    return pps.OptimizationProblem(f, np.zeros(D, np.float32), list(f.default_params) or None,
                                   lb=np.full(D, -4.0, np.float32), ub=np.full(D, 5.0, np.float32))


def _solve(pps, name, D, n, seed):
    sol = pps.solve(_problem(pps, name, D), pps.ParallelSyncPSOKernel(n), maxiters=60, seed=seed)
    return sol.u, sol.objective, np.asarray(sol.original)


def _swarms(pps, b):
    for k in range(8):
        b.add(_problem(pps, ("sphere", "rastrigin", "ackley", "rosenbrock")[k % 4], 20 + k), 3000 + k, maxiters=50,
              seed=k)
    return b


def _results(b, count):
    b.run()
    return [b.result(k) for k in range(count)]


class _Fits:
    """A batch of fits of 16 units: one cooperative launch that holds 16 SMs for about a second."""

    def __init__(self, pps):
        self.b = pps.Batch()
        for k in range(8):
            self.b.add(pps.ode.synthetic_fit("lv", k)[0], 256, maxiters=20000, seed=k)

    def run(self):
        return _results(self.b, 8)

    def close(self):
        self.b.close()


class _Async:
    """A run against private global bests: a plain launch of 16 blocks for about a second."""

    def __init__(self, pps):
        self.sw = pps.Swarm(_problem(pps, "ackley", 4), 4096, seed=1)

    def run(self):
        self.sw.init().async_run(1500000)
        return [self.sw.gbest()]

    def close(self):
        self.sw.close()


@pytest.mark.parametrize("work", [_Fits, _Async])
def test_solves_and_batches(pps, monkeypatch, work):
    jobs = [("ackley", 30, 20011, 1), ("rastrigin", 10, 60000, 2), ("rosenbrock", 3, 1000, 3)]
    want = [_solve(pps, *j) for j in jobs]
    held = work(pps)
    with pps.Batch() as swarms:
        held_alone, swarms_alone = held.run(), _results(_swarms(pps, swarms), 8)
        monkeypatch.setenv("PPS_WAIT_POLLS", "8192")  # a few milliseconds
        got, errors = [], []

        def other():
            try:
                got.extend(held.run())
            except Exception as e:  # noqa: BLE001
                errors.append(e)

        t = threading.Thread(target=other)
        t.start()
        time.sleep(0.1)
        rounds = 0
        while rounds == 0 or (t.is_alive() and rounds < 50):
            for j, w in zip(jobs, want):
                g = _solve(pps, *j)
                assert np.array_equal(g[0], w[0]) and g[1] == w[1] and np.array_equal(g[2], w[2]), j
            for g, w in zip(_results(swarms, 8), swarms_alone):
                assert np.array_equal(g[0], w[0]) and g[1:] == w[1:]
            rounds += 1
        t.join()
        assert not errors, errors
        for g, w in zip(got, held_alone):
            assert np.array_equal(g[0], w[0]) and g[1:] == w[1:]
    held.close()
