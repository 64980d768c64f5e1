"""Pooled streams and blocks: more swarms at once than the pool keeps streams,
several threads, snapshots that outlive their swarm, blocks reused by swarms of
other sizes and objectives -- every result equals a first run's."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(pps, name, D):
    return pps.OptimizationProblem(pps.REGISTRY[name], np.zeros(D, np.float32), None, lb=np.full(D, -3, np.float32),
                                   ub=np.full(D, 4, np.float32))


def _run(pps, name, D, n, seed):
    sol = pps.solve(_problem(pps, name, D), pps.ParallelSyncPSOKernel(n), maxiters=12, seed=seed)
    return sol.u, sol.objective, np.asarray(sol.original)


JOBS = [("rastrigin", 3, 40), ("sphere", 17, 3000), ("ackley", 8, 700), ("rosenbrock", 2, 90000), ("ackley", 60, 33)]


def _equal(a, b):
    assert np.array_equal(a[0], b[0]) and a[1] == b[1] and np.array_equal(a[2], b[2])


def test_results_do_not_depend_on_what_the_pools_hold(pps):
    first = [_run(pps, *j, seed=k) for k, j in enumerate(JOBS)]
    swarms = [pps.Swarm(_problem(pps, *JOBS[k % 5][:2]), 50 + k, seed=k).init() for k in range(40)]
    snaps = [sw.positions_on_device() for sw in swarms]
    want = [sw.positions() for sw in swarms]
    for sw in swarms:
        sw.close()
    for k in range(5):
        _equal(_run(pps, *JOBS[k], seed=k), first[k])
    for snap, w in zip(snaps, want):
        assert np.array_equal(snap.numpy(), w.T)


def test_threads(pps):
    first = [_run(pps, *j, seed=k) for k, j in enumerate(JOBS)]
    got, errors = {}, []

    def work(t):
        try:
            for r in range(6):
                k = (t + r) % 5
                got[t, r] = (k, _run(pps, *JOBS[k], seed=k))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    for k, r in got.values():
        _equal(r, first[k])
