"""Batches on several threads whose launches need unlike amounts of shared memory:
every run succeeds and equals the same batch alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fit(pps, steps):  # a save every step: the observations lie in shared memory
    data = np.linspace(0.5, 1.5, 2 * (steps + 1), dtype=np.float32).reshape(-1, 2)
    return pps.ode.lv_problem(data, dt=1e-3, nsteps=steps, save_every=1)


def _swarm(pps, D):
    return pps.OptimizationProblem(pps.REGISTRY["sphere"], np.zeros(D, np.float32), None,
                                   lb=np.full(D, -4.0, np.float32), ub=np.full(D, 5.0, np.float32))


def _check(make, runs, workers=4):
    want = []
    for k in range(len(make)):
        with make[k]() as b:
            b.run()
            want.append(b.result(0))
    errors = []

    def work(k):
        try:
            with make[k]() as b:
                for _ in range(runs):
                    b.run()
                    got = b.result(0)
                    assert np.array_equal(got[0], want[k][0]) and got[1:] == want[k][1:]
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k % len(make),)) for k in range(workers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_units_of_fits(pps):
    def make(steps):
        b = pps.Batch()
        b.add(_fit(pps, steps), 65536, maxiters=0, seed=3)
        return b
    _check([lambda: make(3900), lambda: make(2700)], 1500, workers=8)


@pytest.mark.parametrize("kind", ["fits", "swarms"])
def test_clusters(pps, kind):
    def make(n):
        b = pps.Batch()
        if kind == "fits":
            b.add(_fit(pps, 10), n, maxiters=1, seed=3)
        else:
            b.set_shape(256, 1)
            b.add(_swarm(pps, 5), n, maxiters=1, seed=3)
        return b
    _check([lambda: make(2048), lambda: make(100)], 300)
