"""Batches of closed-form swarms alone (k_batch_resident): every swarm equals
the same swarm solved alone, bit for bit, whatever wave and blocks it gets: few
and many swarms, tiny and large ones, uneven iteration counts, none at all,
unbounded problems; and the batches that keep the streaming form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("sphere", "rosenbrock", "rastrigin", "ackley")


def _problem(pps, name, D, lo=-4.0, hi=5.0):
    f = pps.REGISTRY[name]
    lb, ub = (None, None) if lo is None else (np.full(D, lo, np.float32), np.full(D, hi, np.float32))
    return pps.OptimizationProblem(f, np.linspace(-1.0, 2.0, D).astype(np.float32), list(f.default_params) or None,
                                   lb=lb, ub=ub)


def _check(pps, items, runs=2, **kw):
    """items: (problem, particles, iterations); the batch runs twice, a second run starts over."""
    with pps.Batch() as b:
        for k, (p, n, it) in enumerate(items):
            b.add(p, n, maxiters=it, seed=11 * k, w=0.8, wdamp=0.99, **kw)
        for _ in range(runs):
            b.run()
        for k, (p, n, it) in enumerate(items):
            with pps.Swarm(p, n, seed=11 * k) as sw:
                sw.init()
                sw.sync_run(it, w=0.8, wdamp=0.99, **kw)
                u, c, i = sw.gbest()
                bu, bc, bi = b.result(k)
                assert bi == i and np.float32(bc) == np.float32(c) and np.array_equal(bu, u), (k, n, it)
                want, got = sw.state(), b.state(k)
                for f in want:
                    assert np.array_equal(got[f], want[f], equal_nan=True), (k, p.f.name, p.dim, n, it, f)


def _mix(pps, count, dims, sizes, iters, seed=0):
    r = np.random.default_rng(seed)
    return [(_problem(pps, NAMES[k % 4], int(r.integers(dims[0], dims[1] + 1))),
             int(r.integers(sizes[0], sizes[1] + 1)), int(r.integers(iters[0], iters[1] + 1))) for k in range(count)]


@pytest.mark.parametrize("count,dims,sizes", [(1, (10, 10), (700, 700)), (5, (1, 9), (1, 70)), (40, (2, 64), (256, 2048)),
                                              (300, (2, 40), (100, 900)), (700, (1, 4), (1, 200)),
                                              (6, (90, 140), (4000, 9000))])
def test_equals_the_swarm_alone(pps, count, dims, sizes):
    _check(pps, _mix(pps, count, dims, sizes, (3, 9)))


def test_uneven_iterations_and_none(pps):
    _check(pps, _mix(pps, 60, (2, 30), (50, 1500), (0, 40)))
    _check(pps, [(_problem(pps, "ackley", 7), 33, 0), (_problem(pps, "sphere", 2), 1, 0)])


def test_largest_that_fits_and_beyond(pps):
    fits = (_problem(pps, "sphere", 42), 65536, 2)  # 2.75 M coordinates: every SM
    _check(pps, [fits, (_problem(pps, "rastrigin", 3), 50, 5)], runs=1)
    _check(pps, [(_problem(pps, "sphere", 60), 65536, 2), (_problem(pps, "rastrigin", 3), 50, 5)], runs=1)


def test_runs_that_keep_the_streaming_form(pps):
    _check(pps, _mix(pps, 6, (2, 20), (50, 400), (5, 5)), c1=1e-38)
    _check(pps, [(_problem(pps, "rastrigin", 5, None), 100, 5), (_problem(pps, "sphere", 5, None), 100, 5)])


def test_unbounded(pps):
    _check(pps, [(_problem(pps, n, d, None), 150, 6) for n, d in (("sphere", 5), ("rosenbrock", 12))])
