"""Batches of ODE fits alone: long solves and large fits as units on all SMs
(k_ode_teams), short solves and small fits as one CTA or cluster each
(k_batch_ode).  Every fit equals its solve alone bit for bit on both sides of
the rule, at the edges of a unit, of a CTA and of a cluster."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fit(pps, model, steps, seed):
    from parallelparticleswarms import ode
    every = max(1, steps // 8)
    obs = np.random.default_rng(seed).uniform(0.2, 2.0, (steps // every + 1, 2)).astype(np.float32)
    make = ode.lv_problem if model == "lv" else ode.fhn_problem
    return make(obs, u0=(1.0, 1.0), dt=4.0 / max(steps, 100), nsteps=steps, save_every=every)


def _check(pps, fits):
    with pps.Batch() as b:
        for k, (p, n, iters) in enumerate(fits):
            b.add(p, n, maxiters=iters, seed=3 * k, w=0.75, wdamp=0.99)
        for _ in range(2):  # a second run starts over
            b.run()
        for k, (p, n, iters) in enumerate(fits):
            with pps.Swarm(p, n, seed=3 * k) as sw:
                sw.init()
                sw.sync_run(iters, w=0.75, wdamp=0.99)
                u, c, i = sw.gbest()
                bu, bc, bi = b.result(k)
                assert bi == i and np.float32(bc) == np.float32(c) and np.array_equal(bu, u), (k, n, iters)
                want, got = sw.state(), b.state(k)
                for f in want:
                    assert np.array_equal(got[f], want[f], equal_nan=True), (k, n, iters, f)


def _models(k):
    return "lv" if k % 2 else "fhn"


def test_units_of_one_particle_a_thread(pps):
    sizes = [1, 127, 128, 129, 255, 257, 1000, 5000]
    _check(pps, [(_fit(pps, _models(k), 800, k), n, (5, 1, 0, 4)[k % 4]) for k, n in enumerate(sizes)])


def test_units_of_two_particles_a_thread(pps):
    sizes = [1, 129, 255, 256, 257, 511, 513, 4096, 65535, 20001, 30000]
    _check(pps, [(_fit(pps, _models(k), 800, k), n, (3, 0, 2)[k % 3]) for k, n in enumerate(sizes)])


@pytest.mark.parametrize("steps,sizes", [(1, (1, 300)), (10, (512, 513)), (63, (257, 512)), (64, (257, 512)),
                                         (23, (1024, 2047)), (24, (513, 1025, 2048)), (31, (2049, 4097)), (32, (2049, 9000)),
                                         (10, (20000,)), (400, (128,)), (3, (65536, 1))])
def test_both_sides_of_the_rules(pps, steps, sizes):
    _check(pps, [(_fit(pps, _models(k), steps, k), n, 6 - k) for k, n in enumerate(sizes)])


def test_many_short_fits(pps):
    _check(pps, [(_fit(pps, _models(k), 12, k % 5), 100 + 61 * k, 4) for k in range(40)])


def test_short_solves_time(pps):
    """A unit's phase costs 8 us beside its steps, a CTA's iteration 1: a fit of 10 steps and 128 particles is done
    in a fifth of the time of one of 400 steps, not in a third."""
    def ms(steps):
        with pps.Batch() as b:
            b.add(_fit(pps, "fhn", steps, 0), 128, maxiters=50, seed=1)
            return min(b.run() for _ in range(7))
    assert ms(10) <= 0.2 * ms(400)
