"""Batches of ODE fits alone (k_ode_teams): every fit equals the same fit
solved as a swarm of its own, bit for bit (which the oracle's parity tests
cover), at the edges of a unit of work, with few fits (one particle a thread)
and many (two), uneven iteration counts, no iterations and long observations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(pps, fits):
    with pps.Batch() as b:
        for p, n, iters, seed in fits:
            b.add(p, n, maxiters=iters, seed=seed, w=0.75, wdamp=0.99)
        for _ in range(2):  # a second run starts over
            b.run()
        for k, (p, n, iters, seed) in enumerate(fits):
            with pps.Swarm(p, n, seed=seed) as sw:
                sw.init()
                sw.sync_run(iters, w=0.75, wdamp=0.99)
                u, c, i = sw.gbest()
                bu, bc, bi = b.result(k)
                assert bi == i and np.float32(bc) == np.float32(c) and np.array_equal(bu, u), (k, n, iters)
                want, got = sw.state(), b.state(k)
                for f in want:
                    assert np.array_equal(got[f], want[f], equal_nan=True), (k, n, iters, f)


def _short(pps, model, seed):
    """A fit of 60 steps, 7 saves (models and parameters of the batched workload)."""
    from parallelparticleswarms import ode
    truth = ode.LV_TRUTH if model == "lv" else ode.FHN_TRUTH
    u0 = (1.0, 1.0) if model == "lv" else (-1.0, 1.0)
    obs = ode.trajectory64(model, truth, u0, 0.02, 60, 10) + np.random.default_rng(seed).normal(0, 0.01, (7, 2))
    make = ode.lv_problem if model == "lv" else ode.fhn_problem
    return make(obs.astype(np.float32), dt=0.02, nsteps=60, save_every=10)


def test_unit_edges_one_particle_a_thread(pps):
    sizes = [1, 127, 128, 129, 255, 256, 257, 1000]
    _check(pps, [(_short(pps, "lv" if k % 2 else "fhn", k), n, (0, 1, 5, 9)[k % 4], 7 * k)
                 for k, n in enumerate(sizes)])


def test_unit_edges_two_particles_a_thread(pps):
    sizes = [1, 129, 255, 256, 257, 511, 513, 4096, 65535, 20001, 30000]
    _check(pps, [(_short(pps, "fhn" if k % 2 else "lv", k), n, (6, 0, 3)[k % 3], 5 * k + 1)
                 for k, n in enumerate(sizes)])


def test_many_more_units_than_teams(pps):
    probs = [_short(pps, m, s) for m in ("lv", "fhn") for s in range(3)]
    _check(pps, [(probs[k % 6], 4096 + 37 * k, 3 + k % 2, k) for k in range(90)])


def test_longest_observations(pps):
    """4096 saves: 32 kB of observations a team, so a block holds fewer teams."""
    from parallelparticleswarms import ode
    obs = ode.trajectory64("lv", ode.LV_TRUTH, (1.0, 1.0), 0.002, 4095, 1).astype(np.float32)
    long = ode.lv_problem(obs, dt=0.002, nsteps=4095, save_every=1)
    _check(pps, [(long, 300, 2, 1), (_short(pps, "fhn", 0), 70000 // 2, 2, 2), (long, 33000, 1, 3)])
