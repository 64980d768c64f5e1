"""Which Tsit5 fits take which step kernel: on both sides of each rule's lines
the swarm equals the oracle bit for bit, and few saves or few steps are not
given to the kernels that spread the saves.  For the latter the largest swarm
that those kernels take is timed against a slightly larger one, which has one
thread per particle: without such a rule it took 1.5 to 1.8 times as long."""
import numpy as np
import pytest

from test_gpu_sync_parity import assert_state_equal
from test_ode_oracle import oracle_ode_problem

pytestmark = pytest.mark.gpu


def _fit(pps, model, nsteps, nsaves, adaptive=False, tol=1e-3):
    from parallelparticleswarms import ode
    obs = np.random.default_rng(nsaves).uniform(0.2, 2.0, (nsaves, 2)).astype(np.float32)
    make = ode.lv_problem if model == "lv" else ode.fhn_problem
    prob = make(obs, u0=(1.0, 1.0), dt=3.0 / nsteps, nsteps=nsteps, save_every=1, lb=0.0, ub=3.0, method="tsit5",
                save_dt=3.0 / (nsaves - 1))
    return ode.adaptive(prob, reltol=tol) if adaptive else prob


def _same(pps, orc, prob, n):
    with pps.Swarm(prob, n, seed=4) as sw:
        sw.init()
        ref = orc.OracleSwarm(oracle_ode_problem(orc, prob), n, 4).init()
        for k in (1, 2):
            sw.sync_run(k, w=0.8)
            ref.sync_run(k, w=0.8)
            assert_state_equal(sw, ref, f"{k} iterations")


def _time(pps, prob, n):
    with pps.Swarm(prob, n, seed=1) as sw:
        return min(sw.init().sync_run(64) for _ in range(5))


@pytest.mark.parametrize("saves,n", [(63, 50), (64, 50), (64, 4000), (64, 4001), (101, 8000), (101, 8001), (301, 24001)])
def test_adaptive_lines(pps, orc, saves, n):
    _same(pps, orc, _fit(pps, "fhn", 30, saves, adaptive=True), n)


@pytest.mark.parametrize("model", ["lv", "fhn"])
@pytest.mark.parametrize("saves", [4, 16])
def test_adaptive_few_saves_time(pps, model, saves):
    prob = _fit(pps, model, 30, saves, adaptive=True)
    assert _time(pps, prob, 24000) <= 1.2 * _time(pps, prob, 24320)


# (steps, saves, particles): the first and the last of each row of the rule, and its neighbours
FIXED = [(4, 71, 40), (4, 72, 40), (3, 72, 40), (36, 72, 10240), (36, 72, 10241), (24, 90, 10241), (24, 90, 16001),
         (12, 180, 24000), (12, 180, 24001), (12, 300, 28000), (12, 300, 28001), (400, 801, 10000), (150, 900, 12000), (8, 700, 33), (12, 301, 33),
         (13, 111, 33)]


@pytest.mark.parametrize("steps,saves,n", FIXED)
def test_fixed_step_lines(pps, orc, steps, saves, n):
    _same(pps, orc, _fit(pps, "lv", steps, saves), n)


@pytest.mark.parametrize("model", ["lv", "fhn"])
@pytest.mark.parametrize("steps,saves", [(4, 21), (30, 61)])
def test_fixed_step_few_saves_time(pps, model, steps, saves):
    prob = _fit(pps, model, steps, saves)
    assert _time(pps, prob, 28000) <= 1.2 * _time(pps, prob, 28160)
