"""Fixed-step Tsit5 fits as a pipeline of warps (k_step_tsit5_pipe) and adaptive
ones with several lanes a particle, vs the oracle every iteration: saves that
fall on and between the steps, chunks of 6, 3 and 1 steps, ragged swarms,
solves whose last saves lie past the last step's rounding, and the first fits
that keep the one-thread form.  Same operations in the same order: equal bits."""
import numpy as np
import pytest

from test_gpu_sync_parity import assert_state_equal
from test_ode_oracle import oracle_ode_problem

pytestmark = pytest.mark.gpu


def _fit(pps, model, nsteps, dt, nsaves, save_dt, fit_l=False, seed=0):
    from parallelparticleswarms import ode
    obs = np.random.default_rng(seed).uniform(0.2, 2.0, (nsaves, 2)).astype(np.float32)
    kw = dict(u0=(1.0, 1.0), dt=dt, nsteps=nsteps, save_every=1, lb=0.0, ub=3.0, method="tsit5", save_dt=save_dt)
    return ode.lv_problem(obs, **kw) if model == "lv" else ode.fhn_problem(obs, fit_l=fit_l, **kw)


# (steps, dt, saves, save_dt)
CASES = [(30, 0.1, 301, 0.01), (7, 0.1, 15, 0.05), (7, 0.1, 14, 0.05), (13, 0.1, 90, 0.0143), (12, 0.1, 300, 0.004),
         (6, 0.1, 600, 0.001), (1, 0.5, 50, 0.01), (1, 0.5, 120, 0.004), (5, 0.1, 10, 0.0537), (40, 0.05, 81, 0.025)]


@pytest.mark.parametrize("model,fit_l", [("lv", False), ("fhn", False), ("fhn", True)])
@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}steps-{c[2]}saves")
def test_fixed_step(pps, orc, model, fit_l, case):
    prob = _fit(pps, model, *case, fit_l=fit_l)
    n = 33 if case[0] % 2 else 200
    with pps.Swarm(prob, n, seed=9) as sw:
        sw.init()
        ref = orc.OracleSwarm(oracle_ode_problem(orc, prob), n, 9).init()
        for it in range(4):
            sw.sync_run(1, w=0.8)
            ref.sync_run(1, w=0.8)
            assert_state_equal(sw, ref, f"iteration {it + 1}")
        sw.sync_run(33, w=0.8)
        ref.sync_run(33, w=0.8)
        assert_state_equal(sw, ref, "graph")


@pytest.mark.parametrize("model", ["lv", "fhn"])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 1000])
def test_adaptive_lanes(pps, orc, model, n):
    from parallelparticleswarms import ode
    prob = ode.adaptive(_fit(pps, model, 30, 0.1, 101, 0.03), reltol=1e-4)
    with pps.Swarm(prob, n, seed=2) as sw:
        sw.init()
        ref = orc.OracleSwarm(oracle_ode_problem(orc, prob), n, 2).init()
        for it in range(5):
            sw.sync_run(1)
            ref.sync_run(1)
            assert_state_equal(sw, ref, f"iteration {it + 1}")
