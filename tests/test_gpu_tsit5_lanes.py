"""Adaptive Tsit5 fits whose last block is not full (a block of
k_step_tsit5a_lanes holds 16 particles): whole runs, every iteration chained
to the next by the graph, equal the oracle's bit for bit.  Lanes past the last
particle take no part in it: they read no particle that another warp of the
block writes."""
import numpy as np
import pytest

from test_gpu_sync_parity import assert_state_equal
from test_ode_oracle import oracle_ode_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["lv", "fhn"])
@pytest.mark.parametrize("n", [1, 3, 17, 31, 113])
def test_ragged_swarms(pps, orc, model, n):
    from parallelparticleswarms import ode
    obs = np.random.default_rng(n).uniform(0.2, 2.0, (81, 2)).astype(np.float32)
    make = ode.lv_problem if model == "lv" else ode.fhn_problem
    prob = ode.adaptive(make(obs, u0=(1.0, 1.0), dt=0.1, nsteps=30, save_every=1, lb=0.0, ub=3.0, method="tsit5",
                             save_dt=0.0375))
    with pps.Swarm(prob, n, seed=6) as sw:
        sw.init()
        ref = orc.OracleSwarm(oracle_ode_problem(orc, prob), n, 6).init()
        for k in (1, 40, 3):
            sw.sync_run(k, w=0.8)
            ref.sync_run(k, w=0.8)
            assert_state_equal(sw, ref, f"{k} iterations")
