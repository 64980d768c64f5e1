"""Runs of one and two iterations: a program that watches its swarm.  Whatever
form each run takes (few dims step by step, others in shared memory, one block
or many), alternating them equals the oracle bit for bit; and a swarm that fits
the chip's shared memory takes no longer over such a run than a swarm of three
times the particles, which never enters it."""
import numpy as np
import pytest

from test_gpu_sync_parity import assert_state_equal

pytestmark = pytest.mark.gpu


def _problem(pps, name, D):
    f = pps.REGISTRY[name]
    return pps.OptimizationProblem(f, np.zeros(D, np.float32), list(f.default_params) or None,
                                   lb=np.full(D, -4.0, np.float32), ub=np.full(D, 5.0, np.float32))


@pytest.mark.parametrize("name,oid,prm", [("sphere", 0, []), ("ackley", 3, [20.0, 0.2, 1.0])])
@pytest.mark.parametrize("D,n", [(1, 40), (1, 20000), (2, 65), (2, 300001), (3, 1000), (8, 5003), (9, 5003), (16, 100001),
                                 (17, 1500), (255, 70)])
def test_alternating_runs(pps, orc, name, oid, prm, D, n):
    prob = _problem(pps, name, D)
    ref = orc.OracleSwarm(orc.OracleProblem(oid, D, prob.lb, prob.ub, params=prm), n, 7).init()
    with pps.Swarm(prob, n, seed=7) as sw:
        sw.init()
        for k in (1, 1, 3, 1, 2, 1):
            sw.sync_run(k, w=0.8, wdamp=0.97)
            ref.sync_run(k, w=0.8, wdamp=0.97)
            assert_state_equal(sw, ref, f"{k} iterations")


@pytest.mark.parametrize("n", [1000, 300001])
def test_user_objective(pps, n):
    import user_sources as us
    reg = _problem(pps, "rastrigin", 2)
    with pps.Swarm(reg, n, seed=8) as a, pps.Swarm(reg.remake(f=pps.cuda_objective(us.RASTRIGIN)), n, seed=8) as b:
        a.init()
        b.init()
        for k in (1, 2, 3, 2, 1):
            a.sync_run(k)
            b.sync_run(k)
            sa, sb = a.state(), b.state()
            for f in sa:
                assert np.array_equal(sa[f], sb[f]), (k, f)


@pytest.mark.parametrize("iters", [1, 2])
def test_time(pps, iters):
    def ms(n):
        with pps.Swarm(_problem(pps, "sphere", 2), n, seed=1) as sw:
            sw.init()
            return min(sw.sync_run(iters) for _ in range(9))
    assert ms(1000000) <= ms(3000000)
