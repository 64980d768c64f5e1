"""L-BFGS with the cosines' bounded form and with bounds beyond it (the widest
kernel), vs the oracle particle by particle: equal optima, values, iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,oid,prm", [("rastrigin", 2, [10.0]), ("ackley", 3, [20.0, 0.2, 1.0])])
@pytest.mark.parametrize("D,wide", [(1, False), (2, True), (5, False), (10, True), (11, False), (33, False)])
def test_lbfgs(pps, orc, name, oid, prm, D, wide):
    from parallelparticleswarms import _lib
    lb, ub = np.full(D, -5.0, np.float32), np.full(D, 5.0, np.float32)
    if wide:
        ub[0] = 3e38  # 2 x overflows in the cosine's reduction at such points
    prob = pps.OptimizationProblem(pps.REGISTRY[name], np.zeros(D, np.float32), prm, lb=lb, ub=ub)
    n = 150
    x0 = np.random.default_rng(D).uniform(-4.5, 4.5, (D, n)).astype(np.float32)
    with pps.Swarm(prob, n, seed=1) as sw:
        sw.init()
        sw.set(_lib.FIELD_PBEST, x0)
        sw.local_stage("lbfgs", maxiters=30)
        got = [sw.get(f) for f in (_lib.FIELD_LOCAL_X, _lib.FIELD_LOCAL_F, _lib.FIELD_LOCAL_ITERS)]
    oprob = orc.OracleProblem(oid, D, lb, ub, params=prm)
    x, f, it = orc.lbfgs(oprob, x0, maxiters=30)
    assert np.array_equal(got[2], it) and np.array_equal(got[1], f) and np.array_equal(got[0], x)
