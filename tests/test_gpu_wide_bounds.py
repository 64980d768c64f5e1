"""Cosine objectives with bounds beyond the bounded cosines' limit (2^126), as a
problem without bounds has: the same kernels' forms with the general cosine.
Equal to the oracle bit for bit at every width, and no slower than the
arithmetic explains: the general cosine has 18 instructions for 14, so a form
for the same dims stays well under twice the bounded one's time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRM = {"rastrigin": (2, [10.0]), "ackley": (3, [20.0, 0.2, 1.0])}


def _problem(pps, name, D, hi):
    return pps.OptimizationProblem(pps.REGISTRY[name], np.zeros(D, np.float32), PRM[name][1],
                                   lb=np.full(D, -5.0, np.float32), ub=np.full(D, hi, np.float32))


@pytest.mark.parametrize("name", sorted(PRM))
@pytest.mark.parametrize("D", [1, 3, 4, 7, 9, 16, 17, 32, 33])
def test_lbfgs_equals_the_oracle(pps, orc, name, D):
    from parallelparticleswarms import _lib
    prob, n = _problem(pps, name, D, 3e38), 100
    x0 = np.random.default_rng(D).uniform(-4.5, 4.5, (D, n)).astype(np.float32)
    with pps.Swarm(prob, n, seed=1) as sw:
        sw.init()
        sw.set(_lib.FIELD_PBEST, x0)
        sw.local_stage("lbfgs", maxiters=25)
        got = [sw.get(f) for f in (_lib.FIELD_LOCAL_X, _lib.FIELD_LOCAL_F, _lib.FIELD_LOCAL_ITERS)]
    oprob = orc.OracleProblem(PRM[name][0], D, prob.lb, prob.ub, params=PRM[name][1])
    x, f, it = orc.lbfgs(oprob, x0, maxiters=25)
    assert np.array_equal(got[2], it) and np.array_equal(got[1], f) and np.array_equal(got[0], x)


@pytest.mark.parametrize("name", sorted(PRM))
@pytest.mark.parametrize("D", [2, 4, 8, 10, 16, 24])
def test_lbfgs_time(pps, name, D):
    from parallelparticleswarms import _lib
    n = 20000
    x0 = np.random.default_rng(D).uniform(-4.5, 4.5, (D, n)).astype(np.float32)
    ms = {}
    for hi in (1e30, 3e38):  # no step reaches either bound: the same iterations
        with pps.Swarm(_problem(pps, name, D, hi), n, seed=1) as sw:
            sw.init()
            sw.set(_lib.FIELD_PBEST, x0)
            ms[hi] = min(sw.local_stage("lbfgs", maxiters=50)[3] for _ in range(5))
    assert ms[3e38] <= 2.0 * ms[1e30], ms


@pytest.mark.parametrize("name", sorted(PRM))
@pytest.mark.parametrize("D", [1, 4, 5, 8, 9, 16, 17, 70])
def test_async_equals_the_oracle(pps, orc, name, D):
    from test_gpu_sync_parity import assert_state_equal
    prob = _problem(pps, name, D, 3e38).remake(lb=None, ub=None, u0=np.linspace(-2.0, 3.0, D).astype(np.float32))
    oprob = orc.OracleProblem(PRM[name][0], D, None, None, u0=prob.u0, params=PRM[name][1])
    with pps.Swarm(prob, 70, seed=5) as sw:
        sw.init()
        ref = orc.OracleSwarm(oprob, 70, 5).init(orc.SAMPLER_UNBOUNDED)
        sw.async_run(15, w=0.8, wdamp=0.98)
        ref.async_run(15, lanes=sw.info().async_lanes, w=0.8, wdamp=0.98)
        assert_state_equal(sw, ref, "15 iterations")


@pytest.mark.parametrize("name", sorted(PRM))
@pytest.mark.parametrize("D", [2, 4, 8, 16, 100])
def test_async_time(pps, name, D):
    """The general form against the short one on the same box.  A tiny c1 asks for the general form; it has up to
    87 instructions a dim for 50 and a branch per pair, so three times the short form's time is its limit."""
    n = 100000
    ms = {}
    for c1 in (1.4962, 1e-38):
        with pps.Swarm(_problem(pps, name, D, 5.0), n, seed=1) as sw:
            sw.init()
            ms[c1] = min(sw.async_run(50, c1=c1) for _ in range(5))
    assert ms[1e-38] <= 3.0 * ms[1.4962], ms
