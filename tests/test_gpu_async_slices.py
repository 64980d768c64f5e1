"""The async run's compile-time slices (k_async_slice) vs the oracle: the first
and last dim count of each slice size and lane count, single particles and
ragged swarms, and the runs that keep the general kernel (coefficients too
small to scale, a negative zero as a bound, no bounds).  Same binary32
operations in the same order on both sides: equal bits."""
import numpy as np
import pytest

from test_gpu_sync_parity import assert_state_equal

pytestmark = pytest.mark.gpu

OBJ = {"sphere": (0, []), "rosenbrock": (1, [1.0, 100.0]), "rastrigin": (2, [10.0]), "ackley": (3, [20.0, 0.2, 1.0])}


def _pair(pps, orc, name, D, n, lb, ub, seed=4):
    oid, prm = OBJ[name]
    prob = pps.OptimizationProblem(pps.REGISTRY[name], np.zeros(D, np.float32), prm or None, lb=lb, ub=ub)
    oprob = orc.OracleProblem(oid, D, lb, ub, u0=np.zeros(D, np.float32), params=prm)
    return pps.Swarm(prob, n, seed=seed), orc.OracleSwarm(oprob, n, seed)


def _same(sw, ref, runs=(1, 12), **kw):
    with sw:
        sw.init()
        ref.init()
        for k in runs:
            info = sw.info()
            sw.async_run(k, w=0.8, wdamp=0.98, **kw)
            ref.async_run(k, lanes=info.async_lanes, w=0.8, wdamp=0.98, **kw)
            assert_state_equal(sw, ref, f"{k} iterations")


@pytest.mark.parametrize("name", sorted(OBJ))
@pytest.mark.parametrize("D", [1, 2, 3, 5, 8, 9, 12, 13, 16, 17, 20, 21, 32, 33, 40, 57, 64, 65, 127, 200, 512])
def test_slices(pps, orc, name, D):
    lb, ub = np.full(D, -3.0, np.float32), np.linspace(2.0, 4.0, D).astype(np.float32)
    _same(*_pair(pps, orc, name, D, 131 if D % 2 else 1, lb, ub))


@pytest.mark.parametrize("case", ["tiny c1", "zero c2", "negative zero", "wide", "513 dims"])
def test_general_form_where_the_short_one_does_not_apply(pps, orc, case):
    D = 513 if case == "513 dims" else 6
    lb, ub = np.full(D, -3.0, np.float32), np.full(D, 4.0, np.float32)
    kw = {}
    if case == "tiny c1":
        kw["c1"] = 1e-37
    elif case == "zero c2":
        kw["c2"] = 0.0
    elif case == "negative zero":
        lb[2] = -0.0
    elif case == "wide":
        lb[0], ub[0] = -1e38, 1e38
    _same(*_pair(pps, orc, "rastrigin", D, 100, lb, ub), **kw)
