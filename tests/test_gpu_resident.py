"""Synchronous runs whose state stays in shared memory (k_resident) vs the
oracle, at the sizes where the form changes: one block / several, one thread
per particle / several sharing its dims, the last particles and dims of a
block, the largest swarm that fits the chip and the first that does not.  The
kernel performs the oracle's binary32 operations in the oracle's order, so
every comparison is for equal bits."""
import numpy as np
import pytest

from test_gpu_sync_parity import assert_state_equal

pytestmark = pytest.mark.gpu

OBJ = {"sphere": (0, []), "rosenbrock": (1, [1.0, 100.0]), "rastrigin": (2, [10.0]), "ackley": (3, [20.0, 0.2, 1.0]),
       "shifted_sphere": (7, [0.5, -1.0, 2.0])}


def _pair(pps, orc, name, D, n, seed=3, gpos=False, cons=None):
    oid, prm = OBJ[name]
    prm = prm[:max(D, 1)] if name == "shifted_sphere" else prm
    lb, ub = np.full(D, -4.0, np.float32), np.full(D, 5.0, np.float32)
    prob = pps.OptimizationProblem(pps.REGISTRY[name], np.zeros(D, np.float32), prm or None, lb=lb, ub=ub, cons=cons)
    oprob = orc.OracleProblem(oid, D, lb, ub, params=prm, cons=cons)
    return pps.Swarm(prob, n, seed=seed, gbest_from_position=gpos), orc.OracleSwarm(oprob, n, seed)


# coordinates (dims rounded up to even x particles): 1536 is the last on one
# block; 128 particles of 3 pairs share threads, 1500 of 1 pair do not
SIZES = [(2, 768), (2, 769), (3, 384), (1, 1537), (9, 31), (33, 65), (5, 8191), (2, 200000), (100, 512), (1023, 17),
         (1024, 40)]


@pytest.mark.parametrize("name", sorted(OBJ))
@pytest.mark.parametrize("D,n", SIZES)
def test_runs_match_the_oracle(pps, orc, name, D, n):
    sw, ref = _pair(pps, orc, name, D, n)
    with sw:
        sw.init()
        ref.init()
        for k in (1, 2, 7):  # odd and even counts: the exchange buffers alternate
            sw.sync_run(k, w=0.8, wdamp=0.97)
            ref.sync_run(k, w=0.8, wdamp=0.97)
            assert_state_equal(sw, ref, f"{k} iterations")


@pytest.mark.parametrize("D,n", [(3, 300), (10, 4001), (31, 1000)])
@pytest.mark.parametrize("name", ["rosenbrock", "ackley"])
def test_position_rule_and_constraints(pps, orc, name, D, n):
    sw, ref = _pair(pps, orc, name, D, n, gpos=True)
    with sw:
        sw.init()
        ref.init()
        sw.sync_run(9)
        ref.sync_run(9, gbest_source=orc.GBEST_FROM_POSITION)
        assert_state_equal(sw, ref, "global best from the position")
    cons = np.stack([pps.quadratic_constraint(D, c=-2.0 * D, b=np.ones(D)),
                     pps.quadratic_constraint(D, c=0.25, a=np.linspace(-1.0, 1.0, D))])
    sw, ref = _pair(pps, orc, name, D, n, cons=cons)
    with sw:
        sw.init()
        ref.init()
        sw.sync_run(9)
        ref.sync_run(9)
        assert_state_equal(sw, ref, "constraints")


@pytest.mark.parametrize("name,n", [("sphere", 2_870_000), ("sphere", 3_000_000), ("rastrigin", 1_420_000)])
def test_capacity_edge(pps, orc, name, n):
    """2-D swarms around the most the chip's shared memory holds; beyond it the stepwise run takes over."""
    sw, ref = _pair(pps, orc, name, 2, n)
    with sw:
        sw.init()
        ref.init()
        sw.sync_run(3)
        ref.sync_run(3)
        assert_state_equal(sw, ref, "3 iterations")


@pytest.mark.parametrize("c1,c2", [(1e-38, 1.5), (0.0, 1.5), (1.5, -1e-34)])
def test_coefficients_that_do_not_scale(pps, orc, c1, c2):
    """c 2^-24 is not exact for tiny coefficients: those runs keep the stepwise form."""
    sw, ref = _pair(pps, orc, "rastrigin", 6, 500)
    with sw:
        sw.init()
        ref.init()
        sw.sync_run(5, c1=c1, c2=c2)
        ref.sync_run(5, c1=c1, c2=c2)
        assert_state_equal(sw, ref, "5 iterations")


def test_two_swarms_from_two_threads(pps, orc):
    """Whole-GPU exchanges of two swarms at once: each waits for its own blocks only."""
    import threading
    pairs = [_pair(pps, orc, "ackley", 11, 30000 + k, seed=k) for k in range(2)]
    errors = []

    def go(sw):
        try:
            for _ in range(5):
                sw.sync_run(20)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    for sw, ref in pairs:
        sw.init()
        ref.init().sync_run(100)
    ts = [threading.Thread(target=go, args=(sw,)) for sw, _ in pairs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    for sw, ref in pairs:
        assert_state_equal(sw, ref, "100 iterations")
        sw.close()


@pytest.mark.parametrize("D,n", [(1, 31), (3, 1000), (20, 4097), (33, 20000), (7, 200000)])
@pytest.mark.parametrize("cons", [False, True])
def test_user_objective_matches_the_registered_run(pps, D, n, cons):
    """A source that spells Rastrigin, its position read back from shared memory, against the registered
    kernel: one and several threads per particle, the last pair of an odd dim count, constraints."""
    import user_sources as us
    rows = np.stack([pps.quadratic_constraint(D, c=-2.0 * D, b=np.ones(D))]) if cons else None
    lb, ub = np.full(D, -4.0, np.float32), np.full(D, 5.0, np.float32)
    reg = pps.OptimizationProblem(pps.rastrigin, np.zeros(D, np.float32), [10.0], lb=lb, ub=ub, cons=rows)
    usr = reg.remake(f=pps.cuda_objective(us.RASTRIGIN))
    with pps.Swarm(reg, n, seed=8) as a, pps.Swarm(usr, n, seed=8) as b:
        a.init()
        b.init()
        for k in (1, 2, 9):
            a.sync_run(k)
            b.sync_run(k)
        sa, sb = a.state(), b.state()
        for f in sa:
            assert np.array_equal(sa[f], sb[f]), f
        assert a.gbest()[1:] == b.gbest()[1:] and np.array_equal(a.gbest()[0], b.gbest()[0])
