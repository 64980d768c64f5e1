"""Waits between blocks that give up (PPS_WAIT_POLLS=0 lets each run out at
once): the run reports PPS_ETIMEOUT, nothing of it is offered as a result, and
after a new start the same object runs to the oracle's or the lone swarm's
bits.  The context stays usable throughout."""
import numpy as np
import pytest

from test_gpu_sync_parity import assert_state_equal

pytestmark = pytest.mark.gpu


def _gives_up(pps, call):
    from parallelparticleswarms import _lib
    with pytest.raises(_lib.PPSError) as e:
        call()
    assert e.value.code == _lib.ETIMEOUT


def _problem(pps, name, D):
    f = pps.REGISTRY[name]
    return pps.OptimizationProblem(f, np.zeros(D, np.float32), list(f.default_params) or None,
                                   lb=np.full(D, -4.0, np.float32), ub=np.full(D, 5.0, np.float32))


@pytest.mark.parametrize("D,n", [(3, 1000), (30, 20011)])
def test_resident_run(pps, orc, monkeypatch, D, n):
    prob = _problem(pps, "rastrigin", D)
    ref = orc.OracleSwarm(orc.OracleProblem(2, D, prob.lb, prob.ub, params=[10.0]), n, 3)
    with pps.Swarm(prob, n, seed=3) as sw:
        for _ in range(2):  # a second failure is recovered from like the first
            sw.init()
            sw.sync_run(4)
            monkeypatch.setenv("PPS_WAIT_POLLS", "0")
            _gives_up(pps, lambda: sw.sync_run(6))
            monkeypatch.delenv("PPS_WAIT_POLLS")
            assert sw.info().iteration == 4  # the failed run made no iteration
            for call in (sw.gbest, lambda: sw.sync_run(1), lambda: sw.async_run(1)):
                with pytest.raises(ValueError):  # its state is torn: a new init first
                    call()
            sw.init()
            ref.init()
            for k in (3, 8):
                sw.sync_run(k)
                ref.sync_run(k)
                assert_state_equal(sw, ref, f"{k} iterations after the failure")


def test_user_objective(pps, monkeypatch):
    import user_sources as us
    reg = _problem(pps, "rastrigin", 10)
    with pps.Swarm(reg, 2000, seed=8) as a, pps.Swarm(reg.remake(f=pps.cuda_objective(us.RASTRIGIN)), 2000,
                                                      seed=8) as b:
        b.init()
        monkeypatch.setenv("PPS_WAIT_POLLS", "0")
        _gives_up(pps, lambda: b.sync_run(6))
        monkeypatch.delenv("PPS_WAIT_POLLS")
        a.init().sync_run(9)
        b.init().sync_run(9)
        sa, sb = a.state(), b.state()
        for f in sa:
            assert np.array_equal(sa[f], sb[f]), f


def _fits(pps):
    return [(pps.ode.synthetic_fit("lv" if k % 2 else "fhn", k)[0], 300 + k, 3) for k in range(4)]


def _swarms(pps):
    return [(_problem(pps, name, 12 + k), 2500 + k, 5) for k, name in enumerate(("sphere", "rosenbrock", "rastrigin",
                                                                                  "ackley"))]


@pytest.mark.parametrize("kind", ["fits", "swarms"])
def test_batch(pps, monkeypatch, kind):
    items = _fits(pps) if kind == "fits" else _swarms(pps)
    with pps.Batch() as b:
        for k, (p, n, it) in enumerate(items):
            b.add(p, n, maxiters=it, seed=k)
        b.run()
        want = [b.result(k) for k in range(len(items))]
        monkeypatch.setenv("PPS_WAIT_POLLS", "0")
        _gives_up(pps, b.run)
        monkeypatch.delenv("PPS_WAIT_POLLS")
        for k in range(len(items)):  # neither the failed run's values nor the last good run's
            with pytest.raises(ValueError):
                b.result(k)
            with pytest.raises(ValueError):
                b.state(k)
        b.run()
        for k, w in enumerate(want):
            got = b.result(k)
            assert np.array_equal(got[0], w[0]) and got[1:] == w[1:], k
