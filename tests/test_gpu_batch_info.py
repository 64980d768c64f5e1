"""What pps_batch_info and pps_swarm_info_get report: the block that ran, and
every byte of device memory that a batch or a swarm keeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(pps, D, name="sphere"):
    f = pps.REGISTRY[name]
    return pps.OptimizationProblem(f, np.zeros(D, np.float32), list(f.default_params) or None,
                                   lb=np.full(D, -4.0, np.float32), ub=np.full(D, 5.0, np.float32))


def _state(D, n):
    up = lambda v: (v + 255) // 256 * 256  # noqa: E731
    ld = (n + 31) // 32 * 32
    return 3 * up(4 * D * ld) + 2 * up(4 * ld)


def test_bytes_of_a_batch(pps):
    sizes = [(10, 700), (33, 5000)]
    with pps.Batch() as b:
        for D, n in sizes:
            b.add(_problem(pps, D), n, maxiters=3)
        state = sum(_state(D, n) for D, n in sizes)
        words = sum(4 * (4 * D + 3) for D, _ in sizes)  # bounds, start point, global best, result
        queued = b.info()["device_bytes"]
        # beside them a descriptor of a few hundred bytes per swarm, and no second place for the inputs
        assert state + words < queued < state + words + 1024 * len(sizes)
        b.run()
        assert b.info()["device_bytes"] > queued  # the run's tables


def test_block_of_a_batch(pps):
    with pps.Batch() as b:  # small swarms share an SM: blocks of at most half its threads
        for k in range(40):
            b.add(_problem(pps, 10), 300 + k, maxiters=3)
        b.run()
        assert 32 <= b.info()["threads"] <= 256
        b.set_shape(512, 2)
        b.run()
        assert (b.info()["threads"], b.info()["ppt"]) == (512, 2)
    with pps.Batch() as b:  # a long fit: units of 128 threads, one particle each while they are few
        b.add(pps.ode.synthetic_fit("lv", 0)[0], 5000, maxiters=2)
        b.run()
        assert (b.info()["threads"], b.info()["ppt"]) == (128, 1)
        b.add(pps.ode.synthetic_fit("lv", 1)[0], 65536, maxiters=2)
        b.run()
        assert b.info()["threads"] in (256, 384, 512) and b.info()["ppt"] == 2
    with pps.Batch() as b:  # short fits: a CTA of half the particles, two a thread
        data = np.ones((2, 2), np.float32)
        b.add(pps.ode.lv_problem(data, nsteps=10, save_every=10), 500, maxiters=2)
        b.run()
        assert (b.info()["threads"], b.info()["ppt"]) == (256, 2)


def test_bytes_of_a_swarm(pps):
    with pps.Swarm(_problem(pps, 3), 64, seed=1) as one, pps.Swarm(_problem(pps, 30), 20011, seed=1) as many:
        npad = (20011 + 63) // 64 * 64
        assert one.info().device_bytes < many.info().device_bytes
        assert many.info().device_bytes > 4 * (3 * 30 + 2) * npad + 2 * 152 * (2 + 30) * 8  # the exchange words too
