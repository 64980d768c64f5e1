"""Performance cases of the particle-swarm engine: what its users have it do,
through the package's public entry points.

Kinds of case, and what each stands for in real use:

  solve      ``solve(prob, alg)`` from a fresh problem to the solution with every
             particle's final position read: the call most programs make, from
             the three-parameter fit of a few hundred particles up.  ``alg`` is
             "sync" (ParallelSyncPSOKernel) or "queue" (ParallelPSOKernel with
             the shared global best, the reference's default); ``cons`` adds the
             penalty path with one quadratic constraint.
  restart    a program that keeps its cache and solves again: ``reinit_`` and
             ``solve_``, then every personal best's cost.
  async      ParallelPSOKernel(global_update=False): the whole run against
             private global bests, on a kept cache.
  monitor    a swarm advanced one iteration at a time while the program watches
             the global best, then the whole state read.
  hybrid     HybridPSO: the swarm, then a local optimiser on every particle, all
             local optima read.
  ode        ode_pso: one fit of an ODE model's parameters to a trajectory.
  ode_batch  many such fits of uneven size in one batched launch.
  batch      many uneven closed-form swarms in one batched launch.
  mlp        the neural-network fit on the tensor cores (577 parameters).
  served     a stream of mixed requests given to a running server, all results
             collected.
  user       an objective given as CUDA C source, on a kept cache.

Sizes are those of the repository's tests and benchmark (3-D Rosenbrock with
1000 particles; 2^20 x 100-D Rastrigin; 65,536 x 10-D local stages; 10,000
particles on the Lotka-Volterra benchmark; fits of 256-4096 particles; swarms
of 2-64 dims; the served mix) and generic ones between them.
"""
from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "parallelparticleswarms.jl_gb300"))

import parallelparticleswarms as pps  # noqa: E402
from parallelparticleswarms import _lib, mlp, ode  # noqa: E402

W, C1, C2 = 0.7298, 1.4962, 1.4962  # the library's defaults

BOX = {"sphere": (-5.0, 5.0), "rosenbrock": (-5.0, 5.0), "rastrigin": (-5.12, 5.12), "ackley": (-5.0, 5.0)}
OBJECTIVES = ("sphere", "rosenbrock", "rastrigin", "ackley")

# A least-squares objective with a periodic term, its centres and weights in the
# problem's data: the form in which a user's own function reaches the engine.
USER_SOURCE = """
PPS_DEVICE float pps_objective(pps_point x, int dim, const float* p, const float* data, long long ndata) {
  float s = 0.0f;
  for (int i = 0; i < dim; ++i) {
    const float t = x[i] - data[i];
    s = s + data[dim + i] * (t * t);
    s = s + p[0] * (1.0f - pps_cos2pi(t));
  }
  return s;
}
"""
# the same objective with its fold, which the synchronous step evaluates in registers
USER_STREAM = "#define PPS_HAS_STREAM 1\n" + USER_SOURCE + """
typedef struct { float s; } pps_stream;
PPS_DEVICE void pps_stream_start(pps_stream* st, int dim, const float* p, const float* data, long long ndata) {
  st->s = 0.0f;
}
PPS_DEVICE void pps_stream_add(pps_stream* st, int d, float v, int dim, const float* p, const float* data,
                               long long ndata) {
  const float t = v - data[d];
  st->s = st->s + data[dim + d] * (t * t);
  st->s = st->s + p[0] * (1.0f - pps_cos2pi(t));
}
PPS_DEVICE float pps_stream_finish(const pps_stream* st, int dim, const float* p, const float* data, long long ndata) {
  return st->s;
}
"""


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the reference's regression problem: the smallest call, all latency
        {"name": "solve_small", "kind": "solve", "alg": "sync", "objective": "rosenbrock", "n": 1000, "dim": 3,
         "iters": 500, "cons": False},
        # an ordinary fit through the default algorithm, ragged sizes
        {"name": "solve_ordinary", "kind": "solve", "alg": "queue", "objective": "ackley", "n": 20011, "dim": 30,
         "iters": 300, "cons": False},
        # the headline swarm: every iteration streams 2.1 GB
        {"name": "restart_large", "kind": "restart", "objective": "rastrigin", "n": 1 << 20, "dim": 100, "iters": 200},
        # private global bests: the whole run in one launch
        {"name": "async_mid", "kind": "async", "objective": "rastrigin", "n": 200000, "dim": 100, "iters": 300},
        # a few watched iterations
        {"name": "monitor", "kind": "monitor", "objective": "rastrigin", "n": 10007, "dim": 25, "iters": 6},
        # the local-stage workload of the benchmark
        {"name": "hybrid_lbfgs", "kind": "hybrid", "local": "lbfgs", "objective": "ackley", "n": 65536, "dim": 10,
         "iters": 200, "local_iters": 100},
        # the reference's Lotka-Volterra benchmark: Tsit5, 301 saves
        {"name": "ode_tsit5", "kind": "ode", "model": "lv", "method": "tsit5", "n": 10000, "iters": 100},
        # RK4 fits of uneven size together
        {"name": "ode_batch", "kind": "ode_batch", "fits": 128, "iters": 100},
        # closed-form swarms of uneven size together
        {"name": "batch_swarms", "kind": "batch", "swarms": 256, "iters": 500},
        {"name": "mlp_fit", "kind": "mlp", "n": 16384, "samples": 1024, "iters": 50},
        {"name": "served_mix", "kind": "served", "requests": 64},
        {"name": "user_source", "kind": "user", "stream": False, "n": 100003, "dim": 20, "iters": 200},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng: random.Random):
    kind = rng.choice(["solve", "solve", "solve", "restart", "async", "monitor", "hybrid", "ode", "ode_batch", "batch",
                       "mlp", "served", "user"])
    obj = rng.choice(OBJECTIVES)
    if kind == "solve":
        n, dim = _log_int(rng, 200, 200000), _log_int(rng, 2, 128)
        iters = min(_log_int(rng, 50, 1000), max(50, (1 << 31) // (n * dim)))
        return {"kind": kind, "alg": rng.choice(["sync", "queue"]), "objective": obj, "n": n, "dim": dim,
                "iters": iters, "cons": rng.random() < 0.2}
    if kind == "restart":
        n, dim = _log_int(rng, 100000, 1 << 20), _log_int(rng, 10, 100)
        return {"kind": kind, "objective": obj, "n": n, "dim": dim, "iters": _log_int(rng, 50, 200)}
    if kind == "async":
        n, dim = _log_int(rng, 1000, 400000), _log_int(rng, 2, 128)
        iters = min(_log_int(rng, 50, 1000), max(50, (1 << 32) // (n * dim)))
        return {"kind": kind, "objective": obj, "n": n, "dim": dim, "iters": iters}
    if kind == "monitor":
        return {"kind": kind, "objective": obj, "n": _log_int(rng, 500, 50000), "dim": _log_int(rng, 2, 64),
                "iters": rng.randint(2, 8)}
    if kind == "hybrid":
        return {"kind": kind, "local": rng.choice(["lbfgs", "bfgs"]), "objective": obj, "n": _log_int(rng, 500, 65536),
                "dim": rng.randint(2, 12), "iters": _log_int(rng, 50, 200), "local_iters": rng.randint(20, 100)}
    if kind == "ode":
        return {"kind": kind, "model": rng.choice(["lv", "fhn"]),
                "method": rng.choice(["rk4", "tsit5", "tsit5", "tsit5_adaptive"]), "n": _log_int(rng, 500, 20000),
                "iters": _log_int(rng, 30, 100)}
    if kind == "ode_batch":
        return {"kind": kind, "fits": _log_int(rng, 8, 200), "iters": _log_int(rng, 30, 100)}
    if kind == "batch":
        return {"kind": kind, "swarms": _log_int(rng, 16, 512), "iters": _log_int(rng, 100, 500)}
    if kind == "mlp":
        return {"kind": kind, "n": _log_int(rng, 500, 16384), "samples": 128 * rng.randint(1, 12),
                "iters": _log_int(rng, 10, 50)}
    if kind == "served":
        return {"kind": kind, "requests": _log_int(rng, 8, 96)}
    return {"kind": "user", "stream": rng.random() < 0.5, "n": _log_int(rng, 1000, 200000),
            "dim": _log_int(rng, 2, 64), "iters": _log_int(rng, 50, 300)}


# ------------------------------------------------------------------ inputs
def _problem(objective, dim, cons=False):
    lo, hi = BOX[objective]
    f = pps.REGISTRY[objective]
    rows = None
    if cons:  # stay inside the ball of the box's half width: x . x <= r^2 dim / 4
        rows = pps.quadratic_constraint(dim, c=-0.25 * hi * hi * dim, b=np.ones(dim))
    return pps.OptimizationProblem(f, np.zeros(dim, np.float32), list(f.default_params) or None,
                                   lb=np.full(dim, lo, np.float32), ub=np.full(dim, hi, np.float32), cons=rows)


def _ode_rhs(model, p, u, v, l=0.5):
    if model == "lv":
        return p[0] * u - p[1] * u * v, -p[2] * v + p[3] * u * v
    return u - u ** 3 / 3 - v + l, p[2] * (u + p[0] - p[1] * v)


def _trajectories(model, p, u0, dt, nsteps, every):
    """float64 RK4 of many parameter sets at once: (saves, 2, sets)."""
    u, v = np.full(p.shape[1], u0[0]), np.full(p.shape[1], u0[1])
    out = [(u, v)]
    for s in range(1, nsteps + 1):
        a1, b1 = _ode_rhs(model, p, u, v)
        a2, b2 = _ode_rhs(model, p, u + 0.5 * dt * a1, v + 0.5 * dt * b1)
        a3, b3 = _ode_rhs(model, p, u + 0.5 * dt * a2, v + 0.5 * dt * b2)
        a4, b4 = _ode_rhs(model, p, u + dt * a3, v + dt * b3)
        u = u + dt / 6 * (a1 + 2 * a2 + 2 * a3 + a4)
        v = v + dt / 6 * (b1 + 2 * b2 + 2 * b3 + b4)
        if s % every == 0:
            out.append((u, v))
    return np.array(out)


def _fits(model, count, rng, noise=0.01):
    """``count`` RK4 fits of the batched workload: truth within 20 % of the usual parameters, noisy observations."""
    truth = np.array(ode.LV_TRUTH if model == "lv" else ode.FHN_TRUTH)
    p = truth[:, None] * rng.uniform(0.8, 1.2, (truth.size, count))
    if model == "lv":
        obs = _trajectories("lv", p, (1.0, 1.0), 0.01, 1000, 10)
    else:
        obs = _trajectories("fhn", p, (-1.0, 1.0), 0.01, 2000, 10)
    obs = (obs + rng.normal(0.0, noise, obs.shape)).astype(np.float32)
    make = ode.lv_problem if model == "lv" else ode.fhn_problem
    return [make(np.ascontiguousarray(obs[:, :, k])) for k in range(count)]


def _ode_problem(model, method, rng):
    """One fit: RK4 as in the batched workload, Tsit5 as in the reference's benchmarks (301 saves on [0, 3])."""
    if method == "rk4":
        return _fits(model, 1, rng)[0]
    truth = np.array(ode.LV_TRUTH if model == "lv" else ode.FHN_TRUTH)
    p = truth[:, None] * rng.uniform(0.9, 1.1, (truth.size, 1))
    obs = _trajectories(model, p, (1.0, 1.0), 0.0025, 1200, 4)[:, :, 0].astype(np.float32)
    if model == "lv":
        prob = ode.lv_problem(obs, u0=(1.0, 1.0), dt=0.1, nsteps=30, save_every=1, lb=0.0, ub=10.0, method="tsit5",
                              save_dt=0.01)
    else:
        prob = ode.fhn_problem(obs, u0=(1.0, 1.0), dt=0.1, nsteps=30, save_every=1, l=0.0, lb=0.0, ub=5.0,
                               method="tsit5", save_dt=0.01, fit_l=True)
    return ode.adaptive(prob) if method == "tsit5_adaptive" else prob


def _seed(rng):
    return int(rng.integers(0, 1 << 62))


def prepare(case, seed):
    rng = np.random.default_rng([seed, 2024])
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "solve":
        st["prob"] = _problem(case["objective"], case["dim"], case["cons"])
        st["alg"] = (pps.ParallelSyncPSOKernel(case["n"]) if case["alg"] == "sync"
                     else pps.ParallelPSOKernel(case["n"], global_update=True))
        st["seed"] = _seed(rng)
    elif kind in ("restart", "async"):
        alg = (pps.ParallelSyncPSOKernel(case["n"]) if kind == "restart"
               else pps.ParallelPSOKernel(case["n"], global_update=False))
        st["cache"] = pps.init(_problem(case["objective"], case["dim"]), alg, seed=_seed(rng))
    elif kind == "monitor":
        st["swarm"] = pps.Swarm(_problem(case["objective"], case["dim"]), case["n"], seed=_seed(rng))
    elif kind == "hybrid":
        local = pps.SimpleLBFGS() if case["local"] == "lbfgs" else pps.BFGS()
        alg = pps.HybridPSO(pps.ParallelSyncPSOKernel(case["n"]), local)
        st["cache"] = pps.init(_problem(case["objective"], case["dim"]), alg, seed=_seed(rng))
    elif kind == "ode":
        st["swarm"] = pps.Swarm(_ode_problem(case["model"], case["method"], rng), case["n"], seed=_seed(rng))
    elif kind == "ode_batch":
        nl = (case["fits"] + 1) // 2
        probs = _fits("lv", nl, rng) + _fits("fhn", case["fits"] - nl, rng)
        b = pps.Batch()
        for k, p in enumerate(probs):
            b.add(p, (256, 1024, 4096)[k % 3], maxiters=case["iters"], seed=_seed(rng))
        st["batch"], st["count"] = b, len(probs)
    elif kind == "batch":
        b = pps.Batch()
        for k in range(case["swarms"]):
            # the mix of sizes is the batch's, the samples are the seed's
            h = random.Random(7919 * case["swarms"] + k)
            b.add(_problem(OBJECTIVES[k % 4], h.randint(2, 64)), h.randint(256, 2048), maxiters=case["iters"],
                  seed=_seed(rng))
        st["batch"], st["count"] = b, case["swarms"]
    elif kind == "mlp":
        data, _ = mlp.teacher_task(case["samples"], seed=int(rng.integers(0, 1 << 31)))
        st["swarm"] = pps.Swarm(mlp.mlp_problem(data), case["n"], seed=_seed(rng))
    elif kind == "served":
        st["server"] = pps.Server(memory_budget=2 << 30, max_launches=16)
        fits = _fits("lv", case["requests"] // 4 + 1, rng)
        reqs = []
        for k in range(case["requests"]):
            h = random.Random(104729 * case["requests"] + k)
            n, iters, dim = h.randint(256, 16384), h.randint(100, 2000), h.randint(2, 64)
            prob = fits[k // 4] if k % 4 == 3 else _problem(("rosenbrock", "rastrigin", "ackley")[k % 4], dim)
            reqs.append((prob, n, iters, _seed(rng)))
        st["requests"] = reqs
    else:
        dim = case["dim"]
        f = pps.cuda_objective(USER_STREAM if case["stream"] else USER_SOURCE)
        data = np.concatenate([rng.uniform(-2.0, 2.0, dim), rng.uniform(0.5, 2.0, dim)]).astype(np.float32)
        prob = pps.OptimizationProblem(f, np.zeros(dim, np.float32), [2.5], lb=np.full(dim, -5.0, np.float32),
                                       ub=np.full(dim, 5.0, np.float32), data=data)
        st["cache"] = pps.init(prob, pps.ParallelSyncPSOKernel(case["n"]), seed=_seed(rng))
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "solve":
        sol = pps.solve(st["prob"], st["alg"], maxiters=case["iters"], seed=st["seed"])
        return {"u": sol.u, "objective": sol.objective, "positions": np.asarray(sol.original)}
    if kind in ("restart", "async", "user"):
        cache = st["cache"]
        pps.reinit_(cache)
        sol = pps.solve_(cache, maxiters=case["iters"])
        return {"u": sol.u, "objective": sol.objective, "pcost": cache.swarm.get(_lib.FIELD_PCOST)}
    if kind == "monitor":
        sw = st["swarm"].init()
        watched = []
        for _ in range(case["iters"]):
            sw.sync_run(1)
            watched.append(sw.gbest()[1])
        u, cost, idx = sw.gbest()
        return {"watched": np.array(watched, np.float32), "u": u, "idx": idx, "state": sw.state()}
    if kind == "hybrid":
        cache = st["cache"]
        pps.reinit_(cache)
        sol = pps.solve_(cache, maxiters=case["iters"], local_maxiters=case["local_iters"])
        return {"u": sol.u, "objective": sol.objective, "local_x": cache.swarm.get(_lib.FIELD_LOCAL_X),
                "local_f": cache.swarm.get(_lib.FIELD_LOCAL_F)}
    if kind == "ode":
        sw = st["swarm"].init()
        sw.sync_run(case["iters"])
        u, cost, idx = sw.gbest()
        return {"u": u, "cost": cost, "idx": idx, "pbest": sw.get(_lib.FIELD_PBEST), "pcost": sw.get(_lib.FIELD_PCOST)}
    if kind in ("ode_batch", "batch"):
        st["batch"].run()
        return _results([st["batch"].result(k) for k in range(st["count"])])
    if kind == "mlp":
        sw = st["swarm"].init()
        sw.sync_run(case["iters"])
        u, cost, idx = sw.gbest()
        return {"u": u, "cost": cost, "idx": idx, "pcost": sw.get(_lib.FIELD_PCOST)}
    tickets = [st["server"].submit(p, n, maxiters=it, seed=s) for p, n, it, s in st["requests"]]
    return _results([st["server"].wait(t)[:3] for t in tickets])


def _results(rs):
    return {"u": np.concatenate([r[0] for r in rs]), "cost": np.array([r[1] for r in rs], np.float32),
            "idx": np.array([r[2] for r in rs], np.int64)}


# ------------------------------------------------------------------ work
# floating-point operations of one coordinate's update and of its objective term
_UPDATE = 10
_TERM = {"sphere": 2, "rosenbrock": 8, "rastrigin": 15, "ackley": 15, "user": 18}
_ON_CHIP = 128e6  # bytes of state that the L2 keeps between two iterations


def _swarm_work(n, dim, iters, objective):
    """A synchronous run: a state beyond the L2 streams through memory every
    iteration (read x, v, pbest, pcost; write x, v, pcost), a smaller one is
    made and left once (x, v, pbest, pcost)."""
    per_pass = 4.0 * (5 * dim + 2) * n
    once = 4.0 * (3 * dim + 2) * n
    return {"bytes": per_pass * iters if 12.0 * n * dim > _ON_CHIP else once,
            "flops": float(n) * dim * iters * (_UPDATE + _TERM[objective])}


def _rk4_flops(model, n, iters):
    return float(n) * (iters + 1) * (1000 if model == "lv" else 2000) * (40 if model == "lv" else 52)


def _add(a, b):
    return {k: a[k] + b[k] for k in a}


def work(case):
    kind = case["kind"]
    if kind in ("solve", "restart", "monitor"):
        w = _swarm_work(case["n"], case["dim"], case["iters"], case["objective"])
        if kind == "solve":
            w["bytes"] += 4.0 * case["n"] * case["dim"]  # the positions read
        return w
    if kind == "user":
        return _swarm_work(case["n"], case["dim"], case["iters"], "user")
    if kind == "async":  # private global bests: the state needs no pass per iteration at any size
        w = _swarm_work(case["n"], case["dim"], case["iters"], case["objective"])
        return {"bytes": 4.0 * (3 * case["dim"] + 2) * case["n"], "flops": w["flops"]}
    if kind == "hybrid":
        D, n = case["dim"], case["n"]
        w = _swarm_work(n, D, case["iters"], case["objective"])
        # one local iteration: two-loop recursion of history 10 (or the Jacobian update), gradient, two values;
        # about half of the allowed iterations are taken
        per = (8 * 10 * D if case["local"] == "lbfgs" else 8 * D * D) + 4 * D * _TERM[case["objective"]]
        return _add(w, {"bytes": 4.0 * n * (2 * D + 1), "flops": 0.5 * n * case["local_iters"] * per})
    if kind == "ode":
        n, it = case["n"], case["iters"]
        if case["method"] == "rk4":
            flops = _rk4_flops(case["model"], n, it)
        else:  # 30 steps of six stages, 301 saves of the continuous extension
            flops = float(n) * (it + 1) * (30 * 6 * 22 + 301 * 34)
        return {"bytes": 4.0 * n * 14, "flops": flops}
    if kind == "ode_batch":
        tot, nl = {"bytes": 0.0, "flops": 0.0}, (case["fits"] + 1) // 2
        for k in range(case["fits"]):
            n = (256, 1024, 4096)[k % 3]
            tot = _add(tot, {"bytes": 4.0 * n * 14,
                             "flops": _rk4_flops("lv" if k < nl else "fhn", n, case["iters"])})
        return tot
    if kind == "batch":
        tot = {"bytes": 0.0, "flops": 0.0}
        for k in range(case["swarms"]):
            h = random.Random(7919 * case["swarms"] + k)
            dim, n = h.randint(2, 64), h.randint(256, 2048)
            tot = _add(tot, {"bytes": 4.0 * (3 * dim + 2) * n,
                             "flops": float(n) * dim * case["iters"] * (_UPDATE + _TERM[OBJECTIVES[k % 4]])})
        return tot
    if kind == "mlp":
        n, S, it = case["n"], case["samples"], case["iters"]
        state = 4.0 * (5 * mlp.DIM + 2) * n
        return {"bytes": state * (it if 12.0 * n * mlp.DIM > _ON_CHIP else 1) + 4.0 * 17 * S,
                "flops": float(n) * (it + 1) * S * (2 * 16 * 32 + 32 * 4) + float(n) * mlp.DIM * it * _UPDATE}
    tot = {"bytes": 0.0, "flops": 0.0}
    for k in range(case["requests"]):
        h = random.Random(104729 * case["requests"] + k)
        n, iters, dim = h.randint(256, 16384), h.randint(100, 2000), h.randint(2, 64)
        if k % 4 == 3:
            tot = _add(tot, {"bytes": 4.0 * n * 14, "flops": _rk4_flops("lv", n, iters)})
        else:
            tot = _add(tot, _swarm_work(n, dim, iters, ("rosenbrock", "rastrigin", "ackley")[k % 4]))
    return tot


# ------------------------------------------------------------------ 64-bit values
def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 (Salmon et al., SC'11) over numpy uint64 arrays of 32-bit words."""
    m32 = np.uint64(0xFFFFFFFF)
    s32 = np.uint64(32)
    c0, c1, c2, c3 = np.broadcast_arrays(*(np.asarray(c, np.uint64) for c in (c0, c1, c2, c3)))
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c1, c2, c3 = ((p1 >> s32) ^ c1 ^ np.uint64(k0)), p1 & m32, ((p0 >> s32) ^ c3 ^ np.uint64(k1)), p0 & m32
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return [(c >> np.uint64(8)).astype(np.float64) * 2.0 ** -24 for c in (c0, c1, c2, c3)]


def _value(objective, x):
    """float64 objective of the columns of x (dim, n)."""
    D = x.shape[0]
    if objective == "sphere":
        return (x * x).sum(0)
    if objective == "rosenbrock":
        return (100.0 * (x[1:] - x[:-1] ** 2) ** 2 + (1.0 - x[:-1]) ** 2).sum(0)
    if objective == "rastrigin":
        return 10.0 * D + (x * x - 10.0 * np.cos(2 * np.pi * x)).sum(0)
    return (-20.0 * np.exp(-0.2 * np.sqrt((x * x).sum(0) / D)) - np.exp(np.cos(2 * np.pi * x).sum(0) / D)
            + 20.0 + np.e)


def exact(case, seed):
    """The watched iterations in float64 numpy: the textbook synchronous update
    on the same random stream.  Longer runs amplify the difference between 32
    and 64 bits chaotically, so their outputs have no such value."""
    if case["kind"] != "monitor":
        return None
    rng = np.random.default_rng([seed, 2024])
    sd, n, D = _seed(rng), case["n"], case["dim"]
    lo, hi = (float(np.float32(b)) for b in BOX[case["objective"]])
    i = np.arange(n)
    x = np.empty((D, n))
    for j in range(0, D, 4):
        for h, u in enumerate(_philox(i, j // 4, 0, 0x494E4954, sd)):
            if j + h < D:
                x[j + h] = u * (hi - lo) + lo
    v = np.zeros_like(x)
    p, cost = x.copy(), _value(case["objective"], x)
    pcost = cost.copy()
    watched = []
    for t in range(case["iters"]):
        g = p[:, np.argmin(pcost)].copy()
        for j in range(0, D, 2):
            r = _philox(i, j // 2, t, 0x50534F31, sd)
            for h in range(2):
                d = j + h
                if d < D:
                    v[d] = W * v[d] + C1 * r[2 * h] * (p[d] - x[d]) + C2 * r[2 * h + 1] * (g[d] - x[d])
                    x[d] = np.minimum(np.maximum(x[d] + v[d], lo), hi)
        cost = _value(case["objective"], x)
        better = cost < pcost
        p[:, better], pcost = x[:, better], np.where(better, cost, pcost)
        watched.append(pcost.min())
    return {"watched": np.array(watched), "u": p[:, np.argmin(pcost)].copy(), "idx": None,
            "state": {"x": x, "v": v, "pbest": p, "pcost": pcost, "cost": cost}}
