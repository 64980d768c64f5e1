// pps_batch.cu -- many independent swarms of uneven dimension and size in one
// persistent launch.
//
// The reference solves one problem per solve() call: every iteration of
// vectorized_solve! is a kernel launch plus a host reduction
// (src/lowerlevel_solve.jl:1-36), and parameter_estim_ode! takes about five
// launches and host synchronisations per iteration (src/ode_pso.jl:113-170).
// Small problems leave the GPU idle.  Here one CTA owns one swarm for its
// whole life -- sampling, every synchronous iteration, the global best -- with
// the argmin a block reduction (no atomics, no host round trip), so a batch of
// thousands of swarms is one launch that keeps every SM busy.
//
// Semantics per swarm are exactly pps_sync_run's (same Philox counters, same
// operation order, global best from the personal best), so a swarm's result
// does not depend on the batch it rides in: bit-identical alone and in a mix.
//
// Scheduling: CTAs are issued longest-estimated-work first (LPT), so the long
// swarms start early and the short ones fill the tail.  The block size and
// particles per thread come from an autotuner that times the candidates on
// the batch itself (a few iterations each) and caches the winner per batch
// shape.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <tuple>
#include <vector>

#include <cooperative_groups.h>

#include "pps_batch.h"
#include "pps_ode.cuh"
#include "pps_vec.cuh"
#include "pps_objgrad.cuh"

namespace pps {

namespace cg = cooperative_groups;

__device__ __forceinline__ unsigned long long wmin64(unsigned long long k) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const unsigned long long o = __shfl_xor_sync(0xffffffffu, k, off);
    k = o < k ? o : k;
  }
  return k;
}

struct BatchSmem {
  unsigned long long red[33];
  unsigned long long win_key;  // this CTA's best key, read by the other CTAs of the cluster
  int win_fromx;               // its deferred-pbest flag
  float gcost;
};

// block-wide argmin; every thread returns the winning key
__device__ __forceinline__ unsigned long long block_min(unsigned long long key, unsigned long long* red) {
  key = wmin64(key);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __syncthreads();  // red may still be read from the previous call
  if (lane == 0) red[warp] = key;
  __syncthreads();
  if (warp == 0) {
    unsigned long long k = (lane < (int)(blockDim.x >> 5)) ? red[lane] : ~0ull;
    k = wmin64(k);
    if (lane == 0) red[32] = k;
  }
  __syncthreads();
  return red[32];
}

// The swarm-wide argmin.  One CTA: the block reduction.  A cluster of C
// CTAs: each CTA publishes its block minimum (and the winner's pending
// personal-best flag) in shared memory, the hardware cluster barrier makes it
// visible, and every CTA reads all C entries through distributed shared
// memory, so all of them agree on the winner.  `from_x` says whether the
// winner's personal best is its position (improved this iteration).
__device__ __forceinline__ unsigned long long swarm_min(unsigned long long key, BatchSmem& S, const uint8_t* flag,
                                                        int64_t pb, int C, int* from_x) {
  const unsigned long long local = block_min(key, S.red);
  if (C == 1) {
    *from_x = (local != ~0ull) ? flag[(int64_t)(uint32_t)local - pb] : 0;
    return local;
  }
  if (threadIdx.x == 0) {
    S.win_key = local;
    S.win_fromx = (local != ~0ull) ? flag[(int64_t)(uint32_t)local - pb] : 0;
  }
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  unsigned long long best = ~0ull;
  int fx = 0;
  for (int r = 0; r < C; ++r) {
    const BatchSmem* rs = cl.map_shared_rank(&S, r);
    const unsigned long long k = rs->win_key;
    if (k < best) {
      best = k;
      fx = rs->win_fromx;
    }
  }
  *from_x = fx;
  return best;
}

// after the global best has been gathered: no CTA of the swarm may start the
// next iteration (which overwrites positions) or reuse its published key
// before every CTA has read them
__device__ __forceinline__ void swarm_barrier(int C) {
  if (C == 1) {
    __syncthreads();
  } else {
    cg::this_cluster().sync();
  }
}

// particles of this CTA: [pb, pe).  The chunk is a multiple of the block's
// particle width (threads x particles per thread), so every thread of every
// CTA but the last owns the same number of particles.
struct Range {
  int64_t pb, pe;
};
__host__ __device__ __forceinline__ int64_t cta_chunk(int64_t n, int C, int width) {
  return ((n + C - 1) / C + width - 1) / width * width;
}
__device__ __forceinline__ Range cta_range(int64_t n, int C, int rank, int width) {
  const int64_t chunk = cta_chunk(n, C, width);
  Range r;
  r.pb = (int64_t)rank * chunk;
  r.pe = r.pb + chunk < n ? r.pb + chunk : n;
  if (r.pb > n) r.pb = n;
  return r;
}

// rank 0 publishes the swarm's result: in device memory, and when the
// descriptor carries a mailbox in mapped host memory, there too, followed by
// the done flag -- only after every CTA of the swarm has stopped writing
__device__ __forceinline__ void publish_result(const BatchSwarm& sw, const float* sg, float gcost,
                                               unsigned long long win, int rank, int C) {
  swarm_barrier(C);
  if (rank != 0) return;
  for (int d = threadIdx.x; d < sw.dim; d += blockDim.x) {
    sw.g[d] = sg[d];
    if (sw.mail) sw.mail[d] = sg[d];
  }
  if (threadIdx.x == 0) {
    sw.result[0] = gcost;
    sw.result[1] = __uint_as_float((uint32_t)win);
    sw.result[2] = (float)sw.maxiters;
    if (sw.mail) {
      sw.mail[sw.dim] = gcost;
      sw.mail[sw.dim + 1] = __uint_as_float((uint32_t)win);
    }
  }
  if (sw.done) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence_system();
      *reinterpret_cast<volatile int*>(sw.done) = 1;
    }
  }
}

// ---------------------------------------------------------------- separable
template <int OBJ, int PPT>
__device__ void run_swarm(const BatchSwarm& sw, BatchSmem& S, float* sg, float* slb, float* sub, uint8_t* flag,
                          int rank, int C) {
  const int D = sw.dim;
  const int64_t n = sw.n, ld = sw.ld;
  const Range R = cta_range(n, C, rank, (int)blockDim.x * PPT);
  const int64_t pb = R.pb, pe = R.pe;
  const uint32_t k0 = (uint32_t)sw.seed, k1 = (uint32_t)(sw.seed >> 32);
  float* __restrict__ X = sw.X;
  float* __restrict__ V = sw.V;
  float* __restrict__ P = sw.P;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    slb[d] = sw.lb[d];
    sub[d] = sw.ub[d];
  }
  for (int64_t i = pb + threadIdx.x; i < pb + ((pe - pb + 31) / 32 * 32) + 1; i += blockDim.x) flag[i - pb] = 0;
  __syncthreads();
  // ---- init (gpu_init_particles!, src/utils.jl:23-84)
  unsigned long long best = ~0ull;
  for (int64_t i = pb + threadIdx.x; i < pe; i += blockDim.x) {
    Acc<OBJ> acc;
    for (int j = 0; j < D; j += 4) {
      const Rand4 r = philox4x32_10((uint32_t)i, (uint32_t)(j >> 2), 0u, kTagInit, k0, k1);
      const uint32_t rr[4] = {r.a, r.b, r.c, r.d};
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int d = j + h;
        if (d < D) {
          const float u = u01(rr[h]);
          float x;
          if (sw.sampler == PPS_SAMPLER_UNBOUNDED) {
            const float z = sw.u0 ? sw.u0[d] : 0.0f;
            const float a = fabsf(z);
            x = (a > 0.0f) ? __fadd_rn(z, __fmul_rn(u, a)) : u;
          } else {
            x = __fadd_rn(__fmul_rn(u, __fsub_rn(sub[d], slb[d])), slb[d]);
          }
          const int64_t o = (int64_t)d * ld + i;
          X[o] = x;
          V[o] = 0.0f;
          P[o] = x;
          acc.add(sw.op, d, x);
        }
      }
    }
    const float c = finalize<OBJ>(sw.op, acc.s1, acc.s2);
    sw.cost[i] = c;
    sw.pcost[i] = c;
    const unsigned long long k = argmin_key(c, (uint32_t)i);
    best = k < best ? k : best;
  }
  int fromx = 0;
  unsigned long long win = swarm_min(best, S, flag, pb, C, &fromx);
  {
    const uint32_t gi = (uint32_t)win;
    for (int d = threadIdx.x; d < D; d += blockDim.x) sg[d] = P[(int64_t)d * ld + gi];
    if (threadIdx.x == 0) S.gcost = sw.pcost[gi];
  }
  swarm_barrier(C);
  float w = sw.w;
  // ---- synchronous iterations (src/kernels.jl:1-26, src/lowerlevel_solve.jl:1-36)
  // The body is the one of k_sync_step: PPT particles per thread as a vector
  // along the particle axis, dims walked in pairs (one Philox call per
  // particle and pair), the next pair's loads issued before the current pair
  // is computed.
  for (int it = 0; it < sw.maxiters; ++it) {
    const uint32_t t = (uint32_t)it;
    best = ~0ull;
    for (int64_t i0 = pb + (int64_t)threadIdx.x * PPT; i0 < pe; i0 += (int64_t)blockDim.x * PPT) {
      uint8_t fl[PPT];
      bool anyfl = false;
#pragma unroll
      for (int k = 0; k < PPT; ++k) {
        fl[k] = flag[i0 + k - pb];
        anyfl |= fl[k] != 0;
      }
      Acc<OBJ> acc[PPT];
      float xa[PPT], va[PPT], pa[PPT], xb[PPT], vb[PPT], pbv[PPT];
      ldv<PPT>(xa, X + i0);
      ldv<PPT>(va, V + i0);
      ldv<PPT>(pa, P + i0);
      if (D > 1) {
        ldv<PPT>(xb, X + ld + i0);
        ldv<PPT>(vb, V + ld + i0);
        ldv<PPT>(pbv, P + ld + i0);
      }
      for (int j = 0; j < D; j += 2) {
        float nxa[PPT], nva[PPT], npa[PPT], nxb[PPT], nvb[PPT], npb[PPT];
        if (j + 2 < D) {
          const int64_t o = (int64_t)(j + 2) * ld + i0;
          ldv<PPT>(nxa, X + o);
          ldv<PPT>(nva, V + o);
          ldv<PPT>(npa, P + o);
        }
        if (j + 3 < D) {
          const int64_t o = (int64_t)(j + 3) * ld + i0;
          ldv<PPT>(nxb, X + o);
          ldv<PPT>(nvb, V + o);
          ldv<PPT>(npb, P + o);
        }
        Rand4 r[PPT];
#pragma unroll
        for (int k = 0; k < PPT; ++k) r[k] = philox4x32_10((uint32_t)(i0 + k), (uint32_t)(j >> 1), t, kTagStep, k0, k1);
        {
          const int64_t o = (int64_t)j * ld + i0;
          if (anyfl) {
#pragma unroll
            for (int k = 0; k < PPT; ++k) pa[k] = fl[k] ? xa[k] : pa[k];
            stv<PPT>(P + o, pa);
          }
          const float gd = sg[j], lo = slb[j], hi = sub[j];
#pragma unroll
          for (int k = 0; k < PPT; ++k) {
            va[k] = velocity(xa[k], va[k], pa[k], gd, w, sw.c1, sw.c2, u01(r[k].a), u01(r[k].b));
            xa[k] = clamp_lb_ub(__fadd_rn(xa[k], va[k]), lo, hi);
            acc[k].add(sw.op, j, xa[k]);
          }
          stv<PPT>(X + o, xa);
          stv<PPT>(V + o, va);
        }
        if (j + 1 < D) {
          const int64_t o = (int64_t)(j + 1) * ld + i0;
          if (anyfl) {
#pragma unroll
            for (int k = 0; k < PPT; ++k) pbv[k] = fl[k] ? xb[k] : pbv[k];
            stv<PPT>(P + o, pbv);
          }
          const float gd = sg[j + 1], lo = slb[j + 1], hi = sub[j + 1];
#pragma unroll
          for (int k = 0; k < PPT; ++k) {
            vb[k] = velocity(xb[k], vb[k], pbv[k], gd, w, sw.c1, sw.c2, u01(r[k].c), u01(r[k].d));
            xb[k] = clamp_lb_ub(__fadd_rn(xb[k], vb[k]), lo, hi);
            acc[k].add(sw.op, j + 1, xb[k]);
          }
          stv<PPT>(X + o, xb);
          stv<PPT>(V + o, vb);
        }
#pragma unroll
        for (int k = 0; k < PPT; ++k) {
          xa[k] = nxa[k]; va[k] = nva[k]; pa[k] = npa[k];
          xb[k] = nxb[k]; vb[k] = nvb[k]; pbv[k] = npb[k];
        }
      }
#pragma unroll
      for (int k = 0; k < PPT; ++k) {
        const int64_t i = i0 + k;
        const bool valid = i < pe;
        const float c = finalize<OBJ>(sw.op, acc[k].s1, acc[k].s2);
        const float pc = sw.pcost[i];
        const bool imp = valid && c < pc;
        const float npc = imp ? c : pc;
        if (valid) {
          sw.pcost[i] = npc;
          sw.cost[i] = c;
          const unsigned long long key = argmin_key(npc, (uint32_t)i);
          best = key < best ? key : best;
        }
        flag[i - pb] = imp ? 1 : 0;
      }
    }
    win = swarm_min(best, S, flag, pb, C, &fromx);  // also orders this iteration's writes before the gather
    const uint32_t gi = (uint32_t)win;
    for (int d = threadIdx.x; d < D; d += blockDim.x) sg[d] = fromx ? X[(int64_t)d * ld + gi] : P[(int64_t)d * ld + gi];
    if (threadIdx.x == 0) S.gcost = sw.pcost[gi];
    swarm_barrier(C);
    w = __fmul_rn(w, sw.wdamp);
  }
  // ---- canonical state and result
  for (int64_t i = pb + threadIdx.x; i < pe; i += blockDim.x) {
    if (flag[i - pb]) {
      for (int d = 0; d < D; ++d) P[(int64_t)d * ld + i] = X[(int64_t)d * ld + i];
    }
  }
  publish_result(sw, sg, S.gcost, win, rank, C);
}

// ---------------------------------------------------------------- ODE fits
template <int MODEL>
__device__ void run_swarm_ode(const BatchSwarm& sw, BatchSmem& S, float* sg, float* slb, float* sub, uint8_t* flag,
                              float* data, int rank, int C, float one) {
  const int D = sw.dim;
  const int64_t n = sw.n, ld = sw.ld;
  const Range R = cta_range(n, C, rank, 2 * (int)blockDim.x);  // whole trips of two particles per thread
  const int64_t pb = R.pb, pe = R.pe;
  const uint32_t k0 = (uint32_t)sw.seed, k1 = (uint32_t)(sw.seed >> 32);
  const OdeCfg cfg = ode_cfg(sw.op, sw.ndata);
  for (int k = threadIdx.x; k < 2 * cfg.nsaves; k += blockDim.x) data[k] = sw.data[k];
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    slb[d] = sw.lb[d];
    sub[d] = sw.ub[d];
  }
  for (int64_t i = pb + threadIdx.x; i < pe; i += blockDim.x) flag[i - pb] = 0;
  __syncthreads();
  unsigned long long best = ~0ull;
  for (int64_t i = pb + threadIdx.x; i < pe; i += blockDim.x) {
    float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    const Rand4 r = philox4x32_10((uint32_t)i, 0u, 0u, kTagInit, k0, k1);
    const uint32_t rr[4] = {r.a, r.b, r.c, r.d};
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      if (d < D) {
        const float u = u01(rr[d]);
        float xv;
        if (sw.sampler == PPS_SAMPLER_UNBOUNDED) {
          const float z = sw.u0 ? sw.u0[d] : 0.0f;
          const float a = fabsf(z);
          xv = (a > 0.0f) ? __fadd_rn(z, __fmul_rn(u, a)) : u;
        } else {
          xv = __fadd_rn(__fmul_rn(u, __fsub_rn(sub[d], slb[d])), slb[d]);
        }
        x[d] = xv;
        const int64_t o = (int64_t)d * ld + i;
        sw.X[o] = xv;
        sw.V[o] = 0.0f;
        sw.P[o] = xv;
      }
    }
    const float c = ode_loss<MODEL>(x, cfg, data);
    sw.cost[i] = c;
    sw.pcost[i] = c;
    const unsigned long long k = argmin_key(c, (uint32_t)i);
    best = k < best ? k : best;
  }
  int fromx = 0;
  unsigned long long win = swarm_min(best, S, flag, pb, C, &fromx);
  {
    const uint32_t gi = (uint32_t)win;
    for (int d = threadIdx.x; d < D; d += blockDim.x) sg[d] = sw.P[(int64_t)d * ld + gi];
    if (threadIdx.x == 0) S.gcost = sw.pcost[gi];
  }
  swarm_barrier(C);
  float w = sw.w;
  for (int it = 0; it < sw.maxiters; ++it) {
    const uint32_t t = (uint32_t)it;
    best = ~0ull;
    // moves particle i of this CTA's range; its new position in x
    auto move = [&](int64_t i, float (&x)[4]) {
      const bool pending = flag[i - pb] != 0;
      const Rand4 r0 = philox4x32_10((uint32_t)i, 0u, t, kTagStep, k0, k1);
      const Rand4 r1 = philox4x32_10((uint32_t)i, 1u, t, kTagStep, k0, k1);
      const float ra[4] = {u01(r0.a), u01(r0.c), u01(r1.a), u01(r1.c)};
      const float rb[4] = {u01(r0.b), u01(r0.d), u01(r1.b), u01(r1.d)};
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        if (d < D) {
          const int64_t o = (int64_t)d * ld + i;
          float xd = sw.X[o], vd = sw.V[o], pd = sw.P[o];
          if (pending) {
            pd = xd;
            sw.P[o] = pd;
          }
          vd = velocity(xd, vd, pd, sg[d], w, sw.c1, sw.c2, ra[d], rb[d]);
          xd = clamp_lb_ub(__fadd_rn(xd, vd), slb[d], sub[d]);
          sw.X[o] = xd;
          sw.V[o] = vd;
          x[d] = xd;
        }
      }
    };
    // records particle i's cost c: personal best, flag, argmin candidate
    auto settle = [&](int64_t i, float c) {
      const float pc = sw.pcost[i];
      const bool imp = c < pc;
      const float npc = imp ? c : pc;
      sw.pcost[i] = npc;
      sw.cost[i] = c;
      flag[i - pb] = imp ? 1 : 0;
      const unsigned long long key = argmin_key(npc, (uint32_t)i);
      best = key < best ? key : best;
    };
    // two particles per trip, i and i + blockDim.x, their losses packed
    // (ode_loss2: bit-identical to ode_loss of each)
    for (int64_t i = pb + threadIdx.x; i < pe; i += 2 * (int64_t)blockDim.x) {
      const int64_t j = i + blockDim.x;
      float xa[4] = {0.0f, 0.0f, 0.0f, 0.0f}, xb[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      move(i, xa);
      if (j < pe) move(j, xb);
      const float2 c = ode_loss2<MODEL>(xa, xb, cfg, data, one);
      settle(i, c.x);
      if (j < pe) settle(j, c.y);
    }
    win = swarm_min(best, S, flag, pb, C, &fromx);
    const uint32_t gi = (uint32_t)win;
    for (int d = threadIdx.x; d < D; d += blockDim.x)
      sg[d] = fromx ? sw.X[(int64_t)d * ld + gi] : sw.P[(int64_t)d * ld + gi];
    if (threadIdx.x == 0) S.gcost = sw.pcost[gi];
    swarm_barrier(C);
    w = __fmul_rn(w, sw.wdamp);
  }
  for (int64_t i = pb + threadIdx.x; i < pe; i += blockDim.x) {
    if (flag[i - pb]) {
      for (int d = 0; d < D; ++d) sw.P[(int64_t)d * ld + i] = sw.X[(int64_t)d * ld + i];
    }
  }
  publish_result(sw, sg, S.gcost, win, rank, C);
}

// One swarm per cluster of C CTAs (C = 1: a plain CTA).  Dynamic shared
// memory: g, lb, ub (3 * maxdim floats), ODE data (data_floats floats), the
// flags of this CTA's particles (one chunk of bytes).  Separable objectives
// and ODE fits are separate kernels so each gets the registers it needs; both
// take the same arguments (`one`, a run-time 1.0f, is read by the ODE kernel).
template <int PPT>
__global__ void k_batch(const BatchSwarm* __restrict__ descs, const int* __restrict__ order, int C, int maxdim,
                        int data_floats, float one) {
  extern __shared__ float dsm[];
  __shared__ BatchSmem S;
  const int swarm = blockIdx.x / C;
  const int rank = blockIdx.x - swarm * C;  // == cluster block rank: clusters tile the grid in x
  const BatchSwarm sw = descs[order[swarm]];
  float* sg = dsm;
  float* slb = dsm + maxdim;
  float* sub = dsm + 2 * maxdim;
  uint8_t* flag = reinterpret_cast<uint8_t*>(dsm + 3 * maxdim + data_floats);
  switch (sw.objective) {
    case kSphere: run_swarm<kSphere, PPT>(sw, S, sg, slb, sub, flag, rank, C); break;
    case kRosenbrock: run_swarm<kRosenbrock, PPT>(sw, S, sg, slb, sub, flag, rank, C); break;
    case kRastrigin: run_swarm<kRastrigin, PPT>(sw, S, sg, slb, sub, flag, rank, C); break;
    case kAckley: run_swarm<kAckley, PPT>(sw, S, sg, slb, sub, flag, rank, C); break;
    default: break;
  }
}

__global__ void __launch_bounds__(1024, 1) k_batch_ode(const BatchSwarm* __restrict__ descs,
                                                      const int* __restrict__ order, int C, int maxdim,
                                                      int data_floats, float one) {
  extern __shared__ float dsm[];
  __shared__ BatchSmem S;
  const int swarm = blockIdx.x / C;
  const int rank = blockIdx.x - swarm * C;
  const BatchSwarm sw = descs[order[swarm]];
  float* sg = dsm;
  float* slb = dsm + maxdim;
  float* sub = dsm + 2 * maxdim;
  float* data = dsm + 3 * maxdim;
  uint8_t* flag = reinterpret_cast<uint8_t*>(data + data_floats);
  if (sw.objective == kLvFit)
    run_swarm_ode<kOdeLV>(sw, S, sg, slb, sub, flag, data, rank, C, one);
  else if (sw.objective == kFhnFit)
    run_swarm_ode<kOdeFHN>(sw, S, sg, slb, sub, flag, data, rank, C, one);
}

}  // namespace pps

// ---------------------------------------------------------------------------
// host side: shared helpers, the batch object, the autotuner
// ---------------------------------------------------------------------------
namespace pps {

static size_t a256(size_t v) { return (v + 255) / 256 * 256; }

size_t batch_state_bytes(int D, int64_t ld) {
  return a256(sizeof(float) * (size_t)D * ld) * 3 + a256(sizeof(float) * ld) * 2;
}

size_t batch_swarm_bytes(int D, int64_t ld, int64_t ndata) {
  return batch_state_bytes(D, ld) + a256(sizeof(float) * D) * 4 + 256 + a256(sizeof(float) * (size_t)ndata);
}

void batch_carve_state(BatchSwarm& d, char* base) {
  const size_t vec = a256(sizeof(float) * (size_t)d.dim * d.ld), one = a256(sizeof(float) * d.ld);
  d.X = reinterpret_cast<float*>(base);
  d.V = reinterpret_cast<float*>(base + vec);
  d.P = reinterpret_cast<float*>(base + 2 * vec);
  d.pcost = reinterpret_cast<float*>(base + 3 * vec);
  d.cost = reinterpret_cast<float*>(base + 3 * vec + one);
}

void batch_carve(BatchSwarm& d, char* base) {
  const int D = d.dim;
  batch_carve_state(d, base);
  size_t off = batch_state_bytes(D, d.ld);
  auto take = [&](size_t bytes) {
    char* p = base + off;
    off += a256(bytes);
    return p;
  };
  d.lb = reinterpret_cast<float*>(take(sizeof(float) * D));
  d.ub = reinterpret_cast<float*>(take(sizeof(float) * D));
  d.u0 = reinterpret_cast<float*>(take(sizeof(float) * D));
  d.g = reinterpret_cast<float*>(take(sizeof(float) * D));
  d.result = reinterpret_cast<float*>(take(256));
  float* datap = reinterpret_cast<float*>(take(sizeof(float) * (size_t)d.ndata));
  d.data = d.ndata ? datap : nullptr;
}

double batch_work_estimate(const BatchSwarm& d) {
  const double per = is_ode(d.objective) ? (double)ode_cfg(d.op, d.ndata).nsteps * 12.0 : (double)d.dim;
  return (double)d.n * (double)(d.maxiters + 1) * per;
}

int batch_describe(const pps_problem* prob, int64_t n, uint64_t seed, int32_t maxiters, float w, float wdamp,
                   float c1, float c2, BatchSwarm* out, std::vector<float>* host) {
  if (!prob) return set_error(PPS_EINVAL, "problem is NULL");
  const int obj = prob->objective;
  if (!(obj == kSphere || obj == kRosenbrock || obj == kRastrigin || obj == kAckley || is_ode(obj)))
    return set_error(PPS_ENOTSUP, "objective %d is not supported in batches", obj);
  if (prob->dim < 1 || prob->dim > kBatchMaxDim)
    return set_error(PPS_EINVAL, "batched swarms have 1 <= dim <= %d (got %d)", kBatchMaxDim, prob->dim);
  if (prob->ncons != 0)
    return set_error(PPS_ENOTSUP, "constrained problems are solved as swarms of their own, not in batches");
  if (n < 1 || n > kBatchMaxParticles)
    return set_error(PPS_EINVAL, "batched swarms have 1 <= n <= %lld (got %lld)", (long long)kBatchMaxParticles,
                     (long long)n);
  if (maxiters < 0) return set_error(PPS_EINVAL, "maxiters must be >= 0");
  if (prob->nparams < 0 || prob->nparams > 8 || (prob->nparams > 0 && !prob->params))
    return set_error(PPS_EINVAL, "nparams must be in [0, 8]");
  if (!std::isfinite(w) || !std::isfinite(wdamp) || !std::isfinite(c1) || !std::isfinite(c2))
    return set_error(PPS_EINVAL, "coefficients must be finite");
  if (is_ode(obj)) {
    const int rc = ode_check(prob);
    if (rc) return rc;
    if (prob->nparams > 6 && prob->params[6] != 0.0f)
      return set_error(PPS_ENOTSUP, "batched ODE fits integrate with RK4; a Tsit5 fit runs as a swarm of its own");
  }
  const int D = prob->dim;
  bool all_inf = true;
  for (int d = 0; d < D; ++d) {
    const float lo = prob->lb ? prob->lb[d] : -INFINITY, hi = prob->ub ? prob->ub[d] : INFINITY;
    if (std::isnan(lo) || std::isnan(hi) || lo > hi) return set_error(PPS_EINVAL, "bounds of dim %d are invalid", d);
    if (!(std::isinf(lo) && std::isinf(hi))) all_inf = false;
  }
  int sampler = PPS_SAMPLER_UNIFORM;
  if (all_inf) {
    sampler = PPS_SAMPLER_UNBOUNDED;
  } else {
    for (int d = 0; d < D; ++d) {
      const float lo = prob->lb ? prob->lb[d] : -INFINITY, hi = prob->ub ? prob->ub[d] : INFINITY;
      if (!std::isfinite(lo) || !std::isfinite(hi))
        return set_error(PPS_EINVAL, "uniform sampling needs finite bounds (dim %d)", d);
    }
  }
  BatchSwarm d{};
  d.objective = obj;
  d.dim = D;
  d.maxiters = maxiters;
  d.sampler = sampler;
  d.n = n;
  d.ld = (n + 31) / 32 * 32;
  d.w = w;
  d.wdamp = wdamp;
  d.c1 = c1;
  d.c2 = c2;
  d.seed = seed;
  for (int k = 0; k < prob->nparams; ++k) d.op.p[k] = prob->params[k];
  d.op.np = prob->nparams;
  d.op.dim = D;
  d.ndata = is_ode(obj) ? prob->ndata : 0;
  host->clear();
  host->reserve((size_t)3 * D + (size_t)d.ndata);
  for (int k = 0; k < D; ++k) host->push_back(prob->lb ? prob->lb[k] : -INFINITY);
  for (int k = 0; k < D; ++k) host->push_back(prob->ub ? prob->ub[k] : INFINITY);
  for (int k = 0; k < D; ++k) host->push_back(prob->u0 ? prob->u0[k] : 0.0f);
  for (int64_t k = 0; k < d.ndata; ++k) host->push_back(prob->data[k]);
  *out = d;
  return PPS_OK;
}

size_t batch_smem_bytes(int maxdim, int data_floats, int64_t maxchunk) {
  return sizeof(float) * (3 * (size_t)maxdim + (size_t)data_floats) + (size_t)maxchunk + 64;
}

// Shape limits: PPS_BATCH_MAX_CLUSTER (1..16; default 4, ODE fits 4 or 8) caps the
// CTAs a swarm is split over, PPS_ODE_THREADS (128..1024) is the largest block of
// an ODE-fit CTA, then sized to half the fit's particles.  They change how work
// is placed, never what is computed.  Clusters above 8 CTAs are a non-portable
// size.
static int env_int(const char* name, int dflt, int lo, int hi) {
  const char* e = getenv(name);
  const int v = e ? atoi(e) : dflt;
  return (v >= lo && v <= hi) ? v : dflt;
}
static int max_cluster(int dflt) {
  static const int v = env_int("PPS_BATCH_MAX_CLUSTER", 0, 1, 16);
  return v ? v : dflt;
}
// Dims of the reference CTA of the work-based split: a swarm gets one CTA per
// width particles of kBatchDimRef dims (PPS_BATCH_DIM_REF overrides; 0 splits
// by particle count alone).  Measured on 256 swarms of dim U{2..64} and
// U{256..2048} particles, 500 iterations (the autotuner's shape in each case):
// by count 29.7 ms per batch, by work with 8 / 16 / 32 / 64 reference dims
// 23.75 / 27.3 / 23.74 / 27.35 ms.  A swarm's CTAs do not change its result.
constexpr int kBatchDimRef = 32;
static int batch_dim_ref() {
  static const int v = env_int("PPS_BATCH_DIM_REF", kBatchDimRef, 0, 4096);
  return v;
}
static int ode_threads() {  // 0: not given
  static const int v = env_int("PPS_ODE_THREADS", 0, 128, 1024);
  return v;
}
// The shape of an ODE fit's CTAs, two particles per thread and trip (the packed
// RK4 losses).  CTAs of one warp per scheduler spread a fit over more SMs than few
// large ones do: 128 fits of 1000 and 2000 steps, 512 threads and clusters of 4:
// 98 ms, 128 threads and clusters of 8: 58 ms.  But an iteration across a cluster
// waits 4 us for its barriers, and a trip costs 1 us beside its steps, so short
// solves keep the large block: us an iteration, large / small, one fit of 512
// particles and 10 steps 2.2 / 4.8, 60 steps 7.0 / 7.5, 150 steps 15.9 / 12.7; of
// 1024 and 10 steps 3.7 / 4.6, 30 steps 7.7 / 5.7; of 4096 and 30 steps 11.0 /
// 11.6, 60 steps 16.8 / 15.0; 64 of 16384 and 10 steps 43 / 52, 30 steps 73 / 82.
static bool brief_fit(const BatchSwarm& d) {
  return ode_cfg(d.op, d.ndata).nsteps < (d.n <= 512 ? 64 : d.n <= 2048 ? 24 : 32);
}
// Long fits of many particles keep all their threads busy in whatever CTAs, so
// those should spread evenly over the SMs: 256 threads and eight CTAs a fit, or 512
// and four, whichever still gives each CTA an SM of its own; with more fits
// the SMs are full and small CTAs balance best.  Ms, ten iterations beside four
// small swarms, 128 x 8 / 256 x 8 / 512 x 4: 8 LV fits of 8192 particles and 1000
// steps 2.7 / 1.9 / 3.8, 16 of 16384 8.3 / 7.1 / 7.5, 24 of 8192 5.0 / 5.0 / 3.6, 24 FHN 6.2 /
// 6.9 / 4.9, 38 FHN and 400 steps 3.5 / 3.6 / 4.0; us, one LV fit of 3000 and 600 steps with
// a save each, six iterations 1170 / 725 / 1005.
constexpr int64_t kLargeFit = 2048;  // more than one trip of eight CTAs of 128 threads
static bool large_fit(const BatchSwarm& d) { return is_ode(d.objective) && d.n > kLargeFit && !brief_fit(d); }
static int large_fits(const std::vector<BatchSwarm>& descs) {
  int count = 0;
  for (const auto& d : descs) count += large_fit(d);
  return count;
}
static void ode_shape(const BatchSwarm& d, int large, int sm_count, int* threads, int* cluster) {
  const int given = ode_threads();
  bool wide = brief_fit(d) || given;
  int T = 128;
  if (large > 0 && large_fit(d)) {
    if (8 * large <= sm_count)
      T = 256;
    else
      wide = wide || 4 * large <= sm_count - sm_count / 10;
  }
  if (wide) {
    const int64_t half = (d.n + 1) / 2;
    const int most = given ? given : 512;
    T = 128;
    while (T < half && 2 * T <= most) T *= 2;
  }
  const int64_t c = (d.n + 2 * (int64_t)T - 1) / (2 * (int64_t)T);
  const int cmax = max_cluster(wide ? 4 : 8);
  *threads = T;
  *cluster = (int)(c < cmax ? c : cmax);
}

LaunchGroup batch_group_of(const BatchSwarm& d, int threads, int ppt, int spread, int large, int sm_count) {
  LaunchGroup g{};
  const int cmax = max_cluster(4);
  if (is_ode(d.objective)) {
    g.kind = 1;
    ode_shape(d, large, sm_count, &g.T, &g.C);
  } else {
    g.kind = 0;
    g.T = threads;
    const int64_t width = (int64_t)threads * ppt * spread;
    const int dref = batch_dim_ref();
    int64_t c;
    if (dref > 0) {
      // CTAs by work: width particles of dref dims per CTA, so a swarm of many
      // dims spreads over more CTAs than one of few; at least a block's worth
      // of particles per CTA
      c = ((int64_t)d.n * d.dim + width * dref - 1) / (width * dref);
      const int64_t cfull = (d.n + threads - 1) / threads;
      c = c < cfull ? c : cfull;
    } else {
      c = (d.n + width - 1) / width;
    }
    g.C = (int)(c < cmax ? c : cmax);
    if (g.C < 1) g.C = 1;
  }
  return g;
}

static int64_t chunk_of(int64_t n, int C, int width) { return cta_chunk(n, C, width); }

void batch_plan(const std::vector<BatchSwarm>& descs, int threads, int ppt, std::vector<int>* order,
                std::vector<LaunchGroup>* groups, int spread, int sm_count) {
  const int ns = (int)descs.size();
  const int large = large_fits(descs);
  std::map<std::tuple<int, int, int>, std::vector<int>> by;
  for (int k = 0; k < ns; ++k) {
    const LaunchGroup g = batch_group_of(descs[k], threads, ppt, spread, large, sm_count);
    by[std::make_tuple(-g.C, g.kind, g.T)].push_back(k);  // larger clusters first
  }
  order->clear();
  groups->clear();
  for (auto& kv : by) {
    LaunchGroup g{};
    g.C = -std::get<0>(kv.first);
    g.kind = std::get<1>(kv.first);
    g.T = std::get<2>(kv.first);
    g.offset = (int)order->size();
    g.maxdim = 1;
    std::vector<int>& idx = kv.second;
    std::stable_sort(idx.begin(), idx.end(), [&](int a, int c) {
      return batch_work_estimate(descs[a]) > batch_work_estimate(descs[c]);
    });
    for (int k : idx) {
      order->push_back(k);
      g.maxdim = std::max(g.maxdim, descs[k].dim);
      g.data_floats = std::max(g.data_floats, (int)descs[k].ndata);
      g.maxn = std::max(g.maxn, descs[k].n);
    }
    g.count = (int)idx.size();
    groups->push_back(g);
  }
}

constexpr size_t kBatchSmem = 200u << 10;  // dynamic shared memory of a CTA

// Launch a group with clusters of g.C CTAs, or of a smaller size when the
// device cannot co-schedule that many with this block shape.  How a swarm is
// split over CTAs does not change its result (draws are keyed by particle,
// the argmin is over the whole swarm), only its speed.
template <typename Kernel>
static int launch_clustered(Kernel kernel, cudaStream_t stream, const BatchSwarm* ddescs, const int* dorder,
                            const LaunchGroup& g, int width) {
  // the limit is the process's: a constant, so no other thread lowers it before the launch
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBatchSmem);
  if (e != cudaSuccess) return cuda_error(e, "cudaFuncSetAttribute");
  for (int C = g.C; C >= 1; C = (C > 8 ? 8 : C / 2)) {
    const size_t smem = batch_smem_bytes(g.maxdim, g.data_floats, chunk_of(g.maxn, C, width));
    if (smem > kBatchSmem) continue;
    if (C > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(g.count * C));
    cfg.blockDim = dim3((unsigned)g.T);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int active = 0;
    if (C > 1 && (cudaOccupancyMaxActiveClusters(&active, kernel, &cfg) != cudaSuccess || active < 1)) {
      cudaGetLastError();  // clear the query's error and try a smaller cluster
      continue;
    }
    // the last argument is a run-time 1.0f for the packed ODE losses (ode_loss2)
    e = cudaLaunchKernelEx(&cfg, kernel, ddescs, dorder + g.offset, C, g.maxdim, g.data_floats, 1.0f);
    if (e != cudaSuccess) return cuda_error(e, "cudaLaunchKernelEx(batch)");
    return PPS_OK;
  }
  return set_error(PPS_ENOTSUP, "batch needs more shared memory than a CTA has (dim, data or n too large)");
}

int batch_launch_group(cudaStream_t stream, const BatchSwarm* ddescs, const int* dorder, const LaunchGroup& g,
                       int ppt) {
  if (g.kind == 1) return launch_clustered(k_batch_ode, stream, ddescs, dorder, g, 2 * g.T);
  if (ppt == 4) return launch_clustered(k_batch<4>, stream, ddescs, dorder, g, g.T * 4);
  if (ppt == 2) return launch_clustered(k_batch<2>, stream, ddescs, dorder, g, g.T * 2);
  return launch_clustered(k_batch<1>, stream, ddescs, dorder, g, g.T);
}

}  // namespace pps

using namespace pps;

struct pps_batch {
  int device = 0;
  cudaStream_t stream = nullptr;
  static constexpr int kGroupStreams = 5;  // one per cluster size 16, 8, 4, 2, 1
  cudaStream_t gstream[kGroupStreams] = {};
  cudaEvent_t gevent[kGroupStreams] = {};
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  int sm_count = 0;
  std::vector<BatchSwarm> descs;        // device pointers filled at run time
  std::vector<std::vector<float>> host;  // per swarm: lb | ub | u0 | data
  std::vector<size_t> offsets;           // per swarm: arena offset (bytes)
  size_t arena_bytes = 0;
  void* arena = nullptr;
  size_t arena_cap = 0;
  BatchSwarm* ddescs = nullptr;
  int* dorder = nullptr;
  size_t dcap = 0;
  OdeTeams* teams = nullptr;  // ODE fits alone: their units' tables
  BatchResident* resident = nullptr;  // closed-form swarms alone: their waves' tables
  int tuned_threads = 0, tuned_ppt = 0, tuned_spread = 8;
  int last_threads = 0, last_ppt = 0, last_spread = 8;
  int last_groups = 0, last_max_cluster = 0;
  bool ran = false;
  float* io = nullptr;  // device: every swarm's g and result words, then every swarm's inputs
  size_t io_cap = 0;    // floats
  size_t io_floats = 0;  // what the queued swarms need of it
  std::vector<size_t> out_at;    // per swarm: its outputs' place in io
  size_t out_floats = 0;
  std::vector<float> outputs;    // the last run's outputs
};

namespace {

constexpr int kResultWords = 3;  // cost, index bits, iterations

std::mutex g_tune_mu;
std::map<std::string, std::tuple<int, int, int>> g_tune_cache;  // shape -> (threads, ppt, spread)

int prepare(pps_batch* b) {
  const size_t ns = b->descs.size();
  if (b->arena_cap < b->arena_bytes) {
    if (b->arena) cudaFree(b->arena);
    b->arena = nullptr;
    b->arena_cap = 0;
    PPS_CUDA(cudaMalloc(&b->arena, b->arena_bytes));
    b->arena_cap = b->arena_bytes;
  }
  if (b->dcap < ns) {
    if (b->ddescs) cudaFree(b->ddescs);
    if (b->dorder) cudaFree(b->dorder);
    b->ddescs = nullptr;
    b->dorder = nullptr;
    b->dcap = 0;
    PPS_CUDA(cudaMalloc(&b->ddescs, sizeof(BatchSwarm) * ns));
    PPS_CUDA(cudaMalloc(&b->dorder, sizeof(int) * ns));
    b->dcap = ns;
  }
  // every swarm's inputs (lb | ub | u0 | data) in one block written by one
  // copy, and its outputs (g, then the result words) in one read by one copy
  // after the run: a copy per swarm and array took 4 ms of a run of 256 swarms,
  // reading the results one by one 5 ms
  size_t nout = 0;
  for (size_t k = 0; k < ns; ++k) nout += (size_t)b->descs[k].dim + kResultWords;
  const size_t nin = b->io_floats - nout;
  if (b->io_cap < nin + nout) {
    if (b->io) cudaFree(b->io);
    b->io = nullptr;
    b->io_cap = 0;
    PPS_CUDA(cudaMalloc(&b->io, sizeof(float) * (nin + nout)));
    b->io_cap = nin + nout;
  }
  std::vector<float> staged;
  staged.reserve(nin);
  b->out_at.resize(ns);
  b->out_floats = nout;
  char* base = static_cast<char*>(b->arena);
  size_t out = 0;
  for (size_t k = 0; k < ns; ++k) {
    BatchSwarm& d = b->descs[k];
    const int D = d.dim;
    batch_carve_state(d, base + b->offsets[k]);
    d.mail = nullptr;
    d.done = nullptr;
    d.g = b->io + out;
    d.result = d.g + D;
    b->out_at[k] = out;
    out += (size_t)D + kResultWords;
    const float* in = b->io + nout + staged.size();
    d.lb = in;
    d.ub = in + D;
    d.u0 = in + 2 * D;
    if (d.ndata) d.data = in + 3 * D;
    staged.insert(staged.end(), b->host[k].begin(), b->host[k].end());
  }
  PPS_CUDA(cudaMemcpyAsync(b->io + nout, staged.data(), sizeof(float) * nin, cudaMemcpyHostToDevice, b->stream));
  PPS_CUDA(cudaMemcpyAsync(b->ddescs, b->descs.data(), sizeof(BatchSwarm) * ns, cudaMemcpyHostToDevice, b->stream));
  return PPS_OK;
}

// the run's outputs to the host, behind it on b->stream
int read_outputs(pps_batch* b) {
  b->outputs.resize(b->out_floats);
  PPS_CUDA(cudaMemcpyAsync(b->outputs.data(), b->io, sizeof(float) * b->out_floats, cudaMemcpyDeviceToHost, b->stream));
  PPS_CUDA(cudaStreamSynchronize(b->stream));
  return PPS_OK;
}

// every group on its own stream, joined back into b->stream; ev0/ev1 bracket it
int run_groups(pps_batch* b, int threads, int ppt, int spread, int* ngroups, int* maxc) {
  std::vector<int> order;
  std::vector<LaunchGroup> groups;
  batch_plan(b->descs, threads, ppt, &order, &groups, spread, b->sm_count);
  PPS_CUDA(cudaMemcpyAsync(b->dorder, order.data(), sizeof(int) * order.size(), cudaMemcpyHostToDevice, b->stream));
  PPS_CUDA(cudaEventRecord(b->ev0, b->stream));
  int rc = PPS_OK;
  for (size_t k = 0; k < groups.size(); ++k) {
    cudaStream_t st = b->gstream[k % pps_batch::kGroupStreams];
    PPS_CUDA(cudaStreamWaitEvent(st, b->ev0, 0));
    if ((rc = batch_launch_group(st, b->ddescs, b->dorder, groups[k], ppt))) return rc;
    PPS_CUDA(cudaEventRecord(b->gevent[k % pps_batch::kGroupStreams], st));
    PPS_CUDA(cudaStreamWaitEvent(b->stream, b->gevent[k % pps_batch::kGroupStreams], 0));
  }
  PPS_CUDA(cudaEventRecord(b->ev1, b->stream));
  if (ngroups) *ngroups = (int)groups.size();
  if (maxc) {
    *maxc = 1;
    for (const auto& g : groups) *maxc = std::max(*maxc, g.C);
  }
  return PPS_OK;
}

// PPS_BATCH_SHAPE="threads,ppt,spread" (threads 128/256/512, ppt 1/2/4, spread 2/8); other values are ignored
void pinned_shape(int* threads, int* ppt, int* spread) {
  static bool parsed = false;
  static int v[3] = {0, 0, 0};
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  if (!parsed) {
    parsed = true;
    const char* e = getenv("PPS_BATCH_SHAPE");
    int t = 0, p = 0, sp = 0;
    if (e && sscanf(e, "%d,%d,%d", &t, &p, &sp) == 3 && (t == 128 || t == 256 || t == 512) &&
        (p == 1 || p == 2 || p == 4) && (sp == 2 || sp == 8)) {
      v[0] = t;
      v[1] = p;
      v[2] = sp;
    }
  }
  if (v[0]) {
    *threads = v[0];
    *ppt = v[1];
    *spread = v[2];
  }
}

std::string shape_key(const pps_batch* b) {
  // objective mix and coarse size buckets
  int cnt[8] = {0};
  double dims = 0, parts = 0, iters = 0;
  for (const auto& d : b->descs) {
    cnt[std::min(d.objective, 7)]++;
    dims += d.dim;
    parts += (double)d.n;
    iters += d.maxiters;
  }
  const double ns = (double)std::max<size_t>(1, b->descs.size());
  char buf[256];
  snprintf(buf, sizeof(buf), "%d,%d,%d,%d,%d,%d|%d|%d|%d|%d", cnt[0] > 0, cnt[1] > 0, cnt[2] > 0, cnt[3] > 0,
           cnt[4] > 0, cnt[5] > 0, (int)std::log2(1 + dims / ns), (int)std::log2(1 + parts / ns),
           (int)std::log2(1 + iters / ns), (int)std::log2(1.0 + ns));
  return buf;
}

}  // namespace

extern "C" {

int pps_batch_create(pps_batch** out) {
  if (!out) return set_error(PPS_EINVAL, "out is NULL");
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return set_error(PPS_ENODEV, "no CUDA device");
  pps_batch* b = new (std::nothrow) pps_batch();
  if (!b) return set_error(PPS_ENOMEM, "host allocation failed");
  cudaGetDevice(&b->device);
  cudaError_t e = cudaDeviceGetAttribute(&b->sm_count, cudaDevAttrMultiProcessorCount, b->device);
  if (e != cudaSuccess) {
    delete b;
    return cuda_error(e, "cudaDeviceGetAttribute(multiprocessor count)");
  }
  if ((e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking)) != cudaSuccess ||
      (e = cudaEventCreate(&b->ev0)) != cudaSuccess || (e = cudaEventCreate(&b->ev1)) != cudaSuccess) {
    pps_batch_destroy(b);
    return cuda_error(e, "stream/event creation");
  }
  for (int k = 0; k < pps_batch::kGroupStreams; ++k) {
    if ((e = cudaStreamCreateWithFlags(&b->gstream[k], cudaStreamNonBlocking)) != cudaSuccess ||
        (e = cudaEventCreateWithFlags(&b->gevent[k], cudaEventDisableTiming)) != cudaSuccess) {
      pps_batch_destroy(b);
      return cuda_error(e, "stream/event creation");
    }
  }
  *out = b;
  return PPS_OK;
}

int pps_batch_destroy(pps_batch* b) {
  if (!b) return PPS_OK;
  if (b->stream) cudaStreamSynchronize(b->stream);
  for (int k = 0; k < pps_batch::kGroupStreams; ++k) {
    if (b->gstream[k]) {
      cudaStreamSynchronize(b->gstream[k]);
      cudaStreamDestroy(b->gstream[k]);
    }
    if (b->gevent[k]) cudaEventDestroy(b->gevent[k]);
  }
  if (b->arena) cudaFree(b->arena);
  if (b->ddescs) cudaFree(b->ddescs);
  if (b->dorder) cudaFree(b->dorder);
  if (b->io) cudaFree(b->io);
  ode_teams_destroy(b->teams);
  batch_resident_destroy(b->resident);
  if (b->ev0) cudaEventDestroy(b->ev0);
  if (b->ev1) cudaEventDestroy(b->ev1);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
  return PPS_OK;
}

int pps_batch_add(pps_batch* b, const pps_problem* prob, int64_t n, uint64_t seed, int32_t maxiters, float w,
                  float wdamp, float c1, float c2, int32_t* slot) {
  if (!b) return set_error(PPS_EINVAL, "batch is NULL");
  BatchSwarm d;
  std::vector<float> h;
  const int rc = batch_describe(prob, n, seed, maxiters, w, wdamp, c1, c2, &d, &h);
  if (rc) return rc;
  b->offsets.push_back(b->arena_bytes);
  b->arena_bytes += batch_state_bytes(d.dim, d.ld);
  b->io_floats += h.size() + (size_t)d.dim + kResultWords;
  b->descs.push_back(d);
  b->host.push_back(std::move(h));
  b->ran = false;
  if (slot) *slot = (int32_t)(b->descs.size() - 1);
  return PPS_OK;
}

int pps_batch_run(pps_batch* b, float* device_ms) {
  if (!b) return set_error(PPS_EINVAL, "batch is NULL");
  if (b->descs.empty()) return set_error(PPS_EINVAL, "batch is empty");
  int dev = -1;
  cudaGetDevice(&dev);
  if (dev != b->device) PPS_CUDA(cudaSetDevice(b->device));
  b->ran = false;  // no results until this run's are complete
  int rc = prepare(b);
  if (rc) return rc;
  const int ns = (int)b->descs.size();
  bool all_ode = true, none_ode = true;
  for (const auto& d : b->descs) (is_ode(d.objective) ? none_ode : all_ode) = false;
  int pinned = b->tuned_threads, pin_ppt = 0, pin_spread = 0;
  if (!pinned) pinned_shape(&pinned, &pin_ppt, &pin_spread);
  if (all_ode || (none_ode && !pinned)) {
    // fits alone, and closed-form swarms alone whose block shape nobody has
    // fixed, have forms of their own, with nothing to tune
    if (all_ode && !b->teams && !(b->teams = ode_teams_create())) return set_error(PPS_ENOMEM, "host allocation failed");
    if (none_ode && !b->resident && !(b->resident = batch_resident_create()))
      return set_error(PPS_ENOMEM, "host allocation failed");
    bool taken = false;
    int shape_threads = 0, shape_ppt = 1;
    unsigned int *word = nullptr, timed_out = 0;
    PPS_CUDA(cudaEventRecord(b->ev0, b->stream));
    rc = all_ode ? ode_teams_launch(b->teams, b->stream, b->descs, b->ddescs, b->sm_count, &taken, &word,
                                    &shape_threads, &shape_ppt)
                 : batch_resident_launch(b->resident, b->stream, b->descs, b->host, b->ddescs, b->sm_count, &taken,
                                         &word, &shape_threads);
    if (rc) return rc;
    if (taken) {
      PPS_CUDA(cudaEventRecord(b->ev1, b->stream));
      PPS_CUDA(cudaMemcpyAsync(&timed_out, word, sizeof(timed_out), cudaMemcpyDeviceToHost, b->stream));
      if ((rc = read_outputs(b))) return rc;
      if (device_ms) PPS_CUDA(cudaEventElapsedTime(device_ms, b->ev0, b->ev1));
      if (timed_out) return set_error(PPS_ETIMEOUT, "the batch timed out waiting for a swarm's iteration");
      b->last_threads = shape_threads;
      b->last_ppt = shape_ppt;
      b->ran = true;
      return PPS_OK;
    }
  }
  // autotune the block shape for this batch shape (cached), unless PPS_BATCH_SHAPE
  // pins it for every batch ("threads,ppt,spread", e.g. "256,2,2": reproducible
  // profiles, since the autotuner's timings are not representative under a profiler)
  int threads = b->tuned_threads, ppt = b->tuned_ppt, spread = b->tuned_spread;
  if (!threads) pinned_shape(&threads, &ppt, &spread);
  if (!threads && all_ode) {  // the shape of a fit's CTAs is its own (ode_shape)
    threads = 256;
    ppt = 1;
    spread = 8;
  }
  if (!threads) {
    const std::string key = shape_key(b);
    {
      std::lock_guard<std::mutex> lock(g_tune_mu);
      auto it = g_tune_cache.find(key);
      if (it != g_tune_cache.end()) std::tie(threads, ppt, spread) = it->second;
    }
    if (!threads) {
      // time each candidate on this batch with a few iterations per swarm
      std::vector<BatchSwarm> saved = b->descs;
      for (auto& d : b->descs) d.maxiters = std::min(d.maxiters, 4);
      PPS_CUDA(cudaMemcpyAsync(b->ddescs, b->descs.data(), sizeof(BatchSwarm) * ns, cudaMemcpyHostToDevice, b->stream));
      // block size x particles per thread x particles per thread per
      // iteration: a batch of few swarms runs faster spread over more CTAs
      // (more warps per SM) than over few CTAs that loop over their particles
      const int cand_t[3] = {128, 256, 512};
      const int cand_p[3] = {1, 2, 4};
      const int cand_s[2] = {8, 2};
      float best_ms = 1e30f;
      for (int cs : cand_s) {
        for (int ct : cand_t) {
          for (int cp : cand_p) {
            if ((rc = run_groups(b, ct, cp, cs, nullptr, nullptr))) return rc;
            PPS_CUDA(cudaEventSynchronize(b->ev1));
            float ms = 0.0f;
            PPS_CUDA(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
            if (ms < best_ms) {
              best_ms = ms;
              threads = ct;
              ppt = cp;
              spread = cs;
            }
          }
        }
      }
      b->descs = saved;
      PPS_CUDA(cudaMemcpyAsync(b->ddescs, b->descs.data(), sizeof(BatchSwarm) * ns, cudaMemcpyHostToDevice, b->stream));
      std::lock_guard<std::mutex> lock(g_tune_mu);
      g_tune_cache[key] = std::make_tuple(threads, ppt, spread);
    }
  }
  if ((rc = run_groups(b, threads, ppt, spread, &b->last_groups, &b->last_max_cluster))) return rc;
  if ((rc = read_outputs(b))) return rc;
  if (device_ms) PPS_CUDA(cudaEventElapsedTime(device_ms, b->ev0, b->ev1));
  b->last_threads = threads;
  b->last_ppt = ppt;
  if (all_ode) {
    b->last_threads = 0;
    const int large = large_fits(b->descs);
    for (const auto& d : b->descs)
      b->last_threads = std::max(b->last_threads, batch_group_of(d, threads, ppt, spread, large, b->sm_count).T);
    b->last_ppt = 2;
  }
  b->last_spread = spread;
  b->ran = true;
  return PPS_OK;
}

int pps_batch_set_shape(pps_batch* b, int32_t threads, int32_t ppt) {
  if (!b) return set_error(PPS_EINVAL, "batch is NULL");
  if (threads == 0 && ppt == 0) {
    b->tuned_threads = b->tuned_ppt = 0;
    b->tuned_spread = 8;
    return PPS_OK;
  }
  if (!(threads == 128 || threads == 256 || threads == 512) || !(ppt == 1 || ppt == 2 || ppt == 4))
    return set_error(PPS_EINVAL, "block shape must be threads in {128, 256, 512} and ppt in {1, 2, 4}");
  b->tuned_threads = threads;
  b->tuned_ppt = ppt;
  b->tuned_spread = 8;
  return PPS_OK;
}

int pps_batch_info(pps_batch* b, int32_t* nswarms, int32_t* threads, int32_t* ppt, uint64_t* device_bytes) {
  if (!b) return set_error(PPS_EINVAL, "batch is NULL");
  if (nswarms) *nswarms = (int32_t)b->descs.size();
  if (threads) *threads = b->last_threads;
  if (ppt) *ppt = b->last_ppt;
  if (device_bytes)
    *device_bytes = b->arena_bytes + sizeof(float) * b->io_floats + (sizeof(BatchSwarm) + sizeof(int)) * b->descs.size() +
                    ode_teams_bytes(b->teams) + batch_resident_bytes(b->resident);
  return PPS_OK;
}

int pps_batch_result(pps_batch* b, int32_t slot, float* u, float* cost, int64_t* idx) {
  if (!b) return set_error(PPS_EINVAL, "batch is NULL");
  if (slot < 0 || slot >= (int32_t)b->descs.size()) return set_error(PPS_EINVAL, "slot %d out of range", slot);
  if (!b->ran) return set_error(PPS_EINVAL, "batch has not run");
  const BatchSwarm& d = b->descs[slot];
  const float* o = b->outputs.data() + b->out_at[slot];
  const float* res = o + d.dim;
  if (u) memcpy(u, o, sizeof(float) * d.dim);
  if (cost) *cost = res[0];
  if (idx) {
    uint32_t bits;
    memcpy(&bits, &res[1], 4);
    *idx = (int64_t)bits;
  }
  return PPS_OK;
}

int pps_batch_get_state(pps_batch* b, int32_t slot, int32_t field, float* out) {
  if (!b || !out) return set_error(PPS_EINVAL, "NULL argument");
  if (slot < 0 || slot >= (int32_t)b->descs.size()) return set_error(PPS_EINVAL, "slot %d out of range", slot);
  if (!b->ran) return set_error(PPS_EINVAL, "batch has not run");
  const BatchSwarm& d = b->descs[slot];
  float* dev;
  int rows;
  switch (field) {
    case PPS_FIELD_POSITION: dev = d.X; rows = d.dim; break;
    case PPS_FIELD_VELOCITY: dev = d.V; rows = d.dim; break;
    case PPS_FIELD_PBEST: dev = d.P; rows = d.dim; break;
    case PPS_FIELD_PCOST: dev = d.pcost; rows = 1; break;
    case PPS_FIELD_COST: dev = d.cost; rows = 1; break;
    default: return set_error(PPS_EINVAL, "unknown field %d", field);
  }
  const size_t wb = sizeof(float) * (size_t)d.n;
  PPS_CUDA(cudaMemcpy2DAsync(out, wb, dev, sizeof(float) * (size_t)d.ld, wb, rows, cudaMemcpyDeviceToHost, b->stream));
  PPS_CUDA(cudaStreamSynchronize(b->stream));
  return PPS_OK;
}

}  // extern "C"
