// pps_ode.cu -- one ODE-fit swarm at a time: init and the synchronous step
// for the ode_pso objectives (parameter_estim_ode!, src/ode_pso.jl:113-170).
//
// The reference's loop per iteration: ode_update_particle_states! (:1-24),
// a host broadcast that rebuilds every particle's ODE problem, the DiffEqGPU
// solve, _reduce_losses!, ode_update_particle_costs! (:26-41) and a host
// minimum -- about five launches and five synchronisations.  Here the whole
// iteration is one launch: update, RK4 integration, SSE, personal best and
// the argmin publication fused, one thread per particle (two with packed
// RK4 losses for large swarms), observations in shared memory.
//
// The reference clamps with max(position, lb) on whole SVectors
// (src/ode_pso.jl:18-19), which compares lexicographically; this build
// clamps each parameter (max.(x, lb), min.(x, ub)) as the other kernels do.
#include <cmath>
#include <mutex>

#include "pps_internal.h"
#include "pps_ode.cuh"
#include "pps_publish.cuh"

namespace pps {

constexpr int kOdeThreads = 128;
// The step kernel's launch bounds ask for 4 resident blocks per SM: without
// them the assembler sizes the kernel for full occupancy (32 registers),
// which slows the integrators' dependent chains; with them it takes the 36-56
// registers the integrators use.
constexpr int kOdeStepMinBlocks = 4;
constexpr int kOdeMaxDim = 4;

// dynamic shared memory of a launch: the fixed-step Tsit5 saves' weight table
// (8 floats per save, read as two 128-bit words), then the observations (2
// floats per save)
inline size_t ode_dyn_smem(const OdeCfg& c) {
  return sizeof(float) * (size_t)c.nsaves * (c.method == kOdeTsit5 ? 10 : 2);
}

// the block's dynamic shared memory.  Kernels index it directly so the
// compiler keeps its loads in the shared address space.
extern __shared__ __align__(16) float ode_smem[];
template <int METHOD>
__device__ __forceinline__ const float* ode_observations(const OdeCfg& c) {
  return ode_smem + (METHOD == kOdeTsit5 ? 8 * c.nsaves : 0);
}

// copies the observations to shared memory and builds the save table
// (fixed-step Tsit5 only); every thread calls it, and it ends in a barrier
template <int METHOD>
__device__ __forceinline__ void ode_smem_fill(const OdeCfg& c, const float* __restrict__ data_g) {
  float* data = const_cast<float*>(ode_observations<METHOD>(c));
  for (int k = threadIdx.x; k < 2 * c.nsaves; k += blockDim.x) data[k] = data_g[k];
  if constexpr (METHOD == kOdeTsit5) tsit5_table_build(c, ode_smem, (int)threadIdx.x, (int)blockDim.x);
  __syncthreads();
}

// Particles per thread of the step kernel: 1, or 2 for RK4 losses packed in
// f32x2 (ode_loss2).  The packed form issues half the instructions but its
// dependent chain is slower, so it pays only when the launch is
// throughput-bound: a swarm that fills the GPU several times over, or a
// swarm run by the request server beside other launches.  A smaller swarm
// solved alone, whose launch is latency-bound, keeps one particle per thread.
constexpr int64_t kOdePackedMinParticles = (int64_t)1 << 18;

template <int MODEL, int METHOD>
__device__ __forceinline__ float ode_eval(const float (&x)[kOdeMaxDim], const OdeCfg& c, const float* data,
                                          const float* tab) {
  if constexpr (METHOD == kOdeTsit5) return tsit5_loss_tab<MODEL>(x, c, data, tab);
  else if constexpr (METHOD == kOdeTsit5Adaptive) return tsit5a_loss<MODEL>(x, c, data);
  else return ode_loss<MODEL>(x, c, data);
}

template <int MODEL, int METHOD>
__global__ void __launch_bounds__(kOdeThreads) k_init_ode(SwarmDev s, ObjParams op, OdeCfg cfg,
                                                          const float* __restrict__ data_g, uint64_t seed,
                                                          int sampler, const float* __restrict__ u0) {
  ode_smem_fill<METHOD>(cfg, data_g);
  const float* data = ode_observations<METHOD>(cfg);
  const float* tab = ode_smem;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  const int D = s.dim;
  unsigned long long key = ~0ull;
  if (i < s.npad) {
    const bool valid = i < s.n;
    float x[kOdeMaxDim] = {0.0f, 0.0f, 0.0f, 0.0f};
    const Rand4 r = philox4x32_10((uint32_t)i, 0u, 0u, kTagInit, k0, k1);
    const uint32_t rr[4] = {r.a, r.b, r.c, r.d};
#pragma unroll
    for (int d = 0; d < kOdeMaxDim; ++d) {
      if (d < D) {
        const float u = u01(rr[d]);
        float xv;
        if (sampler == PPS_SAMPLER_UNBOUNDED) {
          const float z = u0 ? u0[d] : 0.0f;
          const float a = fabsf(z);
          xv = (a > 0.0f) ? __fadd_rn(z, __fmul_rn(u, a)) : u;
        } else if (sampler == PPS_SAMPLER_LHS) {
          xv = valid ? lhs_position((uint32_t)i, (uint32_t)s.n, (uint32_t)d, u, s.lb[d], s.ub[d], k0, k1) : 0.0f;
        } else {
          xv = __fadd_rn(__fmul_rn(u, __fsub_rn(s.ub[d], s.lb[d])), s.lb[d]);
        }
        x[d] = valid ? xv : 0.0f;
        const int64_t o = (int64_t)d * s.npad + i;
        s.X[o] = x[d];
        s.V[o] = 0.0f;
        s.P[o] = x[d];
      }
    }
    const float c = valid ? ode_eval<MODEL, METHOD>(x, cfg, data, tab) : __int_as_float(0x7f800000);
    s.cost[i] = c;
    s.pcost[i] = c;
    s.flag[i] = 0;
    if (valid) key = argmin_key(c, (uint32_t)i);
  }
  if (publish_block_min(key, s.st)) finish_iteration(s, false, 0u, s.st->w);
}

// The step of a fixed-step Tsit5 fit as a pipeline of warps over 32 particles.
// A solve is a chain of steps (6 right-hand sides, about 200 cycles each) and,
// off that chain, the saves' dense output -- three quarters of the
// instructions at ten saves a step, which one thread per particle ran in
// between.  Warp 0 moves the particles and takes the steps, a chunk of `K` ahead;
// warps 2-7 take a step each and evaluate its saves from the stages warp 0
// left in shared memory, a lane a particle; warp 1 sums the squared errors in save
// order, the order of tsit5_loss_tab, whose operations these are: equal bits.
// One barrier a chunk; two buffers each between the stages.  While warp 0 takes
// the first chunk the others build the save table.
constexpr int kPipeWarps = 8, kPipeEval = kPipeWarps - 2;
constexpr int kPipeMaxSaves = 96;    // saves of a chunk
constexpr int kPipeMaxSteps = 2048;  // steps of a solve

inline __host__ __device__ size_t pipe_smem(int nsaves, int nsteps, int K) {
  return sizeof(float) * (8 * (size_t)nsaves + 2 * (size_t)nsaves + 2 * (size_t)K * 16 * 32 + 2 * kPipeMaxSaves * 32) +
         sizeof(int) * ((size_t)nsteps + 2);
}

template <int MODEL>
__global__ void __launch_bounds__(kPipeWarps * 32) k_step_tsit5_pipe(SwarmDev s, OdeCfg cfg,
                                                                    const float* __restrict__ data_g, uint64_t seed,
                                                                    float c1, float c2, int from_position, int K) {
  IterState* st = s.st;
  const uint32_t t = st->t;
  const float w = st->w;
  const int D = s.dim, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nsaves = cfg.nsaves, nsteps = cfg.nsteps;
  float* tab = ode_smem;
  float* data = tab + 8 * nsaves;
  float* stages = data + 2 * nsaves;                       // [2][K][16][32]
  float* errors = stages + 2 * K * 16 * 32;                // [2][kPipeMaxSaves][32]
  int* start = reinterpret_cast<int*>(errors + 2 * kPipeMaxSaves * 32);  // first save of each step
  const int64_t i = (int64_t)blockIdx.x * 32 + lane;
  const bool valid = i < s.n;
  const int64_t il = valid ? i : s.n - 1;  // lanes past the last particle follow it and write nothing

  float p[kOdeMaxDim] = {0.0f, 0.0f, 0.0f, 0.0f};
  float l = 0.0f, u0 = cfg.u0a, u1 = cfg.u0b, ka[7], kb[7];
  auto chunk = [&](int c) {  // warp 0: the steps of chunk c
    float* out = stages + (c & 1) * K * 16 * 32 + lane;
    for (int k = 0; k < K; ++k) {
      float n0, n1;
      tsit5_step<MODEL>(p, l, cfg.dt, u0, u1, ka, kb, n0, n1);
      out[0] = u0;
      out[32] = u1;
#pragma unroll
      for (int q = 0; q < 7; ++q) {
        out[(2 + q) * 32] = ka[q];
        out[(9 + q) * 32] = kb[q];
      }
      out += 16 * 32;
      u0 = n0;
      u1 = n1;
      ka[0] = ka[6];
      kb[0] = kb[6];
    }
  };
  if (warp == 0) {
    const Rand4 r0 = philox4x32_10((uint32_t)il, 0u, t, kTagStep, (uint32_t)seed, (uint32_t)(seed >> 32));
    const Rand4 r1 = philox4x32_10((uint32_t)il, 1u, t, kTagStep, (uint32_t)seed, (uint32_t)(seed >> 32));
    const float ra[4] = {u01(r0.a), u01(r0.c), u01(r1.a), u01(r1.c)};  // r1 draws of dims 0..3
    const float rb[4] = {u01(r0.b), u01(r0.d), u01(r1.b), u01(r1.d)};  // r2 draws
    const bool pending = s.flag[il] != 0;
#pragma unroll
    for (int d = 0; d < kOdeMaxDim; ++d) {
      if (d < D) {
        const int64_t o = (int64_t)d * s.npad + il;
        const float xd = s.X[o];
        const float pd = pending ? xd : s.P[o];
        const float v = velocity(xd, s.V[o], pd, s.g[d], w, c1, c2, ra[d], rb[d]);
        p[d] = clamp_lb_ub(__fadd_rn(xd, v), s.lb[d], s.ub[d]);
        __syncwarp();  // lanes that follow the last particle have read it
        if (valid) {
          if (pending) s.P[o] = pd;
          s.X[o] = p[d];
          s.V[o] = v;
        }
      }
    }
    l = ode_l(p, cfg);
    ode_rhs<MODEL>(p, l, u0, u1, ka[0], kb[0]);
    chunk(0);
  } else {
    const int k0 = threadIdx.x - 32, kn = (kPipeWarps - 1) * 32;
    for (int k = k0; k < 2 * nsaves; k += kn) data[k] = data_g[k];
    tsit5_table_build(cfg, tab, k0, kn);
    asm volatile("bar.sync 1, %0;" ::"n"((kPipeWarps - 1) * 32) : "memory");
    // start[n]: the first save whose step is n or later
    for (int m = 1 + k0; m < nsaves; m += kn) {
      const int n = __float_as_int(tab[8 * m]);
      for (int q = m == 1 ? 0 : __float_as_int(tab[8 * (m - 1)]) + 1; q <= n; ++q) start[q] = m;
      if (m == nsaves - 1)
        for (int q = n + 1; q <= nsteps + 1; ++q) start[q] = nsaves;
    }
  }
  __syncthreads();
  // steps up to the last save's; saves past the last step are never reached
  int steps = 0;
  if (nsaves > 1) {
    const int last = __float_as_int(tab[8 * (nsaves - 1)]);
    steps = last + 1 < nsteps ? last + 1 : nsteps;
  }
  const int chunks = (steps + K - 1) / K;
  float acc = 0.0f;
  if (warp == 1) {
    const float e0 = __fsub_rn(data[0], cfg.u0a), e1 = __fsub_rn(data[1], cfg.u0b);
    acc = __fadd_rn(__fmul_rn(e0, e0), __fmul_rn(e1, e1));
  }
  for (int c = 1; c <= chunks + 1; ++c) {
    if (warp == 0) {
      if (c < chunks) chunk(c);
    } else if (warp == 1) {
      if (c >= 2) {
        const int first = (c - 2) * K, end = first + K < steps ? first + K : steps;
        const float* e = errors + (c & 1) * kPipeMaxSaves * 32 + lane;
        const int count = start[end] - start[first];
#pragma unroll 8
        for (int m = 0; m < count; ++m) acc = __fadd_rn(acc, e[m * 32]);
      }
    } else if (c <= chunks) {
      const int first = (c - 1) * K;
      for (int k = warp - 2; k < K && first + k < steps; k += kPipeEval) {
        const float* in = stages + (((c - 1) & 1) * K + k) * 16 * 32 + lane;
        float a[7], b[7];
        const float y0 = in[0], y1 = in[32];
#pragma unroll
        for (int q = 0; q < 7; ++q) {
          a[q] = in[(2 + q) * 32];
          b[q] = in[(9 + q) * 32];
        }
        const int m0 = start[first + k], m1 = start[first + k + 1];
        float* e = errors + ((c - 1) & 1) * kPipeMaxSaves * 32 + (m0 - start[first]) * 32 + lane;
#pragma unroll 2
        for (int m = m0; m < m1; ++m) {
          const float4 ra = reinterpret_cast<const float4*>(tab)[2 * m];
          const float4 rb = reinterpret_cast<const float4*>(tab)[2 * m + 1];
          const float wt[7] = {ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
          const float x0 = __fsub_rn(data[2 * m], tsit5_dense_w(y0, cfg.dt, wt, a));
          const float x1 = __fsub_rn(data[2 * m + 1], tsit5_dense_w(y1, cfg.dt, wt, b));
          *e = __fadd_rn(__fmul_rn(x0, x0), __fmul_rn(x1, x1));
          e += 32;
        }
      }
    }
    __syncthreads();
  }
  unsigned long long key = ~0ull;
  if (warp == 1 && valid) {
    float pc = s.pcost[i];
    const bool improved = acc < pc;
    pc = improved ? acc : pc;
    s.pcost[i] = pc;
    s.cost[i] = acc;
    s.flag[i] = improved ? 1 : 0;
    key = argmin_key(pc, (uint32_t)i);
  }
  if (publish_block_min(key, st)) finish_iteration(s, from_position != 0, t + 1u, __fmul_rn(w, st->wdamp));
}

// The step of an adaptive Tsit5 fit with L lanes per particle: all take every
// step, each evaluates every L-th save (tsit5a_loss), so a swarm too small for one
// particle per thread to fill the schedulers gets L times the warps.  Lanes past
// the last particle (whole groups of L) go straight to the publication: one
// that followed a real particle would read it while its own lanes, in another
// warp, write it.
template <int MODEL, int L>
__global__ void __launch_bounds__(kOdeThreads) k_step_tsit5a_lanes(SwarmDev s, OdeCfg cfg,
                                                                const float* __restrict__ data_g, uint64_t seed,
                                                                float c1, float c2, int from_position) {
  IterState* st = s.st;
  const uint32_t t = st->t;
  const float w = st->w;
  const int D = s.dim;
  ode_smem_fill<kOdeTsit5Adaptive>(cfg, data_g);
  const float* data = ode_observations<kOdeTsit5Adaptive>(cfg);
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / L;
  const bool lead = (threadIdx.x & (L - 1)) == 0, valid = i < s.n;
  bool pending = false;
  float x[kOdeMaxDim] = {}, v[kOdeMaxDim] = {}, p[kOdeMaxDim] = {};
  float pc0 = 0.0f, c = 0.0f;
  if (valid) {
    const Rand4 r0 = philox4x32_10((uint32_t)i, 0u, t, kTagStep, (uint32_t)seed, (uint32_t)(seed >> 32));
    const Rand4 r1 = philox4x32_10((uint32_t)i, 1u, t, kTagStep, (uint32_t)seed, (uint32_t)(seed >> 32));
    const float ra[4] = {u01(r0.a), u01(r0.c), u01(r1.a), u01(r1.c)};  // r1 draws of dims 0..3
    const float rb[4] = {u01(r0.b), u01(r0.d), u01(r1.b), u01(r1.d)};  // r2 draws
    pending = s.flag[i] != 0;
#pragma unroll
    for (int d = 0; d < kOdeMaxDim; ++d) {
      if (d < D) {
        const int64_t o = (int64_t)d * s.npad + i;
        const float xd = s.X[o];
        p[d] = pending ? xd : s.P[o];
        v[d] = velocity(xd, s.V[o], p[d], s.g[d], w, c1, c2, ra[d], rb[d]);
        x[d] = clamp_lb_ub(__fadd_rn(xd, v[d]), s.lb[d], s.ub[d]);
      }
    }
    pc0 = s.pcost[i];
    c = tsit5a_loss<MODEL, L>(x, cfg, data);
  }
  __syncwarp();  // every lane of the particle, all in one warp, has read it
  unsigned long long key = ~0ull;
  if (valid && lead) {
#pragma unroll
    for (int d = 0; d < kOdeMaxDim; ++d) {
      if (d < D) {
        const int64_t o = (int64_t)d * s.npad + i;
        if (pending) s.P[o] = p[d];
        s.X[o] = x[d];
        s.V[o] = v[d];
      }
    }
    const bool improved = c < pc0;
    const float pc = improved ? c : pc0;
    s.pcost[i] = pc;
    s.cost[i] = c;
    s.flag[i] = improved ? 1 : 0;
    key = argmin_key(pc, (uint32_t)i);
  }
  if (publish_block_min(key, st)) finish_iteration(s, from_position != 0, t + 1u, __fmul_rn(w, st->wdamp));
}

template <int MODEL, int METHOD, int PPT>
__global__ void __launch_bounds__(kOdeThreads, kOdeStepMinBlocks) k_sync_step_ode(SwarmDev s, ObjParams op, OdeCfg cfg,
                                                               const float* __restrict__ data_g, uint64_t seed,
                                                               float c1, float c2, int from_position, float one) {
  static_assert(PPT == 1 || (PPT == 2 && METHOD == kOdeRk4), "two particles per thread: RK4 only");
  __shared__ float sg[kOdeMaxDim], slb[kOdeMaxDim], sub[kOdeMaxDim];
  IterState* st = s.st;
  const uint32_t t = st->t;
  const float w = st->w;
  const int D = s.dim;
  if (threadIdx.x < D) {
    sg[threadIdx.x] = s.g[threadIdx.x];
    slb[threadIdx.x] = s.lb[threadIdx.x];
    sub[threadIdx.x] = s.ub[threadIdx.x];
  }
  ode_smem_fill<METHOD>(cfg, data_g);
  const float* data = ode_observations<METHOD>(cfg);
  const float* tab = ode_smem;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  // this thread's particles: i0 (and i0 + blockDim.x) of the block's tile
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x * PPT + threadIdx.x;
  float x[PPT][kOdeMaxDim];
#pragma unroll
  for (int q = 0; q < PPT; ++q) {
    const int64_t i = i0 + (int64_t)q * blockDim.x;
#pragma unroll
    for (int d = 0; d < kOdeMaxDim; ++d) x[q][d] = 0.0f;
    if (i >= s.npad) continue;
    const bool pending = s.flag[i] != 0;
    const Rand4 r0 = philox4x32_10((uint32_t)i, 0u, t, kTagStep, k0, k1);
    const Rand4 r1 = philox4x32_10((uint32_t)i, 1u, t, kTagStep, k0, k1);
    const float ra[4] = {u01(r0.a), u01(r0.c), u01(r1.a), u01(r1.c)};  // r1 draws of dims 0..3
    const float rb[4] = {u01(r0.b), u01(r0.d), u01(r1.b), u01(r1.d)};  // r2 draws
#pragma unroll
    for (int d = 0; d < kOdeMaxDim; ++d) {
      if (d < D) {
        const int64_t o = (int64_t)d * s.npad + i;
        float xd = s.X[o];
        float vd = s.V[o];
        float pd = s.P[o];
        if (pending) {
          pd = xd;
          s.P[o] = pd;
        }
        vd = velocity(xd, vd, pd, sg[d], w, c1, c2, ra[d], rb[d]);
        xd = clamp_lb_ub(__fadd_rn(xd, vd), slb[d], sub[d]);
        s.X[o] = xd;
        s.V[o] = vd;
        x[q][d] = xd;
      }
    }
  }
  float c[PPT];
  if constexpr (PPT == 2) {
    const float2 cc = ode_loss2<MODEL>(x[0], x[1], cfg, data, one);
    c[0] = cc.x;
    c[1] = cc.y;
  } else {
    c[0] = ode_eval<MODEL, METHOD>(x[0], cfg, data, tab);
  }
  unsigned long long key = ~0ull;
#pragma unroll
  for (int q = 0; q < PPT; ++q) {
    const int64_t i = i0 + (int64_t)q * blockDim.x;
    if (i >= s.npad) continue;
    const bool valid = i < s.n;
    float pc = s.pcost[i];
    const bool improved = valid && c[q] < pc;
    pc = improved ? c[q] : pc;
    s.pcost[i] = pc;
    s.cost[i] = c[q];
    s.flag[i] = improved ? 1 : 0;
    if (valid) {
      const unsigned long long k = argmin_key(pc, (uint32_t)i);
      key = k < key ? k : key;
    }
  }
  if (publish_block_min(key, st)) finish_iteration(s, from_position != 0, t + 1u, __fmul_rn(w, st->wdamp));
}

// model x integrator
#define PPS_DISPATCH_ODE(obj, method, MACRO)                              \
  do {                                                                    \
    const bool lv_ = (obj) == kLvFit;                                     \
    if ((method) == kOdeTsit5) {                                          \
      if (lv_) MACRO(kOdeLV, kOdeTsit5); else MACRO(kOdeFHN, kOdeTsit5);  \
    } else if ((method) == kOdeTsit5Adaptive) {                           \
      if (lv_) MACRO(kOdeLV, kOdeTsit5Adaptive);                          \
      else MACRO(kOdeFHN, kOdeTsit5Adaptive);                             \
    } else {                                                              \
      if (lv_) MACRO(kOdeLV, kOdeRk4); else MACRO(kOdeFHN, kOdeRk4);      \
    }                                                                     \
  } while (0)

int ode_check(const pps_problem* prob) {
  if (prob->dim < 1 || prob->dim > kOdeMaxDim)
    return set_error(PPS_EINVAL, "ODE fits have at most %d parameters (got %d)", kOdeMaxDim, prob->dim);
  if (prob->objective == kLvFit && prob->dim != 4)
    return set_error(PPS_EINVAL, "the Lotka-Volterra fit has 4 parameters (got %d)", prob->dim);
  if (prob->objective == kFhnFit && prob->dim != 3 && prob->dim != 4)
    return set_error(PPS_EINVAL, "the FitzHugh-Nagumo fit has 3 parameters, or 4 with l (got %d)", prob->dim);
  if (prob->nparams < 5 || !prob->params)
    return set_error(PPS_EINVAL, "ODE fits take params = [u0_1, u0_2, dt, nsteps, save_every(, l)]");
  if (prob->objective == kFhnFit && prob->dim == 3 && prob->nparams < 6)
    return set_error(PPS_EINVAL, "the FitzHugh-Nagumo fit of 3 parameters needs params[5] = l");
  if (!prob->data || prob->ndata < 2 || (prob->ndata & 1) || prob->ndata / 2 > kOdeMaxSaves)
    return set_error(PPS_EINVAL, "ODE fit needs data of 2 * nsaves floats, 1 <= nsaves <= %d", kOdeMaxSaves);
  const float method = prob->nparams > 6 ? prob->params[6] : 0.0f;
  if (method != (float)kOdeRk4 && method != (float)kOdeTsit5 && method != (float)kOdeTsit5Adaptive)
    return set_error(PPS_EINVAL, "ODE fit: params[6] (method) is 0 (RK4), 1 (Tsit5) or 2 (adaptive Tsit5)");
  if (method == (float)kOdeTsit5Adaptive) {
    // params = [u0_1, u0_2, dt (first step), reltol, abstol, l, 2, save_dt]
    const float dt0 = prob->params[2], rtol = prob->params[3], atol = prob->params[4];
    const float save_dt = prob->nparams > 7 ? prob->params[7] : 0.0f;
    if (!(dt0 > 0.0f) || !std::isfinite(dt0) || !(rtol > 0.0f) || !std::isfinite(rtol) || !(atol > 0.0f) ||
        !std::isfinite(atol))
      return set_error(PPS_EINVAL, "adaptive Tsit5 needs a first step dt > 0, reltol > 0 and abstol > 0 (finite)");
    if (!(save_dt > 0.0f) || !std::isfinite(save_dt) || !std::isfinite((prob->ndata / 2 - 1) * save_dt))
      return set_error(PPS_EINVAL, "ODE fit with Tsit5 needs params[7] = save_dt > 0");
    return PPS_OK;
  }
  const float nsteps = prob->params[3], every = prob->params[4];
  if (!(prob->params[2] > 0.0f) || !(nsteps >= 1.0f) || !(every >= 1.0f) || nsteps != (float)(int)nsteps ||
      every != (float)(int)every)
    return set_error(PPS_EINVAL, "ODE fit needs dt > 0 and integral nsteps, save_every >= 1");
  if (method == (float)kOdeTsit5) {
    const float save_dt = prob->nparams > 7 ? prob->params[7] : 0.0f;
    if (!(save_dt > 0.0f) || !std::isfinite(save_dt))
      return set_error(PPS_EINVAL, "ODE fit with Tsit5 needs params[7] = save_dt > 0");
    if ((double)(prob->ndata / 2 - 1) * save_dt > (double)nsteps * prob->params[2] * (1.0 + 1e-6))
      return set_error(PPS_EINVAL, "ODE fit: (nsaves - 1) * save_dt exceeds nsteps * dt");
    return PPS_OK;
  }
  if ((prob->ndata / 2 - 1) * (int64_t)every > (int64_t)nsteps)
    return set_error(PPS_EINVAL, "ODE fit: (nsaves - 1) * save_every exceeds nsteps");
  return PPS_OK;
}

static OdeCfg cfg_of(pps_swarm* s) { return ode_cfg(s->op, s->od.ndata); }

template <int MODEL, int METHOD>
__global__ void k_eval_ode(ObjParams op, OdeCfg cfg, const float* __restrict__ data_g, const float* __restrict__ x,
                           int64_t npts, int64_t stride, float* __restrict__ f);

// The fixed-step Tsit5 kernels' dynamic shared-memory limit is raised once
// per device to the largest observations + save table (init precedes every
// captured run of a swarm, so captured launches need no attribute call); the
// other methods stay within the default 48 KB (2 floats per save).
constexpr int kPipeSmemMax = 200 << 10;

static int ode_set_smem_limit() {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  PPS_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return set_error(PPS_ENOTSUP, "device %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (done[dev]) return PPS_OK;
  const int smem = (int)(sizeof(float) * 10 * kOdeMaxSaves);
#define PPS_ODE_SMEM(M)                                                                                         \
  PPS_CUDA(cudaFuncSetAttribute(k_init_ode<M, kOdeTsit5>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));      \
  PPS_CUDA(cudaFuncSetAttribute(k_sync_step_ode<M, kOdeTsit5, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)); \
  PPS_CUDA(cudaFuncSetAttribute(k_step_tsit5_pipe<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, kPipeSmemMax));  \
  PPS_CUDA(cudaFuncSetAttribute(k_eval_ode<M, kOdeTsit5>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem))
  PPS_ODE_SMEM(kOdeLV);
  PPS_ODE_SMEM(kOdeFHN);
#undef PPS_ODE_SMEM
  done[dev] = true;
  return PPS_OK;
}

int launch_init_ode(pps_swarm* s, int sampler, const float* u0_dev) {
  const unsigned blocks = (unsigned)((s->dv.npad + kOdeThreads - 1) / kOdeThreads);
  const OdeCfg c = cfg_of(s);
  const size_t dsm = ode_dyn_smem(c);
  if (c.method == kOdeTsit5) {
    const int rc = ode_set_smem_limit();
    if (rc) return rc;
  }
#define L_INIT_ODE(M, I) \
  k_init_ode<M, I><<<blocks, kOdeThreads, dsm, s->stream>>>(s->dv, s->op, c, s->od.data, s->seed, sampler, u0_dev)
  PPS_DISPATCH_ODE(s->objective, c.method, L_INIT_ODE);
#undef L_INIT_ODE
  PPS_CUDA(cudaGetLastError());
  return PPS_OK;
}

// Whether an adaptive fit takes eight lanes per particle.  All lanes take every
// step and share the saves, so it pays where the saves are most of the work,
// and the more particles there are to fill the schedulers the more of it they
// have to be.  One thread / eight lanes, us an iteration, the worse of LV and FHN
// at tolerances 1e-3 and 1e-6 (30 first steps on [0, 3]): 301 saves 500 particles
// 110 / 68, 10000 130 / 94, 24000 0.96 of one thread's time; 201 saves 20000
// 0.99; 101 saves 12000 0.99, 16000 1.18; 61 saves 4000 1.00, 10000 1.07; 41 saves
// 500 1.11; 16 saves 24000 1.91.  So up to kLanesAnyDensity particles 64 saves
// suffice; beyond, a first step has to hold particles / 2400 saves, at
// tolerances that keep the steps near the first one's length.
constexpr int kAdaptiveLanes = 8;
constexpr int kLanesMinSaves = 64;
constexpr int64_t kLanesAnyDensity = 4000, kLanesPerDensity = 2400, kLanesMaxN = 24000;

static bool adaptive_lanes(const OdeCfg& c, int64_t n) {
  if (c.method != kOdeTsit5Adaptive || c.nsaves < kLanesMinSaves || n > kLanesMaxN) return false;
  if (n <= kLanesAnyDensity) return true;
  return c.rtol >= 1e-6f && (double)c.dt * kLanesPerDensity >= 0.999 * (double)c.save_dt * (double)n;
}

// Where the pipelined fixed-step form pays.  What it takes off the chain are the
// saves, what it adds is a fixed part (the table in every block, chunks of one
// warp after the other) and, on large swarms, blocks that do not all fit the SMs
// at once: 32 particles need 52 kB and more.  Its time relative to one thread a
// particle, the worse of LV and FHN (steps x saves a step at particles): 30 x 10 at
// 500 / 10000 / 20000 0.48 / 0.57 / 0.78, 4 x 10 at 500 1.16, 12 x 10 0.81, 24 x 3 at
// 10000 0.97, 24 x 2 1.07, 400 x 2 at 10000 (two rounds of blocks) 1.03, 30 x 3 at
// 15000 / 20000 0.98 / 1.09, 400 x 5 at 15000 (four rounds) 1.19, 18 x 10 at
// 24000 / 28000 0.95 / 1.05, 30 x 10 at 28000 0.89.  Each row: up to so many
// particles, from so many saves, saves a step and steps on, and at most so many
// rounds of resident blocks.
struct PipeRow {
  int64_t n;
  int saves, ratio, steps, rounds;
};
constexpr PipeRow kPipeRows[] = {
    {10240, 72, 2, 4, 1}, {10240, 72, 3, 4, 2}, {16000, 90, 3, 4, 2}, {24000, 180, 5, 12, 3}, {28000, 300, 10, 12, 3}};

static bool pipe_pays(const OdeCfg& c, int64_t particles, size_t smem, int sm_count) {
  // blocks of 256 threads with 64 registers: four an SM, fewer by shared memory (228 kB, 1 kB of it a block's own)
  int64_t per_sm = (int64_t)((228u << 10) / (smem + 1024));
  per_sm = per_sm > 4 ? 4 : per_sm;
  const int64_t blocks = (particles + 31) / 32, wave = per_sm * sm_count;
  const int64_t rounds = (blocks + wave - 1) / wave;
  if (rounds > per_sm + 1) return false;  // few blocks an SM hide little: 400 x 10 at 10000 (three rounds of one) 1.08
  for (const PipeRow& r : kPipeRows)
    if (particles <= r.n && c.nsaves >= r.saves && c.nsaves >= (int64_t)r.ratio * c.nsteps && c.nsteps >= r.steps &&
        rounds <= r.rounds)
      return true;
  return false;
}

// Steps per chunk of the pipelined form, 0 where it is not taken: where it does
// not pay, or a solve has more steps, or a chunk more saves, than it holds.  The
// save table's steps are found as the kernel finds them.
static int pipe_chunk(const OdeCfg& c, int64_t particles, int sm_count) {
  if (c.method != kOdeTsit5 || c.nsteps > kPipeMaxSteps || c.nsaves < 2 * (int64_t)c.nsteps) return 0;
  for (int K : {6, 3, 1}) {
    const size_t smem = pipe_smem(c.nsaves, c.nsteps, K);
    if (smem > (size_t)kPipeSmemMax) continue;
    int most = 0, count = 0, at = 0, n = 0;
    for (int m = 1; m < c.nsaves; ++m) {
      const float tm = (float)m * c.save_dt;
      while (n < c.nsteps && tm > (float)(n + 1) * c.dt) ++n;
      if (n / K != at) {
        at = n / K;
        count = 0;
      }
      if (++count > most) most = count;
    }
    if (most <= kPipeMaxSaves) return pipe_pays(c, particles, smem, sm_count) ? K : 0;
  }
  return 0;
}

int launch_sync_step_ode(pps_swarm* s, float c1, float c2) {
  const OdeCfg c = cfg_of(s);
  const int from_pos = (s->flags & PPS_FLAG_GBEST_FROM_POSITION) ? 1 : 0;
  const bool lv = s->objective == kLvFit;
  if (const int K = pipe_chunk(c, s->dv.n, s->sm_count)) {
    const unsigned blocks = (unsigned)((s->dv.n + 31) / 32);
    const size_t smem = pipe_smem(c.nsaves, c.nsteps, K);
    if (lv)
      k_step_tsit5_pipe<kOdeLV><<<blocks, kPipeWarps * 32, smem, s->stream>>>(s->dv, c, s->od.data, s->seed, c1, c2,
                                                                            from_pos, K);
    else
      k_step_tsit5_pipe<kOdeFHN><<<blocks, kPipeWarps * 32, smem, s->stream>>>(s->dv, c, s->od.data, s->seed, c1, c2,
                                                                             from_pos, K);
    PPS_CUDA(cudaGetLastError());
    return PPS_OK;
  }
  if (adaptive_lanes(c, s->dv.n)) {
    constexpr int L = kAdaptiveLanes;
    const unsigned blocks = (unsigned)((s->dv.n * L + kOdeThreads - 1) / kOdeThreads);
    if (lv)
      k_step_tsit5a_lanes<kOdeLV, L><<<blocks, kOdeThreads, ode_dyn_smem(c), s->stream>>>(s->dv, c, s->od.data,
                                                                                         s->seed, c1, c2, from_pos);
    else
      k_step_tsit5a_lanes<kOdeFHN, L><<<blocks, kOdeThreads, ode_dyn_smem(c), s->stream>>>(s->dv, c, s->od.data,
                                                                                          s->seed, c1, c2, from_pos);
    PPS_CUDA(cudaGetLastError());
    return PPS_OK;
  }
  const bool served = !s->owns_memory;  // state carved from a server's arena
  const int ppt = (c.method == kOdeRk4 && (s->dv.npad >= kOdePackedMinParticles || served)) ? 2 : 1;
  const int64_t tile = (int64_t)kOdeThreads * ppt;
  const unsigned blocks = (unsigned)((s->dv.npad + tile - 1) / tile);
  const size_t dsm = ode_dyn_smem(c);
  // the last argument, 1.0f, is the packed losses' run-time one
#define L_STEP_ODE(M, I)                                                                                   \
  do {                                                                                                     \
    if (I == kOdeRk4 && ppt == 2)                                                                          \
      k_sync_step_ode<M, kOdeRk4, 2><<<blocks, kOdeThreads, dsm, s->stream>>>(s->dv, s->op, c, s->od.data, \
                                                                              s->seed, c1, c2, from_pos,  \
                                                                              1.0f);                      \
    else                                                                                                   \
      k_sync_step_ode<M, I, 1><<<blocks, kOdeThreads, dsm, s->stream>>>(s->dv, s->op, c, s->od.data,       \
                                                                        s->seed, c1, c2, from_pos, 1.0f);  \
  } while (0)
  PPS_DISPATCH_ODE(s->objective, c.method, L_STEP_ODE);
#undef L_STEP_ODE
  PPS_CUDA(cudaGetLastError());
  return PPS_OK;
}

template <int MODEL, int METHOD>
__global__ void k_eval_ode(ObjParams op, OdeCfg cfg, const float* __restrict__ data_g, const float* __restrict__ x,
                           int64_t npts, int64_t stride, float* __restrict__ f) {
  ode_smem_fill<METHOD>(cfg, data_g);
  const float* data = ode_observations<METHOD>(cfg);
  const float* tab = ode_smem;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npts) return;
  float p[kOdeMaxDim] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int d = 0; d < kOdeMaxDim; ++d)
    if (d < op.dim) p[d] = x[(int64_t)d * stride + i];
  f[i] = ode_eval<MODEL, METHOD>(p, cfg, data, tab);
}

int launch_eval_ode(const ObjParams& op, const ObjData& od, int objective, const float* x, int64_t npts,
                    int64_t stride, float* f, cudaStream_t stream) {
  const unsigned blocks = (unsigned)((npts + 127) / 128);
  const OdeCfg c = ode_cfg(op, od.ndata);
  const size_t dsm = ode_dyn_smem(c);
  if (c.method == kOdeTsit5) {
    const int rc = ode_set_smem_limit();
    if (rc) return rc;
  }
#define L_EVAL_ODE(M, I) k_eval_ode<M, I><<<blocks, 128, dsm, stream>>>(op, c, od.data, x, npts, stride, f)
  PPS_DISPATCH_ODE(objective, c.method, L_EVAL_ODE);
#undef L_EVAL_ODE
  PPS_CUDA(cudaGetLastError());
  return PPS_OK;
}

}  // namespace pps
