// pps_ode_teams.cu -- a batch of ODE fits (RK4) as units of work placed on the
// SMs by their cost.
//
// A unit is 128 threads' worth of consecutive particles of one fit (two
// particles a thread, their losses packed, or one); a fit's phase is its
// sampling (phase 0) or one synchronous iteration.  One block per SM holds up
// to 8 teams of 128 threads -- one warp on each of the SM's four schedulers --
// and every team owns units for the whole run, chosen on the host so that all
// SMs carry the same cost (longest first onto the least loaded SM).  A fit's
// units lie on many SMs; the team that finishes a phase's last unit gathers
// the global best and opens the next phase.
//
// What bounds such a batch is the FP32 pipe and, with few fits, the Runge-Kutta
// chain of one particle; what it lost before was balance.  With one CTA or
// cluster per fit (k_batch_ode) an SM that held two large FitzHugh-Nagumo CTAs
// took twice as long as one that held one, and every iteration waits for its
// slowest CTA.  Measured, ms a batch of 128 / 32 mixed fits (100 iterations):
// one cluster of up to 4 x 512 threads a fit 98 / 42, of up to 8 x 128 threads
// 58 / 27, units handed out dynamically over the GPU 60 / 21 (the units in
// flight spread unevenly over the SMs), a block's units shared by its teams
// 52 / 18, this form 50 / 17.
//
// The grid is cooperative, so a team may wait for the others of its fit; a
// wait that gives up (`looks` looks) sets the run's error word.  Positions,
// velocities, personal bests and costs pass between SMs through L2: written
// before a device fence and the phase's counter, read past L1.  Each fit's
// result equals its solve alone, bit for bit (Philox by particle, the argmin
// over the whole fit).
#include <algorithm>
#include <cmath>
#include <functional>
#include <new>
#include <queue>
#include <utility>

#include "pps_batch.h"
#include "pps_ode.cuh"
#include "pps_publish.cuh"

namespace pps {

constexpr int kTeam = 128;
constexpr int kMaxTeams = 8;
constexpr size_t kOdeTeamSmem = 200u << 10;  // observations of a block's teams
constexpr unsigned int kOdeTeamLooks = 1u << 30;  // many minutes: phases of very long fits end in seconds

// control words of one fit, zero at launch; the entry behind the last fit holds the run's error word in `phase`
struct OdeCtl {
  unsigned long long inv_key;  // ~ the phase's lowest argmin key so far
  unsigned int phase;          // the phase that is open
  unsigned int done;           // units of it finished
  float w;                     // its inertia
  unsigned int pad[11];
};

struct OdeUnit {
  int fit, unit;
};

__device__ __forceinline__ void team_barrier(int team) {
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kTeam) : "memory");
}

// one phase of one unit by one team
template <int MODEL, bool PACK>
__device__ __forceinline__ void ode_unit(const BatchSwarm& sw, OdeCtl* c, unsigned int phase, int unit,
                                         const OdeCfg& cfg, const float* data, float one, int team, int tid,
                                         unsigned long long* red) {
  const int D = sw.dim;
  const int64_t n = sw.n, ld = sw.ld;
  constexpr int Q = PACK ? 2 : 1;
  const int64_t i0 = (int64_t)unit * (kTeam * Q) + tid;
  const uint32_t k0 = (uint32_t)sw.seed, k1 = (uint32_t)(sw.seed >> 32);
  float x[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
  if (phase == 0) {  // gpu_init_particles!, src/utils.jl:23-84
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int64_t i = i0 + q * kTeam;
      if (i >= n) continue;
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
            xv = __fadd_rn(__fmul_rn(u, __fsub_rn(sw.ub[d], sw.lb[d])), sw.lb[d]);
          }
          x[q][d] = xv;
          const int64_t o = (int64_t)d * ld + i;
          sw.X[o] = xv;
          sw.V[o] = 0.0f;
        }
      }
    }
  } else {  // ode_update_particle_states!, src/ode_pso.jl:1-24
    const uint32_t t = phase - 1u;
    const float w = __ldcg(&c->w);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int64_t i = i0 + q * kTeam;
      if (i >= n) continue;
      const Rand4 r0 = philox4x32_10((uint32_t)i, 0u, t, kTagStep, k0, k1);
      const Rand4 r1 = philox4x32_10((uint32_t)i, 1u, t, kTagStep, k0, k1);
      const float ra[4] = {u01(r0.a), u01(r0.c), u01(r1.a), u01(r1.c)};
      const float rb[4] = {u01(r0.b), u01(r0.d), u01(r1.b), u01(r1.d)};
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        if (d < D) {
          const int64_t o = (int64_t)d * ld + i;
          const float xd = sw.X[o];  // this team's own
          const float v = velocity(xd, sw.V[o], sw.P[o], __ldcg(sw.g + d), w, sw.c1, sw.c2, ra[d], rb[d]);
          const float xn = clamp_lb_ub(__fadd_rn(xd, v), sw.lb[d], sw.ub[d]);
          sw.X[o] = xn;
          sw.V[o] = v;
          x[q][d] = xn;
        }
      }
    }
  }
  float cost[2];
  if constexpr (PACK) {
    const float2 cc = ode_loss2<MODEL>(x[0], x[1], cfg, data, one);  // bit-identical to ode_loss of each
    cost[0] = cc.x;
    cost[1] = cc.y;
  } else {
    cost[0] = ode_loss<MODEL>(x[0], cfg, data);
  }
  unsigned long long best = ~0ull;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int64_t i = i0 + q * kTeam;
    if (i >= n) continue;
    const float pc = phase == 0 ? 0.0f : sw.pcost[i];
    const bool imp = phase == 0 || cost[q] < pc;  // strict <, src/kernels.jl:21-24
    const float npc = imp ? cost[q] : pc;
    sw.cost[i] = cost[q];
    if (imp) {
      sw.pcost[i] = npc;
#pragma unroll
      for (int d = 0; d < 4; ++d)
        if (d < D) sw.P[(int64_t)d * ld + i] = x[q][d];
    }
    const unsigned long long k = argmin_key(npc, (uint32_t)i);
    best = k < best ? k : best;
  }
  // the unit's best into the phase's, and the phase's end
  best = warp_min_u64(best);
  if ((tid & 31) == 0) red[tid >> 5] = best;
  __threadfence();
  team_barrier(team);
  if (tid == 0) {
#pragma unroll
    for (int k = 1; k < kTeam / 32; ++k) best = red[k] < best ? red[k] : best;
    atomicMax(&c->inv_key, ~best);  // inverted, so zeroed memory is "none yet"
    __threadfence();
    const unsigned int units = (unsigned int)((n + kTeam * Q - 1) / (kTeam * Q));
    if (atomicAdd(&c->done, 1u) == units - 1) {
      __threadfence();
      const unsigned long long win = ~atomicExch(&c->inv_key, 0ull);
      const uint32_t gi = (uint32_t)win;
      for (int d = 0; d < D; ++d) sw.g[d] = __ldcg(sw.P + (int64_t)d * ld + gi);
      if ((int)phase == sw.maxiters) {
        sw.result[0] = __ldcg(sw.pcost + gi);
        sw.result[1] = __uint_as_float(gi);
        sw.result[2] = (float)sw.maxiters;
      }
      c->w = phase == 0 ? sw.w : __fmul_rn(__ldcg(&c->w), sw.wdamp);
      c->done = 0u;
      __threadfence();
      atomicExch(&c->phase, phase + 1u);
    }
  }
}

// units: every team's units, team by team (teams of block b: b teams .. b teams
// + teams - 1), offsets[team] .. offsets[team + 1]; next: each unit's next phase
// (zero at launch); looks: kOdeTeamLooks.  `one` is a run-time 1.0f (ode_loss2).
template <bool PACK>
__global__ void __launch_bounds__(kTeam* kMaxTeams, 1)
    k_ode_teams(const BatchSwarm* __restrict__ descs, const OdeUnit* __restrict__ units, const int* __restrict__ offsets,
                unsigned int* next, OdeCtl* ctl, int nfits, int data_floats, unsigned int looks, float one) {
  extern __shared__ float obs[];
  __shared__ unsigned long long red_s[kMaxTeams][kTeam / 32];
  __shared__ int pick_s[kMaxTeams][2];
  const int team = threadIdx.x / kTeam, tid = threadIdx.x - team * kTeam;
  const int gteam = blockIdx.x * (blockDim.x / kTeam) + team;
  const int first = offsets[gteam], count = offsets[gteam + 1] - first;
  float* data = obs + team * data_floats;
  unsigned long long* red = red_s[team];
  int* pick = pick_s[team];
  int loaded = -1, left = count, at = 0;
  while (left > 0) {
    if (tid < 32) {
      // the next of the team's units whose phase is open, from the one after the last
      int got = -1;
      for (unsigned int look = 0; look < looks && got < 0; ++look) {
        for (int base = 0; base < count && got < 0; base += 32) {
          int e = at + base + tid;
          bool ready = false;
          if (base + tid < count) {
            if (e >= count) e -= count;
            const unsigned int p = next[first + e];
            const int fit = units[first + e].fit;
            ready = (int)p <= descs[fit].maxiters &&
                    *reinterpret_cast<volatile unsigned int*>(&ctl[fit].phase) >= p;
          }
          const unsigned int m = __ballot_sync(0xffffffffu, ready);
          if (m) got = __shfl_sync(0xffffffffu, e, __ffs(m) - 1);
        }
        if (got < 0) __nanosleep(100);
      }
      __threadfence();  // the phase's state, written by other teams, is visible from here
      if (tid == 0) {
        pick[0] = got;
        pick[1] = got < 0 ? 0 : (int)next[first + got];
        if (got < 0) atomicExch(&ctl[nfits].phase, 1u);
      }
    }
    team_barrier(team);
    const int e = pick[0];
    const unsigned int phase = (unsigned int)pick[1];
    if (e < 0) return;
    const OdeUnit u = units[first + e];
    const BatchSwarm& sw = descs[u.fit];
    const OdeCfg cfg = ode_cfg(sw.op, sw.ndata);
    if (loaded != u.fit) {
      for (int k = tid; k < 2 * cfg.nsaves; k += kTeam) data[k] = sw.data[k];
      loaded = u.fit;
    }
    team_barrier(team);
    if (sw.objective == kLvFit)
      ode_unit<kOdeLV, PACK>(sw, ctl + u.fit, phase, u.unit, cfg, data, one, team, tid, red);
    else
      ode_unit<kOdeFHN, PACK>(sw, ctl + u.fit, phase, u.unit, cfg, data, one, team, tid, red);
    if (tid == 0) next[first + e] = phase + 1u;
    if ((int)phase == sw.maxiters) --left;
    at = e + 1 == count ? 0 : e + 1;
    team_barrier(team);  // pick, red and next are settled
  }
}

// ---------------------------------------------------------------- host side
// relative cost of one particle's phase: steps of about 30 (LV) or 46 (FHN) FP32 operations
static double phase_cost(const BatchSwarm& d) {
  return (double)ode_cfg(d.op, d.ndata).nsteps * (d.objective == kLvFit ? 30.0 : 46.0);
}

// Units of one particle a thread per SM up to which that form is taken: its
// chain is shorter (LV 85 cycles a step against 119 packed) and an SM with one
// to three such units is bound by the chain (8 fits: 12.3 ms against 14.8
// packed); more fill the pipe, where packing halves the instructions issued
// (700 fits, 30 iterations: 78 ms against 83).
constexpr int kOdeScalarUnits = 3;

// Whether the units beat one CTA or cluster per fit (k_batch_ode) for this batch,
// by estimates of both in us.  A phase of a unit costs 2.3 us of its SM beside its
// steps (state through L2, fence, counters, the next phase's gather) and at least
// 8 from end to end; a trip of a CTA costs 1.0 and 1.2, a cluster's barriers
// 3.5.  So short solves and fits that one CTA holds are better off with the CTA,
// long and large ones with the units, which also fill the SMs evenly.  Measured,
// ms a batch of 50 iterations, clusters / units: 1 fit of 128 particles and 10 steps
// 0.16 / 0.42, 400 steps 1.27 / 1.40; 64 of 1024 and 60 steps 0.62 / 0.86, 400
// steps 2.51 / 2.30; 600 of 4096 and 10 steps 4.4 / 8.5, 60 steps 11.6 / 13.2; 200 of
// 4096 and 150 steps 9.3 / 8.5; 16 of 16384 and 10 steps 1.44 / 1.09; 1 of 65536 and
// 400 steps 43 / 2.6.  Over 219 such batches the estimates' choice is within 5 %
// of the better form in all but a few, and those within 16 %.
static bool units_pay(const std::vector<BatchSwarm>& descs, int64_t total1, int64_t total2, bool pack, int sm_count) {
  double chain_u = 0.0, load_u = 0.0, chain_c = 0.0, load_c = 0.0, most = 0.0, ctas = 0.0;
  for (const auto& d : descs) {
    const LaunchGroup g = batch_group_of(d, 256, 1);
    const double steps = ode_cfg(d.op, d.ndata).nsteps, phases = d.maxiters + 1.0, q = g.T / 128.0;
    const double units = (double)((d.n + kTeam * (pack ? 2 : 1) - 1) / (kTeam * (pack ? 2 : 1)));
    const double trips = (double)((d.n + 2 * (int64_t)g.T * g.C - 1) / (2 * (int64_t)g.T * g.C));
    most = std::max(most, phases);
    chain_u = std::max(chain_u, phases * (pack ? steps * 0.0575 + 9.0 : steps * 0.05));
    load_u += phases * units * (pack ? steps * 0.04 + 2.3 : steps * 0.03);
    chain_c = std::max(chain_c, phases * (trips * (steps * std::max(0.0575, 0.052 * q) + 0.6 + 0.6 * q) +
                                          (g.C > 1 ? 3.5 : 0.0)));
    load_c += phases * g.C * q * trips * (steps * 0.052 + 1.0);
    ctas += g.C * q;
  }
  // whole units and CTAs per SM
  const double sm = sm_count, per_u = (double)(pack ? total2 : total1) / sm, per_c = ctas / sm;
  const double u = pack ? std::max(chain_u, load_u / sm + 3.0 * most)
                        : std::max(chain_u, load_u / sm * std::ceil(per_u) / per_u) + most * (8.0 + per_u);
  const double c = std::max(chain_c, load_c / sm * (per_c > 1.0 ? std::ceil(per_c) / per_c : 1.0));
  return u < c;
}

struct OdeTeams {
  void* mem = nullptr;
  size_t cap = 0;
};
OdeTeams* ode_teams_create() { return new (std::nothrow) OdeTeams(); }
void ode_teams_destroy(OdeTeams* t) {
  if (!t) return;
  if (t->mem) cudaFree(t->mem);
  delete t;
}

size_t ode_teams_bytes(const OdeTeams* t) { return t ? t->cap : 0; }

int ode_teams_launch(OdeTeams* t, cudaStream_t stream, const std::vector<BatchSwarm>& descs, const BatchSwarm* ddescs,
                     int sm_count, bool* taken, unsigned int** error_word, int* threads, int* ppt) {
  *taken = false;
  const int nf = (int)descs.size();
  int64_t total1 = 0, total2 = 0;
  int data_floats = 0;
  for (const auto& d : descs) {
    total1 += (d.n + kTeam - 1) / kTeam;
    total2 += (d.n + 2 * kTeam - 1) / (2 * kTeam);
    data_floats = std::max(data_floats, (int)d.ndata);
  }
  const bool pack = total1 > (int64_t)kOdeScalarUnits * sm_count;
  const int64_t total = pack ? total2 : total1;
  if (total > (1 << 22) || !units_pay(descs, total1, total2, pack, sm_count)) return PPS_OK;
  const int width = kTeam * (pack ? 2 : 1);
  int teams = kMaxTeams;
  while (teams > 1 && sizeof(float) * (size_t)data_floats * teams > kOdeTeamSmem) --teams;
  const int blocks = (int)std::min<int64_t>(sm_count, total);
  teams = (int)std::min<int64_t>(teams, (total + blocks - 1) / blocks);
  // longest fits first, each unit onto the least loaded block, within it onto the least loaded team
  std::vector<int> by(nf);
  for (int k = 0; k < nf; ++k) by[k] = k;
  std::stable_sort(by.begin(), by.end(), [&](int a, int b) {
    return phase_cost(descs[a]) * (descs[a].maxiters + 1) > phase_cost(descs[b]) * (descs[b].maxiters + 1);
  });
  using Load = std::pair<double, int>;
  std::priority_queue<Load, std::vector<Load>, std::greater<Load>> load;
  for (int b = 0; b < blocks; ++b) load.push({0.0, b});
  std::vector<std::vector<OdeUnit>> own((size_t)blocks * teams);
  std::vector<double> team_load((size_t)blocks * teams, 0.0);
  for (int k : by) {
    const double cost = phase_cost(descs[k]) * (descs[k].maxiters + 1);
    const int units = (int)((descs[k].n + width - 1) / width);
    for (int u = 0; u < units; ++u) {
      const Load l = load.top();
      load.pop();
      double* tl = &team_load[(size_t)l.second * teams];
      const int tm = (int)(std::min_element(tl, tl + teams) - tl);
      own[(size_t)l.second * teams + tm].push_back(OdeUnit{k, u});
      tl[tm] += cost;
      load.push({l.first + cost, l.second});
    }
  }
  std::vector<OdeUnit> units;
  std::vector<int> offsets;
  units.reserve((size_t)total);
  for (const auto& o : own) {
    offsets.push_back((int)units.size());
    units.insert(units.end(), o.begin(), o.end());
  }
  offsets.push_back((int)units.size());
  // control words, each unit's next phase, then the tables
  const size_t bctl = sizeof(OdeCtl) * ((size_t)nf + 1);
  const size_t bnext = (sizeof(unsigned int) * (size_t)total + 63) / 64 * 64;
  const size_t bunits = (sizeof(OdeUnit) * (size_t)total + 63) / 64 * 64;
  const size_t need = bctl + bnext + bunits + sizeof(int) * offsets.size();
  if (t->cap < need) {
    if (t->mem) cudaFree(t->mem);
    t->mem = nullptr;
    t->cap = 0;
    PPS_CUDA(cudaMalloc(&t->mem, need));
    t->cap = need;
  }
  char* m = static_cast<char*>(t->mem);
  OdeCtl* ctl = reinterpret_cast<OdeCtl*>(m);
  unsigned int* next = reinterpret_cast<unsigned int*>(m + bctl);
  OdeUnit* du = reinterpret_cast<OdeUnit*>(m + bctl + bnext);
  int* doff = reinterpret_cast<int*>(m + bctl + bnext + bunits);
  PPS_CUDA(cudaMemsetAsync(m, 0, bctl + bnext, stream));
  PPS_CUDA(cudaMemcpyAsync(du, units.data(), sizeof(OdeUnit) * units.size(), cudaMemcpyHostToDevice, stream));
  PPS_CUDA(cudaMemcpyAsync(doff, offsets.data(), sizeof(int) * offsets.size(), cudaMemcpyHostToDevice, stream));
  const size_t smem = sizeof(float) * (size_t)data_floats * teams;
  auto kernel = pack ? k_ode_teams<true> : k_ode_teams<false>;
  // the limit is the process's: a constant, so no other thread lowers it before the launch
  PPS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kOdeTeamSmem));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)(teams * kTeam));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;  // every team resident, or the launch fails
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, ddescs, (const OdeUnit*)du, (const int*)doff, next, ctl, nf,
                                           data_floats, wait_polls(kOdeTeamLooks), 1.0f);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return PPS_OK;
  }
  if (e != cudaSuccess) return cuda_error(e, "cudaLaunchKernelEx(k_ode_teams)");
  *error_word = &ctl[nf].phase;
  *threads = teams * kTeam;
  *ppt = pack ? 2 : 1;
  *taken = true;
  return PPS_OK;
}

}  // namespace pps
