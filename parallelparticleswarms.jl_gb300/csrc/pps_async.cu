// pps_async.cu -- ParallelPSOKernel(global_update = false): the whole
// iteration loop inside one launch (src/kernels.jl:196-225,
// src/lowerlevel_solve.jl:95-121).
//
// Semantics.  Every particle starts from the swarm's global best and keeps a
// private copy that it replaces whenever its own personal best beats it
// (src/kernels.jl:215-218).  Once that has happened the private copy IS the
// personal best (the personal best only improves from then on and each
// improvement beats the copy again), so the private state is one flag:
// g_private = own ? pbest : g_start.  w is damped in-kernel (:219).  The run
// ends with the argmin over personal bests (src/lowerlevel_solve.jl:119-120).
//
// GB300 design.  A particle's state lives in registers for the whole run: a
// group of `lanes` threads (a power of two dividing 32) shares one particle,
// each lane holding an even-length slice of its dims (x, v, pbest), so
// D = 100 uses 8 lanes of 14 dims and 48 registers of state.  The objective
// is summed per lane in dim order and the lane sums are combined by an XOR
// butterfly, which yields the balanced pairwise tree in dim order on every
// lane (IEEE addition is commutative), so all lanes take the same
// personal-best decision.  Nothing but the start and end state touches HBM.
#include <cmath>

#include <cuda_runtime.h>

#include "pps_internal.h"
#include "pps_pair.cuh"
#include "pps_publish.cuh"

namespace pps {

constexpr int kAsyncThreads = 256;

// The argmin over the personal bests at the end of a run and the publication
// of the final global best by the last block (src/lowerlevel_solve.jl:119-120).
__device__ __forceinline__ void async_publish(const SwarmDev& s, unsigned long long key, uint32_t t_next, float w) {
  // every flag is clear now, so the winner's vector is its personal best
  if (publish_block_min(key, s.st)) finish_iteration(s, false, t_next, w);
}

// The run with every lane's slice exactly S dims (a compile-time count) and
// the general form's arithmetic in fewer instructions: the draws'
// loop-invariant rounds carried (PhiloxIteration), the draws' scale in the
// coefficients (draw24), a pair's update and cosines in packed f32x2
// (pps_pair.cuh), its bounds and g in one 128-bit and one 64-bit load,
// two-instruction clamps.  Dims past the last are moved as zeros inside [0, 0]
// and left out of the sums, so a pair needs no branch and the assembler
// interleaves the pairs' dependent chains.  Every lane's values and sums are
// k_async's, bit for bit.
// What bounds it is instruction issue and the integer and FP32 pipes behind
// it.  200,000 x 100-D Rastrigin, 100 iterations: k_async 7.30 ms (87
// instructions per dim and warp, a branch per pair, 58 % of the issue slots
// used), this form unpacked 4.68 ms, packed 4.51 ms (50 instructions, 62 %).
// Two blocks of 128 registers an SM; asking for one or three: 4.89 / 4.73 ms.
template <int OBJ, int S, int BLOCKS>
__global__ void __launch_bounds__(kAsyncThreads, BLOCKS) k_async_slice(SwarmDev s, ObjParams op, PhiloxKeys keys, int iters,
                                                                float c1s, float c2s, int lanes, float one) {
  extern __shared__ __align__(16) float sm[];
  const int D = s.dim;
  const int np = lanes * (S / 2);
  float4* sb = reinterpret_cast<float4*>(sm);
  float2* sg = reinterpret_cast<float2*>(sb + np);
  IterState* st = s.st;
  const uint32_t t0 = st->t;
  const float wdamp = st->wdamp;
  const float gcost0 = st->gcost;
  for (int j = threadIdx.x; j < np; j += blockDim.x) {
    const bool a = 2 * j < D, b = 2 * j + 1 < D;
    sg[j] = make_float2(a ? s.g[2 * j] : 0.0f, b ? s.g[2 * j + 1] : 0.0f);
    sb[j] = make_float4(a ? s.lb[2 * j] : 0.0f, a ? s.ub[2 * j] : 0.0f, b ? s.lb[2 * j + 1] : 0.0f,
                        b ? s.ub[2 * j + 1] : 0.0f);
  }
  __syncthreads();

  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i = gtid / lanes;
  const int lane = (int)(gtid - i * lanes);
  const bool active = i < s.n;
  const int64_t il = active ? i : (s.n - 1);  // inactive threads mirror a real particle
  const uint32_t gil = (uint32_t)(s.first + il);
  const int d0 = lane * S;
  int cnt = D - d0;
  cnt = cnt < 0 ? 0 : (cnt > S ? S : cnt);
  using namespace pair32;
  float2 x[S / 2], v[S / 2], p[S / 2];
  const bool pending = s.flag[il] != 0;
#pragma unroll
  for (int k = 0; k < S; k += 2) {
    const int64_t o = (int64_t)(d0 + k) * s.npad + il;
    const bool a = k < cnt, b = k + 1 < cnt;
    x[k / 2] = make_float2(a ? s.X[o] : 0.0f, b ? s.X[o + s.npad] : 0.0f);
    v[k / 2] = make_float2(a ? s.V[o] : 0.0f, b ? s.V[o + s.npad] : 0.0f);
    p[k / 2] = pending ? x[k / 2] : make_float2(a ? s.P[o] : 0.0f, b ? s.P[o + s.npad] : 0.0f);
  }
  float pc = s.pcost[il];
  float cc = s.cost[il];
  bool own = false;
  float w = st->w;
  const unsigned full = 0xffffffffu;
  PhiloxParticle pp;
  pp.start(gil, keys);
  sb += d0 / 2;
  sg += d0 / 2;
  const float2 c1 = dup(c1s), c2 = dup(c2s), one2 = dup(one), mone2 = dup(-one);

  for (int it = 0; it < iters; ++it) {
    PhiloxIteration pi;
    pi.start(pp, t0 + (uint32_t)it, keys);
    const float2 w2 = dup(w);
    Acc<OBJ, true> acc;
#pragma unroll
    for (int k = 0; k < S; k += 2) {
      const Rand4 r = pi.draw((uint32_t)((d0 + k) >> 1), keys);
      const float2 g = sg[k / 2];
      const float4 b = sb[k / 2];
      const float2 X = x[k / 2], P = p[k / 2];
      const float2 G = own ? P : g;
      const float2 V = velocity24x2(X, v[k / 2], P, G, w2, c1, c2, r, one2, mone2);
      float2 Y = add(X, V);
      Y.x = clamp_box(Y.x, b.x, b.y);
      Y.y = clamp_box(Y.y, b.z, b.w);
      x[k / 2] = Y;
      v[k / 2] = V;
      // the lane's objective sums in dim order, dims past the last left out
      if constexpr (OBJ == kRastrigin || OBJ == kAckley) {
        const float2 m = moved_terms<OBJ>(op, Y, mone2);
        if (k < cnt) add_term<OBJ>(acc, Y.x, m.x);
        if (k + 1 < cnt) add_term<OBJ>(acc, Y.y, m.y);
      } else {
        Acc<OBJ, true> next = acc;
        next.add(op, k, Y.x);
        if (k < cnt) acc = next;
        next = acc;
        next.add(op, k + 1, Y.y);
        if (k + 1 < cnt) acc = next;
      }
    }
    if constexpr (OBJ == kRosenbrock) {
      // the term of the lane's last dim couples to the next lane's first dim
      const float xn = __shfl_down_sync(full, x[0].x, 1);
      if (cnt > 0 && d0 + cnt < D) acc.add(op, 1, xn);
    }
    float s1 = acc.s1, s2 = acc.s2;
    for (int off = 1; off < lanes; off <<= 1) {
      s1 = __fadd_rn(s1, __shfl_xor_sync(full, s1, off));
      s2 = __fadd_rn(s2, __shfl_xor_sync(full, s2, off));
    }
    cc = finalize<OBJ>(op, s1, s2);
    if (cc < pc) {
      pc = cc;
#pragma unroll
      for (int k = 0; k < S / 2; ++k) p[k] = x[k];
    }
    own = own || (pc < gcost0);
    w = __fmul_rn(w, wdamp);
  }

  if (active) {
#pragma unroll
    for (int k = 0; k < S; k += 2) {
      const int64_t o = (int64_t)(d0 + k) * s.npad + i;
      if (k < cnt) {
        s.X[o] = x[k / 2].x;
        s.V[o] = v[k / 2].x;
        s.P[o] = p[k / 2].x;
      }
      if (k + 1 < cnt) {
        s.X[o + s.npad] = x[k / 2].y;
        s.V[o + s.npad] = v[k / 2].y;
        s.P[o + s.npad] = p[k / 2].y;
      }
    }
    if (lane == 0) {
      s.pcost[i] = pc;
      s.cost[i] = cc;
      s.flag[i] = 0;
    }
  }
  async_publish(s, (active && lane == 0) ? argmin_key(pc, gil) : ~0ull, t0 + (uint32_t)iters, w);
}

// The general form: slices up to S dims, any bounds and coefficients.
template <int OBJ, int S>
__global__ void __launch_bounds__(kAsyncThreads) k_async(SwarmDev s, ObjParams op, PhiloxKeys keys,
                                                          int iters, float c1, float c2, int lanes,
                                                          int slice) {
  extern __shared__ float sm[];
  const int D = s.dim;
  float* sg = sm;
  float* slb = sm + D;
  float* sub = sm + 2 * D;
  IterState* st = s.st;
  const uint32_t t0 = st->t;
  const float w0 = st->w;
  const float wdamp = st->wdamp;
  const float gcost0 = st->gcost;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    sg[d] = s.g[d];
    slb[d] = s.lb[d];
    sub[d] = s.ub[d];
  }
  __syncthreads();

  const int64_t gtid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i = gtid / lanes;
  const int lane = (int)(gtid - i * lanes);
  const bool active = i < s.n;
  const int64_t il = active ? i : (s.n - 1);  // inactive threads mirror a real particle
  const uint32_t gil = (uint32_t)(s.first + il);  // its index in the whole swarm (a shard's is offset)
  const int d0 = lane * slice;
  int cnt = D - d0;
  cnt = cnt < 0 ? 0 : (cnt > slice ? slice : cnt);
  float x[S], v[S], p[S];
  const bool pending = s.flag[il] != 0;
#pragma unroll
  for (int k = 0; k < S; ++k) {
    if (k < cnt) {
      const int64_t o = (int64_t)(d0 + k) * s.npad + il;
      x[k] = s.X[o];
      v[k] = s.V[o];
      p[k] = pending ? x[k] : s.P[o];
    }
  }
  float pc = s.pcost[il];
  float cc = s.cost[il];
  bool own = false;
  float w = w0;
  const unsigned full = 0xffffffffu;

  for (int it = 0; it < iters; ++it) {
    const uint32_t t = t0 + (uint32_t)it;
#pragma unroll
    for (int k = 0; k < S; k += 2) {
      if (k < cnt) {
        const Rand4 r = philox4x32_10(gil, (uint32_t)((d0 + k) >> 1), t, kTagStep, keys);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int kk = k + h;
          if (kk < cnt) {
            const int d = d0 + kk;
            const float gd = own ? p[kk] : sg[d];
            const float r1 = u01(h ? r.c : r.a), r2 = u01(h ? r.d : r.b);
            v[kk] = velocity(x[kk], v[kk], p[kk], gd, w, c1, c2, r1, r2);
            x[kk] = clamp_lb_ub(__fadd_rn(x[kk], v[kk]), slb[d], sub[d]);
          }
        }
      }
    }
    // per-lane objective sums in dim order
    Acc<OBJ> acc;
#pragma unroll
    for (int k = 0; k < S; ++k)
      if (k < cnt) acc.add(op, k, x[k]);
    if constexpr (OBJ == kRosenbrock) {
      // the term of the lane's last dim couples to the next lane's first dim
      const float xn = __shfl_down_sync(full, x[0], 1);
      if (cnt > 0 && d0 + cnt < D) acc.add(op, 1, xn);
    }
    float s1 = acc.s1, s2 = acc.s2;
    for (int off = 1; off < lanes; off <<= 1) {
      s1 = __fadd_rn(s1, __shfl_xor_sync(full, s1, off));
      s2 = __fadd_rn(s2, __shfl_xor_sync(full, s2, off));
    }
    cc = finalize<OBJ>(op, s1, s2);
    if (cc < pc) {
      pc = cc;
#pragma unroll
      for (int k = 0; k < S; ++k)
        if (k < cnt) p[k] = x[k];
    }
    own = own || (pc < gcost0);
    w = __fmul_rn(w, wdamp);
  }

  if (active) {
#pragma unroll
    for (int k = 0; k < S; ++k) {
      if (k < cnt) {
        const int64_t o = (int64_t)(d0 + k) * s.npad + i;
        s.X[o] = x[k];
        s.V[o] = v[k];
        s.P[o] = p[k];
      }
    }
    if (lane == 0) {
      s.pcost[i] = pc;
      s.cost[i] = cc;
      s.flag[i] = 0;
    }
  }
  async_publish(s, (active && lane == 0) ? argmin_key(pc, gil) : ~0ull, t0 + (uint32_t)iters, w);
}

int async_lanes(int dim, int* slice) {
  int lanes = 1;
  if (dim > 16) {
    const int need = (dim + 15) / 16;
    while (lanes < need) lanes <<= 1;
    if (lanes > 32) lanes = 32;
  }
  int S = (dim + lanes - 1) / lanes;
  S += S & 1;
  if (slice) *slice = S;
  return lanes;
}

// whether the shorter arithmetic of the pair forms is exact for this run: the
// coefficients scale (coef_scales), no bound is a negative zero (clamp_box) and
// the cosines' arguments stay below cos2pi_box's limit
bool box_cosines(int objective, const ObjParams& op, int dim, const float* lb, const float* ub) {
  if (objective != kRastrigin && objective != kAckley) return true;
  const float k = objective == kAckley ? fabsf(op.np > 2 ? op.p[2] : 1.0f) : 1.0f;
  for (int d = 0; d < dim; ++d) {
    const float m = fmaxf(fabsf(lb[d]), fabsf(ub[d]));
    if (!(m < kCosBoxLimit) || !(m * k < kCosBoxLimit)) return false;
  }
  return true;
}
bool pair_form(int objective, const ObjParams& op, int dim, const float* lb, const float* ub, float c1, float c2) {
  if (!coef_scales(c1) || !coef_scales(c2)) return false;
  for (int d = 0; d < dim; ++d)
    if ((lb[d] == 0.0f && std::signbit(lb[d])) || (ub[d] == 0.0f && std::signbit(ub[d]))) return false;
  return box_cosines(objective, op, dim, lb, ub);
}
bool pair_form(const pps_swarm* s, float c1, float c2) {
  return pair_form(s->objective, s->op, s->dv.dim, s->host_lb, s->host_ub, c1, c2);
}

template <int OBJ>
static int launch_async_obj(pps_swarm* s, int iters, float c1, float c2, int lanes, int slice) {
  const int64_t threads = s->dv.npad * lanes;
  const int64_t blocks = (threads + kAsyncThreads - 1) / kAsyncThreads;
  const PhiloxKeys keys = philox_round_keys(s->seed);
  const size_t smem = 3 * sizeof(float) * (size_t)lanes * slice;
  const float c1s = c1 * 0x1p-24f, c2s = c2 * 0x1p-24f;
  // Blocks an SM (registers a thread): two, and in short runs three or four for
  // slices of 4 to 8 where the grid has more than one round of two (two rounds for
  // slices of 4).  There the loads of the state count, which more warps overlap: 10^6
  // x 8-D sphere, us a run of 1 / 5 iterations, two blocks 115 / 156, three 90 / 122,
  // k_async 91 / 132.  From ten to twenty iterations on the registers count for more:
  // 300 iterations of 160,000 to 10^6 particles take 1 to 6 % longer with three or four.
  // Up to three iterations take k_async where the grid is that long and where a slice has at
  // most four dims: 10^6 x 5-D, one iteration 62, three blocks 67; 10,000 x 3-D 24 and 26.
  const int64_t round = 2 * (int64_t)s->sm_count;
  const bool many = iters <= 8 && blocks > (slice == 4 ? 2 : 1) * round;
#define L_SLICE_B(S, B) \
  k_async_slice<OBJ, S, B><<<(unsigned)blocks, kAsyncThreads, smem, s->stream>>>(s->dv, s->op, keys, iters, c1s, c2s, lanes, 1.0f)
#define L_SLICE(S)                                      \
  case S:                                               \
    if constexpr (S >= 4 && S <= 8) {                   \
      if (many) {                                       \
        L_SLICE_B(S, S == 4 ? 4 : 3);                   \
        break;                                          \
      }                                                 \
    }                                                   \
    L_SLICE_B(S, 2);                                    \
    break
  const bool brief = iters <= 3 && (slice <= 4 || (slice <= 8 && blocks > 2 * round));
  if (slice <= 16 && !brief && pair_form(s, c1, c2)) {
    if constexpr (OBJ >= kBeale) {  // closed forms of at most two dims
      switch (slice) { L_SLICE(2); }
    } else {
      switch (slice) {
        L_SLICE(2);
        L_SLICE(4);
        L_SLICE(6);
        L_SLICE(8);
        L_SLICE(10);
        L_SLICE(12);
        L_SLICE(14);
        L_SLICE(16);
      }
    }
  } else {
    // the smallest form that holds the slice: its loops are unrolled to S
    // (unbounded Rastrigin, 100,000 particles, 50 iterations, us at 4 / 16 / 100
    // dims: all in the form for 32 343 / 628 / 4211, in these 96 / 355 / 1997)
    const size_t general = 3 * sizeof(float) * (size_t)s->dv.dim;
#define L_GENERAL(S) \
  k_async<OBJ, S><<<(unsigned)blocks, kAsyncThreads, general, s->stream>>>(s->dv, s->op, keys, iters, c1, c2, lanes, slice)
    if constexpr (OBJ >= kBeale) {
      L_GENERAL(4);
    } else {
      if (slice <= 4) L_GENERAL(4);
      else if (slice <= 8) L_GENERAL(8);
      else if (slice <= 16) L_GENERAL(16);
      else L_GENERAL(32);
    }
  }
#undef L_SLICE
#undef L_SLICE_B
#undef L_GENERAL
  PPS_CUDA(cudaGetLastError());
  return PPS_OK;
}

int launch_async(pps_swarm* s, int iters, float c1, float c2, int* lanes_out) {
  int slice = 0;
  const int lanes = async_lanes(s->dv.dim, &slice);
  if (slice > 32) return set_error(PPS_ENOTSUP, "async run supports dim <= 1024 (got %d)", s->dv.dim);
  if (lanes_out) *lanes_out = lanes;
  switch (s->objective) {
    case kSphere: return launch_async_obj<kSphere>(s, iters, c1, c2, lanes, slice);
    case kRosenbrock: return launch_async_obj<kRosenbrock>(s, iters, c1, c2, lanes, slice);
    case kRastrigin: return launch_async_obj<kRastrigin>(s, iters, c1, c2, lanes, slice);
    case kAckley: return launch_async_obj<kAckley>(s, iters, c1, c2, lanes, slice);
    case kBeale: return launch_async_obj<kBeale>(s, iters, c1, c2, lanes, slice);
    case kBooth: return launch_async_obj<kBooth>(s, iters, c1, c2, lanes, slice);
    case kHimmelblau: return launch_async_obj<kHimmelblau>(s, iters, c1, c2, lanes, slice);
    case kQuadratic: return launch_async_obj<kQuadratic>(s, iters, c1, c2, lanes, slice);
    case kBoundaryQuadratic: return launch_async_obj<kBoundaryQuadratic>(s, iters, c1, c2, lanes, slice);
    case kShiftedSphere: return launch_async_obj<kShiftedSphere>(s, iters, c1, c2, lanes, slice);
    default: return set_error(PPS_ENOTSUP, "objective %d has no async kernel", s->objective);
  }
}

}  // namespace pps
