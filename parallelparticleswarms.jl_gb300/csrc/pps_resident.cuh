// pps_resident.cuh -- a whole synchronous run of one swarm inside one launch,
// the swarm's state resident in shared memory.
//
// Same particles, draws, operation order, strict `<`, lowest-index argmin and
// global best as one k_sync_step launch per iteration (src/kernels.jl:127-177,
// src/lowerlevel_solve.jl:1-65), so the state after a run is bit-identical.
//
// What bounds the launch-per-iteration form for a swarm that fits the chip is
// neither bandwidth nor arithmetic but latency: a launch per iteration (about
// 5 us), a thread walking every dim of its particles in sequence with an L2
// round trip per pair, and few warps.  Here:
//   - each block owns `chunk` consecutive particles for the whole run; x, v
//     and pbest live in its shared memory as float2 (dims 2j, 2j+1) at
//     [j][particle], so a pair is one 64-bit access per array;
//   - with fewer particles than threads, `groups` threads share a particle's
//     pairs (SPLIT): they move the coordinates and leave the costly objective
//     terms (the cosines) in shared memory, and one thread per particle then
//     sums the terms in dim order -- the order the streaming accumulators use;
//   - blocks agree on the global best once per iteration through 64-bit words
//     in global memory that carry a 32-bit value and the 32-bit sequence
//     number of the exchange, so a reader that sees the number has the value
//     and no fence or counter stands between them.  Every block posts its own
//     best and that particle's vector together; one warp per block gathers the
//     posts.  Two buffers alternate: a block can only be one exchange ahead of
//     another, since it needs the other's post to go on.  The grid is a
//     cooperative launch, so every block is resident.
// A user objective (kUserObjective, compiled by NVRTC) reads the new position
// back through its accessor, so its state lies at [dim][particle]; the
// read-back is from shared memory instead of L2.
// The wait for a post is bounded: poll_limit polls, and start_limit in the first
// exchange: a cooperative launch promises that the blocks can all be resident,
// not that they start together while other work holds SMs (on a GB300 they did,
// beside a batch of fits and beside an async run of a second).  A wait that gives up sets
// IterState::status bit 3 and the block leaves the loop.
#pragma once
#include "pps_pair.cuh"
#include "pps_publish.cuh"

namespace pps {

struct ResidentArgs {
  int chunk;          // particles of a block
  int blocks;         // blocks that share the swarm
  int groups;         // threads that share a particle's pairs
  int iters;
  uint32_t t0;
  float w0, wdamp;
  float c1s, c2s;     // c1 2^-24, c2 2^-24 (draw24)
  int from_position;
  uint32_t seq0;      // sequence number before the first exchange
  unsigned int start_limit;  // polls of the first exchange
  unsigned int poll_limit;   // polls of the others
  float one;          // 1.0f (pps_pair.cuh)
  unsigned long long* xch;  // exchange of several blocks: two buffers of resident_words
  unsigned int* status;     // a wait that gives up sets kStatusResidentTimeout here
};

// objectives whose terms are computed while moving in the SPLIT form
template <int OBJ>
constexpr bool kTermsMoved = OBJ == kRastrigin || OBJ == kAckley;

// Threads of a block: up to 512, with 128 registers each, while a block has at
// most so many particles, else up to 1024 with 64.  Us an iteration, 512 / 1024:
// Ackley 20011 x 30 3.9 / 4.3, Rastrigin 10007 x 25 2.6 / 3.1, 10000 x 100 5.0 /
// 5.4, Rosenbrock 65536 x 10 3.5 / 3.9, but sphere 100003 x 20 (658 particles a
// block) 5.65 / 5.5, Rastrigin 250000 x 10 (1645) 10.1 / 8.9.
constexpr int kResidentThreads = 512;
constexpr int kResidentMaxThreads = 1024;
// polls of one word before a wait gives up: each is at least an L2 round trip
// (several hundred cycles), so seconds -- between blocks that all run, no
// exchange takes milliseconds
constexpr unsigned int kResidentPollLimit = 1u << 23;
// the first exchange of a launch, and every one of a user objective, which may
// take its own time and unevenly: minutes
constexpr unsigned int kResidentStartLimit = 1u << 29;

// shared memory of a block: bounds (float4 per pair), g (float2 per pair),
// x, v, pbest (float2 per pair and particle), the moved terms, pcost, flags
__host__ __device__ inline size_t resident_smem(int dim, int chunk, bool terms) {
  const size_t np = (size_t)(dim + 1) / 2;
  return 16 * np + 8 * np + 8 * np * (size_t)chunk * (terms ? 4 : 3) + 4 * (size_t)chunk +
         ((size_t)chunk + 15) / 16 * 16;
}

// 64-bit words of an exchange's one buffer: each block's key (two words:
// cost and index), packed so a warp polls whole lines, then the vectors; even,
// so the second buffer's keys too start on the 16 bytes their loads need
__host__ __device__ inline size_t resident_words(int blocks, int dim) {
  return ((size_t)blocks * (2 + (size_t)dim) + 1) / 2 * 2;
}

__device__ __forceinline__ unsigned long long resident_word(uint32_t value, uint32_t seq) {
  return ((unsigned long long)value << 32) | (unsigned long long)seq;
}

// minimum of the warp's 64-bit keys by two 32-bit hardware reductions
__device__ __forceinline__ unsigned long long warp_min_key(unsigned long long k) {
  const uint32_t hi = (uint32_t)(k >> 32), lo = (uint32_t)k;
  const uint32_t m = __reduce_min_sync(0xffffffffu, hi);
  const uint32_t i = __reduce_min_sync(0xffffffffu, hi == m ? lo : 0xffffffffu);
  return ((unsigned long long)m << 32) | (unsigned long long)i;
}

__device__ __forceinline__ void post_word(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// waits for the word of exchange `seq`; false after `limit` polls without it
__device__ __forceinline__ bool await_word(const unsigned long long* p, uint32_t seq, unsigned int limit,
                                           uint32_t* value) {
  for (unsigned int n = 0; n < limit; ++n) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    if ((uint32_t)v == seq) {
      *value = (uint32_t)(v >> 32);
      return true;
    }
  }
  return false;
}
// The lowest of the blocks' keys of exchange `seq`, by one warp: each lane
// polls its up to kPollSlots keys with all loads in flight, so a round costs
// one L2 round trip whatever the number of blocks (one word after the other:
// 4.8 us an iteration at 152 blocks for 2.0).  ok: every key arrived.
constexpr int kPollSlots = 5;  // 160 blocks a round
__device__ __forceinline__ unsigned long long await_keys(const unsigned long long* keys, int blocks, uint32_t seq,
                                                         unsigned int limit, bool* ok) {
  const int lane = threadIdx.x & 31;
  unsigned long long best = ~0ull;
  for (int base = 0; base < blocks; base += 32 * kPollSlots) {
    unsigned int missing = 0u;
#pragma unroll
    for (int i = 0; i < kPollSlots; ++i)
      if (base + 32 * i + lane < blocks) missing |= 1u << i;
    for (unsigned int n = 0; missing && n < limit; ++n) {
      unsigned long long a[kPollSlots], b[kPollSlots];
#pragma unroll
      for (int i = 0; i < kPollSlots; ++i) {
        a[i] = b[i] = 0ull;
        if (missing & (1u << i)) {
          const unsigned long long* p = keys + 2 * (size_t)(base + 32 * i + lane);
          asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(a[i]), "=l"(b[i]) : "l"(p) : "memory");
        }
      }
#pragma unroll
      for (int i = 0; i < kPollSlots; ++i) {
        if ((missing & (1u << i)) && (uint32_t)a[i] == seq && (uint32_t)b[i] == seq) {
          missing &= ~(1u << i);
          const unsigned long long k = (a[i] & 0xffffffff00000000ull) | (b[i] >> 32);
          best = k < best ? k : best;
        }
      }
    }
    if (missing) *ok = false;
  }
  return warp_min_key(best);
}

// the objective of a user source at particle p, its position in rows
#ifdef PPS_USER_SOURCE
__device__ __forceinline__ float user_value(const float2* X, int p, int chunk, int D, const float* prm8,
                                            const ObjParams& op) {
  return pps_objective(pps_point{reinterpret_cast<const float*>(X) + p, chunk}, D, prm8, op.data, op.ndata);
}
#else
__device__ __forceinline__ float user_value(const float2*, int, int, int, const float*, const ObjParams&) {
  return 0.0f;
}
#endif

// a pair's x, v or pbest: float2 at [pair][particle], or ROWS: floats at [dim][particle]
template <bool ROWS>
__device__ __forceinline__ float2 pair_get(const float2* A, int j, int p, int chunk) {
  if constexpr (ROWS) {
    const float* f = reinterpret_cast<const float*>(A) + 2 * j * chunk + p;
    return make_float2(f[0], f[chunk]);
  } else {
    return A[j * chunk + p];
  }
}
template <bool ROWS>
__device__ __forceinline__ void pair_put(float2* A, int j, int p, int chunk, float2 v) {
  if constexpr (ROWS) {
    float* f = reinterpret_cast<float*>(A) + 2 * j * chunk + p;
    f[0] = v.x;
    f[chunk] = v.y;
  } else {
    A[j * chunk + p] = v;
  }
}
template <bool ROWS>
__device__ __forceinline__ float coord_get(const float2* A, int d, int p, int chunk) {
  return reinterpret_cast<const float*>(A)[ROWS ? d * chunk + p : 2 * ((d >> 1) * chunk + p) + (d & 1)];
}

// The run of swarm `s` by the a.blocks blocks that hold it, this one block
// `rank` of them.  s.flag and s.st may be NULL (a batched swarm): no pending
// copies, and the global best goes to `result` (cost, index bits, iterations).
// `prm8`: a user objective's 8 parameters in shared memory.  UNROLL: pairs a
// thread moves between two loop tests.
template <int OBJ, bool SPLIT, bool CONS, int UNROLL = 1>
__device__ __forceinline__ void resident_run(const SwarmDev& s, const ObjParams& op, const PhiloxKeys& keys,
                                             const ResidentArgs& a, int rank, float* result = nullptr,
                                             const float* prm8 = nullptr) {
  static_assert(SPLIT || !(CONS || OBJ == kUserObjective), "constraints and user objectives are summed in a phase of their own");
  constexpr bool ROWS = OBJ == kUserObjective;
  extern __shared__ __align__(16) float rsm[];
  __shared__ unsigned long long red[2][32];
  __shared__ unsigned long long win_s;
  __shared__ int bail;
  const int D = s.dim, np = (D + 1) >> 1, chunk = a.chunk;
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = T >> 5;
  const int64_t first = (int64_t)rank * chunk;
  int cnt = (int)(s.n - first < (int64_t)chunk ? s.n - first : (int64_t)chunk);
  cnt = cnt < 0 ? 0 : cnt;
  constexpr bool TERMS = SPLIT && kTermsMoved<OBJ>;

  float4* bnd = reinterpret_cast<float4*>(rsm);
  float2* g2 = reinterpret_cast<float2*>(bnd + np);
  float2* X = g2 + np;
  float2* V = X + np * chunk;
  float2* P = V + np * chunk;
  float2* TM = P + np * chunk;
  float* pcost = reinterpret_cast<float*>(TM + (TERMS ? np * chunk : 0));
  unsigned char* flag = reinterpret_cast<unsigned char*>(pcost + chunk);
  float* gs = reinterpret_cast<float*>(g2);

  for (int j = tid; j < np; j += T) {
    const bool two = 2 * j + 1 < D;
    g2[j] = make_float2(s.g[2 * j], two ? s.g[2 * j + 1] : 0.0f);
    bnd[j] = make_float4(s.lb[2 * j], s.ub[2 * j], two ? s.lb[2 * j + 1] : 0.0f, two ? s.ub[2 * j + 1] : 0.0f);
  }
  for (int p = tid; p < cnt; p += T) {
    pcost[p] = s.pcost[first + p];
    flag[p] = s.flag ? s.flag[first + p] : 0;
  }
  if (tid == 0) bail = 0;
  // 32 particles of a pair row at a time, dealt to all warps: rows alone leave
  // most warps idle where the dims are few (a 2-D swarm has one row)
  const int tiles = (cnt + 31) >> 5, moves = tiles * np;
  for (int m = warp; m < moves; m += nw) {
    const int j = m / tiles, p = ((m - j * tiles) << 5) + lane;
    if (p < cnt) {
      const int64_t o = (int64_t)(2 * j) * s.npad + first + p;
      const bool two = 2 * j + 1 < D;
      pair_put<ROWS>(X, j, p, chunk, make_float2(s.X[o], two ? s.X[o + s.npad] : 0.0f));
      pair_put<ROWS>(V, j, p, chunk, make_float2(s.V[o], two ? s.V[o + s.npad] : 0.0f));
      pair_put<ROWS>(P, j, p, chunk, make_float2(s.P[o], two ? s.P[o + s.npad] : 0.0f));
    }
  }
  __syncthreads();

  const int G = SPLIT ? a.groups : 1;
  int p0 = tid, g0 = 0;
  if (SPLIT && G > 1) {
    g0 = tid / chunk;
    p0 = g0 < G ? tid - g0 * chunk : cnt;
  }
  const int stride = (SPLIT && G > 1) ? chunk : T;  // one particle per thread when pairs are shared
  using namespace pair32;
  const float2 c1 = dup(a.c1s), c2 = dup(a.c2s), one2 = dup(a.one), mone2 = dup(-a.one);
  float w = a.w0;
  unsigned long long win = ~0ull, prev = ~0ull;
  bool have_prev = false;
  PhiloxParticle pp;
  pp.start((uint32_t)(first + p0), keys);

  for (int it = 0; it < a.iters; ++it) {
    const uint32_t t = a.t0 + (uint32_t)it;
    const int par = it & 1;
    unsigned long long best = ~0ull;
    auto settle = [&](int p, float c) {
      const float pc = pcost[p];
      const bool imp = c < pc;  // strict <, src/kernels.jl:21-24
      const float npc = imp ? c : pc;
      if (imp) pcost[p] = c;
      flag[p] = imp ? 1 : 0;
      if (it == a.iters - 1) s.cost[first + p] = c;
      const unsigned long long k = argmin_key(npc, (uint32_t)(first + p));
      best = k < best ? k : best;
    };
    // ---- move (src/kernels.jl:1-26)
    for (int p = p0; p < cnt; p += stride) {
      if (chunk > T) pp.start((uint32_t)(first + p), keys);  // else the thread's one particle
      PhiloxIteration pi;
      pi.start(pp, t, keys);
      const bool fl = flag[p] != 0;
      const float2 w2 = dup(w);
      Acc<OBJ, true> acc;
#pragma unroll UNROLL
      for (int j = g0; j < np; j += G) {
        const Rand4 r = pi.draw((uint32_t)j, keys);
        const float2 x = pair_get<ROWS>(X, j, p, chunk);
        float2 q = pair_get<ROWS>(P, j, p, chunk);
        if (fl) {  // the personal-best copy deferred from the last iteration
          q = x;
          pair_put<ROWS>(P, j, p, chunk, q);
        }
        const float4 b = bnd[j];
        const float2 v =
            velocity24x2(x, pair_get<ROWS>(V, j, p, chunk), q, g2[j], w2, c1, c2, r, one2, mone2);
        float2 y = add(x, v);
        y.x = clamp_box(y.x, b.x, b.y);
        y.y = clamp_box(y.y, b.z, b.w);
        pair_put<ROWS>(X, j, p, chunk, y);
        pair_put<ROWS>(V, j, p, chunk, v);
        const bool two = 2 * j + 1 < D;
        if constexpr (ROWS) {
        } else if constexpr (TERMS) {
          TM[j * chunk + p] = moved_terms<OBJ>(op, y, mone2);
        } else if constexpr (!SPLIT && kTermsMoved<OBJ>) {
          const float2 m = moved_terms<OBJ>(op, y, mone2);
          add_term<OBJ>(acc, y.x, m.x);
          if (two) add_term<OBJ>(acc, y.y, m.y);
        } else if constexpr (!SPLIT) {
          acc.add(op, 2 * j, y.x);
          if (two) acc.add(op, 2 * j + 1, y.y);
        }
      }
      if constexpr (!SPLIT) settle(p, finalize<OBJ>(op, acc.s1, acc.s2));
    }
    // ---- sum the terms in dim order
    if constexpr (SPLIT) {
      __syncthreads();
      for (int p = tid; p < cnt; p += T) {
        Acc<OBJ, true> acc;
        ConsAcc ca;
        if constexpr (CONS) ca.start(s.cons, s.ncons, D);
        auto add = [&](int d, float x, float term) {
          if constexpr (TERMS) {
            add_term<OBJ>(acc, x, term);
          } else if constexpr (!ROWS) {
            acc.add(op, d, x);
          }
          if constexpr (CONS) ca.add(s.cons, s.ncons, D, d, x);
        };
        const int full = D >> 1;
        if (!ROWS || s.ncons > 0) {  // a user objective reads its position itself
#pragma unroll 4
          for (int j = 0; j < full; ++j) {
            const float2 x = pair_get<ROWS>(X, j, p, chunk), m = TERMS ? TM[j * chunk + p] : x;
            add(2 * j, x.x, m.x);
            add(2 * j + 1, x.y, m.y);
          }
          if (D & 1) {
            const float2 x = pair_get<ROWS>(X, full, p, chunk), m = TERMS ? TM[full * chunk + p] : x;
            add(D - 1, x.x, m.x);
          }
        }
        float c;
        if constexpr (ROWS) {
          c = user_value(X, p, chunk, D, prm8, op);
        } else {
          c = finalize<OBJ>(op, acc.s1, acc.s2);
        }
        if (CONS && (!ROWS || s.ncons > 0)) c = __fadd_rn(c, penalty(ca, s.ncons, __uint2float_rn((uint32_t)(first + p) + 2u)));
        settle(p, c);
      }
    }
    // ---- the block's best
    best = warp_min_key(best);
    if (lane == 0) red[par][warp] = best;
    __syncthreads();
    const unsigned long long mine = warp_min_key(lane < nw ? red[par][lane] : ~0ull);
    const int lp = (int)((int64_t)(uint32_t)mine - first);  // its particle (meaningless when mine is ~0)
    const bool none = mine == ~0ull;
    const float2* src = nullptr;  // its vector: the position if it improved just now, else the personal best
    if (!none) src = (a.from_position || flag[lp]) ? X : P;
    // ---- agree on the global best
    const uint32_t seq = a.seq0 + 1u + (uint32_t)it;
    // (a user objective's limits are the same, and the choice alone took its kernel
    // from 1.97 to 2.32 ms for 200 iterations of 100,003 x 20-D)
    const unsigned int limit = !ROWS && it == 0 ? a.start_limit : a.poll_limit;
    const int nb = a.blocks;
    unsigned long long* kw = a.xch + (size_t)par * resident_words(nb, D);  // keys
    unsigned long long* vw = kw + 2 * (size_t)nb;                          // vectors
    if (nb == 1) {
      win = mine;
      for (int d = tid; d < D; d += T) gs[d] = coord_get<ROWS>(src, d, lp, chunk);
    } else {
      if (tid == 0) {
        post_word(kw + 2 * (size_t)rank, resident_word((uint32_t)(mine >> 32), seq));
        post_word(kw + 2 * (size_t)rank + 1, resident_word((uint32_t)mine, seq));
      }
      if (!none)
        for (int d = tid; d < D; d += T)
          post_word(vw + (size_t)rank * D + d,
                    resident_word(__float_as_uint(coord_get<ROWS>(src, d, lp, chunk)), seq));
    }
    if (nb > 1 && warp == 0) {
      bool ok = true;
      const unsigned long long k = await_keys(kw, nb, seq, limit, &ok);
      ok = __all_sync(0xffffffffu, ok);
      // nobody's personal best beat the last global best: its vector stands
      if (ok && (a.from_position || !have_prev || k != prev)) {
        const unsigned long long* v = vw + (size_t)((int64_t)(uint32_t)k / chunk) * D;
        for (int d = lane; d < D && ok; d += 32) {
          uint32_t bits = 0u;
          ok = await_word(v + d, seq, limit, &bits);
          gs[d] = __uint_as_float(bits);
        }
        ok = __all_sync(0xffffffffu, ok);
      }
      if (lane == 0) {
        win_s = k;
        if (!ok) {
          bail = 1;
          atomicOr(a.status, kStatusResidentTimeout);
        }
      }
    }
    __syncthreads();
    if (nb > 1) {
      win = win_s;
      if (bail) return;
      prev = win;
      have_prev = true;
    }
    w = __fmul_rn(w, a.wdamp);
  }

  // ---- the state back to global memory, personal bests canonical
  for (int m = warp; m < moves; m += nw) {
    const int j = m / tiles, p = ((m - j * tiles) << 5) + lane;
    if (p < cnt) {
      const bool fl = flag[p] != 0;
      const int64_t o = (int64_t)(2 * j) * s.npad + first + p;
      const float2 x = pair_get<ROWS>(X, j, p, chunk), v = pair_get<ROWS>(V, j, p, chunk);
      const float2 q = fl ? x : pair_get<ROWS>(P, j, p, chunk);
      s.X[o] = x.x;
      s.V[o] = v.x;
      s.P[o] = q.x;
      if (2 * j + 1 < D) {
        s.X[o + s.npad] = x.y;
        s.V[o + s.npad] = v.y;
        s.P[o + s.npad] = q.y;
      }
    }
  }
  for (int p = tid; p < cnt; p += T) {
    s.pcost[first + p] = pcost[p];
    if (s.flag) s.flag[first + p] = 0;
  }
  if (rank == 0) {
    for (int d = tid; d < D; d += T) s.g[d] = gs[d];
    if (tid == 0) {
      const uint32_t o = (uint32_t)(win >> 32);
      const float gcost = __uint_as_float((o & 0x80000000u) ? (o ^ 0x80000000u) : ~o);
      if (result) {
        result[0] = gcost;
        result[1] = __uint_as_float((uint32_t)win);
        result[2] = (float)a.iters;
      } else {
        s.st->gcost = gcost;
        s.st->gidx = (uint32_t)win;
        s.st->key = ~0ull;
        s.st->count = 0u;
        s.st->tile_next = 0u;
        s.st->t = a.t0 + (uint32_t)a.iters;
        s.st->w = w;
        s.st->wdamp = a.wdamp;
      }
    }
  }
}

}  // namespace pps
