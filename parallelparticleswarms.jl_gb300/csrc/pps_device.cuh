// pps_device.cuh -- device-side primitives shared by every PSO kernel.
//
// Random stream: Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) with the
// counter layout
//   update draws: ctr = {particle, dim/2, iteration, PPS_TAG_STEP}, key = seed
//                 out = {r1[2j], r2[2j], r1[2j+1], r2[2j+1]}
//   init draws:   ctr = {particle, dim/4, 0, PPS_TAG_INIT},   out[k] -> dim 4j+k
// so a draw depends only on (seed, particle, dim, iteration) -- never on the
// block, slot or launch that computes it.  The reference draws r1, r2 with
// rand() (src/kernels.jl:3,8) and positions with rand() (src/utils.jl:1-5).
//
// Arithmetic: the library is compiled with -fmad=false, so every + and * is a
// single IEEE binary32 operation in the order written; fused multiply-adds are
// spelled __fmaf_rn where the algorithm uses them.  cos(2 pi x), sin(2 pi x)
// and exp(x) are this project's own: exact reduction y = 2x = n + r (|r|<=1/2)
// followed by a minimax polynomial (cos, below) or the Taylor series of
// sin(pi r) / cos(pi r) with coefficients pi^k/k! rounded to binary32 (sin),
// and Cody-Waite reduction by ln 2 followed by the Taylor series of exp.
// Accuracy: <= 1.66 ulp (cos), <= 1.7 ulp (sin), <= 0.9 ulp (exp).
#pragma once
#ifdef __CUDACC_RTC__
// NVRTC (the kernels of a user objective) has no standard headers
typedef unsigned char uint8_t;
typedef unsigned int uint32_t;
typedef unsigned long long uint64_t;
typedef long long int64_t;
#else
#include <cstdint>

#include <cuda_runtime.h>
#endif

namespace pps {

constexpr uint32_t kTagInit = 0x494E4954u;  // "INIT"
constexpr uint32_t kTagStep = 0x50534F31u;  // "PSO1"
constexpr uint32_t kTagLhs = 0x4C485331u;   // "LHS1"

// samplers (the values of include/pps.h's PPS_SAMPLER_*)
constexpr int kSamplerUniform = 1;
constexpr int kSamplerUnbounded = 2;
constexpr int kSamplerLhs = 3;

enum Objective : int {
  kSphere = 0,
  kRosenbrock = 1,
  kRastrigin = 2,
  kAckley = 3,
  kLvFit = 4,
  kFhnFit = 5,
  kMlp = 6,
  kShiftedSphere = 7,
  kBeale = 16,
  kBooth = 17,
  kHimmelblau = 18,
  kQuadratic = 19,
  kBoundaryQuadratic = 20,
};

// a user objective (compiled by NVRTC with its source): f and, when the source
// defines PPS_HAS_GRADIENT, pps_gradient(x, dim, p, data, ndata, g) returning f
constexpr int kUserObjective = 255;

// ---------------------------------------------------------------- Philox
struct Rand4 {
  uint32_t a, b, c, d;
};

__device__ __forceinline__ Rand4 philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                               uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * (uint64_t)c0;
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * (uint64_t)c2;
    const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0;
    const uint32_t n1 = (uint32_t)p1;
    const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1;
    const uint32_t n3 = (uint32_t)p0;
    c0 = n0;
    c1 = n1;
    c2 = n2;
    c3 = n3;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return Rand4{c0, c1, c2, c3};
}

// The round keys of a Philox4x32-10 key (k0 + r W0, k1 + r W1, r = 0..9),
// computed once on the host: a kernel that takes them by value reads them
// from its parameter bank instead of stepping the key schedule in every call.
struct PhiloxKeys {
  uint32_t k[20];
};
#ifndef __CUDACC_RTC__
inline PhiloxKeys philox_round_keys(uint64_t seed) {
  PhiloxKeys K;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  for (int r = 0; r < 10; ++r) {
    K.k[2 * r] = k0;
    K.k[2 * r + 1] = k1;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return K;
}
#endif
__device__ __forceinline__ Rand4 philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                               const PhiloxKeys& K) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * (uint64_t)c0;
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * (uint64_t)c2;
    const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ K.k[2 * r];
    const uint32_t n1 = (uint32_t)p1;
    const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c3 ^ K.k[2 * r + 1];
    const uint32_t n3 = (uint32_t)p0;
    c0 = n0;
    c1 = n1;
    c2 = n2;
    c3 = n3;
  }
  return Rand4{c0, c1, c2, c3};
}

// The update draws of one particle with everything that does not depend on
// the dim pair computed ahead: in the first three rounds of counter
// {particle, j, t, tag} five of the six products depend on the particle or
// on the particle and the iteration alone, so a loop over pairs (and over
// iterations) carries them instead of redoing them: 16 wide multiplications a
// call for 20.  The words are those of philox4x32_10(particle, j, t, kTagStep, K).
struct PhiloxParticle {
  uint32_t a1, b1, l0;
  __device__ __forceinline__ void start(uint32_t particle, const PhiloxKeys& K) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * (uint64_t)particle;
    const uint64_t q1 = (uint64_t)0xCD9E8D57u * (uint64_t)((uint32_t)(p0 >> 32) ^ kTagStep ^ K.k[1]);
    a1 = (uint32_t)(q1 >> 32) ^ K.k[2];
    b1 = (uint32_t)q1 ^ K.k[4];
    l0 = (uint32_t)p0 ^ K.k[3];
  }
};
struct PhiloxIteration {
  uint32_t h1, sh, sl, l0, b1;
  __device__ __forceinline__ void start(const PhiloxParticle& P, uint32_t t, const PhiloxKeys& K) {
    const uint64_t p1 = (uint64_t)0xCD9E8D57u * (uint64_t)t;
    const uint64_t s0 = (uint64_t)0xD2511F53u * (uint64_t)(P.a1 ^ (uint32_t)p1);
    h1 = (uint32_t)(p1 >> 32) ^ K.k[0];
    sh = (uint32_t)(s0 >> 32) ^ K.k[5];
    sl = (uint32_t)s0;
    l0 = P.l0;
    b1 = P.b1;
  }
  __device__ __forceinline__ Rand4 draw(uint32_t j, const PhiloxKeys& K) const {
    const uint64_t q0 = (uint64_t)0xD2511F53u * (uint64_t)(h1 ^ j);
    const uint64_t s1 = (uint64_t)0xCD9E8D57u * (uint64_t)((uint32_t)(q0 >> 32) ^ l0);
    uint32_t c0 = (uint32_t)(s1 >> 32) ^ b1, c1 = (uint32_t)s1, c2 = sh ^ (uint32_t)q0, c3 = sl;
#pragma unroll
    for (int r = 3; r < 10; ++r) {
      const uint64_t p0 = (uint64_t)0xD2511F53u * (uint64_t)c0;
      const uint64_t p1 = (uint64_t)0xCD9E8D57u * (uint64_t)c2;
      c0 = (uint32_t)(p1 >> 32) ^ c1 ^ K.k[2 * r];
      c1 = (uint32_t)p1;
      c2 = (uint32_t)(p0 >> 32) ^ c3 ^ K.k[2 * r + 1];
      c3 = (uint32_t)p0;
    }
    return Rand4{c0, c1, c2, c3};
  }
};

__device__ __forceinline__ float u01(uint32_t bits) {
  return __fmul_rn(__uint2float_rn(bits >> 8), 0x1p-24f);
}

// ---------------------------------------------------------------- Latin hypercube
// Latin hypercube sampling (McKay, Beckman & Conover, Technometrics 1979),
// the reference's init(...; sampler = LatinHypercubeSample()) (QMC samples
// read by the init kernel, src/init.jl:15-34, src/utils.jl:86-112): in each
// dim the n strata [k/n, (k+1)/n) are dealt to the particles by a random
// permutation and each particle draws uniformly inside its stratum.  The
// permutation of dim d is computed per particle, with no sort: a 4-round
// balanced Feistel network on 2h-bit values (2^(2h) >= n) whose round keys
// are one Philox draw of (d, seed), restricted to [0, n) by cycle-walking
// (Black & Rogaway, "Ciphers with arbitrary finite domains", CT-RSA 2002).
// The walk from i < n returns below n within the cycle through i, so it ends
// after at most 2^(2h) - n + 1 rounds (fewer than 4 expected).
__device__ __forceinline__ uint32_t lhs_round(uint32_t r, uint32_t key) {
  uint32_t x = r ^ key;
  x *= 0xD2511F53u;
  x ^= x >> 15;
  x *= 0xCD9E8D57u;
  x ^= x >> 13;
  return x;
}
__device__ __forceinline__ uint32_t lhs_feistel(uint32_t v, int h, const Rand4& key) {
  const uint32_t mask = (1u << h) - 1u;
  uint32_t L = v >> h, R = v & mask;
  const uint32_t k[4] = {key.a, key.b, key.c, key.d};
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint32_t nl = R;
    R = L ^ (lhs_round(R, k[r]) & mask);
    L = nl;
  }
  return (L << h) | R;
}
// the stratum of particle i (< n) in dim d
__device__ __forceinline__ uint32_t lhs_stratum(uint32_t i, uint32_t n, uint32_t d, uint32_t k0, uint32_t k1) {
  int bits = 0;
  while (bits < 32 && (1ull << bits) < (unsigned long long)n) ++bits;
  const int h = bits < 2 ? 1 : (bits + 1) / 2;
  const Rand4 key = philox4x32_10(d, 0u, 0u, kTagLhs, k0, k1);
  const unsigned long long domain = 1ull << (2 * h);
  uint32_t v = i;
  for (unsigned long long it = 0; it < domain; ++it) {
    v = lhs_feistel(v, h, key);
    if (v < n) return v;
  }
  return i;  // not reached (see above)
}
// x = ((stratum + u) / n) (ub - lb) + lb
__device__ __forceinline__ float lhs_position(uint32_t i, uint32_t n, uint32_t d, float u, float lo, float hi,
                                              uint32_t k0, uint32_t k1) {
  const float t = __fdiv_rn(__fadd_rn(__uint2float_rn(lhs_stratum(i, n, d, k0, k1)), u), __uint2float_rn(n));
  return __fadd_rn(__fmul_rn(t, __fsub_rn(hi, lo)), lo);
}

// ---------------------------------------------------------------- math
__device__ __forceinline__ float cospi_poly(float a) {  // cos(pi a), 0 <= a <= 1/4
  const float z = __fmul_rn(a, a);
  float p = 0x1.f9d38ap-10f;             //  pi^12/12!
  p = __fmaf_rn(p, z, -0x1.a6d1f2p-6f);  // -pi^10/10!
  p = __fmaf_rn(p, z, 0x1.e1f506p-3f);   //  pi^8/8!
  p = __fmaf_rn(p, z, -0x1.55d3c8p+0f);  // -pi^6/6!
  p = __fmaf_rn(p, z, 0x1.03c1f0p+2f);   //  pi^4/4!
  p = __fmaf_rn(p, z, -0x1.3bd3ccp+2f);  // -pi^2/2!
  return __fmaf_rn(p, z, 1.0f);
}
__device__ __forceinline__ float sinpi_poly(float b) {  // sin(pi b), 0 <= b <= 1/4
  const float z = __fmul_rn(b, b);
  float p = -0x1.e30750p-8f;             // -pi^11/11!
  p = __fmaf_rn(p, z, 0x1.507834p-4f);   //  pi^9/9!
  p = __fmaf_rn(p, z, -0x1.32d2ccp-1f);  // -pi^7/7!
  p = __fmaf_rn(p, z, 0x1.466bc6p+1f);   //  pi^5/5!
  p = __fmaf_rn(p, z, -0x1.4abbcep+2f);  // -pi^3/3!
  p = __fmaf_rn(p, z, 0x1.921fb6p+1f);   //  pi
  return __fmul_rn(p, b);
}
__device__ __forceinline__ bool is_odd_integer(float n) {
  return __fmul_rn(rintf(__fmul_rn(n, 0.5f)), 2.0f) != n;
}
// cos(2 pi x): y = 2x = n + r with n = rint(y), |r| <= 1/2, and
// cos(pi y) = (-1)^n cos(pi a), a = |r|, with
//   cos(pi a) = (1/4 - a^2) (4 + z P(z)),  z = a^2,
// P a degree-3 minimax fit of (cos(pi sqrt z) / (1/4 - z) - 4) / z on
// [0, 1/4] (relative error 0.07 ulp; oracle/cospi_coefficients.py).  The
// factor 1/4 - a^2 is one fused multiply-add, so the zero at a = 1/2 keeps
// its relative accuracy, and 4 (1/4 - a^2) is exact.  Max error 1.66 ulp
// over every binary32 a in [0, 1/2].  (Taking n and its parity from the
// 1.5 * 2^23 round trip instead of rint measured slower: 0.3917 vs 0.3872 ms
// per sync step, 2.80e9 vs 2.99e9 async particle-iterations/s.)
constexpr float kCosP0 = -0x1.de9e60p+1f, kCosP1 = 0x1.472a8ap+0f, kCosP2 = -0x1.d47d94p-3f,
                kCosP3 = 0x1.8c391ap-6f;
__device__ __forceinline__ float cos2pi(float x) {
  const float y = __fadd_rn(x, x);
  const float n = rintf(y);
  const uint32_t odd = is_odd_integer(n) ? 1u : 0u;
  const float a = fabsf(__fsub_rn(y, n));
  const float z = __fmul_rn(a, a);
  float q = __fmaf_rn(kCosP3, z, kCosP2);
  q = __fmaf_rn(q, z, kCosP1);
  q = __fmaf_rn(q, z, kCosP0);
  const float p = __fmaf_rn(-a, a, 0.25f);
  const float c = __fmaf_rn(p, __fmul_rn(z, q), __fmul_rn(4.0f, p));
  return __uint_as_float(__float_as_uint(c) ^ (odd << 31));
}
// cos2pi for |x| < 2^126, the same value bit for bit in 14 instructions and one
// conversion for 18 and two: x = m + f with m = rint(x) and f exact, h =
// min(|f|, 1/2 - |f|) = a / 2 (exact: 1/2 - |f| is only taken where |f| >=
// 1/4), and cos(2 pi x) is negative exactly where |f| > 1/4 (n odd above).
// The polynomial is cos2pi's with z = 4 h^2 and its powers of two moved into
// the constants and the last step, which changes no rounding: 4p = 1 - 16 h^2
// is one fused multiply-add, c = 4p (z q / 4) + 4p.  From 2^127 on cos2pi's 2x
// overflows and it returns NaN, which this form would not: the limit stays below.
constexpr float kCosBoxLimit = 0x1p+126f;
__device__ __forceinline__ float cos2pi_box(float x) {
  const float f = fabsf(__fsub_rn(x, rintf(x)));
  const float h = fminf(f, __fsub_rn(0.5f, f));
  const float z = __fmul_rn(h, h);
  float q = __fmaf_rn(64.0f * kCosP3, z, 16.0f * kCosP2);
  q = __fmaf_rn(q, z, 4.0f * kCosP1);
  q = __fmaf_rn(q, z, kCosP0);
  const float p4 = __fmaf_rn(__fmul_rn(-16.0f, h), h, 1.0f);
  const float c = __fmaf_rn(p4, __fmul_rn(z, q), p4);
  return __uint_as_float((__float_as_uint(c) & 0x7fffffffu) | (__float_as_uint(__fsub_rn(0.25f, f)) & 0x80000000u));
}
__device__ __forceinline__ float sin2pi(float x) {
  const float y = __fadd_rn(x, x);
  const float n = rintf(y);
  const float r = __fsub_rn(y, n);
  const float a = fabsf(r);
  float s = (a <= 0.25f) ? sinpi_poly(a) : cospi_poly(__fsub_rn(0.5f, a));
  if (r < 0.0f) s = -s;
  return is_odd_integer(n) ? -s : s;
}
__device__ __forceinline__ float exp_f(float x) {
  if (x != x) return x;
  if (x > 88.72283f) return __int_as_float(0x7f800000);
  if (x < -87.33654f) return 0.0f;
  const float k = rintf(__fmul_rn(x, 0x1.715476p+0f));
  float r = __fmaf_rn(-k, 0x1.62e430p-1f, x);
  r = __fmaf_rn(-k, -0x1.05c610p-29f, r);
  float p = 0x1.a01a02p-13f;
  p = __fmaf_rn(p, r, 0x1.6c16c2p-10f);
  p = __fmaf_rn(p, r, 0x1.111112p-7f);
  p = __fmaf_rn(p, r, 0x1.555556p-5f);
  p = __fmaf_rn(p, r, 0x1.555556p-3f);
  p = __fmaf_rn(p, r, 0.5f);
  p = __fmaf_rn(p, r, 1.0f);
  p = __fmaf_rn(p, r, 1.0f);
  const int ki = (int)k;
  if (ki > 127) return __fmul_rn(__fmul_rn(p, __int_as_float(0x7f000000)), 2.0f);
  return __fmul_rn(p, __int_as_float((ki + 127) << 23));
}

// ln(x) for the adaptive integrators' step-size controller, this project's own
// (identical bits in the oracle's orc_log): x = 2^e m with m in (sqrt(1/2),
// sqrt(2)], ln m = 2 atanh(s) = 2 (s + s^3/3 + ... + s^9/9), s = (m-1)/(m+1)
// (|s| <= 0.1716, the series' remainder below 2^-28), plus e ln 2 with the
// Cody-Waite split of exp_f.  x <= 0 or NaN gives NaN, 0 -inf, +inf +inf;
// subnormal x is scaled into the normal range first.
__device__ __forceinline__ float log_f(float x) {
  if (!(x > 0.0f)) return (x == 0.0f) ? __int_as_float(0xff800000) : __int_as_float(0x7fc00000);
  if (x == __int_as_float(0x7f800000)) return x;
  int e = 0;
  if (x < 0x1p-126f) {
    x = __fmul_rn(x, 0x1p+24f);
    e = -24;
  }
  const int b = __float_as_int(x);
  e += (b >> 23) - 127;
  float m = __int_as_float((b & 0x007fffff) | 0x3f800000);
  if (m > 0x1.6a09e6p+0f) {
    m = __fmul_rn(m, 0.5f);
    e += 1;
  }
  const float sv = __fdiv_rn(__fsub_rn(m, 1.0f), __fadd_rn(m, 1.0f));
  const float z = __fmul_rn(sv, sv);
  float q = 0x1.c71c72p-3f;          // 2/9
  q = __fmaf_rn(q, z, 0x1.249250p-2f);  // 2/7
  q = __fmaf_rn(q, z, 0x1.99999ap-2f);  // 2/5
  q = __fmaf_rn(q, z, 0x1.555556p-1f);  // 2/3
  q = __fmaf_rn(q, z, 2.0f);
  const float lm = __fmul_rn(sv, q);
  const float ef = __int2float_rn(e);
  return __fmaf_rn(ef, 0x1.62e430p-1f, __fmaf_rn(ef, -0x1.05c610p-29f, lm));
}

// ---------------------------------------------------------------- constraints
// calc_penalty (src/utils.jl:320-372) for the registered constraint form
// g_k(x) = c_k + sum_i a_ki x_i + b_ki x_i^2 (rows of `cons`: c_k, a_k[dim],
// b_k[dim]).  ConsAcc streams the dims like Acc; penalty() turns the k
// constraint values into h(iter) (sum theta(q) + sum theta(q) q^gamma(q)),
// q = max.(g, 0), h = sqrt, theta_default / gamma_default (:320-338).  The
// reference compares a Float32 with the Float64 literals 0.001 and 0.1; no
// binary32 lies in [0.001, 0.001f) or in (0.1, 0.1f), so q < 0.001 is
// q < 0.001f and q <= 0.1 is q < 0.1f.
constexpr int kMaxCons = 4;

struct ConsAcc {
  float g[kMaxCons];
  __device__ __forceinline__ void start(const float* __restrict__ cons, int ncons, int dim) {
#pragma unroll
    for (int k = 0; k < kMaxCons; ++k) g[k] = (k < ncons) ? cons[(size_t)k * (1 + 2 * dim)] : 0.0f;
  }
  __device__ __forceinline__ void add(const float* __restrict__ cons, int ncons, int dim, int d, float x) {
    const float x2 = __fmul_rn(x, x);
#pragma unroll
    for (int k = 0; k < kMaxCons; ++k) {
      if (k < ncons) {
        const float* row = cons + (size_t)k * (1 + 2 * dim);
        g[k] = __fadd_rn(g[k], __fadd_rn(__fmul_rn(__ldg(row + 1 + d), x), __fmul_rn(__ldg(row + 1 + dim + d), x2)));
      }
    }
  }
};

__device__ __forceinline__ float theta_default(float q) {
  return q < 0.001f ? 10.0f : (q < 0.1f ? 20.0f : (q <= 1.0f ? 100.0f : 300.0f));
}

__device__ __forceinline__ float penalty(const ConsAcc& a, int ncons, float iter) {
  float q[kMaxCons];
#pragma unroll
  for (int k = 0; k < kMaxCons; ++k) q[k] = (a.g[k] < 0.0f) ? 0.0f : a.g[k];  // max.(g, 0), NaN kept
  float pen = 0.0f;
#pragma unroll
  for (int k = 0; k < kMaxCons; ++k)
    if (k < ncons) pen = __fadd_rn(pen, theta_default(q[k]));
#pragma unroll
  for (int k = 0; k < kMaxCons; ++k) {
    if (k < ncons) {
      const float pw = (q[k] < 1.0f) ? q[k] : __fmul_rn(q[k], q[k]);  // q^gamma_default(q)
      pen = __fadd_rn(pen, __fmul_rn(theta_default(q[k]), pw));
    }
  }
  return __fmul_rn(__fsqrt_rn(iter), pen);
}

// orderable image of a cost (NaN above +inf) packed with the particle index:
// the minimum key is the lowest cost, lowest index on ties.
__device__ __forceinline__ unsigned long long argmin_key(float c, uint32_t idx) {
  uint32_t o;
  if (c != c) {
    o = 0xFFFFFFFFu;
  } else {
    const uint32_t b = __float_as_uint(c);
    o = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  }
  return ((unsigned long long)o << 32) | (unsigned long long)idx;
}

// max.(x, lb) then min.(x, ub) (src/kernels.jl:15-16)
__device__ __forceinline__ float clamp_lb_ub(float x, float lo, float hi) {
  x = (x < lo) ? lo : x;
  x = (x > hi) ? hi : x;
  return x;
}

// The same in two instructions where neither a bound nor the position is a
// negative zero (which lo = +0 would turn positive): NaN stays NaN.
__device__ __forceinline__ float clamp_box(float x, float lo, float hi) {
  float y;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(x), "f"(lo));
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(y), "f"(hi));
  return y;
}

// the velocity update of src/kernels.jl:2-9 in Julia's broadcast order:
// ((w*v) + ((c1*r1)*(p-x))) + ((c2*r2)*(g-x))
__device__ __forceinline__ float velocity(float x, float v, float p, float g, float w, float c1,
                                          float c2, float r1, float r2) {
  const float a = __fmul_rn(w, v);
  const float b = __fmul_rn(__fmul_rn(c1, r1), __fsub_rn(p, x));
  const float c = __fmul_rn(__fmul_rn(c2, r2), __fsub_rn(g, x));
  return __fadd_rn(__fadd_rn(a, b), c);
}

// A draw's 24-bit integer m = bits >> 8, for updates that take c1s = c1 2^-24 and
// c2s = c2 2^-24 (pps_pair.cuh): c1 (m 2^-24) and (c1 2^-24) m are the same
// real product, so they round to the same value wherever c1s is exact
// (coef_scales), and the draw's own multiplication by 2^-24 goes.
__device__ __forceinline__ float draw24(uint32_t bits) { return __uint2float_rn(bits >> 8); }
// whether c 2^-24 is exact (c is 0 or large enough that it stays normal)
__host__ __device__ inline bool coef_scales(float c) { return c == 0.0f || c >= 0x1p-100f || c <= -0x1p-100f; }

// ---------------------------------------------------------------- objectives
// Objective parameters, passed by value to every kernel.
struct ObjParams {
  float p[8];
  int np;
  int dim;
  const float* data;  // a user objective's data buffer on the device (NULL otherwise)
  long long ndata;
};
__device__ __forceinline__ float prm(const ObjParams& o, int k, float dflt) {
  return (k < o.np) ? o.p[k] : dflt;
}

// Streaming accumulator over dims d = 0..D-1 (separable and chained
// objectives).  add(d, x) must be called in increasing d.  BOX: the cosines'
// arguments are below 2^126 (box_cosines), cos2pi_box takes them.
template <int OBJ, bool BOX = false>
struct Acc {
  float s1 = 0.0f, s2 = 0.0f, prev = 0.0f;
  __device__ __forceinline__ void add(const ObjParams& o, int d, float x) {
    if constexpr (OBJ == kSphere) {
      s1 = __fadd_rn(s1, __fmul_rn(x, x));
    } else if constexpr (OBJ == kRosenbrock) {
      // res += p2*(x[i+1]-x[i]^2)^2 + (p1-x[i])^2  (test/regression.jl:12-18)
      if (d > 0) {
        const float t = __fsub_rn(x, __fmul_rn(prev, prev));
        const float u = __fsub_rn(prm(o, 0, 1.0f), prev);
        s1 = __fadd_rn(s1, __fadd_rn(__fmul_rn(prm(o, 1, 100.0f), __fmul_rn(t, t)), __fmul_rn(u, u)));
      }
      prev = x;
    } else if constexpr (OBJ == kRastrigin) {
      s1 = __fadd_rn(s1, __fsub_rn(__fmul_rn(x, x), __fmul_rn(prm(o, 0, 10.0f), BOX ? cos2pi_box(x) : cos2pi(x))));
    } else if constexpr (OBJ == kAckley) {
      const float kx = __fmul_rn(prm(o, 2, 1.0f), x);
      s1 = __fadd_rn(s1, __fmul_rn(x, x));
      s2 = __fadd_rn(s2, BOX ? cos2pi_box(kx) : cos2pi(kx));
    } else if constexpr (OBJ == kShiftedSphere) {
      const float t = __fsub_rn(x, prm(o, d, 0.0f));  // test/constraints.jl:7
      s1 = __fadd_rn(s1, __fmul_rn(t, t));
    } else if constexpr (OBJ == kMlp) {
      // evaluated by the tensor-core kernel after the position update
    } else {
      // closed-form low-dimensional objectives keep x1, x2
      if (d == 0) s1 = x;
      if (d == 1) s2 = x;
    }
  }
};

__device__ __forceinline__ float sq(float a) { return __fmul_rn(a, a); }

// combine slice sums s1, s2 into the objective value
template <int OBJ>
__device__ __forceinline__ float finalize(const ObjParams& o, float s1, float s2) {
  const float Df = (float)o.dim;
  if constexpr (OBJ == kRastrigin) {
    return __fadd_rn(__fmul_rn(prm(o, 0, 10.0f), Df), s1);
  } else if constexpr (OBJ == kAckley) {
    const float a = prm(o, 0, 20.0f), b = prm(o, 1, 0.2f);
    const float t1 = __fmul_rn(-a, exp_f(__fmul_rn(-b, __fsqrt_rn(__fdiv_rn(s1, Df)))));
    const float t2 = exp_f(__fdiv_rn(s2, Df));
    return __fadd_rn(__fadd_rn(__fsub_rn(t1, t2), a), 0x1.5bf0a8p+1f);
  } else if constexpr (OBJ == kBeale) {
    // (1.5 - x1 + x1 x2)^2 + (2.25 - x1 + x1 x2^2)^2 + (2.625 - x1 + x1 x2^3)^2
    const float x1 = s1, x2 = s2, x22 = sq(x2), x23 = __fmul_rn(x22, x2);
    const float a = __fadd_rn(__fsub_rn(1.5f, x1), __fmul_rn(x1, x2));
    const float b = __fadd_rn(__fsub_rn(2.25f, x1), __fmul_rn(x1, x22));
    const float c = __fadd_rn(__fsub_rn(2.625f, x1), __fmul_rn(x1, x23));
    return __fadd_rn(__fadd_rn(sq(a), sq(b)), sq(c));
  } else if constexpr (OBJ == kBooth) {
    // (x1 + 2 x2 - 7)^2 + (2 x1 + x2 - 5)^2
    const float a = __fsub_rn(__fadd_rn(s1, __fmul_rn(2.0f, s2)), 7.0f);
    const float b = __fsub_rn(__fadd_rn(__fmul_rn(2.0f, s1), s2), 5.0f);
    return __fadd_rn(sq(a), sq(b));
  } else if constexpr (OBJ == kHimmelblau) {
    // (x1^2 + x2 - 11)^2 + (x1 + x2^2 - 7)^2
    const float a = __fsub_rn(__fadd_rn(sq(s1), s2), 11.0f);
    const float b = __fsub_rn(__fadd_rn(s1, sq(s2)), 7.0f);
    return __fadd_rn(sq(a), sq(b));
  } else if constexpr (OBJ == kQuadratic) {
    // p1 (x1 - 1)^2 + (x2 + 2)^2
    return __fadd_rn(__fmul_rn(prm(o, 0, 1.0f), sq(__fsub_rn(s1, 1.0f))), sq(__fadd_rn(s2, 2.0f)));
  } else if constexpr (OBJ == kBoundaryQuadratic) {
    return sq(__fadd_rn(s1, 1.0f));  // (x1 + 1)^2
  } else {
    return s1;
  }
}

}  // namespace pps
