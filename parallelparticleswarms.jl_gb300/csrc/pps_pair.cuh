// pps_pair.cuh -- two dims of a particle per instruction: the update and the
// cosine objectives' terms in Blackwell's packed f32x2 arithmetic, each lane
// the scalar operation sequence (velocity with draw24, cos2pi_box), so
// bit-identical to it.
//
// The assembler contracts a packed multiply whose only use is a packed add
// into one fused operation, which rounds once where two operations round
// twice.  So a product is only ever added as fma(product, one, other) with
// `one` a run-time 1.0f (or mone = -1.0f for a difference) that the compiler
// cannot see through: product * 1 is exact.
#pragma once
#include "pps_device.cuh"

namespace pps {
namespace pair32 {

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }  // of sums only

// velocity() of a pair with draw r (r.a, r.b: first dim; r.c, r.d: second) and
// the coefficients times 2^-24
__device__ __forceinline__ float2 velocity24x2(float2 x, float2 v, float2 p, float2 g, float2 w, float2 c1s, float2 c2s,
                                               const Rand4& r, float2 one, float2 mone) {
  const float2 a = mul(w, v);
  const float2 b = mul(mul(c1s, make_float2(draw24(r.a), draw24(r.c))), fma(x, mone, p));
  const float2 c = mul(mul(c2s, make_float2(draw24(r.b), draw24(r.d))), fma(x, mone, g));
  return fma(fma(a, one, b), one, c);
}

// cos2pi_box of a pair
__device__ __forceinline__ float2 cos2pi_box2(float2 x, float2 mone) {
  const float2 f = fma(make_float2(rintf(x.x), rintf(x.y)), mone, x);
  const float fx = fabsf(f.x), fy = fabsf(f.y);
  const float2 h = make_float2(fminf(fx, __fsub_rn(0.5f, fx)), fminf(fy, __fsub_rn(0.5f, fy)));
  const float2 z = mul(h, h);
  float2 q = fma(dup(64.0f * kCosP3), z, dup(16.0f * kCosP2));
  q = fma(q, z, dup(4.0f * kCosP1));
  q = fma(q, z, dup(kCosP0));
  const float2 p4 = fma(mul(dup(-16.0f), h), h, dup(1.0f));
  const float2 c = fma(p4, mul(z, q), p4);
  return make_float2(
      __uint_as_float((__float_as_uint(c.x) & 0x7fffffffu) | (__float_as_uint(__fsub_rn(0.25f, fx)) & 0x80000000u)),
      __uint_as_float((__float_as_uint(c.y) & 0x7fffffffu) | (__float_as_uint(__fsub_rn(0.25f, fy)) & 0x80000000u)));
}

// the terms of Rastrigin (whole) and Ackley (the cosine) at a pair
template <int OBJ>
__device__ __forceinline__ float2 moved_terms(const ObjParams& op, float2 x, float2 mone) {
  if constexpr (OBJ == kRastrigin) {
    return fma(mul(dup(prm(op, 0, 10.0f)), cos2pi_box2(x, mone)), mone, mul(x, x));
  } else {
    return cos2pi_box2(mul(dup(prm(op, 2, 1.0f)), x), mone);
  }
}
template <int OBJ, typename A>
__device__ __forceinline__ void add_term(A& acc, float x, float term) {
  if constexpr (OBJ == kRastrigin) {
    acc.s1 = __fadd_rn(acc.s1, term);
  } else {
    acc.s1 = __fadd_rn(acc.s1, __fmul_rn(x, x));
    acc.s2 = __fadd_rn(acc.s2, term);
  }
}

}  // namespace pair32
}  // namespace pps
