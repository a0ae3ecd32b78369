// fq_lanes.cuh -- Fq arithmetic by several lanes of a warp, for chains that a lone
// warp works through (the last steps of the multi-scalar multiplication).
#pragma once
#include "fq.cuh"

namespace pp {
namespace {

// A field element spread over six lanes, one 64-bit digit each: five of them in a
// warp.  A lone warp's multiply is bound by its 288 wide products in a row (1.0 us);
// spread like this each lane makes 48, and the six reduction steps' exchanges bound
// it (0.43 us).  Elements are below 2^384 = 9.84 q, not reduced: a product of
// a < x q and b < y q is below (0.1016 x y + 1) q.
struct digit {
  uint32_t l, h;
  int32_t c;  // what lies above the digit, signed, until norm
};
constexpr uint32_t kSpread = 6;
constexpr uint64_t kFqNegInv64 = 0x89f3fffcfffcfffdull;  // -1 / q mod 2^64
__constant__ uint32_t c_fq_multiple[3][12] = {  // q, 2q, 3q
    {0xffffaaabu, 0xb9feffffu, 0xb153ffffu, 0x1eabfffeu, 0xf6b0f624u, 0x6730d2a0u, 0xf38512bfu, 0x64774b84u, 0x434bacd7u, 0x4b1ba7b6u, 0x397fe69au, 0x1a0111eau},
    {0xffff5556u, 0x73fdffffu, 0x62a7ffffu, 0x3d57fffdu, 0xed61ec48u, 0xce61a541u, 0xe70a257eu, 0xc8ee9709u, 0x869759aeu, 0x96374f6cu, 0x72ffcd34u, 0x340223d4u},
    {0xffff0001u, 0x2dfcffffu, 0x13fbffffu, 0x5c03fffcu, 0xe412e26cu, 0x359277e2u, 0xda8f383eu, 0x2d65e28eu, 0xc9e30686u, 0xe152f722u, 0xac7fb3ceu, 0x4e0335beu}};

struct Spread {
  uint32_t lane, k, base;  // digit k of the element whose lanes start at base
  uint32_t el;             // which of the five; lanes 30 and 31 hold nothing
  uint32_t q[3][2];        // digits of q, 2q, 3q
  __device__ __forceinline__ Spread()
      : lane(threadIdx.x & 31), k(lane % kSpread), base(lane - k), el(lane / kSpread) {
#pragma unroll
    for (int m = 0; m < 3; ++m) q[m][0] = c_fq_multiple[m][2 * k], q[m][1] = c_fq_multiple[m][2 * k + 1];
  }
  // carries moved up until every digit is whole (the value is in [0, 2^384))
  __device__ __forceinline__ digit norm(digit d) const {
    for (uint32_t it = 0; it < kSpread; ++it) {
      const int32_t in = __shfl_up_sync(0xffffffffu, d.c, 1);
      const int32_t c = k ? in : 0;
      d.l = add_cc(d.l, (uint32_t)c);
      d.h = addc_cc(d.h, (uint32_t)(c >> 31));
      d.c = (int32_t)addc((uint32_t)(c >> 31), 0);
      if (!__any_sync(0xffffffffu, d.c != 0 && k < kSpread - 1 && lane < 5 * kSpread)) break;
    }
    d.c = 0;
    return d;
  }
  // t (5 words) = (a1 a0) (b1 b0)
  static __device__ __forceinline__ void product(uint32_t t[5], uint32_t a0, uint32_t a1, uint32_t b0,
                                                 uint32_t b1) {
    const uint64_t lo = (uint64_t)a0 * b0, hi = (uint64_t)a1 * b1, p = (uint64_t)a0 * b1;
    uint32_t x0 = (uint32_t)p, x1 = (uint32_t)(p >> 32);
    x0 = madlo_cc(a1, b0, x0);
    x1 = madhic_cc(a1, b0, x1);
    const uint32_t x2 = addc(0, 0);
    t[0] = (uint32_t)lo;
    t[1] = add_cc((uint32_t)(lo >> 32), x0);
    t[2] = addc_cc((uint32_t)hi, x1);
    t[3] = addc_cc((uint32_t)(hi >> 32), x2);
    t[4] = addc(0, 0);
  }
  // a b / 2^384 mod q, carries left in c (at most 3).  The statements stand in the
  // order in which a lone warp should issue them: exchanges first, the products
  // that do not wait for them after.
  __device__ __forceinline__ digit mul(const digit &a, const digit &b) const {
    uint32_t b0[kSpread], b1[kSpread], P[5], t[5] = {0, 0, 0, 0, 0};
#pragma unroll
    for (uint32_t i = 0; i < kSpread; ++i) {
      b0[i] = __shfl_sync(0xffffffffu, b.l, base + i);
      b1[i] = __shfl_sync(0xffffffffu, b.h, base + i);
    }
    product(P, a.l, a.h, b0[0], b1[0]);
#pragma unroll
    for (uint32_t i = 0; i < kSpread; ++i) {
      t[0] = add_cc(t[0], P[0]);
      t[1] = addc_cc(t[1], P[1]);
      t[2] = addc_cc(t[2], P[2]);
      t[3] = addc_cc(P[3], 0);
      t[4] = addc(P[4], 0);
      // m = (lowest digit) (-1 / q) mod 2^64
      const uint64_t p = (uint64_t)t[0] * (uint32_t)kFqNegInv64;
      const uint32_t m0 = __shfl_sync(0xffffffffu, (uint32_t)p, base);
      const uint32_t m1 = __shfl_sync(0xffffffffu,
                                      (uint32_t)(p >> 32) + t[0] * (uint32_t)(kFqNegInv64 >> 32) +
                                          t[1] * (uint32_t)kFqNegInv64,
                                      base);
      if (i + 1 < kSpread) product(P, a.l, a.h, b0[i + 1 < kSpread ? i + 1 : 0], b1[i + 1 < kSpread ? i + 1 : 0]);
      // t += m q, then one digit down: the lowest is zero
      const uint64_t x = (uint64_t)q[0][1] * m0;
      t[0] = madlo_cc(q[0][0], m0, t[0]);
      t[1] = madhic_cc(q[0][0], m0, t[1]);
      t[2] = madloc_cc(q[0][1], m1, t[2]);
      t[3] = madhic_cc(q[0][1], m1, t[3]);
      t[4] = addc(t[4], 0);
      const uint32_t n0 = __shfl_down_sync(0xffffffffu, t[0], 1);
      const uint32_t x0 = madlo_cc(q[0][0], m1, (uint32_t)x), x1 = madhic_cc(q[0][0], m1, (uint32_t)(x >> 32));
      const uint32_t x2 = addc(0, 0);
      t[1] = add_cc(t[1], x0);
      t[2] = addc_cc(t[2], x1);
      t[3] = addc_cc(t[3], x2);
      t[4] = addc(t[4], 0);
      const uint32_t n1 = __shfl_down_sync(0xffffffffu, t[1], 1);
      t[0] = add_cc(t[2], k < kSpread - 1 ? n0 : 0);
      t[1] = addc_cc(t[3], k < kSpread - 1 ? n1 : 0);
      t[2] = addc(t[4], 0);
    }
    return {t[0], t[1], (int32_t)t[2]};
  }
  __device__ __forceinline__ digit from(const digit &a, uint32_t src) const {  // of another element
    digit r;
    r.l = __shfl_sync(0xffffffffu, a.l, src * kSpread + k);
    r.h = __shfl_sync(0xffffffffu, a.h, src * kSpread + k);
    r.c = __shfl_sync(0xffffffffu, a.c, src * kSpread + k);
    return r;
  }
  static __device__ __forceinline__ digit add(digit a, const digit &b) {
    a.l = add_cc(a.l, b.l);
    a.h = addc_cc(a.h, b.h);
    a.c = (int32_t)addc((uint32_t)a.c, (uint32_t)b.c);
    return a;
  }
  static __device__ __forceinline__ digit sub(digit a, const digit &b) {
    a.l = sub_cc(a.l, b.l);
    a.h = subc_cc(a.h, b.h);
    a.c = (int32_t)subc((uint32_t)a.c, (uint32_t)b.c);
    return a;
  }
  __device__ __forceinline__ digit multiple(uint32_t m) const { return {q[m - 1][0], q[m - 1][1], 0}; }
  // a - e q, 0 <= the result < 1.04 q: e from the top digit's upper bits (0 <= a <
  // 8 q, carries pending): 157 / 2^20 is 0.3 % below 2^16 / (q's top word)
  __device__ __forceinline__ digit reduce(const digit &a) const {
    const int32_t e = (int32_t)(((uint32_t)a.c << 16) | (a.h >> 16)) * 157 >> 20;
    const uint32_t n = __shfl_sync(0xffffffffu, e > 0 ? (uint32_t)e : 0u, base + kSpread - 1);
    const uint64_t p0 = (uint64_t)n * q[0][0], p1 = (uint64_t)n * q[0][1] + (p0 >> 32);
    return sub(a, {(uint32_t)p0, (uint32_t)p1, (int32_t)(p1 >> 32)});
  }
};
// lanes of element el among the bits of a ballot
__device__ __forceinline__ bool element_all(uint32_t ballot, uint32_t el) {
  const uint32_t mask = ((1u << kSpread) - 1) << (kSpread * el);
  return (ballot & mask) == mask;
}
__device__ __forceinline__ digit sel_digit(bool c, const digit &a, const digit &b) {
  return {c ? a.l : b.l, c ? a.h : b.h, c ? a.c : b.c};
}

}  // namespace
}  // namespace pp
