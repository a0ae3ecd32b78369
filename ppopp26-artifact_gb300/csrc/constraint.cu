// constraint.cu -- PLONK quotient-constraint operators: element-wise terms
// over the points of the extended domain, computed from the LDE outputs.
//
// Each output point costs 18 (permutation, fused) to ~80 (gate) multiplies
// against 448 / 736 bytes of HBM traffic, so both kernels are integer-multiply
// bound by a factor of 5-40 over HBM.  They are plain element-wise loops: one
// thread per point, scalars staged once per block.
//
// Multiplies by a scalar of the call take the four-part constant form
// (fr_mul_const4, 82 wide products against 112; the parts are prepared once per
// block or call), squares the squaring (84), sums of products one reduction for
// all (fr_mac17), small integers fr_mul_small.  Values are lazy (below 2r)
// between loads and the store: fr_mul and fr_sqr of lazy values are below 1.82 r
// (4 r^2 / 2^256), and canonical again when one factor is below r and the other
// below 2r.  The kernels keep the integer-multiply pipe 78 - 82 % busy.  GB300,
// 2^20 points: permutation terms 228 us, gate 1074 us (other scalars than the
// prover's integers 1166 us); both together 1307 us, against 1722 us with
// fr_mul throughout, canonical additions and small integers by additions.
#include "common.cuh"

namespace pp {
namespace {

constexpr int kThreads = 256;

struct PermArgs {
  const fr *x, *w[4], *z, *z_next, *sigma[4], *mod, *l1;
  const fr *alpha, *beta, *gamma, *k[3], *one;
};

enum : int { kIdentity = 1, kCopy = 2, kTermOne = 4, kAll = 7 };

// The scalars as shared constants, four parts each: alpha, beta, beta k_1..3.
enum : int { kCAlpha, kCBeta, kCBetaK, kPermConsts = kCBetaK + 3 };

__device__ __forceinline__ void stage_perm_constants(const PermArgs &a, fr *sc, int terms) {
  if (threadIdx.x < 4 * kPermConsts) {
    const int c = threadIdx.x >> 2;
    const bool used = c == kCAlpha || c == kCBeta ? (terms & (kIdentity | kCopy)) != 0 : (terms & kIdentity) != 0;
    if (used) {
      fr k = ld_fr(c == kCAlpha ? a.alpha : a.beta);
      if (c >= kCBetaK) k = fr_mul(k, ld_fr(a.k[c - kCBetaK]));
      st_fr(sc + threadIdx.x, fr_mul(k, fr_const4_factor(threadIdx.x & 3)));
    }
  }
  __syncthreads();
}

// prod_j (u_j * beta * c_j + w_j + gamma) below 2r: the identity product uses
// u_j = x and c = (1, k1, k2, k3); the copy product u_j = sigma_j and c_j = 1.
// wg[j] = w_j + gamma, unreduced.
__device__ __forceinline__ fr identity_product(const fr &x, const fr wg[4], const fr *sc) {
  fr acc = fr_add_lazy(mul_shared_const(x, sc + 4 * kCBeta), wg[0]);
#pragma unroll
  for (int j = 1; j < 4; ++j)
    acc = fr_mul(acc, fr_add_lazy(mul_shared_const(x, sc + 4 * (kCBetaK + j - 1)), wg[j]));
  return acc;
}

__device__ __forceinline__ fr copy_product(const PermArgs &a, uint64_t i, const fr wg[4], const fr *sc) {
  fr acc = fr_add_lazy(mul_shared_const(ldcs_fr(a.sigma[0] + i), sc + 4 * kCBeta), wg[0]);
#pragma unroll
  for (int j = 1; j < 4; ++j)
    acc = fr_mul(acc, fr_add_lazy(mul_shared_const(ldcs_fr(a.sigma[j] + i), sc + 4 * kCBeta), wg[j]));
  return acc;
}

template <int TERMS>
__global__ void __launch_bounds__(kThreads, 2) k_perm_quotient(const PermArgs a, fr *result,
                                                               uint64_t n) {
  __shared__ __align__(16) fr sc[4 * kPermConsts];
  stage_perm_constants(a, sc, TERMS);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    fr wg[4];
    if (TERMS & (kIdentity | kCopy)) {
      const fr gamma = ldg_fr(a.gamma);
#pragma unroll
      for (int j = 0; j < 4; ++j) wg[j] = fr_add_raw(ldcs_fr(a.w[j] + i), gamma);
    }
    const fr one = (TERMS & kTermOne) ? ldg_fr(a.one) : fr_zero();
    fr r;
    if (TERMS == kAll) {
      // (id * z - cp * z_next) * alpha + mod + (z - one) * l1: alpha once
      const fr z = ldcs_fr(a.z + i);
      const fr id = fr_mul(identity_product(ldcs_fr(a.x + i), wg, sc), z);
      const fr cp = fr_mul(copy_product(a, i, wg, sc), ldcs_fr(a.z_next + i));
      r = fr_add_lazy(mul_shared_const(fr_sub_lazy(id, cp), sc + 4 * kCAlpha), ldcs_fr(a.mod + i));
      r = fr_canon(fr_add_lazy(r, fr_mul(fr_sub_lazy(z, one), ldcs_fr(a.l1 + i))));
    } else if (TERMS == kIdentity) {
      r = fr_mul(identity_product(ldcs_fr(a.x + i), wg, sc), ldcs_fr(a.z + i));
      r = fr_canon(mul_shared_const(r, sc + 4 * kCAlpha));
    } else if (TERMS == kCopy) {
      const fr cp = fr_mul(copy_product(a, i, wg, sc), ldcs_fr(a.z_next + i));
      r = fr_add_raw(ld_fr(result + i), ldcs_fr(a.mod + i));
      r = fr_canon(fr_sub_lazy(r, mul_shared_const(cp, sc + 4 * kCAlpha)));
    } else {
      r = fr_add(ld_fr(result + i), fr_mul(fr_sub(ldcs_fr(a.z + i), one), ldcs_fr(a.l1 + i)));
    }
    st_fr(result + i, r);
  }
}

// ------------------------------------------------------------------- gate
struct GateArgs {
  const fr *v[PP_GATE_NV];
  const fr *s[PP_GATE_NS];
  uint32_t sbox_alpha;  // 2 <= sbox_alpha < 2^31
};

// x^e below 2r for 2 <= e < 2^31, square and multiply from the top set bit
__device__ __forceinline__ fr pow_small(const fr &x, uint32_t e) {
  fr r = x;
  for (int b = 30 - __clz(e); b >= 0; --b) {
    r = fr_sqr(r);
    if ((e >> b) & 1) r = fr_mul(r, x);
  }
  return r;
}

// small multiples by additions, canonical (k_gate_prepare's comparison)
__device__ __forceinline__ fr dbl(const fr &x) { return fr_add(x, x); }
__device__ __forceinline__ fr mul3(const fr &x) { return fr_add(dbl(x), x); }
__device__ __forceinline__ fr mul4(const fr &x) { return dbl(dbl(x)); }
__device__ __forceinline__ fr mul9(const fr &x) { return fr_add(dbl(mul4(x)), x); }
__device__ __forceinline__ fr mul18(const fr &x) { return dbl(mul9(x)); }
__device__ __forceinline__ fr mul81(const fr &x) { return mul9(mul9(x)); }
__device__ __forceinline__ fr mul83(const fr &x) { return fr_add(mul81(x), dbl(x)); }

// The gate runs as three launches so that each keeps its live values in
// fewer registers (more resident warps): the range and logic terms are
// written first, then the arithmetic and public-input terms and the fixed-
// and variable-base group additions are added.

// The constants of the gate kernels, prepared once per call by k_gate_prepare
// in the four-part form: products of the call's scalars, with each gate's
// challenge multiplied in (Kxx below: the reference's kappa names), so that a
// sum of terms needs no further multiply by it.  `small` says whether four, one,
// two, three, nine, eighteen, eightyone and eightythree hold those integers, as
// the prover passes them.  Then the kernels take SMALL = true: multiplies by
// them become fr_mul_small.  Any other values take SMALL = false, the
// expression as written.
enum : int {
  kRangeCu, kRangeSq, kRangeOne, kRangeK,  // three one two kappa.. range_challenge
  kLogicQu, kLogicCu, kLogicQuad,          // the last: three one two logic_challenge
  kFbK, kFbCu, kFbOne, kFbSq, kPd, kPa, kVbSq, kVbOne, kVbK,
  kOneSq, kFour, kEighteen, kEightyone, kTwo83, kThree, kNine,  // SMALL = false only
  kGateConsts
};
struct GateScalars {
  fr c[4 * kGateConsts];
  int small;
};

// constant c is the product of these scalars (PP_GATE_NS: the factor 1)
#define GS(name) PP_GATE_S_##name
constexpr int kNone = PP_GATE_NS, kGateFactors = 5;
__constant__ unsigned char c_gate_factors[kGateConsts][kGateFactors] = {
    {GS(THREE), GS(ONE), GS(TWO), GS(KAPPA_CU_RANGE), GS(RANGE_CHALLENGE)},
    {GS(THREE), GS(ONE), GS(TWO), GS(KAPPA_SQ_RANGE), GS(RANGE_CHALLENGE)},
    {GS(THREE), GS(ONE), GS(TWO), GS(RANGE_CHALLENGE), kNone},
    {GS(THREE), GS(ONE), GS(TWO), GS(KAPPA_RANGE), GS(RANGE_CHALLENGE)},
    {GS(KAPPA_QU_LOGIC), GS(LOGIC_CHALLENGE), kNone, kNone, kNone},
    {GS(KAPPA_CU_LOGIC), GS(LOGIC_CHALLENGE), kNone, kNone, kNone},
    {GS(THREE), GS(ONE), GS(TWO), GS(LOGIC_CHALLENGE), kNone},
    {GS(KAPPA_FB), GS(FB_CHALLENGE), kNone, kNone, kNone},
    {GS(KAPPA_CU_FB), GS(FB_CHALLENGE), kNone, kNone, kNone},
    {GS(ONE), GS(ONE), GS(FB_CHALLENGE), kNone, kNone},
    {GS(KAPPA_SQ_FB), GS(FB_CHALLENGE), kNone, kNone, kNone},
    {GS(P_D), kNone, kNone, kNone, kNone},
    {GS(P_A), kNone, kNone, kNone, kNone},
    {GS(KAPPA_SQ_VB), GS(VB_CHALLENGE), kNone, kNone, kNone},
    {GS(VB_CHALLENGE), kNone, kNone, kNone, kNone},
    {GS(KAPPA_VB), GS(VB_CHALLENGE), kNone, kNone, kNone},
    {GS(ONE), GS(ONE), kNone, kNone, kNone},
    {GS(FOUR), kNone, kNone, kNone, kNone},
    {GS(EIGHTEEN), kNone, kNone, kNone, kNone},
    {GS(EIGHTYONE), kNone, kNone, kNone, kNone},
    {GS(TWO), GS(EIGHTYTHREE), kNone, kNone, kNone},
    {GS(THREE), kNone, kNone, kNone, kNone},
    {GS(NINE), kNone, kNone, kNone, kNone},
};
#undef GS

// one thread per part of a constant
__global__ void __launch_bounds__(128) k_gate_prepare(const GateArgs a, GateScalars *out) {
  __shared__ __align__(16) fr sc[PP_GATE_NS + 1];
  const uint32_t t = threadIdx.x;
  if (t < PP_GATE_NS) st_fr(sc + t, ldg_fr(a.s[t]));
  if (t == PP_GATE_NS) st_fr(sc + t, fr_one());
  __syncthreads();
  if (t < 4 * kGateConsts) {
    fr k = lds_fr(sc + c_gate_factors[t >> 2][0]);
#pragma unroll 1
    for (int f = 1; f < kGateFactors; ++f) k = fr_mul(k, lds_fr(sc + c_gate_factors[t >> 2][f]));
    st_fr(out->c + t, fr_mul(k, fr_const4_factor(t & 3)));
  }
  if (t == 127) {
    const fr one = fr_one();
    auto is = [&](int s, const fr &v) { return fr_eq(lds_fr(sc + s), v); };
    out->small = is(PP_GATE_S_ONE, one) && is(PP_GATE_S_TWO, dbl(one)) && is(PP_GATE_S_THREE, mul3(one)) &&
                 is(PP_GATE_S_FOUR, mul4(one)) && is(PP_GATE_S_NINE, mul9(one)) &&
                 is(PP_GATE_S_EIGHTEEN, mul18(one)) && is(PP_GATE_S_EIGHTYONE, mul81(one)) &&
                 is(PP_GATE_S_EIGHTYTHREE, mul83(one));
  }
}
static_assert(4 * kGateConsts < 127, "k_gate_prepare: one thread per part, the last compares");

// copies the prepared constants to shared memory
__device__ __forceinline__ void stage_constants(const GateScalars *g, fr *sc) {
  if (threadIdx.x < 4 * kGateConsts) st_fr(sc + threadIdx.x, ldg_fr(g->c + threadIdx.x));
  __syncthreads();
}

#define MC(x, c) mul_shared_const(x, sc + 4 * (c))
#define V(name) ldcs_fr(a.v[PP_GATE_V_##name] + i)

// The host launches both forms; the one whose SMALL does not match the
// scalars returns at once.
template <bool SMALL>
__global__ void __launch_bounds__(kThreads, 2) k_gate_range_logic(const GateArgs a,
                                                               const GateScalars *gs, fr *out,
                                                               uint64_t n) {
  if ((__ldg(&gs->small) != 0) != SMALL) return;
  __shared__ __align__(16) fr sc[4 * kGateConsts];
  stage_constants(gs, sc);
  // x times one of the gate's integers, below 2r
  const auto times = [&](const fr &x, uint32_t k, int c) { return SMALL ? fr_mul_small(x, k) : MC(x, c); };
  const auto pow4 = [](const fr &x) { return fr_sqr(fr_sqr(x)); };
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const fr a_ = V(A), b = V(B), c = V(C), d = V(D), dn = V(D_NEXT);
    const fr a4 = times(a_, 4, kFour), b4 = times(b, 4, kFour);
    const fr c4 = times(c, 4, kFour), d4 = times(d, 4, kFour);

    // range gate: four 2-bit quads, quad(x) = x^4 three one two
    fr t = MC(pow4(fr_sub_lazy(a4, dn)), kRangeCu);
    t = fr_add_lazy(t, MC(pow4(fr_sub_lazy(a_, b4)), kRangeSq));
    t = fr_add_lazy(t, MC(pow4(fr_sub_lazy(c, d4)), kRangeOne));
    t = fr_add_lazy(t, MC(pow4(fr_sub_lazy(b, c4)), kRangeK));
    fr acc = fr_mul(t, V(RANGE));

    // logic gate
    const fr da = fr_sub_lazy(a4, V(A_NEXT)), db = fr_sub_lazy(b4, V(B_NEXT));
    const fr w = fr_add_lazy(da, db), e = fr_sub_lazy(dn, d4);
    const fr da2 = fr_sqr(da);
    const fr u = fr_mul(times(fr_sub_lazy(c4, times(w, 18, kEighteen)), 81, kEightyone), c);
    const fr inner = fr_sub_lazy(times(w, 81, kEightyone),
                                 fr_add_lazy(u, times(fr_add_lazy(da2, da2), 18, kEighteen)));
    const fr A = fr_sub_lazy(times(fr_add_lazy(e, w), 3, kThree), times(fr_mul(inner, c), 166, kTwo83));
    const fr B = fr_mul(fr_sub_lazy(times(e, 9, kNine), times(w, 3, kThree)), V(Q_C));
    fr l = MC(fr_add_lazy(A, B), kLogicQu);
    l = fr_add_lazy(l, MC(fr_sub_lazy(c, fr_mul(da, db)), kLogicCu));
    l = fr_add_lazy(l, MC(fr_add_lazy(fr_add_lazy(pow4(e), fr_sqr(da2)), pow4(db)), kLogicQuad));
    st_fr(out + i, fr_add(acc, fr_mul(l, V(LOGIC))));
  }
}

__global__ void __launch_bounds__(kThreads, 2) k_gate_arith(const GateArgs a, fr *out, uint64_t n) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    // arithmetic gate (with the x^alpha S-box terms) and public inputs: eight
    // products of a value below 2r and a canonical one, one reduction (their
    // sum is below 16 r^2, as fr_redc17 allows)
    uint32_t s[17];
#pragma unroll
    for (int k = 0; k < 17; ++k) s[k] = 0;
    const fr a_ = V(A), b = V(B);
    fr_mac17(s, pow_small(a_, a.sbox_alpha), V(Q_HL));
    fr_mac17(s, a_, V(Q_L));
    fr_mac17(s, pow_small(b, a.sbox_alpha), V(Q_HR));
    fr_mac17(s, b, V(Q_R));
    fr_mac17(s, fr_mul(a_, b), V(Q_M));
    const fr d = V(D);
    fr_mac17(s, pow_small(d, a.sbox_alpha), V(Q_H4));
    fr_mac17(s, d, V(Q_4));
    fr_mac17(s, V(C), V(Q_O));
    const fr ar = fr_add_raw(fr_redc17(s), V(Q_C));
    st_fr(out + i, fr_add(fr_add(ld_fr(out + i), fr_mul(ar, V(Q_ARITH))), V(PI)));
  }
}

template <bool SMALL>
__global__ void __launch_bounds__(kThreads, 2) k_gate_groups(const GateArgs a,
                                                          const GateScalars *gs, fr *out,
                                                          uint64_t n) {
  if ((__ldg(&gs->small) != 0) != SMALL) return;
  __shared__ __align__(16) fr sc[4 * kGateConsts];
  stage_constants(gs, sc);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const fr a_ = V(A), b = V(B), c = V(C);
    const fr an = V(A_NEXT), bn = V(B_NEXT), dn = V(D_NEXT);
    const fr bc = fr_mul(b, c);
    fr f, g;
    {
      // fixed-base group addition
      const fr dn2 = fr_sqr(dn), qldn = fr_mul(V(Q_L), dn);
      fr qr2 = fr_mul(dn2, V(Q_R));
      if (!SMALL) qr2 = MC(qr2, kOneSq);  // one one = 1 when SMALL
      const fr abc_pd = MC(fr_mul(a_, bc), kPd);
      fr u = fr_sub_lazy(fr_sub_lazy(bn, fr_mul(abc_pd, bn)),
                         fr_sub_lazy(fr_mul(qr2, b), fr_mul(MC(qldn, kPa), a_)));
      f = MC(u, kFbCu);
      u = fr_sub_lazy(fr_add_lazy(an, fr_mul(abc_pd, an)), fr_add_lazy(fr_mul(qldn, b), fr_mul(qr2, a_)));
      f = fr_add_lazy(f, MC(u, kFbSq));
      f = fr_add_lazy(f, MC(fr_mul(dn2, dn), kFbOne));
      f = fr_add_lazy(f, MC(fr_sub_lazy(c, fr_mul(V(Q_C), dn)), kFbK));
      f = fr_mul(f, V(FIXED_GROUP_ADD));
    }
    {
      // variable-base group addition
      const fr d = V(D);
      const fr h = MC(fr_mul(bc, dn), kPd);
      fr u = fr_sub_lazy(fr_sub_lazy(fr_mul(b, d), MC(fr_mul(a_, c), kPa)), fr_sub_lazy(bn, fr_mul(h, bn)));
      g = MC(u, kVbSq);
      u = fr_sub_lazy(fr_add_raw(dn, bc), fr_add_lazy(an, fr_mul(h, an)));
      g = fr_add_lazy(g, MC(u, kVbK));
      g = fr_add_lazy(g, MC(fr_sub_lazy(dn, fr_mul(a_, d)), kVbOne));
      g = fr_mul(g, V(VARIABLE_GROUP_ADD));
    }
    st_fr(out + i, fr_add(fr_add(ld_fr(out + i), f), g));
  }
}
#undef MC
#undef V

bool aligned16(const void *p) { return p && (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// one thread per point (at most 2^31 - 1 blocks; the kernels stride beyond): 2^22 points'
// permutation terms took 1.45 ms so, 1.85 ms with at most 8 blocks per SM
unsigned grid_for(uint64_t n) {
  const uint64_t want = (n + kThreads - 1) / kThreads;
  return (unsigned)(want < 0x7fffffffull ? want : 0x7fffffffull);
}

// which fields each term reads
int check_perm(const pp_perm_quotient_args *a, int terms, const void *result, const char *who) {
  if (!a || !aligned16(result)) {
    set_error("%s: arguments and a 16-byte aligned result are required", who);
    return PP_E_INVAL;
  }
  bool ok = aligned16(a->alpha) || !(terms & (kIdentity | kCopy));
  if (terms & (kIdentity | kCopy)) ok = ok && aligned16(a->beta) && aligned16(a->gamma);
  for (int j = 0; j < 4; ++j) {
    if (terms & (kIdentity | kCopy)) ok = ok && aligned16(a->w[j]);
    if (terms & kCopy) ok = ok && aligned16(a->sigma[j]);
  }
  if (terms & kIdentity) {
    ok = ok && aligned16(a->x) && aligned16(a->z);
    for (int j = 0; j < 3; ++j) ok = ok && aligned16(a->k[j]);
  }
  if (terms & kCopy) ok = ok && aligned16(a->mod) && aligned16(a->z_next);
  if (terms & kTermOne) ok = ok && aligned16(a->z) && aligned16(a->l1) && aligned16(a->one);
  if (!ok) {
    set_error("%s: a required input is missing or not 16-byte aligned", who);
    return PP_E_INVAL;
  }
  return PP_OK;
}

template <int TERMS>
int perm_launch(const pp_perm_quotient_args *a, void *result, uint64_t n, void *stream,
                const char *who) {
  if (n == 0) return PP_OK;
  const int st = check_perm(a, TERMS, result, who);
  if (st) return st;
  PermArgs p;
  p.x = static_cast<const fr *>(a->x);
  for (int j = 0; j < 4; ++j) {
    p.w[j] = static_cast<const fr *>(a->w[j]);
    p.sigma[j] = static_cast<const fr *>(a->sigma[j]);
  }
  p.z = static_cast<const fr *>(a->z);
  p.z_next = static_cast<const fr *>(a->z_next);
  p.mod = static_cast<const fr *>(a->mod);
  p.l1 = static_cast<const fr *>(a->l1);
  p.alpha = static_cast<const fr *>(a->alpha);
  p.beta = static_cast<const fr *>(a->beta);
  p.gamma = static_cast<const fr *>(a->gamma);
  for (int j = 0; j < 3; ++j) p.k[j] = static_cast<const fr *>(a->k[j]);
  p.one = static_cast<const fr *>(a->one);
  k_perm_quotient<TERMS><<<grid_for(n), kThreads, 0, (cudaStream_t)stream>>>(
      p, static_cast<fr *>(result), n);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}

}  // namespace
}  // namespace pp

extern "C" int pp_quotient_identity(const pp_perm_quotient_args *a, void *d_result, uint64_t n,
                                    void *stream) {
  return pp::perm_launch<pp::kIdentity>(a, d_result, n, stream, "pp_quotient_identity");
}

extern "C" int pp_quotient_copy(const pp_perm_quotient_args *a, void *d_result, uint64_t n,
                                void *stream) {
  return pp::perm_launch<pp::kCopy>(a, d_result, n, stream, "pp_quotient_copy");
}

extern "C" int pp_quotient_term_one(const pp_perm_quotient_args *a, void *d_result, uint64_t n,
                                    void *stream) {
  return pp::perm_launch<pp::kTermOne>(a, d_result, n, stream, "pp_quotient_term_one");
}

extern "C" int pp_quotient_permutation(const pp_perm_quotient_args *a, void *d_result, uint64_t n,
                                       void *stream) {
  return pp::perm_launch<pp::kAll>(a, d_result, n, stream, "pp_quotient_permutation");
}

extern "C" int pp_gate_constraint(const pp_gate_args *a, void *d_out, uint64_t n, void *stream) {
  if (n == 0) return PP_OK;
  if (!a || !pp::aligned16(d_out)) {
    pp::set_error("pp_gate_constraint: arguments and a 16-byte aligned output are required");
    return PP_E_INVAL;
  }
  if (a->sbox_alpha < 2 || a->sbox_alpha >= (int64_t{1} << 31)) {
    pp::set_error("pp_gate_constraint: sbox_alpha = %lld outside [2, 2^31)",
                  (long long)a->sbox_alpha);
    return PP_E_INVAL;
  }
  pp::GateArgs g;
  for (int j = 0; j < PP_GATE_NV; ++j) {
    if (!pp::aligned16(a->v[j])) {
      pp::set_error("pp_gate_constraint: vector %d is missing or not 16-byte aligned", j);
      return PP_E_INVAL;
    }
    g.v[j] = static_cast<const pp::fr *>(a->v[j]);
  }
  for (int j = 0; j < PP_GATE_NS; ++j) {
    if (!pp::aligned16(a->s[j])) {
      pp::set_error("pp_gate_constraint: scalar %d is missing or not 16-byte aligned", j);
      return PP_E_INVAL;
    }
    g.s[j] = static_cast<const pp::fr *>(a->s[j]);
  }
  g.sbox_alpha = (uint32_t)a->sbox_alpha;
  cudaStream_t s = (cudaStream_t)stream;
  int st = PP_OK;
  auto *gs = static_cast<pp::GateScalars *>(pp::workspace_get(sizeof(pp::GateScalars), s, 8, &st));
  if (st) return st;
  pp::k_gate_prepare<<<1, 128, 0, s>>>(g, gs);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  // one thread per point; of each pair, the form that does not match the
  // scalars returns at once
  const unsigned grid = pp::grid_for(n);
  pp::fr *out = static_cast<pp::fr *>(d_out);
  pp::k_gate_range_logic<true><<<grid, pp::kThreads, 0, s>>>(g, gs, out, n);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  pp::k_gate_range_logic<false><<<grid, pp::kThreads, 0, s>>>(g, gs, out, n);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  pp::k_gate_arith<<<grid, pp::kThreads, 0, s>>>(g, out, n);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  pp::k_gate_groups<true><<<grid, pp::kThreads, 0, s>>>(g, gs, out, n);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  pp::k_gate_groups<false><<<grid, pp::kThreads, 0, s>>>(g, gs, out, n);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}
