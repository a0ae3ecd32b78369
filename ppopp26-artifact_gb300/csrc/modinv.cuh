// modinv.cuh -- modular inverse by Bernstein-Yang divsteps ("Fast
// constant-time gcd computation and modular inversion", D. J. Bernstein and
// B.-Y. Yang, TCHES 2019), in the variable-time form: runs of zero low bits
// of g are skipped at once, and the loop ends as soon as g is 0.  Variable
// time is fine here (public prover data).
//
// divstep(delta, f, g), f odd:
//   delta > 0 and g odd:  (1 - delta, g, (g - f) / 2)
//   g odd:                (1 + delta, f, (g + f) / 2)
//   g even:               (1 + delta, f, g / 2)
// Starting from (1, M, x) it reaches g = 0 with f = +-gcd(M, x) = +-1 within
// floor((49 * 256 + 57) / 17) = 741 steps for 256-bit inputs, and within
// 1101 for 381-bit ones.  Starting from delta = 1/2 instead it takes fewer: at most
// 590 and 879 (P. Wuille and G. Maxwell, "Bounds on divsteps iterations in safegcd",
// 2021).
//
// B divsteps depend only on the low B + 2 bits of f and g, so they run on
// one machine word each and record a 2x2 integer matrix T with
// 2^B [f', g'] = T [f, g]; |u| + |v| <= 2^B and |q| + |r| <= 2^B.  T is then
// applied to the full f, g (the division by 2^B is exact) and to the pair
// d, e with f = d x, g = e x (mod M), where the division by 2^B is done mod
// M by first adding the multiple of M that clears the low B bits.
//
// Numbers are NL limbs of B bits, least significant first; limbs below the
// top one are in [0, 2^B) and the top limb carries the sign.  Two widths:
// B = 30 on 32-bit words with 64-bit sums (the GPU form: every limb product
// is one 32 x 32 -> 64-bit multiply-add) and B = 62 on 64-bit words with
// 128-bit sums (a 64-bit host CPU's form; on a GB300 it took 1.2 to 1.6 times
// the 30-bit form's time, a binary GCD 1.6 to 4.6 times).
//
// GB300, 30-bit form: a lone thread inverts in 19.4 us (Fr) and 33.3 us (Fq); 34.5
// and 57.1 us one divstep at a time with d and e reduced after each batch.  One per lane,
// 9728 warps: 0.65 and 1.18 ns (0.96 and 1.89).
#pragma once
#include <cstdint>

namespace pp {

template <typename L>
struct LimbTraits;
template <>
struct LimbTraits<int32_t> {
  using U = uint32_t;
  using A = int64_t;  // sums of limb products
  static constexpr int B = 30;
};
template <>
struct LimbTraits<int64_t> {
  using U = uint64_t;
  using A = __int128;
  static constexpr int B = 62;
};

template <typename L, int NL>
struct SLimbs {
  L l[NL];
};

// modulus in B-bit limbs and M^-1 mod 2^B
template <typename L, int NL>
struct ModulusB {
  L m[NL];
  typename LimbTraits<L>::U inv;
};

PP_HD int ctz_word(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __ffs((int)x) - 1;
#else
  return __builtin_ctz(x);
#endif
}
PP_HD int ctz_word(uint64_t x) {
#ifdef __CUDA_ARCH__
  return __ffsll((long long)x) - 1;
#else
  return __builtin_ctzll(x);
#endif
}

// ---- B divsteps on the low words.  Returns the updated D = delta - 1/2; T in u..r.
// A divstep with delta <= 0 keeps f and adds it to an odd g before halving, so up to
// 1/2 - delta = -D of them in a row come to one: g + w f with the w that clears the
// low bits, w = -g / f modulo a power of two; f (f^2 - 2) = -1 / f modulo 2^6 for odd
// f, since (f^2 - 1)^2 is a multiple of 64.  One with delta > 0 is an exchange
// (f, g) -> (g, -f), delta -> -delta, and such a step.
template <typename L>
PP_HD int divsteps_word(int D, typename LimbTraits<L>::U f0, typename LimbTraits<L>::U g0,
                        L &u_out, L &v_out, L &q_out, L &r_out) {
  using U = typename LimbTraits<L>::U;
  constexpr int B = LimbTraits<L>::B;
  U u = 1, v = 0, q = 0, r = 1;
  int left = B;
  for (;;) {
    const int z = ctz_word(g0 | ((U)~(U)0 << left));  // a run of zero bits, at most `left`
    g0 >>= z;
    u <<= z;
    v <<= z;
    D += z;
    left -= z;
    if (left == 0) break;
    if (D >= 0) {
      D = -D - 1;
      U t = f0;
      f0 = g0;
      g0 = 0 - t;
      t = u;
      u = q;
      q = 0 - t;
      t = v;
      v = r;
      r = 0 - t;
    }
    int bits = -D < left ? -D : left;
    if (bits > 6) bits = 6;
    const U w = (f0 * g0 * (f0 * f0 - 2)) & (((U)1 << bits) - 1);
    g0 += w * f0;
    q += w * u;
    r += w * v;
  }
  u_out = (L)u;
  v_out = (L)v;
  q_out = (L)q;
  r_out = (L)r;
  return D;
}

// [f, g] = T [f, g] / 2^B (exact)
template <typename L, int NL>
PP_HD void apply_fg(SLimbs<L, NL> &f, SLimbs<L, NL> &g, L u, L v, L q, L r) {
  using A = typename LimbTraits<L>::A;
  using U = typename LimbTraits<L>::U;
  constexpr int B = LimbTraits<L>::B;
  constexpr U MASK = ((U)1 << B) - 1;
  A cf = (A)u * f.l[0] + (A)v * g.l[0];
  A cg = (A)q * f.l[0] + (A)r * g.l[0];
  cf >>= B;
  cg >>= B;
#pragma unroll
  for (int i = 1; i < NL; ++i) {
    cf += (A)u * f.l[i] + (A)v * g.l[i];
    cg += (A)q * f.l[i] + (A)r * g.l[i];
    f.l[i - 1] = (L)((U)cf & MASK);
    g.l[i - 1] = (L)((U)cg & MASK);
    cf >>= B;
    cg >>= B;
  }
  f.l[NL - 1] = (L)cf;
  g.l[NL - 1] = (L)cg;
}

// x, or -x where neg is all ones, plus M where mask is all ones
template <typename L, int NL>
PP_HD void negate_add(SLimbs<L, NL> &x, L neg, L mask, const ModulusB<L, NL> &M) {
  using U = typename LimbTraits<L>::U;
  constexpr int B = LimbTraits<L>::B;
  constexpr U MASK = ((U)1 << B) - 1;
  L c = 0;
#pragma unroll
  for (int i = 0; i < NL; ++i) {
    c += ((x.l[i] ^ neg) - neg) + (M.m[i] & mask);
    if (i < NL - 1) {
      x.l[i] = (L)((U)c & MASK);
      c >>= B;
    } else {
      x.l[i] = c;
    }
  }
}

// [d, e] = T [d, e] / 2^B mod M, d and e in (-2M, M) before and after: with M added to
// negative ones u d + v e lies within 2^B M of 0 (|u| + |v| <= 2^B), and the multiple
// of M that clears the low B bits, taken in (-2^B M, 0], leaves (-2^(B+1) M, 2^B M).
template <typename L, int NL>
PP_HD void apply_de(SLimbs<L, NL> &d, SLimbs<L, NL> &e, L u, L v, L q, L r,
                    const ModulusB<L, NL> &M) {
  using A = typename LimbTraits<L>::A;
  using U = typename LimbTraits<L>::U;
  constexpr int B = LimbTraits<L>::B;
  constexpr U MASK = ((U)1 << B) - 1;
  const L sd = d.l[NL - 1] < 0 ? -1 : 0, se = e.l[NL - 1] < 0 ? -1 : 0;
  A cd = (A)u * d.l[0] + (A)v * e.l[0];
  A ce = (A)q * d.l[0] + (A)r * e.l[0];
  L md = (u & sd) + (v & se), me = (q & sd) + (r & se);
  md -= (L)(((U)cd * M.inv + (U)md) & MASK);
  me -= (L)(((U)ce * M.inv + (U)me) & MASK);
  cd += (A)md * M.m[0];
  ce += (A)me * M.m[0];
  cd >>= B;
  ce >>= B;
#pragma unroll
  for (int i = 1; i < NL; ++i) {
    cd += (A)u * d.l[i] + (A)v * e.l[i] + (A)md * M.m[i];
    ce += (A)q * d.l[i] + (A)r * e.l[i] + (A)me * M.m[i];
    d.l[i - 1] = (L)((U)cd & MASK);
    e.l[i - 1] = (L)((U)ce & MASK);
    cd >>= B;
    ce >>= B;
  }
  d.l[NL - 1] = (L)cd;
  e.l[NL - 1] = (L)ce;
}

template <typename L, int NL>
PP_HD bool is_zero_limbs(const SLimbs<L, NL> &x) {
  L o = 0;
#pragma unroll
  for (int i = 0; i < NL; ++i) o |= x.l[i];
  return o == 0;
}

// x^-1 mod M for 0 <= x < M, M an odd prime; 0 -> 0.  max_batches bounds the
// loop: it must cover the divstep bound of the modulus's size (741 for
// 256-bit inputs, 1101 for 381-bit ones) in batches of B.  An input that does
// not finish within them (not below M) gives 0.
template <typename L, int NL>
PP_HD SLimbs<L, NL> modinv_divsteps(const SLimbs<L, NL> &x, const ModulusB<L, NL> &M,
                                    int max_batches) {
  using U = typename LimbTraits<L>::U;
  constexpr int B = LimbTraits<L>::B;
  SLimbs<L, NL> f, g, d, e;
#pragma unroll
  for (int i = 0; i < NL; ++i) {
    f.l[i] = M.m[i];
    g.l[i] = x.l[i];
    d.l[i] = 0;
    e.l[i] = 0;
  }
  e.l[0] = 1;
  if (is_zero_limbs(g)) return d;
  int D = 0;
  bool done = false;
  for (int b = 0; b < max_batches && !done; ++b) {
    L u, v, q, r;
    const U f0 = (U)f.l[0] | ((U)f.l[1] << B);
    const U g0 = (U)g.l[0] | ((U)g.l[1] << B);
    D = divsteps_word<L>(D, f0, g0, u, v, q, r);
    apply_fg(f, g, u, v, q, r);
    apply_de(d, e, u, v, q, r, M);
    done = is_zero_limbs(g);
  }
  if (!done) {
#pragma unroll
    for (int i = 0; i < NL; ++i) d.l[i] = 0;
    return d;
  }
  // f = +-1: x^-1 = +-d, d in (-2M, M)
  negate_add(d, (L)0, d.l[NL - 1] < 0 ? (L)-1 : (L)0, M);
  const L neg = f.l[NL - 1] < 0 ? (L)-1 : (L)0;
  negate_add(d, neg, (L)0, M);
  negate_add(d, (L)0, d.l[NL - 1] < 0 ? (L)-1 : (L)0, M);
  return d;
}

// 32-bit words <-> B-bit limbs (non-negative values)
template <typename L, int NW, int NL>
PP_HD SLimbs<L, NL> words_to_limbs(const uint32_t w[NW]) {
  using U = typename LimbTraits<L>::U;
  constexpr int B = LimbTraits<L>::B;
  constexpr int UB = 8 * (int)sizeof(U);
  SLimbs<L, NL> x;
#pragma unroll
  for (int i = 0; i < NL; ++i) {
    U acc = 0;
    const int bit = B * i;
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // a limb of at most 62 bits spans at most 3 words
      const int wi = bit / 32 + k;
      if (wi < NW) {
        const int sh = wi * 32 - bit;  // word wi's position within the limb
        const U wv = w[wi];
        if (sh >= 0) {
          if (sh < UB) acc |= wv << sh;
        } else {
          acc |= wv >> (-sh);
        }
      }
    }
    x.l[i] = (L)(acc & (((U)1 << B) - 1));
  }
  return x;
}

template <typename L, int NW, int NL>
PP_HD void limbs_to_words(const SLimbs<L, NL> &x, uint32_t w[NW]) {
  using U = typename LimbTraits<L>::U;
  constexpr int B = LimbTraits<L>::B;
#pragma unroll
  for (int k = 0; k < NW; ++k) {
    const int bit = 32 * k;
    const int li = bit / B, sh = bit % B;
    uint64_t v = (uint64_t)((U)x.l[li] >> sh);
    // bits of the next limb(s) above position B - sh
    if (li + 1 < NL && B - sh < 32) v |= (uint64_t)(U)x.l[li + 1] << (B - sh);
    if (li + 2 < NL && 2 * B - sh < 32) v |= (uint64_t)(U)x.l[li + 2] << (2 * B - sh);
    w[k] = (uint32_t)v;
  }
}

}  // namespace pp
