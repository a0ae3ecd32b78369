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
// Steps in a row are divisions.  After an exchange at delta the next steps keep f, and
// the first delta + 1/2 of them (with delta at a half) add f to g or not, as g is odd
// or even, and halve it: together they add the w f, 0 <= w < 2^(delta + 1/2), that makes
// g divisible by 2^(delta + 1/2), so
//   (f, g) -> (g, w g - f),  w = f / g (mod 2^(delta + 1/2)),  and g's zero bits go;
// as g then has at least that many of them, delta is positive again and the next
// division follows.  A division is three multiply-adds (f and g, and the two columns of
// their coefficients), however many steps it stands for.
//
// B divsteps depend only on the low B + 2 bits of f and g, so they run on
// one machine word each and record a 2x2 integer matrix T with
// 2^B [f', g'] = T [f, g]; |u| + |v| <= 2^B and |q| + |r| <= 2^B.  T is then
// applied to the full f, g (the division by 2^B is exact) and to the pair
// d, e with f = d x, g = e x (mod M), where the division by 2^B is done mod
// M by first adding the multiple of M that clears the low B bits.  That multiple is
// taken from [-2^(B-1), 2^(B-1)) M, so a batch adds at most M / 2 to the larger of |d|
// and |e|: they stay below (1 + batches / 2) M and are not reduced until the end.
//
// Numbers are NL limbs of B bits, least significant first; limbs below the
// top one are in [0, 2^B) and the top limb carries the sign.  Two widths:
// B = 30 on 32-bit words with 64-bit sums (the GPU form: every limb product
// is one 32 x 32 -> 64-bit multiply-add) and B = 62 on 64-bit words with
// 128-bit sums (a 64-bit host CPU's form; on a GB300 it took 1.2 to 1.6 times
// the 30-bit form's time, a binary GCD 1.6 to 4.6 times).
//
// GB300, 30-bit form: a lone thread that only inverts takes 20.0 us (Fr) and 34.6 us
// (Fq), 32 lanes with a value each 28.4 and 47.1; the lone thread took 34.5 and 57.1 us
// one divstep at a time with d and e reduced after each batch.
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

// a b + s; on the device one instruction, whatever the compiler makes of the sum.  For the
// products by T, not for those by M's limbs, which are constants: the permutation product
// of 2^13 rows, half of it the inversion, takes 66.9 us so, 69.2 with no product and 72.4
// with all of them written like this.
PP_HD int64_t mad_limbs(int32_t a, int32_t b, int64_t s) {
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(s));
  return r;
#else
  return (int64_t)a * b + s;
#endif
}
PP_HD __int128 mad_limbs(int64_t a, int64_t b, __int128 s) { return (__int128)a * b + s; }

// B divsteps as a matrix: f' = (u f + v g) / 2^B, g' = (q f + r g) / 2^B
template <typename L>
struct DivMatrix {
  L u, v, q, r;
};

// x / y modulo 2^bits, or 2^10 where that is less; y odd.  3 y with its second bit
// flipped is 1 / y modulo 2^5 (P. Montgomery's start), one of Newton's steps makes that
// ten bits.  Longer quotients are rare: a branch for them costs each division more (lone
// thread 22.3 against 18.5 us, with products by M's limbs as mad_limbs) than finishing
// them in a second piece.
template <typename U>
PP_HD U quotient_mod2(U x, U y, int bits) {
  const U inv = (3 * y) ^ 2;
  return (x * inv) * (2 - y * inv) & (((U)1 << (bits < 10 ? bits : 10)) - 1);
}

// ---- B divsteps on the low words; D is delta - 1/2
template <typename L>
PP_HD void divide_batch(int &D, typename LimbTraits<L>::U f, typename LimbTraits<L>::U g, DivMatrix<L> &T) {
  using U = typename LimbTraits<L>::U;
  // f and g are fF F + fG G and gF F + gG G over a power of two, F and G the words given
  U fF = 1, fG = 0, gF = 0, gG = 1;
  int left = LimbTraits<L>::B;
  for (;;) {
    // g's zero bits, at most `left` of them
    const int zeros = ctz_word(g | (U)1 << left);
    g >>= zeros;
    fF <<= zeros;
    fG <<= zeros;
    D += zeros;
    left -= zeros;
    if (left == 0) break;
    // the next division, (f, g) -> (g, w g - f); or, with D < 0, the rest of a long one
    // or of one that the batch before began, (f, g) -> (f, w f + g)
    const bool next = D >= 0;
    const U b = next ? 0 - f : g, bF = next ? 0 - fF : gF, bG = next ? 0 - fG : gG;
    f = next ? g : f, fF = next ? gF : fF, fG = next ? gG : fG;
    D = next ? -1 - D : D;
    const U w = quotient_mod2<U>(0 - b, f, -D < left ? -D : left);
    g = w * f + b;
    gF = w * fF + bF;
    gG = w * fG + bG;
  }
  T = {(L)fF, (L)fG, (L)gF, (L)gG};
}

// [x, y] = T [x, y] / 2^B: exact (f and g), or modulo M.  A limb's products are summed
// before the carry joins them, so the chain along the limbs is two additions a limb.
template <bool EXACT, typename L, int NL>
PP_HD void apply_batch(SLimbs<L, NL> &x, SLimbs<L, NL> &y, const DivMatrix<L> &T, const ModulusB<L, NL> &M) {
  using A = typename LimbTraits<L>::A;
  using U = typename LimbTraits<L>::U;
  constexpr int B = LimbTraits<L>::B, PAD = 8 * (int)sizeof(U) - B;
  constexpr U MASK = ((U)1 << B) - 1;
  A sx = (A)T.u * x.l[0] + (A)T.v * y.l[0], sy = (A)T.q * x.l[0] + (A)T.r * y.l[0];
  L mx = 0, my = 0;  // multiples of M
  if (!EXACT) {
    mx = (L)((0 - (U)sx * M.inv) << PAD) >> PAD;
    my = (L)((0 - (U)sy * M.inv) << PAD) >> PAD;
    sx += (A)mx * M.m[0];
    sy += (A)my * M.m[0];
  }
#pragma unroll
  for (int i = 1; i < NL; ++i) {
    A px = mad_limbs(T.v, y.l[i], mad_limbs(T.u, x.l[i], 0)), py = mad_limbs(T.r, y.l[i], mad_limbs(T.q, x.l[i], 0));
    if (!EXACT) {
      px += (A)mx * M.m[i];
      py += (A)my * M.m[i];
    }
    sx = (sx >> B) + px;
    sy = (sy >> B) + py;
    x.l[i - 1] = (L)((U)sx & MASK);
    y.l[i - 1] = (L)((U)sy & MASK);
  }
  sx >>= B;
  sy >>= B;
  x.l[NL - 1] = (L)sx;
  y.l[NL - 1] = (L)sy;
}

// sign x modulo M, in [0, 5/4 M), for |x| < 20 M and sign = 1 or -1.  The multiple of M
// comes from the top limbs: t is at most sign x / 2^s and less than 2 below it (1 where
// sign is 1), M / 2^s lies between the modulus's top limb and one more, and the quotient
// is rounded down towards the side where nothing is taken too often.  What is left is
// below 1 + 22 / (top limb) times M, and the smallest top limb is 115.
template <typename L, int NL>
PP_HD void reduce_once_signed(SLimbs<L, NL> &x, L sign, const ModulusB<L, NL> &M) {
  using A = typename LimbTraits<L>::A;
  using U = typename LimbTraits<L>::U;
  constexpr int B = LimbTraits<L>::B;
  constexpr U MASK = ((U)1 << B) - 1;
  const L top = M.m[NL - 1], t = sign < 0 ? -1 - x.l[NL - 1] : x.l[NL - 1];
  const L k = t < 0 ? -((top - 1 - t) / top) : t / (top + 1);
  A c = 0;
#pragma unroll
  for (int i = 0; i < NL; ++i) {
    c += (A)sign * x.l[i] - (A)k * M.m[i];
    if (i < NL - 1) {
      x.l[i] = (L)((U)c & MASK);
      c >>= B;
    } else {
      x.l[i] = (L)c;
    }
  }
}

template <typename L, int NL>
PP_HD bool is_zero_limbs(const SLimbs<L, NL> &x) {
  L o = 0;
#pragma unroll
  for (int i = 0; i < NL; ++i) o |= x.l[i];
  return o == 0;
}

// x^-1 mod M, in [0, 5/4 M), for 0 <= x < M, M an odd prime; 0 -> 0.  The loop ends
// when g is 0; max_batches (at most 38) only stops an input that is not below M, which
// then gives 0, and covers the divstep bound of the modulus's size.
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
    DivMatrix<L> T;
    divide_batch<L>(D, (U)f.l[0] | ((U)f.l[1] << B), (U)g.l[0] | ((U)g.l[1] << B), T);
    apply_batch<true>(f, g, T, M);
    apply_batch<false>(d, e, T, M);
    done = is_zero_limbs(g);
  }
  if (!done) {
#pragma unroll
    for (int i = 0; i < NL; ++i) d.l[i] = 0;
    return d;
  }
  // f = +-1: x^-1 = +-d
  reduce_once_signed(d, f.l[NL - 1] < 0 ? (L)-1 : (L)1, M);
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
