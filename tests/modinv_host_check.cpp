// Host-side check of the divstep inversion (csrc/modinv.cuh) at both limb widths:
//  * a batch's matrix and delta equal those of single divsteps, from every kind of state
//    a batch can start in (odd f; g odd, even, zero in its low bits; delta of both signs);
//  * the 2-adic quotient at every width up to its ten bits;
//  * inverses of both fields against the binary GCD, for random values, values whose
//    first divisions are long (M modulo high powers of two), near 0 and near M.
// Built and run by tests/test_modinv_host.py.
#include <cstdio>
#include <random>

#include "../ppopp26-artifact_gb300/csrc/fq.cuh"

using namespace pp;

static std::mt19937_64 rng(9);

// one divstep at a time, from the definition, with delta = D + 1/2
template <typename L>
static int single_steps(int D, typename LimbTraits<L>::U f, typename LimbTraits<L>::U g, DivMatrix<L> &T) {
  using U = typename LimbTraits<L>::U;
  U u = 1, v = 0, q = 0, r = 1;
  for (int i = 0; i < LimbTraits<L>::B; ++i) {
    if (D >= 0 && (g & 1)) {  // (1 - delta, g, (g - f) / 2)
      const U of = f, ou = u, ov = v;
      f = g, u = 2 * q, v = 2 * r;
      g = (g - of) >> 1, q = q - ou, r = r - ov;
      D = -D;  // 1 - (D + 1/2) = -D + 1/2
    } else {
      if (g & 1) g += f, q += u, r += v;
      g >>= 1, u *= 2, v *= 2;
      D += 1;
    }
  }
  T = {(L)u, (L)v, (L)q, (L)r};
  return D;
}

template <typename L>
static long check_batches(long n) {
  using U = typename LimbTraits<L>::U;
  long bad = 0;
  for (long it = 0; it < n; ++it) {
    const U f = (U)rng() | 1;
    U g = (U)rng();
    if (it % 4 == 1) g <<= rng() % LimbTraits<L>::B;
    if (it % 4 == 2) g = f * (U)(rng() % 64) + ((U)(rng() & 1) << (rng() % (8 * sizeof(U))));
    if (it % 64 == 3) g = 0;
    const int D = (int)(rng() % 81) - 40;
    DivMatrix<L> a, b;
    int Da = D;
    divide_batch<L>(Da, f, g, a);
    const int Db = single_steps<L>(D, f, g, b);
    bad += Da != Db || a.u != b.u || a.v != b.v || a.q != b.q || a.r != b.r;
    for (int bits = 1; bits <= LimbTraits<L>::B; ++bits) {  // ten of them at most
      const U w = quotient_mod2<U>(g, f, bits), mask = ((U)1 << (bits < 10 ? bits : 10)) - 1;
      bad += w > mask || ((w * f - g) & mask) != 0;
    }
  }
  return bad;
}

int main() {
  long bad = check_batches<int32_t>(20000) + check_batches<int64_t>(20000);
  const uint32_t r[8] = {PP_R0, PP_R1, PP_R2, PP_R3, PP_R4, PP_R5, PP_R6, PP_R7};
  const uint32_t q[12] = {PP_Q0, PP_Q1, PP_Q2, PP_Q3, PP_Q4, PP_Q5, PP_Q6, PP_Q7, PP_Q8, PP_Q9, PP_Q10, PP_Q11};
  for (long it = 0; it < 6000; ++it) {
    fr x = fr_zero();
    fq y = fq_zero();
    const uint32_t kind = it % 4, cut = 1 + rng() % 254, cutq = 1 + rng() % 380;
    for (int i = 0; i < 8; ++i) x.v[i] = kind == 0 ? (uint32_t)rng() : r[i];
    for (int i = 0; i < 12; ++i) y.v[i] = kind == 0 ? (uint32_t)rng() : q[i];
    // kinds 1 and 2: the modulus with its upper bits changed, or only its lower bits
    for (uint32_t b = cut; kind > 0 && kind < 3 && b < 255; ++b)
      if (kind == 2 || (rng() & 1)) x.v[b / 32] &= ~(1u << (b % 32));
    for (uint32_t b = cutq; kind > 0 && kind < 3 && b < 381; ++b)
      if (kind == 2 || (rng() & 1)) y.v[b / 32] &= ~(1u << (b % 32));
    if (kind == 3) {  // near 0 and near the modulus, and single bits
      x = fr_zero(), y = fq_zero();
      x.v[0] = y.v[0] = (uint32_t)(rng() % 5);
      if (rng() & 1) x.v[cut / 32] = 1u << (cut % 32), y.v[cutq / 32] = 1u << (cutq % 32);
      if (x.v[7] == 0x40000000u) x.v[7] = 0x20000000u;
      if (rng() & 1) x = fr_neg(x), y = fq_neg(y);
    }
    x.v[7] &= 0x7fffffffu;
    y.v[11] &= 0x1fffffffu;
    fr_reduce_once(x.v);
    fq_reduce_once(y.v);
    const fr ix = fr_inv_binary(x);
    bad += !fr_eq(fr_inv_divsteps<int32_t>(x), ix) || !fr_eq(fr_inv_divsteps<int64_t>(x), ix);
    bad += !fr_is_zero(x) && !fr_eq(fr_mul(x, ix), fr_one());
    const fq iy = fq_inv(y);
    bad += !fq_eq(fq_inv_divsteps<int32_t>(y), iy) || !fq_eq(fq_inv_divsteps<int64_t>(y), iy);
    bad += !fq_is_zero(y) && !fq_eq(fq_mul(y, iy), fq_one());
  }
  std::printf("mismatches %ld\n", bad);
  return bad ? 1 : 0;
}
