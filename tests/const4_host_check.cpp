// Host-side check of the canonical four-part constant multiply (fr_mul_const4<false>,
// csrc/fr.cuh) and of the division's replay that relies on it: products equal fr_mul's
// and lie below r, also where the lazy form leaves r or a little more (multipliers whose
// low part sums vanish modulo 2^96, small states), and the state of the replay,
// coefficient plus product, stays below 2r.  Built and run by tests/test_const4_host.py.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../ppopp26-artifact_gb300/csrc/fr.cuh"

using namespace pp;

static std::mt19937_64 rng(5);

static fr small(uint64_t v) { return fr{{(uint32_t)v, (uint32_t)(v >> 32), 0, 0, 0, 0, 0, 0}}; }
static fr random_fr() {
  fr a;
  for (int i = 0; i < 8; ++i) a.v[i] = (uint32_t)rng();
  a.v[7] &= 0x7fffffffu;
  fr_reduce_once(a.v);
  return a;
}
// raw words near 0, near r, of few words or random
static fr edge() {
  const uint64_t k = rng() % 9;
  switch (rng() % 6) {
    case 0: return small(k);
    case 1: return fr_sub(fr_zero(), small(k));
    case 2: {  // one bit, or a run of them below it
      fr a = fr_zero();
      const uint32_t bit = rng() % 254;
      a.v[bit / 32] = 1u << (bit % 32);
      return k & 1 ? a : fr_sub(a, small(1));
    }
    case 3: {  // only the low words
      fr a = random_fr();
      for (uint32_t i = 1 + rng() % 7; i < 8; ++i) a.v[i] = 0;
      return a;
    }
    default: return random_fr();
  }
}
static bool below(const fr &a, const fr &b) {  // a < b
  for (int i = 7; i >= 0; --i)
    if (a.v[i] != b.v[i]) return a.v[i] < b.v[i];
  return false;
}

int main(int argc, char **argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 100000;
  const fr r = {{PP_R0, PP_R1, PP_R2, PP_R3, PP_R4, PP_R5, PP_R6, PP_R7}};
  const fr two_r = fr_add_raw(r, r);
  const fr half = fr_inv(fr_add(fr_one(), fr_one()));
  // raw words of a shift c for which a state of 2^63 times -c leaves more than r
  const fr found = {{0x7c31db70u, 0x9740630cu, 0xfd27b6a3u, 0xfb947fc7u, 0x4df03793u, 0xedd0f968u, 0x4d011e3cu,
                     0x6b3587f0u}};
  long bad = 0;
  for (long it = 0; it < n; ++it) {
    fr m = fr_zero();  // Montgomery form: small integers and their halves, edges, random
    const int kind = it % 4;
    if (kind == 0) {
      for (uint64_t k = rng() % 200; k > 0; --k) m = fr_add(m, fr_one());
      if (rng() & 1) m = fr_mul(m, half);
      if (rng() & 1) m = fr_sub(fr_zero(), m);
    } else {
      m = kind == 1 ? edge() : kind == 2 ? random_fr() : fr_sub(fr_zero(), found);
    }
    fr w[4];
    for (int p = 0; p < 4; ++p) w[p] = fr_mul(m, fr_const4_factor(p));
    fr s = fr_zero(), want = fr_zero();
    for (int step = 0; step < 12; ++step) {
      bad += !fr_eq(fr_canon(s), want) || !below(fr_canon(s), r);
      const fr prod = fr_mul_const4<false>(s, w);
      bad += !fr_eq(prod, fr_mul(want, m)) || !below(prod, r);
      bad += !below(fr_mul_const4(s, w), two_r);
      const fr c = edge();
      s = fr_add_raw(c, prod);
      want = fr_add(c, fr_mul(want, m));
      bad += !below(s, two_r);
    }
  }
  std::printf("checked %ld, mismatches %ld\n", n, bad);
  return bad ? 1 : 0;
}
