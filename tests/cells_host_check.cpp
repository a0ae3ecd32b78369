// Host-side check of the carry-chained field multiplies (csrc/fr.cuh,
// csrc/fq.cuh): products, squares and lazy products against the row forms,
// which fr_host_check and g1_host_check hold against the oracle.  Operands are
// random and built from all-ones and all-zero limbs, so every carry link is
// exercised.  Built and run by tests/test_cells_host.py.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../ppopp26-artifact_gb300/csrc/fq.cuh"

using namespace pp;

static std::mt19937_64 rng(7);

template <typename T, int N>
static T operand(int kind) {
  T a;
  for (int i = 0; i < N; ++i) {
    const uint32_t r = (uint32_t)rng();
    a.v[i] = kind == 0 ? r : kind == 1 ? (r & 1 ? 0xffffffffu : 0u) : (r & 3 ? r : 0xffffffffu);
  }
  return a;
}

int main(int argc, char **argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 100000;
  long bad = 0;
  for (long it = 0; it < n; ++it) {
    fr a = operand<fr, 8>(it % 3), b = operand<fr, 8>((it / 3) % 3);
    const fr wide = a;  // any 256-bit value: what the lazy multiply accepts
    a.v[7] &= 0x7fffffffu;
    b.v[7] &= 0x7fffffffu;
    fr_reduce_once(a.v);
    fr_reduce_once(b.v);
    if (it == 0) a = fr_zero();
    if (it == 1) b = a = fr_sub(fr_zero(), fr_one());
    const fr want = fr_mul_row9(a, b);
    bad += !fr_eq(fr_mul_cells(a, b), want);
    bad += !fr_eq(fr_sqr(a), fr_mul_row9(a, a));
    fr wc = fr_canon(fr_mul_row9<true>(wide, b));
    bad += !fr_eq(fr_canon(fr_mul_cells<true>(wide, b)), wc);

    fq x = operand<fq, 12>(it % 3), y = operand<fq, 12>((it / 3) % 3);
    x.v[11] &= 0x1fffffffu;
    y.v[11] &= 0x1fffffffu;
    fq_reduce_once(x.v);
    fq_reduce_once(y.v);
    if (it == 0) x = fq_zero();
    if (it == 1) x = y = fq_sub(fq_zero(), fq_one());
    bad += !fq_eq(fq_mul(x, y), fq_mul_rows<0, 0>(x, y));
    bad += !fq_eq(fq_sqr(x), fq_mul_rows<0, 0>(x, x));
  }
  std::printf("checked %ld, mismatches %ld\n", n, bad);
  return bad ? 1 : 0;
}
