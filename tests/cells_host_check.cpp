// Host-side check of the carry-chained field multiplies (csrc/fr.cuh,
// csrc/fq.cuh): products, squares and lazy products against the row forms,
// which fr_host_check and g1_host_check hold against the oracle, and the
// four-part constant multiply and the small multiples against their definitions.  Operands are
// random and built from limbs 0, 1, 2^32 - 1 and 2^32 - 2, which reach the
// carry links that random limbs meet once in 2^32 products.  Built and run by tests/test_cells_host.py.
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
    const uint32_t edge[4] = {0u, 0xffffffffu, 1u, 0xfffffffeu};
    a.v[i] = kind == 0 ? r : kind == 1 ? edge[r & 3] : (r & 4 ? r : edge[r & 3]);
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

    // the four-part product: result 2^96 = sum of (64-bit part) w_p (mod r),
    // and below r + 2^-30 r
    fr w[4], sum = fr_zero(), p96 = fr_zero();
    p96.v[3] = 1;
    for (int p = 0; p < 4; ++p) {
      w[p] = operand<fr, 8>((it / 9 + p) % 3);
      w[p].v[7] &= 0x7fffffffu;
      fr_reduce_once(w[p].v);
      if (it == 2) w[p] = fr_sub(fr_zero(), fr_one());
      fr part = fr_zero();
      part.v[0] = wide.v[2 * p];
      part.v[1] = wide.v[2 * p + 1];
      sum = fr_add(sum, fr_mul_row9(fr_mul_row9(part, fr_rr()), w[p]));
    }
    const fr four = fr_mul_const4(wide, w);
    bad += four.v[7] > PP_R7 || !fr_eq(fr_mul_row9(fr_mul_row9(fr_canon(four), fr_rr()), p96), sum);

    // small multiples of a lazy value (below 2r): k x (mod r), below 1.002 r
    fr lazy = wide;
    lazy.v[7] %= 0xe7db4ea6u;
    if (it == 3) lazy = fr{{0x00000001u, 0xfffffffeu, 0xfffcb7fdu, 0xa77b4805u, 0x1343b00au, 0x6673b010u,
                            0x533afa90u, 0xe7db4ea6u}};  // 2r - 1
    const uint32_t k = it % 2 ? 2 + (uint32_t)(rng() % 255) : 256 - (uint32_t)(it % 7);
    const fr small = fr_mul_small(lazy, k);
    fr multiple = fr_zero();
    for (int bit = 8; bit >= 0; --bit) {
      multiple = fr_add(multiple, multiple);
      if ((k >> bit) & 1) multiple = fr_add(multiple, fr_canon(lazy));
    }
    bad += small.v[7] >= 0x74100000u || !fr_eq(fr_canon(small), multiple);
    // squares and products of lazy values stay lazy
    bad += !fr_eq(fr_canon(fr_sqr(lazy)), fr_mul_row9(fr_canon(lazy), fr_canon(lazy)));
    bad += !fr_eq(fr_canon(fr_mul_cells(lazy, lazy)), fr_mul_row9(fr_canon(lazy), fr_canon(lazy)));

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
