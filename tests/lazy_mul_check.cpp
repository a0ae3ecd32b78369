// Host-side check of fr_mul's contract for two factors below 2r (csrc/fr.cuh): congruent
// to the canonical product and below 1.82 r.  Built and run by tests/test_lazy_mul_host.py.
#include <cstdio>
#include <random>

#include "../ppopp26-artifact_gb300/csrc/fr.cuh"

using namespace pp;

int main() {
  std::mt19937_64 rng(3);
  const fr two_r_less_1 = {{0x00000001u, 0xfffffffeu, 0xfffcb7fdu, 0xa77b4805u, 0x1343b00au, 0x6673b010u, 0x533afa90u,
                            0xe7db4ea6u}};
  long bad = 0;
  const long n = 200000;
  for (long it = 0; it < n; ++it) {
    fr x[2];
    for (fr &a : x) {
      for (int i = 0; i < 8; ++i) a.v[i] = (uint32_t)rng();
      a.v[7] %= 0xe7db4ea6u;  // below 2r
      if (rng() % 16 == 0) a = two_r_less_1;
    }
    const fr want = fr_mul_row9(fr_canon(x[0]), fr_canon(x[1])), got = fr_mul(x[0], x[1]);
    bad += !fr_eq(fr_canon(got), want) || got.v[7] > 0xd2fd545eu;  // 1.82 r's top word
    bad += !fr_eq(fr_mul(x[0], fr_canon(x[1])), want);
  }
  std::printf("checked %ld, mismatches %ld\n", n, bad);
  return bad ? 1 : 0;
}
