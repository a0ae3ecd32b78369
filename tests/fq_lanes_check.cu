// Checks the products over spread elements (csrc/fq_lanes.cuh) against fq_mul, on
// random operands and on operands built from limbs 0, 1, 2^32 - 1 and 2^32 - 2,
// whose carries random limbs meet once in 2^64 products; a value and its
// negative meet in a sum and a difference.  Built and run by
// tests/test_gpu_fq_lanes.py.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "../ppopp26-artifact_gb300/csrc/fq_lanes.cuh"

using namespace pp;

__device__ digit scatter(const Spread &s, const fq &a) {
  digit d = {0, 0, 0};
  for (uint32_t k = 0; k < kSpread; ++k)
    if (s.k == k) d.l = a.v[2 * k], d.h = a.v[2 * k + 1];
  return d;
}
__device__ fq gather(const digit &d, uint32_t el) {
  fq v;
  for (uint32_t k = 0; k < kSpread; ++k) {
    v.v[2 * k] = __shfl_sync(0xffffffffu, d.l, el * kSpread + k);
    v.v[2 * k + 1] = __shfl_sync(0xffffffffu, d.h, el * kSpread + k);
  }
  return fq_mul(v, fq_one());
}

// one warp: elements 5 w .. 5 w + 4 of the operands, canonical values
__global__ void check(const fq *a, const fq *b, unsigned long long *bad) {
  const Spread s;
  const uint32_t el = s.lane / kSpread < 5 ? s.lane / kSpread : 4;
  const uint64_t i = (uint64_t)blockIdx.x * 5 + el;
  const digit x = scatter(s, a[i]), y = scatter(s, b[i]);
  const digit p = s.norm(s.mul(x, y));
  const digit sum = s.norm(Spread::add(x, y));                                        // < 2 q
  const digit dif = s.norm(Spread::sub(Spread::add(x, s.multiple(1)), y));            // < 2 q
  const digit red = s.norm(s.reduce(Spread::sub(Spread::add(Spread::add(sum, sum), s.multiple(2)), dif)));
  const digit big = s.norm(s.mul(sum, s.norm(Spread::add(dif, dif))));                // 2 q by 4 q
  for (uint32_t e = 0; e < 5; ++e) {
    const fq u = a[(uint64_t)blockIdx.x * 5 + e], v = b[(uint64_t)blockIdx.x * 5 + e];
    const fq g[5] = {gather(p, e), gather(sum, e), gather(dif, e), gather(red, e), gather(big, e)};
    const uint32_t top = __shfl_sync(0xffffffffu, red.h, e * kSpread + kSpread - 1);
    if (s.lane) continue;
    const fq ws = fq_add(u, v), wd = fq_sub(u, v);
    const fq want[5] = {fq_mul(u, v), ws, wd, fq_sub(fq_dbl(ws), wd), fq_mul(ws, fq_dbl(wd))};
    for (int k = 0; k < 5; ++k)
      if (!fq_eq(g[k], want[k])) atomicAdd(bad, 1ull);
    if (top > (uint32_t)(1.03 * PP_Q11)) atomicAdd(bad, 1ull);  // reduce's bound
  }
}

int main() {
  const uint64_t n = 5 * 40000;
  std::mt19937_64 rng(11);
  std::vector<fq> a(n), b(n);
  const uint32_t edge[4] = {0u, 0xffffffffu, 1u, 0xfffffffeu};
  for (uint64_t i = 0; i < n; ++i)
    for (fq *x : {&a[i], &b[i]}) {
      const uint64_t kind = x == &a[i] ? i % 3 : i / 3 % 4;
      for (int w = 0; w < 12; ++w) {
        const uint32_t r = (uint32_t)rng();
        x->v[w] = kind == 0 ? r : kind == 1 ? edge[r & 3] : (r & 4 ? r : edge[r & 3]);
      }
      x->v[11] &= 0x1fffffffu;
      fq_reduce_once(x->v);
      if (kind == 3) *x = i & 4 ? a[i] : fq_neg(a[i]);
    }
  a[0] = b[0] = fq_zero();
  a[1] = b[1] = fq_neg(fq_one());
  fq *da, *db;
  unsigned long long *dbad, bad = 1;
  if (cudaMalloc(&da, n * sizeof(fq)) || cudaMalloc(&db, n * sizeof(fq)) || cudaMalloc(&dbad, 8)) return 2;
  cudaMemcpy(da, a.data(), n * sizeof(fq), cudaMemcpyHostToDevice);
  cudaMemcpy(db, b.data(), n * sizeof(fq), cudaMemcpyHostToDevice);
  cudaMemset(dbad, 0, 8);
  check<<<(unsigned)(n / 5), 32>>>(da, db, dbad);
  if (cudaMemcpy(&bad, dbad, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  std::printf("checked %llu, mismatches %llu\n", (unsigned long long)n, bad);
  return bad ? 1 : 0;
}
