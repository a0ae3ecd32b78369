// scan.cu -- grand product (exclusive prefix product), evaluation and division
// by (X + c) as blocked scans.
//
// The reference runs these as lg N Hillis-Steele launches over the whole
// vector (mont_arithmetic.cu:165-212, :305-361): O(N log N) multiplies and
// HBM traffic, plus a <<<1,1>>> squaring launch per step for division.  Here
// each is two launches with O(N) multiplies and two passes over HBM:
//  1. every thread folds a contiguous chunk of K elements into one summary
//     (a product for the grand product; the value S_start for S_end = 0 of the
//     backward recurrence S_i = p_i + m*S_{i+1} behind both evaluation, m = x,
//     and division, m = -c); a block-wide scan over the 256 thread summaries
//     gives every thread its in-block carry and the block its summary
//     (evaluation needs only the summary);
//  2. every block folds the summaries of the blocks before it (grand product)
//     or after it (division) and each thread replays its chunk with the exact
//     carry; evaluation composes all block maps in one block.
// Field arithmetic is exact, so the grouping does not change any result.
#include <cuda.h>

#include "common.cuh"
#include "ntt.cuh"
#include "scan.cuh"

#include <mutex>

namespace pp {

// Blocks per SM each operator's geometry aims for (scan_geom): longer chunks
// cut the summaries to scan, more blocks hide more latency.  Swept over 1, 2,
// 3 and 4 on GB300 (us at 2^20 / 2^22 / 2^24): division 2 (58 / 139 / 453; with the
// general maps before it 77 / 170 / 529, 1: 72 / 171 / 559, 4: 115 / 207 / 546).
// Evaluation has its own geometry (k_eval_tree), and so has the permutation product
// (k_perm_local).
constexpr uint32_t kGpBlocksPerSm = 2, kDivBlocksPerSm = 2;
// The grand product's chains grow with n while its block trees do not: us with
// 2 / 3 / 4 blocks per SM at 2^20 57.4 / 57.4 / 65.6, at 2^22 159.5 / 156.1 /
// 162.0, at 2^24 563 / 547 / 545.
inline uint32_t gp_blocks_per_sm(uint64_t n) {
  return n <= (1ull << 21) ? kGpBlocksPerSm : n <= (1ull << 23) ? 3 : 4;
}

// ---------------------------------------------------------------- helpers
__device__ __forceinline__ void sts_fr(fr *p, const fr &v) { st_fr(p, v); }

// Block scans are work-efficient (Blelloch, "Prefix sums and their
// applications", 1990): an up-sweep and a down-sweep over a balanced tree,
// 2(n-1) combines for n = blockDim.x (a power of two) instead of the n log n
// of a Hillis-Steele or warp-shuffle scan -- each combine here is one or two
// field multiplies.  All blocks of these launches are resident at once, so
// the scans' multiply count, not their depth, is what they cost: warp-shuffle
// scans (9 dependent steps instead of 16) made the 2^20 grand product,
// evaluation and division 13-36 % slower on GB300.

// A warp's view of its 32 chunks (lane l owns the K contiguous elements from
// (gt0 + l) K): tiles of kTileElems elements per lane go through shared memory,
// so global accesses are whole 64-byte segments (a lane reading its own chunk
// touches 32 lines per instruction), and the next tile's cp.async copies run
// while this one is multiplied.  In-place kernels write their results into the
// tile and store it the same way: with plain accesses each load hits the line
// the previous iteration's store went to, and the replay loops ran 2 to 9x
// slower depending on how the compiler placed the two (carry-chained multiply,
// 2^20 / 2^24: grand product 189 / 2885 us with plain accesses, 57 / 547 us
// through the tiles; division 221 / 5686 us, 77 / 529 us).
constexpr uint32_t kTileElems = 2, kTileUnits = 32 * 2 * kTileElems;  // 16-byte units per tile

// 16 bytes, or 16 zero bytes when !valid (src is not read then)
__device__ __forceinline__ void cp_async16(uint4 *dst, const uint4 *src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

struct ChunkTiles {
  uint4 *buf;     // 2 tiles of this warp
  uint64_t base;  // first element of lane 0's chunk
  uint64_t n, k;
  uint32_t tiles;  // tiles per chunk

  __device__ __forceinline__ ChunkTiles(uint4 *sm, uint32_t warp, uint64_t gt0, uint64_t n_, uint64_t k_)
      : buf(sm + warp * 2 * kTileUnits), base(gt0 * k_), n(n_), k(k_),
        tiles((uint32_t)((k_ + kTileElems - 1) / kTileElems)) {}

  // unit p of row r: conflict-free for a lane's own row and for whole segments
  static __device__ __forceinline__ uint32_t at(uint32_t r, uint32_t p) {
    return r * 4 + (p ^ ((r >> 1) & 3));
  }
  // element of unit u of tile t; n when it lies past the chunk or the vector
  // (its tile slot reads as zero and is not stored)
  __device__ __forceinline__ uint64_t elem(uint32_t u, uint32_t t) const {
    const uint64_t off = (uint64_t)t * kTileElems + ((u & 3) >> 1);
    const uint64_t i = base + (u >> 2) * k + off;
    return off < k && i < n ? i : n;
  }
  __device__ __forceinline__ void load(const fr *p, uint32_t t, uint32_t slot) const {
    const uint32_t lane = threadIdx.x & 31;
    uint4 *s = buf + slot * kTileUnits;
#pragma unroll
    for (uint32_t q = 0; q < kTileUnits / 32; ++q) {
      const uint32_t u = q * 32 + lane;
      const uint64_t i = elem(u, t);
      const bool valid = i < n;
      cp_async16(s + at(u >> 2, u & 3), reinterpret_cast<const uint4 *>(p + (valid ? i : 0)) + (u & 1), valid);
    }
  }
  __device__ __forceinline__ void store(fr *p, uint32_t t, uint32_t slot) const {
    const uint32_t lane = threadIdx.x & 31;
    const uint4 *s = buf + slot * kTileUnits;
#pragma unroll
    for (uint32_t q = 0; q < kTileUnits / 32; ++q) {
      const uint32_t u = q * 32 + lane;
      const uint64_t i = elem(u, t);
      if (i < n) reinterpret_cast<uint4 *>(p + i)[u & 1] = s[at(u >> 2, u & 3)];
    }
  }
  // element e of this lane's row of the tile in `slot`
  __device__ __forceinline__ fr get(uint32_t slot, uint32_t e) const {
    const uint4 *s = buf + slot * kTileUnits;
    const uint32_t lane = threadIdx.x & 31;
    const uint4 a = s[at(lane, 2 * e)], b = s[at(lane, 2 * e + 1)];
    return fr{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
  }
  __device__ __forceinline__ void put(uint32_t slot, uint32_t e, const fr &v) const {
    uint4 *s = buf + slot * kTileUnits;
    const uint32_t lane = threadIdx.x & 31;
    s[at(lane, 2 * e)] = make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]);
    s[at(lane, 2 * e + 1)] = make_uint4(v.v[4], v.v[5], v.v[6], v.v[7]);
  }

  // body(step, tile, slot) for steps 0 .. tiles-1 in the order tile_of(step);
  // with out, the tile is stored there after its body
  template <typename Order, typename Body>
  __device__ __forceinline__ void run(const fr *in, fr *out, Order tile_of, Body body) const {
    load(in, tile_of(0u), 0);
    cp_async_commit();
#pragma unroll 1
    for (uint32_t s = 0; s < tiles; ++s) {
      if (s + 1 < tiles) load(in, tile_of(s + 1), (s + 1) & 1);
      cp_async_commit();
      cp_async_wait<1>();  // this step's tile has landed
      __syncwarp();
      const uint32_t t = tile_of(s);
      body(s, t, s & 1);
      __syncwarp();
      if (out) {
        store(out, t, s & 1);
        __syncwarp();
      }
    }
  }
};
constexpr uint32_t kTileSmemUnits = (kScanThreads / 32) * 2 * kTileUnits;  // 32 KiB
static_assert(kTileSmemUnits * sizeof(uint4) >= 2 * kScanThreads * sizeof(fr),
              "the block scans reuse the tiles' shared memory");

// sum p[lo + i] x^i over this lane's chunk (lo = its first element; elements
// past the vector read as zero) from pw[k] = x^k, k <= 16, in shared memory: groups of
// 16 coefficients are dot products with one reduction each (fr_mac17 /
// fr_redc17), joined by Horner steps with x^16.  Whole warps only.
__device__ __forceinline__ fr chunk_dot(const ChunkTiles &ct, const fr *p, const fr *pw) {
  constexpr uint32_t TG = 16 / kTileElems;  // tiles per group
  const uint32_t ng = (ct.tiles + TG - 1) / TG, top = ct.tiles - (ng - 1) * TG;
  fr L = fr_zero();
  uint32_t acc[17];
#pragma unroll
  for (int k = 0; k < 17; ++k) acc[k] = 0;
  // groups from the top down, the tiles of a group upwards
  const auto order = [&](uint32_t s) {
    return s < top ? (ng - 1) * TG + s : (ng - 2 - (s - top) / TG) * TG + (s - top) % TG;
  };
  ct.run(p, nullptr, order, [&](uint32_t, uint32_t t, uint32_t slot) {
    const uint32_t e0 = (t % TG) * kTileElems;
#pragma unroll
    for (uint32_t e = 0; e < kTileElems; ++e)
      fr_mac17(acc, ct.get(slot, e), lds_fr(pw + e0 + e));
    if (t % TG == TG - 1 || t == ct.tiles - 1) {  // the group's last tile
      const fr S = fr_redc17(acc);
      L = t / TG == ng - 1 ? S : fr_add(fr_mul(L, lds_fr(pw + 16)), S);
#pragma unroll
      for (int k = 0; k < 17; ++k) acc[k] = 0;
    }
  });
  return L;
}

// pw[k] = x^k, k <= 16, by the 32 lanes of one warp: four doubling steps
// (lanes 2^j < k <= 2^(j+1) take x^(k - 2^j) x^(2^j)); lanes 0..16 store
__device__ __forceinline__ void warp_power_table17(const fr &x, fr *pw) {
  const uint32_t lane = threadIdx.x & 31;
  fr v = lane == 0 ? fr_one() : x;
#pragma unroll 1
  for (uint32_t h = 1; h <= 8; h <<= 1) {
    fr lowv, hv;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      lowv.v[w] = __shfl_sync(0xffffffffu, v.v[w], (int)(lane >= h ? lane - h : 0));
      hv.v[w] = __shfl_sync(0xffffffffu, v.v[w], (int)h);
    }
    if (lane > h && lane <= 2 * h) v = fr_mul(lowv, hv);
  }
  if (lane <= 16) sts_fr(pw + lane, v);
}

// Exclusive prefix product over a block of 256 threads (commutative): returns
// the product of the v of the threads before this one; *total receives the
// product of all.  A work-efficient up-sweep over the lowest three tree levels
// leaves the products of the 32 runs of 8; one warp scans those with shuffles
// (5 steps), and a three-level down-sweep hands the run prefixes back down.  11
// dependent multiplies against 17 for the full up- and down-sweep: the block
// scan is latency-bound (few threads multiply at each level).
__device__ __forceinline__ fr shfl_up_fr(const fr &v, int o) {
  fr r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = __shfl_up_sync(0xffffffffu, v.v[i], o);
  return r;
}

__device__ fr block_exclusive_product(const fr &v, fr *s, fr *total) {
  const uint32_t t = threadIdx.x;
  static_assert(kScanThreads == 256, "32 runs of 8");
  sts_fr(s + t, v);
  __syncthreads();
#pragma unroll 1
  for (uint32_t d = 1; d < 8; d <<= 1) {
    const uint32_t idx = (t + 1) * 2 * d - 1;
    if (idx < 256) sts_fr(s + idx, fr_mul(lds_fr(s + idx - d), lds_fr(s + idx)));
    __syncthreads();
  }
  if (t < 32) {
    fr inc = lds_fr(s + 8 * t + 7);
#pragma unroll 1
    for (int o = 1; o < 32; o <<= 1) {
      const fr u = shfl_up_fr(inc, o);
      if ((int)t >= o) inc = fr_mul(u, inc);
    }
    const fr ex = shfl_up_fr(inc, 1);
    sts_fr(s + 8 * t + 7, t ? ex : fr_one());
    if (t == 31) sts_fr(total, inc);
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t d = 4; d >= 1; d >>= 1) {
    const uint32_t idx = (t + 1) * 2 * d - 1;
    if (idx < 256) {
      const fr left = lds_fr(s + idx - d), before = lds_fr(s + idx);
      sts_fr(s + idx - d, before);
      sts_fr(s + idx, fr_mul(before, left));
    }
    __syncthreads();
  }
  return lds_fr(s + t);
}

// Two scans over a block of 256 threads at once: afterwards s1[t] is the product
// of the a of the threads before t and s2[255 - t] the product of the b of the
// threads after t; total[0] and total[1] hold the products of all a and all b.
// Half of the threads work on each array: three up-sweep levels, one warp
// scanning the 32 run products, three down-sweep levels, as
// block_exclusive_product: 38 warp-wide multiplies for both scans, 11 deep.  Two
// warp-shuffle (Kogge-Stone) scans took 100, 9 deep, a quarter of the
// permutation product's multiplies.
__device__ void block_scan_pair(const fr &a, const fr &b, fr *s1, fr *s2, fr *total) {
  static_assert(kScanThreads == 256, "32 runs of 8");
  const uint32_t t = threadIdx.x, h = t & 127;
  fr *s = t < 128 ? s1 : s2;
  sts_fr(s1 + t, a);
  sts_fr(s2 + 255 - t, b);
  __syncthreads();
#pragma unroll 1
  for (uint32_t d = 1; d < 8; d <<= 1) {
    const uint32_t idx = (h + 1) * 2 * d - 1;
    if (idx < 256) sts_fr(s + idx, fr_mul(lds_fr(s + idx - d), lds_fr(s + idx)));
    __syncthreads();
  }
  if (h < 32) {
    fr inc = lds_fr(s + 8 * h + 7);
#pragma unroll 1
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const fr u = shfl_up_fr(inc, o);
      if (h >= o) inc = fr_mul(u, inc);
    }
    const fr ex = shfl_up_fr(inc, 1);
    sts_fr(s + 8 * h + 7, h ? ex : fr_one());
    if (h == 31) sts_fr(total + (t >> 7), inc);
  }
  __syncthreads();
#pragma unroll 1
  for (uint32_t d = 4; d >= 1; d >>= 1) {
    const uint32_t idx = (h + 1) * 2 * d - 1;
    if (idx < 256) {
      const fr left = lds_fr(s + idx - d), before = lds_fr(s + idx);
      sts_fr(s + idx - d, before);
      sts_fr(s + idx, fr_mul(before, left));
    }
    __syncthreads();
  }
}

// Composition of affine maps f_t(x) = a_t + b_t x over the block: afterwards thread
// 0's (a, b) and sa[0], sb[0] hold f_0 o f_1 o ... o f_255.  Reversed order
// u = 255 - t, where the running composition is G_u = g_u o G_{u-1}.
// NAMED: the block also has a helper warp past the first 256 threads that
// does not take part, so the threads synchronise on a named barrier instead of
// __syncthreads.
template <bool NAMED>
__device__ __forceinline__ void scan_sync() {
  if (NAMED) asm volatile("bar.sync 1, 256;" ::: "memory");
  else __syncthreads();
}

template <bool NAMED = false>
__device__ void block_affine_compose(fr &a, fr &b, fr *sa, fr *sb) {
  const int t = threadIdx.x, n = kScanThreads;
  const int u = n - 1 - t;
  sts_fr(sa + u, a);
  sts_fr(sb + u, b);
  scan_sync<NAMED>();
  // combine(left = earlier in u, right = later in u) = right o left
  for (int d = 1; d < n; d <<= 1) {
    const int idx = (t + 1) * 2 * d - 1;
    if (idx < n) {
      const fr la = lds_fr(sa + idx - d), lb = lds_fr(sb + idx - d), ra = lds_fr(sa + idx), rb = lds_fr(sb + idx);
      sts_fr(sa + idx, fr_add(ra, fr_mul(rb, la)));
      sts_fr(sb + idx, fr_mul(rb, lb));
    }
    scan_sync<NAMED>();
  }
  // sa[n-1], sb[n-1] = G_{n-1} = F_0
  if (t == 0) {
    a = lds_fr(sa + n - 1);
    b = lds_fr(sb + n - 1);
    sts_fr(sa, a);
    sts_fr(sb, b);
  }
  scan_sync<NAMED>();
}

// ------------------------------------------------------------ grand product
__device__ __forceinline__ void gp_local_body(const fr *__restrict__ in, const ScanGeom &g,
                                              fr *__restrict__ thread_excl,
                                              fr *__restrict__ block_total, uint32_t blk, uint4 *sm) {
  fr *s = reinterpret_cast<fr *>(sm);
  const uint64_t gt = blk * (uint64_t)kScanThreads + threadIdx.x;
  const ChunkTiles ct(sm, threadIdx.x >> 5, gt - (threadIdx.x & 31), g.n, g.k);
  // elements past the vector read as zero: only lanes after the last element
  // see those products, and nothing reads theirs
  fr p = fr_one();
  ct.run(in, nullptr, [](uint32_t st) { return st; }, [&](uint32_t, uint32_t t, uint32_t slot) {
#pragma unroll
    for (uint32_t e = 0; e < kTileElems; ++e)
      if (e == 0 || t * kTileElems + e < g.k) p = t + e ? fr_mul(p, ct.get(slot, e)) : ct.get(slot, e);
  });
  __syncthreads();
  // the tiles are free: the scan takes their first 8 KiB, the total what follows
  fr *total = s + kScanThreads;
  const fr excl = block_exclusive_product(p, s, total);
  if (gt < g.threads) st_fr(thread_excl + gt, excl);
  if (threadIdx.x == 0) st_fr(block_total + blk, lds_fr(total));
}

__global__ void __launch_bounds__(kScanThreads) k_gp_local(const fr *__restrict__ in, ScanGeom g,
                                                            fr *__restrict__ thread_excl,
                                                            fr *__restrict__ block_total) {
  __shared__ uint4 sm[kTileSmemUnits];
  gp_local_body(in, g, thread_excl, block_total, blockIdx.x, sm);
}

// out_excl[i] = prod_{j<i} in[j] and/or out_incl[i] = prod_{j<=i} in[j]; either
// output may be null or alias `in` (each element is read before it is written)
__device__ __forceinline__ void gp_apply_body(const fr *in, fr *out_excl, fr *out_incl,
                                              const ScanGeom &g, const fr *__restrict__ thread_excl,
                                              const fr *__restrict__ block_total, uint32_t blk,
                                              uint4 *sm) {
  // product of the totals of all earlier blocks
  fr *s = reinterpret_cast<fr *>(sm);
  fr p = fr_one();
  for (uint32_t b = threadIdx.x; b < blk; b += blockDim.x) p = fr_mul(p, ld_fr(block_total + b));
  sts_fr(s + threadIdx.x, p);
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sts_fr(s + threadIdx.x, fr_mul(lds_fr(s + threadIdx.x), lds_fr(s + threadIdx.x + o)));
    __syncthreads();
  }
  const fr block_prefix = lds_fr(s);
  __syncthreads();  // the tiles reuse s
  const uint64_t gt = blk * (uint64_t)kScanThreads + threadIdx.x;
  const uint64_t lo = gt * g.k;
  fr run = gt < g.threads ? fr_mul(block_prefix, ld_fr(thread_excl + gt)) : fr_one();
  const ChunkTiles ct(sm, threadIdx.x >> 5, gt - (threadIdx.x & 31), g.n, g.k);
  // the tile leaves with the exclusive products (or, without out_excl, the
  // inclusive ones); when both are wanted the lanes store the inclusive ones
  ct.run(in, out_excl ? out_excl : out_incl, [](uint32_t st) { return st; },
         [&](uint32_t, uint32_t t, uint32_t slot) {
#pragma unroll
           for (uint32_t e = 0; e < kTileElems; ++e) {
             const uint64_t i = (uint64_t)t * kTileElems + e;
             if (e == 0 || i < g.k) {
               const fr v = ct.get(slot, e);
               if (out_excl) ct.put(slot, e, run);
               run = fr_mul(run, v);
               if (!out_excl) ct.put(slot, e, run);
               else if (out_incl && lo + i < g.n) st_fr(out_incl + lo + i, run);
             }
           }
         });
}

__global__ void __launch_bounds__(kScanThreads) k_gp_apply(const fr *in, fr *out_excl, fr *out_incl,
                                                            ScanGeom g,
                                                            const fr *__restrict__ thread_excl,
                                                            const fr *__restrict__ block_total) {
  __shared__ uint4 sm[kTileSmemUnits];
  gp_apply_body(in, out_excl, out_incl, g, thread_excl, block_total, blockIdx.x, sm);
}

// Batched grand products: the blocks of all jobs are numbered consecutively
// (block_start = prefix sums); each block finds its job and runs the body.
__device__ __forceinline__ uint32_t find_job(const uint32_t *__restrict__ start, uint32_t count,
                                             uint32_t b) {
  uint32_t lo = 0, hi = count;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (start[mid] <= b) lo = mid;
    else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(kScanThreads) k_gp_local_batch(const GpBatchJob *__restrict__ jobs,
                                                                  const uint32_t *__restrict__ start,
                                                                  uint32_t count) {
  __shared__ uint4 sm[kTileSmemUnits];
  const uint32_t j = find_job(start, count, blockIdx.x);
  const GpBatchJob jb = jobs[j];
  gp_local_body(jb.in, jb.g, jb.thread_excl, jb.block_total, blockIdx.x - start[j], sm);
}

__global__ void __launch_bounds__(kScanThreads) k_gp_apply_batch(const GpBatchJob *__restrict__ jobs,
                                                                  const uint32_t *__restrict__ start,
                                                                  uint32_t count) {
  __shared__ uint4 sm[kTileSmemUnits];
  const uint32_t j = find_job(start, count, blockIdx.x);
  const GpBatchJob jb = jobs[j];
  gp_apply_body(jb.in, jb.out, nullptr, jb.g, jb.thread_excl, jb.block_total, blockIdx.x - start[j],
                sm);
}

int gp_batch_launch(const GpBatchJob *d_jobs, const uint32_t *d_block_start, uint32_t count,
                    uint32_t total_blocks, cudaStream_t stream) {
  if (!total_blocks) return PP_OK;
  k_gp_local_batch<<<total_blocks, kScanThreads, 0, stream>>>(d_jobs, d_block_start, count);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  k_gp_apply_batch<<<total_blocks, kScanThreads, 0, stream>>>(d_jobs, d_block_start, count);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}

struct PermArgs {
  const fr *w[3];
  const fr *sigma[3];
  const fr *params;     // beta, gamma, k1, k2, k3
  const fr *omega_pow;  // w^i, i < n
  fr *z;                // output; holds the in-block terms until the last pass
};

// Copy-constraint grand product z_i = prod_{j<i} num_j / den_j, computed as
//   z_i = (prod_{j<i} num_j) * (prod_{j>=i} den_j) / (prod_j den_j):
// a prefix product of the numerators and a suffix product of the
// denominators, both blocked scans, and one field inversion for the whole
// vector instead of one per block.  A zero denominator makes its ratio 0
// (num := 0, den := 1), the field-inverse-of-zero-is-zero convention.
//
// A block takes 1024 rows, 4 consecutive ones per thread.  Inside a block the
// term is q_i = (numerators of the block before i) (denominators of the block
// from i on), and z_i = q_i c_b with one factor c_b per block: the numerators
// of the earlier blocks times the denominators of the later ones over all of
// them.  So the first pass leaves one vector of terms (in z) and the last one
// multiplies it by a per-block constant; the vectors of numerators and
// denominators, and the two replays over them, are gone.
//
// Values are below 2r throughout (fr_mul of two such values is below 1.82 r,
// since 4 r^2 / 2^256 < 1.82 r); the last pass stores them canonical.  The
// products by beta and beta k_j take the four-part constant form.
//
// GB300, 2^20 rows, us: first pass / carry / last pass 257 / 55 / 110 with
// numerators and denominators kept in memory, 221 / 33 / 21 so (561 -> 285 per
// call with the general multiply's rows counted in; with an inversion 7 us longer 3, 4
// and 5 rows per thread took 293, 292 and 308, at 2^22 1029, 1002 and 1005).
constexpr uint32_t kPermRows = 4, kPermBlockRows = kPermRows * kScanThreads;
constexpr uint32_t kPermSlots = 2 * kPermRows * 2 * kScanThreads;  // 16-byte units: 64 KiB

// x k + w + gamma below 2r, from canonical w and gamma
__device__ __forceinline__ fr perm_factor(const fr &xk, const fr &w, const fr &gamma) {
  return fr_add_lazy(xk, fr_add_raw(w, gamma));
}

// Pass 1: the block's terms q_i into z, the block's products of numerators and
// of denominators.
__global__ void __launch_bounds__(kScanThreads, 2)
    k_perm_local(const PermArgs a, uint64_t n, fr *__restrict__ block_num, fr *__restrict__ block_den) {
  extern __shared__ uint4 slots[];
  __shared__ __align__(16) fr s1[kScanThreads], s2[kScanThreads];
  __shared__ __align__(16) fr s_total[2];
  __shared__ __align__(16) fr s_k[16];  // beta, beta k1, beta k2, beta k3 in four parts each
  const uint32_t t = threadIdx.x;
  if (t < 16) {
    fr k = ld_fr(a.params);
    if (t >> 2) k = fr_mul(k, ld_fr(a.params + 1 + (t >> 2)));
    sts_fr(s_k + t, fr_mul(k, fr_const4_factor(t & 3)));
  }
  __syncthreads();
  const auto slot = [&](uint32_t j) { return slots + j * 2 * kScanThreads + t; };
  const auto put = [&](uint32_t j, const fr &v) {
    slot(j)[0] = make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]);
    slot(j)[kScanThreads] = make_uint4(v.v[4], v.v[5], v.v[6], v.v[7]);
  };
  const auto get = [&](uint32_t j) {
    const uint4 u = slot(j)[0], v = slot(j)[kScanThreads];
    return fr{{u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w}};
  };
  const uint64_t row0 = (blockIdx.x * (uint64_t)kScanThreads + t) * kPermRows;
  fr N = fr_one(), D = fr_one();
#pragma unroll 1
  for (uint32_t j = 0; j < kPermRows; ++j) {
    const uint64_t i = row0 + j;
    put(j, N);  // numerators of this thread before row j
    fr den = fr_one();
    if (i < n) {
      const fr gamma = ld_fr(a.params + 1);
      const fr wi = ldcs_fr(a.omega_pow + i);
      fr x = ldcs_fr(a.w[0] + i);
      fr num = perm_factor(mul_shared_const(wi, s_k + 4), x, gamma);
      den = perm_factor(mul_shared_const(ldcs_fr(a.sigma[0] + i), s_k), x, gamma);
#pragma unroll 1
      for (uint32_t c = 1; c < 3; ++c) {
        x = ldcs_fr(a.w[c] + i);
        num = fr_mul(num, perm_factor(mul_shared_const(wi, s_k + 4 + 4 * c), x, gamma));
        den = fr_mul(den, perm_factor(mul_shared_const(ldcs_fr(a.sigma[c] + i), s_k), x, gamma));
      }
      if (fr_is_zero(fr_canon(den))) {
        num = fr_zero();
        den = fr_one();
      }
      N = j ? fr_mul(N, num) : num;
    }
    put(kPermRows + j, den);
  }
#pragma unroll 1
  for (uint32_t j = kPermRows; j-- > 0;) {
    D = j + 1 < kPermRows ? fr_mul(D, get(kPermRows + j)) : get(kPermRows + j);
    put(j, j ? fr_mul(get(j), D) : D);
  }
  block_scan_pair(N, D, s1, s2, s_total);
  const fr T = fr_mul(lds_fr(s1 + t), lds_fr(s2 + kScanThreads - 1 - t));
#pragma unroll 1
  for (uint32_t j = 0; j < kPermRows && row0 + j < n; ++j) st_fr(a.z + row0 + j, fr_mul(get(j), T));
  if (t == 0) {
    st_fr(block_num + blockIdx.x, lds_fr(s_total));
    st_fr(block_den + blockIdx.x, lds_fr(s_total + 1));
  }
}

// Pass 2, one block of two halves: in place, block_num[b] := the product of the
// numerators of the blocks before b (first half of the threads), block_den[b]
// := the product of the denominators of the blocks after b, divided by all
// denominators (second half, over the blocks in reverse).
__global__ void __launch_bounds__(2 * kScanThreads) k_perm_carry(fr *block_num, fr *block_den, uint32_t nb) {
  __shared__ __align__(16) fr sw[2][kScanThreads / 32];
  __shared__ __align__(16) fr s_inv;
  const uint32_t half = threadIdx.x / kScanThreads, t = threadIdx.x % kScanThreads;
  const uint32_t lane = t & 31, w = t >> 5;
  constexpr uint32_t nw = kScanThreads / 32;
  fr *v = half ? block_den : block_num;
  const auto at = [&](uint32_t l) { return half ? nb - 1 - l : l; };
  const uint32_t per = (nb + kScanThreads - 1) / kScanThreads;
  const uint32_t lo = t * per < nb ? t * per : nb, hi = lo + per < nb ? lo + per : nb;
  fr P = fr_one();
  for (uint32_t l = lo; l < hi; ++l) P = l > lo ? fr_mul(P, ld_fr(v + at(l))) : ld_fr(v + at(l));
  // inclusive scan of the half's 256 products
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const fr u = shfl_up_fr(P, o);
    if (lane >= o) P = fr_mul(u, P);
  }
  if (lane == 31) sts_fr(&sw[half][w], P);
  __syncthreads();
  if (w == 0) {
    fr x = lane < nw ? lds_fr(&sw[half][lane]) : fr_one();
    for (uint32_t o = 1; o < nw; o <<= 1) {
      const fr u = shfl_up_fr(x, o);
      if (lane >= o) x = fr_mul(u, x);
    }
    if (lane < nw) sts_fr(&sw[half][lane], x);
  }
  __syncthreads();
  // one inversion for the vector (no denominator is zero), beside the
  // numerators' half, which does not need it
  if (threadIdx.x == kScanThreads) sts_fr(&s_inv, fr_inv_fast(fr_canon(lds_fr(&sw[1][nw - 1]))));
  fr run = shfl_up_fr(P, 1);
  if (lane == 0) run = w ? lds_fr(&sw[half][w - 1]) : fr_one();
  else if (w) run = fr_mul(run, lds_fr(&sw[half][w - 1]));
  if (half) {
    asm volatile("bar.sync 1, 256;" ::: "memory");  // the second half: s_inv is there
    run = fr_mul(run, lds_fr(&s_inv));
  }
  for (uint32_t l = lo; l < hi; ++l) {
    const fr x = ld_fr(v + at(l));
    st_fr(v + at(l), run);
    if (l + 1 < hi) run = fr_mul(run, x);
  }
}

// Pass 3: z_i = q_i c_b
__global__ void __launch_bounds__(kScanThreads)
    k_perm_apply(fr *z, uint64_t n, const fr *__restrict__ block_num, const fr *__restrict__ block_den) {
  __shared__ __align__(16) fr s_c[4];
  if (threadIdx.x < 4) {
    const fr c = fr_mul(ld_fr(block_num + blockIdx.x), ld_fr(block_den + blockIdx.x));
    sts_fr(s_c + threadIdx.x, fr_mul(c, fr_const4_factor(threadIdx.x)));
  }
  __syncthreads();
  fr w[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) w[p] = lds_fr(s_c + p);
  const uint64_t i0 = blockIdx.x * (uint64_t)kPermBlockRows + threadIdx.x;
#pragma unroll 1
  for (uint32_t j = 0; j < kPermRows; ++j) {
    const uint64_t i = i0 + j * kScanThreads;
    if (i < n) st_fr(z + i, fr_canon(fr_mul_const4(ld_fr(z + i), w)));
  }
}

// --------------------------------------------- backward affine recurrence
// S_i = p_i + m * S_{i+1}: a thread's chunk [lo, hi) is the map
// S_lo = L + m^(hi-lo) * S_hi with L its Horner value.  m^K for the full
// chunk length K is shared by the block: only a shorter (last) chunk computes
// its own power.

// per-block map.  Launched with kScanThreads + 32 threads: the extra warp
// computes m^K while the others evaluate their chunks (chunk_dot, after the
// first warp's table of m^0 .. m^16), which do not need it.
__global__ void __launch_bounds__(kScanThreads + 32, 2) k_affine_local(const fr *__restrict__ p, ScanGeom g,
                                                                     const fr *__restrict__ m_ptr,
                                                                     fr *block_a, fr *block_b) {
  __shared__ uint4 sm[kTileSmemUnits];  // the chunks' tiles, then the scan
  fr *sa = reinterpret_cast<fr *>(sm), *sb = sa + kScanThreads;
  __shared__ fr s_mk;
  __shared__ __align__(16) fr s_pw[17];  // m^k, k <= 16, for the chunks' dot products
  const fr m = ld_fr(m_ptr);
  if (threadIdx.x >= kScanThreads) {
    if (threadIdx.x == kScanThreads) s_mk = fr_pow_u64(m, g.k);
    __syncthreads();
    return;  // the scan below synchronises the other 256 threads by name
  }
  if (threadIdx.x < 32) warp_power_table17(m, s_pw);
  asm volatile("bar.sync 1, 256;" ::: "memory");
  const uint64_t gt = blockIdx.x * (uint64_t)kScanThreads + threadIdx.x;
  const uint64_t lo = gt * g.k < g.n ? gt * g.k : g.n;
  const uint64_t hi = lo + g.k < g.n ? lo + g.k : g.n;
  const ChunkTiles ct(sm, threadIdx.x >> 5, gt - (threadIdx.x & 31), g.n, g.k);
  const fr L = chunk_dot(ct, p, s_pw);
  __syncthreads();  // m^K ready, tiles free
  fr a = L, b = hi - lo == g.k ? s_mk : hi > lo ? fr_pow_u64(m, hi - lo) : fr_one();
  block_affine_compose<true>(a, b, sa, sb);
  if (threadIdx.x == 0) {
    st_fr(block_a + blockIdx.x, a);
    st_fr(block_b + blockIdx.x, b);
  }
}

// ordered composition of the block maps [first, count) (from one block of
// threads); returns the composed map's a (the value applied to S = 0) and b.
__device__ void compose_blocks(const fr *block_a, const fr *block_b, uint32_t first,
                               uint32_t count, fr &A, fr &B, fr *sa, fr *sb) {
  const uint32_t span = count > first ? count - first : 0;
  const uint32_t per = (span + blockDim.x - 1) / blockDim.x;
  const uint32_t lo = first + threadIdx.x * per;
  const uint32_t hi = lo + per < count ? lo + per : count;
  // sequential composition over [lo, hi): f_lo o ... o f_{hi-1}
  fr a = fr_zero(), b = fr_one();
  for (uint32_t i = hi; i > lo; --i) {  // prepend f_{i-1}
    const fr ai = ld_fr(block_a + i - 1), bi = ld_fr(block_b + i - 1);
    a = fr_add(ai, fr_mul(bi, a));
    b = fr_mul(bi, b);
  }
  block_affine_compose(a, b, sa, sb);
  A = lds_fr(sa);
  B = lds_fr(sb);
}

// Division: every S.  The vector counts as padded with zeros to whole chunks and
// blocks (S = 0 past its end), so each chunk's map is x -> L + q x with the same
// q = m^K and each block's x -> A + Q x, Q = q^256: a combine of two neighbours is one
// multiply by a known power instead of two, and a sum over all later blocks is a
// weighted sum without a chain.  us at 2^20 / 2^22 / 2^24: 77 / 170 / 529 with general
// maps (two multiplies per combine, 24 and 18 deep), 58 / 139 / 453 so.
// Powers, by the helper warp beside the chunks; block 0 leaves them for the apply:
struct DivPowers {
  fr q[33];     // q^a
  fr q32[9];    // q^(32 b)
  fr Q[33];     // Q^a
  fr Q32[17];   // Q^(32 b): up to 512 blocks
};
// pw[k] = x^k for k <= 2^steps (at most 32), by the lanes of one warp
__device__ __forceinline__ void warp_powers(const fr &x, uint32_t steps, fr *pw) {
  const uint32_t lane = threadIdx.x & 31;
  // lane l makes x^(l + 1): in step h lanes h .. 2h - 1 take x^(l + 1 - h) x^h
  fr v = x;
#pragma unroll 1
  for (uint32_t h = 1; h < 1u << steps; h <<= 1) {
    fr low, hv;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      low.v[w] = __shfl_sync(0xffffffffu, v.v[w], (int)(lane >= h ? lane - h : 0));
      hv.v[w] = __shfl_sync(0xffffffffu, v.v[w], (int)h - 1);
    }
    if (lane >= h && lane < 2 * h) v = fr_mul(low, hv);
  }
  if (lane < 1u << steps) sts_fr(pw + lane + 1, v);
  if (lane == 0) sts_fr(pw, fr_one());
  __syncwarp();
}

__device__ __forceinline__ fr shfl_down_fr(const fr &v, int o) {
  fr r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = __shfl_down_sync(0xffffffffu, v.v[i], o);
  return r;
}

// thread_s[t] = S at the end of thread t's chunk if it is 0 at the end of its block,
// block_s[b] = S at the start of block b likewise
__global__ void __launch_bounds__(kScanThreads + 32, 2)
    k_div_local(const fr *__restrict__ p, ScanGeom g, const fr *__restrict__ c_ptr, fr *thread_s, fr *block_s,
                DivPowers *powers) {
  __shared__ uint4 sm[kTileSmemUnits];
  __shared__ __align__(16) fr s_pw[17];  // m^k, k <= 16, for the chunks' dot products
  __shared__ __align__(16) fr s_q[33], s_q32[9], s_Q[33], s_Q32[17], s_warp[kScanThreads / 32];
  const fr m = fr_neg(ld_fr(c_ptr));
  if (threadIdx.x >= kScanThreads) {
    warp_powers(fr_pow_u64(m, g.k), 5, s_q);
    warp_powers(lds_fr(s_q + 32), 3, s_q32);
    __syncthreads();
    if (blockIdx.x == 0) {
      const uint32_t lane = threadIdx.x & 31;
      warp_powers(lds_fr(s_q32 + 8), 5, s_Q);
      warp_powers(lds_fr(s_Q + 32), 4, s_Q32);
      for (uint32_t i = lane; i < 33; i += 32) {
        st_fr(powers->q + i, lds_fr(s_q + i));
        st_fr(powers->Q + i, lds_fr(s_Q + i));
      }
      if (lane < 9) st_fr(powers->q32 + lane, lds_fr(s_q32 + lane));
      if (lane < 17) st_fr(powers->Q32 + lane, lds_fr(s_Q32 + lane));
    }
    return;
  }
  if (threadIdx.x < 32) warp_power_table17(m, s_pw);
  asm volatile("bar.sync 1, 256;" ::: "memory");
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t gt = blockIdx.x * (uint64_t)kScanThreads + threadIdx.x;
  const ChunkTiles ct(sm, warp, gt - lane, g.n, g.k);
  fr I = chunk_dot(ct, p, s_pw);
  __syncthreads();  // the powers are there
  // I = S at the lane's start if 0 at the warp's end
#pragma unroll 1
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const fr next = shfl_down_fr(I, o);
    if (lane + o < 32) I = fr_add(I, fr_mul(next, lds_fr(s_q + o)));
  }
  if (lane == 0) sts_fr(s_warp + warp, I);
  asm volatile("bar.sync 1, 256;" ::: "memory");
  // the same over the warps, by every warp
  constexpr uint32_t nw = kScanThreads / 32;
  fr W = lds_fr(s_warp + (lane & (nw - 1)));
#pragma unroll 1
  for (uint32_t o = 1; o < nw; o <<= 1) {
    const fr next = shfl_down_fr(W, o);
    if ((lane & (nw - 1)) + o < nw) W = fr_add(W, fr_mul(next, lds_fr(s_q32 + o)));
  }
  fr C;  // at this warp's end
#pragma unroll
  for (int w = 0; w < 8; ++w) C.v[w] = __shfl_sync(0xffffffffu, W.v[w], warp + 1 < nw ? warp + 1 : 0);
  if (warp + 1 == nw) C = fr_zero();
  const fr after = shfl_down_fr(I, 1);
  const fr S = fr_mul(C, lds_fr(s_q + 31 - lane));
  if (gt < g.threads) st_fr(thread_s + gt, lane == 31 ? S : fr_add(after, S));
  if (threadIdx.x == 0) st_fr(block_s + blockIdx.x, W);
}

// The exact S at the block's end, then at the chunk's, then the chunk replayed: m as
// a four-part constant.  The product is canonical, so S, its unreduced sum with a
// coefficient, is below 2r as fr_canon needs.
__global__ void __launch_bounds__(kScanThreads, 2)
    k_div_apply(fr *inout, ScanGeom g, const fr *__restrict__ c_ptr, const fr *__restrict__ thread_s,
                const fr *__restrict__ block_s, const DivPowers *__restrict__ powers) {
  __shared__ uint4 sm[kTileSmemUnits];
  __shared__ __align__(16) fr s_m[4], s_warp[kScanThreads / 32];
  const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t < 4) sts_fr(s_m + t, fr_mul(fr_neg(ld_fr(c_ptr)), fr_const4_factor(t)));
  // sum over the later blocks b of block_s[b] Q^(b - this - 1)
  fr sum = fr_zero();
  for (uint32_t j = t; blockIdx.x + 1 + j < g.blocks; j += kScanThreads) {
    const fr w = fr_mul(ldg_fr(powers->Q + (j & 31)), ldg_fr(powers->Q32 + (j >> 5)));
    sum = fr_add(sum, fr_mul(w, ldg_fr(block_s + blockIdx.x + 1 + j)));
  }
#pragma unroll 1
  for (uint32_t o = 16; o > 0; o >>= 1) sum = fr_add(sum, shfl_down_fr(sum, o));
  if (lane == 0) sts_fr(s_warp + warp, sum);
  // q^(255 - t)
  const fr weight = fr_mul(ldg_fr(powers->q + 31 - lane), ldg_fr(powers->q32 + kScanThreads / 32 - 1 - warp));
  __syncthreads();
  fr end = lds_fr(s_warp);
#pragma unroll 1
  for (uint32_t w = 1; w < kScanThreads / 32; ++w) end = fr_add(end, lds_fr(s_warp + w));
  const uint64_t gt = blockIdx.x * (uint64_t)kScanThreads + t;
  // past the vector S = 0 and elements read as zero, so s stays 0 there
  fr s = gt < g.threads ? fr_add(ld_fr(thread_s + gt), fr_mul(weight, end)) : fr_zero();
  fr m[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) m[k] = lds_fr(s_m + k);
  const ChunkTiles ct(sm, warp, gt - lane, g.n, g.k);
  const uint32_t last = ct.tiles - 1;
  ct.run(inout, inout, [&](uint32_t st) { return last - st; }, [&](uint32_t, uint32_t tile, uint32_t slot) {
#pragma unroll
    for (int e = (int)kTileElems - 1; e >= 0; --e)
      if (e == 0 || tile * kTileElems + e < g.k) {
        const fr pi = ct.get(slot, e);
        ct.put(slot, e, fr_canon(s));  // q_i = S_(i+1)
        s = fr_add_raw(pi, fr_mul_const4<false>(s, m));
      }
  });
}

__global__ void __launch_bounds__(kScanThreads) k_eval_final(const fr *__restrict__ block_a,
                                                              const fr *__restrict__ block_b,
                                                              uint32_t count, fr *y) {
  __shared__ __align__(16) fr sa[kScanThreads], sb[kScanThreads];
  fr A, B;
  compose_blocks(block_a, block_b, 0, count, A, B, sa, sb);
  if (threadIdx.x == 0) st_fr(y, A);
}

// ------------------------------------------------------------ evaluation
// y = sum_i p_i x^i in one launch.
//  * Thread t of block b takes the K contiguous coefficients from (256 b + t) K
//    and evaluates them: L = sum_{i<K} p_{(256 b + t) K + i} x^i, as dot
//    products of groups of 16 coefficients with x^0 .. x^15 (one reduction per
//    group, chunk_dot) joined by Horner steps with x^16.  The first Horner warp
//    builds x^0 .. x^16 first.  K is chosen as for the other scans (scan_geom;
//    blocks per SM below).
//  * Its term is L x^(K t) x^(256 K b).  Thread weights come from two 16-entry
//    tables, x^(K a) and x^(16 K a) for a < 16 (x^(K t) = one product of an
//    entry of each); the block's weight x^(256 K b) is one power.  Two helper
//    warps compute the tables and that power while the other eight run their
//    Horner chains.
//  * Weighted terms are summed with field additions (warp shuffles, then the
//    warps' sums); the block stores its sum times its weight, and the block
//    that finishes last (a ticket counter) adds the block sums into y.
// After the chains, a thread does two multiplies; every other step is an
// addition.  A binary fold of the same terms (L_u + x^(K s) L_(u+s)) needs
// eight dependent multiplies per block and as many more in the last block.
// The sum's grouping does not change the value: field addition is exact.
// Blocks per SM: 1 up to 2^21 coefficients, 2 above.  At 2^20 the helpers'
// powers (a chain of about 25 dependent multiplies, slowed by the Horner warps
// that share their SM) end after the chains, so fewer Horner warps per SM
// finish the block sooner (30.8 against 32.9 us); at 2^22 and 2^24 the chains
// are the longer part and two blocks per SM are faster (70.3 against 73.9 us,
// 223 against 246 us).
constexpr uint32_t kEvalBlocksPerSmSmall = 1, kEvalBlocksPerSm = 2;
constexpr uint64_t kEvalSmallMax = 1ull << 21;
constexpr uint32_t kEvalHelperWarps = 2;
// Horner threads per block (with the two helper warps on top).  128 per block
// (fewer Horner warps beside the helpers, twice the coefficients per thread)
// was slower: 37.9 against 35.5 us at 2^20, 85.2 against 82.8 us at 2^22.
constexpr uint32_t kEvalHorner = 256;

__device__ __forceinline__ fr ldcg_fr(const fr *p) {
  const uint4 *q = reinterpret_cast<const uint4 *>(p);
  uint4 a = __ldcg(q), b = __ldcg(q + 1);
  return fr{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}

__device__ __forceinline__ fr shfl_xor_fr(const fr &v, int o) {
  fr r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = __shfl_xor_sync(0xffffffffu, v.v[i], o);
  return r;
}

// sum over the 32 lanes of a warp (every lane gets it)
__device__ __forceinline__ fr warp_sum_fr(fr v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fr_add(v, shfl_xor_fr(v, o));
  return v;
}

template <uint32_t HT>
__global__ void __launch_bounds__(HT + 32 * kEvalHelperWarps)
    k_eval_tree(const fr *__restrict__ p, ScanGeom g, const fr *__restrict__ xp,
                fr *__restrict__ block_val, uint32_t *__restrict__ ticket, fr *__restrict__ y) {
  static_assert(HT % 32 == 0 && HT <= 256, "Horner threads: whole warps, at most 256");
  constexpr uint32_t kHelpers = 32 * kEvalHelperWarps, kWarps = HT / 32;
  __shared__ uint4 sm[kWarps * 2 * kTileUnits];
  __shared__ __align__(16) fr tab[32];  // tab[a] = x^(K a), tab[16 + a] = x^(16 K a), a < 16
  __shared__ fr s_wb;     // x^(HT K b)
  __shared__ __align__(16) fr s_pw[17]; // x^k, k <= 16, for the Horner threads' dot products
  __shared__ __align__(16) fr s_warp[kWarps];
  __shared__ uint32_t s_last;
  // warps 0 and 1 are the helpers
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t t = threadIdx.x - kHelpers, warp = t >> 5;  // Horner thread and warp
  const fr x = ld_fr(xp);
  fr L = fr_zero();
  if (threadIdx.x < 32) {
    // the tables: lane a < 16 raises x^K to a, lane 16 + a raises x^(16 K) to a
    const fr v = fr_pow_u64(x, g.k);
    fr u = v;
#pragma unroll 1
    for (int i = 0; i < 4; ++i) u = fr_sqr(u);
    sts_fr(tab + lane, fr_pow_u64(lane < 16 ? v : u, lane & 15));
  } else if (threadIdx.x < kHelpers) {
    // the block's weight: (x^(HT K))^b
    fr v = fr_pow_u64(x, g.k);
#pragma unroll 1
    for (uint32_t i = 1; i < HT; i <<= 1) v = fr_sqr(v);
    v = fr_pow_u64(v, blockIdx.x);
    if (lane == 0) s_wb = v;
  } else {
    // the first Horner warp builds x^0 .. x^16; the Horner threads wait for
    // it on a named barrier (the helper warps do not)
    if (warp == 0) warp_power_table17(x, s_pw);
    asm volatile("bar.sync 1, %0;" ::"n"(HT) : "memory");
    const ChunkTiles ct(sm, warp, (uint64_t)blockIdx.x * HT + t - lane, g.n, g.k);
    L = chunk_dot(ct, p, s_pw);
  }
  __syncthreads();  // the tables, the block weight and the chunk values are ready
  if (threadIdx.x >= kHelpers) {
    const fr w = fr_mul(lds_fr(tab + (t & 15)), lds_fr(tab + 16 + (t >> 4)));  // x^(K t)
    const fr sum = warp_sum_fr(fr_mul(L, w));
    if (lane == 0) sts_fr(s_warp + warp, sum);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    fr v = warp_sum_fr(lane < kWarps ? lds_fr(s_warp + lane) : fr_zero());
    if (lane == 0) {
      st_fr(block_val + blockIdx.x, fr_mul(v, s_wb));
      __threadfence();
      s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (!s_last) return;
  // the last block: y = the sum of the gridDim.x weighted block sums
  __threadfence();
  if (threadIdx.x >= kHelpers) {
    fr acc = fr_zero();
    for (uint32_t b = t; b < gridDim.x; b += HT) acc = fr_add(acc, ldcg_fr(block_val + b));
    acc = warp_sum_fr(acc);
    if (lane == 0) sts_fr(s_warp + warp, acc);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const fr v = warp_sum_fr(lane < kWarps ? lds_fr(s_warp + lane) : fr_zero());
    if (lane == 0) {
      st_fr(y, v);
      *ticket = 0;
    }
  }
}

__global__ void k_zero1(fr *y) { st_fr(y, fr_zero()); }

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static uint32_t perm_blocks(uint64_t n) { return (uint32_t)((n + kPermBlockRows - 1) / kPermBlockRows); }

// scan_geom's rule with kEvalHorner threads per block
static ScanGeom eval_geom(uint64_t n) {
  const uint32_t bps = n <= kEvalSmallMax ? kEvalBlocksPerSmSmall : kEvalBlocksPerSm;
  ScanGeom g;
  g.n = n;
  const uint64_t target = (uint64_t)device_sm_count() * bps * kEvalHorner;
  g.k = (n + target - 1) / target;
  if (g.k < 4) g.k = 4;
  g.threads = (n + g.k - 1) / g.k;
  g.blocks = (uint32_t)((g.threads + kEvalHorner - 1) / kEvalHorner);
  return g;
}

size_t gp_perm_workspace(uint64_t n) { return 2 * (size_t)perm_blocks(n) * sizeof(fr); }
size_t div_workspace(uint64_t n) {
  const ScanGeom g = scan_geom(n, kDivBlocksPerSm);
  return (g.threads + g.blocks) * sizeof(fr) + sizeof(DivPowers);
}
// block sums, then the ticket counter in a slot of its own
size_t eval_workspace(uint64_t n) { return ((size_t)eval_geom(n).blocks + 1) * sizeof(fr); }

}  // namespace pp

using pp::fr;

extern "C" int pp_gp_scan(const void *d_in, void *d_excl, void *d_incl, uint64_t n, void *stream) {
  if (n == 0) return PP_OK;
  if (!d_in || !pp::aligned16(d_in) || (d_excl && !pp::aligned16(d_excl)) ||
      (d_incl && !pp::aligned16(d_incl)) || (!d_excl && !d_incl)) {
    pp::set_error("pp_gp_scan: need a 16-byte aligned input and at least one aligned output");
    return PP_E_INVAL;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const pp::ScanGeom g = pp::scan_geom(n, pp::gp_blocks_per_sm(n));
  int st = PP_OK;
  fr *ws = static_cast<fr *>(
      pp::workspace_get((g.threads + g.blocks) * sizeof(fr), s, 1, &st));
  if (st) return st;
  fr *thread_excl = ws, *block_total = ws + g.threads;
  pp::k_gp_local<<<g.blocks, pp::kScanThreads, 0, s>>>(static_cast<const fr *>(d_in), g, thread_excl,
                                                       block_total);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  pp::k_gp_apply<<<g.blocks, pp::kScanThreads, 0, s>>>(
      static_cast<const fr *>(d_in), static_cast<fr *>(d_excl), static_cast<fr *>(d_incl), g,
      thread_excl, block_total);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}

extern "C" int pp_gp_prefix(void *d_inout, uint64_t n, void *stream) {
  if (n && (!d_inout || !pp::aligned16(d_inout))) {
    pp::set_error("pp_gp_prefix: buffer must be a 16-byte aligned device pointer");
    return PP_E_INVAL;
  }
  return pp_gp_scan(d_inout, d_inout, nullptr, n, stream);
}

extern "C" int pp_div_xplusc(void *d_inout, uint64_t n, const void *d_c, void *stream) {
  if (n == 0) return PP_OK;
  if (!d_inout || !d_c || !pp::aligned16(d_inout) || !pp::aligned16(d_c)) {
    pp::set_error("pp_div_xplusc: buffers must be 16-byte aligned device pointers");
    return PP_E_INVAL;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const pp::ScanGeom g = pp::scan_geom(n, pp::kDivBlocksPerSm);
  int st = PP_OK;
  static_assert(sizeof(pp::DivPowers) % sizeof(fr) == 0, "in whole elements");
  fr *ws = static_cast<fr *>(pp::workspace_get(pp::div_workspace(n), s, 1, &st));
  if (st) return st;
  fr *thread_s = ws, *block_s = ws + g.threads;
  pp::DivPowers *powers = reinterpret_cast<pp::DivPowers *>(block_s + g.blocks);
  const fr *c = static_cast<const fr *>(d_c);
  pp::k_div_local<<<g.blocks, pp::kScanThreads + 32, 0, s>>>(static_cast<const fr *>(d_inout), g, c,
                                                            thread_s, block_s, powers);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  pp::k_div_apply<<<g.blocks, pp::kScanThreads, 0, s>>>(static_cast<fr *>(d_inout), g, c, thread_s,
                                                        block_s, powers);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}

extern "C" int pp_eval(const void *d_poly, uint64_t n, const void *d_x, void *d_y, void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (!d_y || !pp::aligned16(d_y) || (n && (!d_poly || !d_x || !pp::aligned16(d_poly) ||
                                            !pp::aligned16(d_x)))) {
    pp::set_error("pp_eval: buffers must be 16-byte aligned device pointers");
    return PP_E_INVAL;
  }
  if (n == 0) {
    pp::k_zero1<<<1, 1, 0, s>>>(static_cast<fr *>(d_y));
    PP_COUNT_LAUNCH();
    PP_LAUNCH_CHECK();
    return PP_OK;
  }
  constexpr uint32_t HT = pp::kEvalHorner;
  const pp::ScanGeom g = pp::eval_geom(n);
  const uint32_t nb = g.blocks;
  int st = PP_OK;
  // block sums, then the ticket counter in its own 32-byte slot
  char *ws = static_cast<char *>(pp::workspace_get(pp::eval_workspace(n), s, 1, &st));
  if (st) return st;
  fr *block_val = reinterpret_cast<fr *>(ws);
  uint32_t *ticket = reinterpret_cast<uint32_t *>(ws + nb * sizeof(fr));
  PP_CUDA_TRY(cudaMemsetAsync(ticket, 0, sizeof(uint32_t), s));
  pp::k_eval_tree<HT><<<nb, HT + 32 * pp::kEvalHelperWarps, 0, s>>>(
      static_cast<const fr *>(d_poly), g, static_cast<const fr *>(d_x), block_val, ticket,
      static_cast<fr *>(d_y));
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}

extern "C" int pp_gp_perm(const void *const *d_w, const void *const *d_sigma, const void *d_params,
                          void *d_z, uint32_t lg_n, void *stream) {
  if (!d_w || !d_sigma || !d_params || !d_z || !pp::aligned16(d_params) || !pp::aligned16(d_z)) {
    pp::set_error("pp_gp_perm: null or misaligned pointer");
    return PP_E_INVAL;
  }
  for (int j = 0; j < 3; ++j) {
    if (!d_w[j] || !d_sigma[j] || !pp::aligned16(d_w[j]) || !pp::aligned16(d_sigma[j])) {
      pp::set_error("pp_gp_perm: null or misaligned wire/sigma pointer %d", j);
      return PP_E_INVAL;
    }
  }
  if (lg_n > PP_MAX_LG_N) {
    pp::set_error("pp_gp_perm: lg_n = %u too large", lg_n);
    return PP_E_UNSUPPORTED;
  }
  cudaStream_t s = (cudaStream_t)stream;
  const uint64_t n = 1ull << lg_n;
  const uint32_t nb = pp::perm_blocks(n);
  int st = PP_OK;
  const fr *omega_pow = pp::pow_table(pp::host_root_of_unity((int)lg_n, false), lg_n, &st);
  if (st) return st;
  fr *ws = static_cast<fr *>(pp::workspace_get(pp::gp_perm_workspace(n), s, 1, &st));
  if (st) return st;
  pp::PermArgs a;
  for (int j = 0; j < 3; ++j) {
    a.w[j] = static_cast<const fr *>(d_w[j]);
    a.sigma[j] = static_cast<const fr *>(d_sigma[j]);
  }
  a.params = static_cast<const fr *>(d_params);
  a.omega_pow = omega_pow;
  a.z = static_cast<fr *>(d_z);
  fr *block_num = ws, *block_den = ws + nb;
  constexpr size_t smem = pp::kPermSlots * sizeof(uint4);
  PP_CUDA_TRY(cudaFuncSetAttribute(pp::k_perm_local, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  pp::k_perm_local<<<nb, pp::kScanThreads, smem, s>>>(a, n, block_num, block_den);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  pp::k_perm_carry<<<1, 2 * pp::kScanThreads, 0, s>>>(block_num, block_den, nb);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  pp::k_perm_apply<<<nb, pp::kScanThreads, 0, s>>>(a.z, n, block_num, block_den);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}

// ---------------------------------------------------------------------------
// Evaluation that allocates nothing.
//
// pp_eval takes its block summaries from a per-stream workspace that is
// created with cudaMalloc on first use.  Some callers cannot allow that: a
// serving process that has handed all free device memory to its own pool
// (a fresh cudaMalloc would fail or fragment it), or a latency-critical loop
// where cudaMalloc / cudaFree may synchronise the whole device and stall the
// work of other streams.  For them pp_eval_noalloc keeps its scratch in a
// file-scope device array that exists, for every device that loads this
// library, from module load until process exit:
//   2 * 1024 block summaries of 32 bytes = 64 KiB per device.
// With 16 elements per thread and 256 threads per block that bounds the
// polynomial at 1024 * 256 * 16 = 2^22 coefficients; longer ones are refused
// with PP_E_UNSUPPORTED before any device work.
// ---------------------------------------------------------------------------
namespace pp {

constexpr uint32_t kEvalNoAllocMaxBlocks = 1024;
constexpr uint64_t kEvalNoAllocChunk = 16;
static_assert((uint64_t)kEvalNoAllocMaxBlocks * kScanThreads * kEvalNoAllocChunk == PP_EVAL_NOALLOC_MAX_N,
              "header limit and scratch geometry disagree");

// [0, 1024): affine-map offsets a_b of the blocks, [1024, 2048): factors b_b
static __device__ __align__(256) fr g_eval_noalloc_scratch[2 * kEvalNoAllocMaxBlocks];

// Device address of g_eval_noalloc_scratch per device, with the id of the CUDA
// context it was looked up in.  A device reset (cudaDeviceReset) destroys the
// primary context and the module with it; the next context loads the module
// again, possibly elsewhere, under a new context id.  So the cached address is
// used only while the calling thread's current context has the stored id, and
// looked up again otherwise.
struct NoAllocAddr {
  unsigned long long ctx_id = 0;
  fr *addr = nullptr;
};
static std::mutex g_eval_noalloc_mu;
static NoAllocAddr g_eval_noalloc_addr[64];

// Id of the calling thread's current CUDA context (cuCtxGetCurrent + cuCtxGetId,
// reached through the runtime's driver entry points so that the library does
// not link the driver library), or 0 when there is none or it cannot be read.
static unsigned long long current_context_id() {
  using GetCurrent = CUresult (*)(CUcontext *);
  using GetId = CUresult (*)(CUcontext, unsigned long long *);
  static GetCurrent get_current = nullptr;
  static GetId get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<GetCurrent>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<GetId>(f);
    cudaGetLastError();
  });
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx ||
      get_id(ctx, &id) != CUDA_SUCCESS)
    return 0;
  return id;
}

}  // namespace pp

extern "C" int pp_eval_noalloc(const void *d_poly, uint64_t n, const void *d_x, void *d_y,
                               void *stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (!d_y || !pp::aligned16(d_y) || (n && (!d_poly || !d_x || !pp::aligned16(d_poly) ||
                                            !pp::aligned16(d_x)))) {
    pp::set_error("pp_eval_noalloc: buffers must be 16-byte aligned device pointers");
    return PP_E_INVAL;
  }
  if (n > PP_EVAL_NOALLOC_MAX_N) {
    pp::set_error("pp_eval_noalloc: %llu coefficients exceed the 2^22 its static scratch covers; "
                  "use pp_eval",
                  (unsigned long long)n);
    return PP_E_UNSUPPORTED;
  }
  if (n == 0) {
    pp::k_zero1<<<1, 1, 0, s>>>(static_cast<fr *>(d_y));
    PP_COUNT_LAUNCH();
    PP_LAUNCH_CHECK();
    return PP_OK;
  }
  int dev = 0;
  PP_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    pp::set_error("pp_eval_noalloc: device index %d out of range", dev);
    return PP_E_INVAL;
  }
  fr *scratch = nullptr;
  {
    // set-up on the first call on this device (that device is current), and
    // again after its context changed: the host-side name of the array is not
    // a device address; ask the runtime
    std::lock_guard<std::mutex> lk(pp::g_eval_noalloc_mu);
    pp::NoAllocAddr &slot = pp::g_eval_noalloc_addr[dev];
    const unsigned long long ctx_id = pp::current_context_id();
    if (!slot.addr || ctx_id == 0 || slot.ctx_id != ctx_id) {
      void *p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, pp::g_eval_noalloc_scratch);
      if (e != cudaSuccess) {
        cudaGetLastError();
        pp::set_error("pp_eval_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        return PP_E_CUDA;
      }
      slot.addr = static_cast<fr *>(p);
      // the look-up makes the device's primary context current if none was
      slot.ctx_id = ctx_id ? ctx_id : pp::current_context_id();
    }
    scratch = slot.addr;
  }
  pp::ScanGeom g;
  g.n = n;
  g.k = pp::kEvalNoAllocChunk;
  g.threads = (n + g.k - 1) / g.k;
  g.blocks = (uint32_t)((g.threads + pp::kScanThreads - 1) / pp::kScanThreads);
  // every block summary read by k_eval_final is written by k_affine_local in
  // the same call, so nothing in the array has to be cleared first
  fr *ba = scratch, *bb = scratch + pp::kEvalNoAllocMaxBlocks;
  pp::k_affine_local<<<g.blocks, pp::kScanThreads + 32, 0, s>>>(
      static_cast<const fr *>(d_poly), g, static_cast<const fr *>(d_x), ba, bb);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  pp::k_eval_final<<<1, pp::kScanThreads, 0, s>>>(ba, bb, g.blocks, static_cast<fr *>(d_y));
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}
