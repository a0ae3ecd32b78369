// msm.cu -- BLS12-381 G1 multi-scalar multiplication sum_i s_i P_i on the
// GPU (Pippenger's bucket method with signed digits).
//
// Replaces multi_scalar_mult (PLONK/utils/function.cu:395-411) ->
// cuda::msm_zkp_cuda (PLONK/utils/zkp/cuda/zksnark_msm.cu:48-88, sppark's
// Pippenger with mont = false) + cpu::msm_collect_cpu (zkp/cpu/
// msmcollect.cpp): same inputs (affine points over Fq in Montgomery form,
// scalars as plain 256-bit integers), one Jacobian point out, with the final
// aggregation on the GPU instead of the host.
//
// Pipeline (all on one stream, workspace slot 3):
//   1. digits    one thread per scalar: c-bit windows recoded to signed
//                digits in [-2^(c-1), 2^(c-1)], bucket |d| - 1 per window
//                (W = floor(256 / c) + 1 windows, so any 256-bit scalar is
//                exact); bucket sizes counted with warp-aggregated atomics
//   2. scan      exclusive prefix sum of the W * 2^(c-1) bucket sizes (tiled)
//   3. scatter   (point index, sign) into each bucket's slice: a counting sort
//   4. pairs     while buckets are large, rounds of affine pair sums with shared
//                inversions (k_msm_pairs) halve every bucket's entries
//   5. buckets   the sorted list is cut into equal runs of K entries, one thread
//                each, whatever the bucket sizes: a thread writes the buckets
//                that lie inside its run and leaves a partial sum for the one
//                it shares with the run before and the one after.  A second
//                launch joins each shared bucket's partial sums (one thread
//                for a few, blocks for many: a bucket can hold up to all n
//                points: equal scalars, or the few-bit top window)
//   6. segments  one thread (or two lanes) per run of G buckets: running sums T =
//                sum (j + 1) B and R = sum B over its run
//   7. windows   sum T + G sum_s s R_s with sum_s s R_s = sum_k 2^k Q_k, Q_k
//                the R_s whose index has bit k set: plain sums in chunks, the
//                chunks a warp to an addition, then one warp per window for the Horner
//                chain over k
//   8. final     one warp: Horner over the windows (c doublings each, the
//                independent multiplies of each step on different lanes), one
//                inversion to affine
// Every step is integer-multiply bound (an Fq multiply is ~300 32-bit wide
// products) except the sort, which is a few bytes per point and window.
#include <atomic>
#include <cstring>

#include "common.cuh"
#include "fq_lanes.cuh"
#include "g1.cuh"

namespace pp {
namespace {

constexpr uint32_t kNone = 0xffffffffu;

struct MsmPlan {
  uint32_t c;      // window bits
  uint32_t W;      // windows: W c >= 257, so the top window's carry has a home
  uint32_t B;      // buckets per bucket set, 2^(c-1)
  uint32_t G;      // buckets per aggregation segment
  uint32_t S;      // segments per bucket set, B / G
  uint32_t lgG;    // log2 G
  uint32_t lgS;    // log2 S
  uint32_t chunk;  // terms per thread of the window sums (k_msm_bitsums)
  uint32_t nsets;  // bucket sets: W (one per window), or 1 with window tables
};

// Buckets per segment: the longest run (fewer, cheaper window sums) that still
// gives 2^15 segment threads.  On GB300 this beat fixed 4, 8 and 16 (2^16
// points: 16 -> 4.65 ms, 4 -> 3.92 ms; 2^22: 4 -> 53.2 ms, 16 -> 51.3 ms).
constexpr uint32_t kSegmentMax = 16, kSegmentMin = 4, kSegmentThreads = 1u << 15;
// Segments of four buckets take two lanes each (k_msm_segments4) while those make no
// more than one warp per SM sub-partition (152 SMs, four each): 8192 segments 101 ->
// 74 us, but 20480 segments 131 -> 141.
constexpr uint32_t kPairedLanes = 152 * 128;

// Terms per thread of the window sums (k_msm_bitsums): 8, and 4 where that leaves the
// chip less than full.  With one set of 2^15 buckets 4 terms take 56 us and 8 terms 117.
constexpr uint32_t kChunkMax = 8, kChunkThreads = 1u << 14;

// the rest of a plan once c and the number of bucket sets are fixed
MsmPlan msm_plan_for(uint32_t c, uint32_t nsets) {
  MsmPlan p{};
  p.c = c;
  p.W = 256 / c + 1;
  p.B = 1u << (c - 1);
  p.nsets = nsets;
  p.G = kSegmentMax;  // B >= 32 (c >= 6)
  while (p.G > kSegmentMin && (uint64_t)p.nsets * p.B / p.G < kSegmentThreads) p.G >>= 1;
  p.S = p.B / p.G;
  while ((1u << p.lgG) < p.G) ++p.lgG;
  while ((1u << p.lgS) < p.S) ++p.lgS;
  p.chunk = kChunkMax;
  if ((uint64_t)nsets * (2 + p.lgS) * p.S / (2 * kChunkMax) <= kChunkThreads) p.chunk /= 2;
  return p;
}

// per-size window bits set by pp_msm_g1_set_window_bits (index: ceil(lg n))
std::atomic<uint32_t> g_window_bits[33];

uint32_t ceil_lg(uint64_t n) {
  uint32_t lg = 0;
  while (lg < 32 && (1ull << lg) < n) ++lg;
  return lg;
}

// Window bits.  Scalars below r < 2^255 leave the top window few digit
// values unless c is 13, 16 or 20 (the top window then spans 232, 29678 or
// 29678 values): with other c about n entries share a handful of buckets, or
// one carry window.  Swept on GB300 (2^8..2^24 points, c = 6..20): 13 up to
// 2^19 points, 16 up to 2^23 (2^22: 41.2 against 47.2 ms for 18), 18 beyond (2^24:
// 149.8 against 158.6 for 20).  Below 2^15 points the steps after the bucket sums
// are the larger part, and they shrink with the buckets: 8 up to 2^9 points, 10 up
// to 2^15.  Microseconds with 8 / 10 / 13: 1000 points 825 / 829 / 954, 4096 983 /
// 862 / 980, 2^14 1218 / 1023 / 1073, 2^15 1402 / 1168 / 1196, 2^16 1812 / 1492 /
// 1443.  With 2^7 points and fewer the cost model decides.
//
// The model minimises W (10 n + 14 2^c) Fq multiplies: the bucket sums (one
// mixed add per point and window) against the aggregation (two adds per
// bucket).
MsmPlan msm_plan(uint64_t n) {
  const uint32_t lg = ceil_lg(n);
  const uint32_t forced = g_window_bits[lg].load(std::memory_order_relaxed);
  if (forced) return msm_plan_for(forced, 256 / forced + 1);
  if (lg >= 8) {
    const uint32_t c = lg <= 9 ? 8 : lg <= 15 ? 10 : lg <= 19 ? 13 : lg <= 23 ? 16 : 18;
    return msm_plan_for(c, 256 / c + 1);
  }
  uint32_t best_c = 0;
  double best = 0;
  for (uint32_t c = 6; c <= 20; ++c) {
    const double W = 256 / c + 1;
    const double cost = W * (10.0 * (double)n + 14.0 * (double)(1u << c));
    if (best_c == 0 || cost < best) {
      best = cost;
      best_c = c;
    }
  }
  return msm_plan_for(best_c, 256 / best_c + 1);
}

__device__ __forceinline__ g1a ld_g1a(const g1a *p) {
  const uint4 *q = reinterpret_cast<const uint4 *>(p);
  g1a r;
  uint32_t *w = reinterpret_cast<uint32_t *>(&r);
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const uint4 u = __ldg(q + k);
    w[4 * k] = u.x;
    w[4 * k + 1] = u.y;
    w[4 * k + 2] = u.z;
    w[4 * k + 3] = u.w;
  }
  return r;
}

// bits [off, off + c) of a 256-bit scalar (8 little-endian words), c <= 20
__device__ __forceinline__ uint32_t window_bits(const uint32_t s[8], uint32_t off, uint32_t c) {
  const uint32_t w = off >> 5, sh = off & 31;
  if (w >= 8) return 0;
  uint64_t x = s[w];
  if (w + 1 < 8) x |= (uint64_t)s[w + 1] << 32;
  return (uint32_t)(x >> sh) & ((1u << c) - 1);
}

// atomicAdd(base + key, 1) for every active lane; returns the old value plus the
// lane's rank among its group.  Lanes with the first active lane's key, or that of the
// first of the others, make one atomic together (equal or few scalars: up to all n
// entries fall into a bucket); the rest one each (random ones hardly ever meet).
// With __match_any_sync the digits of 200003 points took 100 us without the
// returned place, 82 so.
__device__ __forceinline__ uint32_t warp_increment(uint32_t *base, uint32_t key) {
  const uint32_t mask = __activemask();
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t g0 = __ballot_sync(mask, key == __shfl_sync(mask, key, __ffs(mask) - 1));
  const uint32_t rest = mask & ~g0;
  const uint32_t g1 = __ballot_sync(mask, key == __shfl_sync(mask, key, __ffs(rest ? rest : mask) - 1)) & rest;
  const uint32_t same = g0 >> lane & 1 ? g0 : g1 >> lane & 1 ? g1 : 1u << lane;
  const uint32_t leader = __ffs(same) - 1;
  uint32_t old = 0;
  if (lane == leader) old = atomicAdd(base + key, (uint32_t)__popc(same));
  old = __shfl_sync(mask, old, leader);
  return old + __popc(same & ((1u << lane) - 1));
}

__global__ void k_msm_digits(const uint32_t *__restrict__ scalars, uint64_t n, MsmPlan p,
                             uint32_t *__restrict__ digits, uint32_t *__restrict__ rank,
                             uint32_t *__restrict__ counts) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t s[8];
    const uint4 a = __ldg(reinterpret_cast<const uint4 *>(scalars) + 2 * i);
    const uint4 b = __ldg(reinterpret_cast<const uint4 *>(scalars) + 2 * i + 1);
    s[0] = a.x, s[1] = a.y, s[2] = a.z, s[3] = a.w, s[4] = b.x, s[5] = b.y, s[6] = b.z, s[7] = b.w;
    uint32_t carry = 0;
    for (uint32_t w = 0; w < p.W; ++w) {
      const uint32_t raw = window_bits(s, w * p.c, p.c) + carry;
      uint32_t mag, sign;
      if (raw > p.B) {  // d = raw - 2^c < 0
        mag = (1u << p.c) - raw;
        sign = 1;
        carry = 1;
      } else {
        mag = raw;
        sign = 0;
        carry = 0;
      }
      uint32_t e = kNone;
      if (mag) {
        const uint32_t bucket = mag - 1;
        e = (bucket << 1) | sign;
        rank[(uint64_t)w * n + i] = warp_increment(counts, (p.nsets > 1 ? w * p.B : 0) + bucket);
      }
      digits[(uint64_t)w * n + i] = e;
    }
  }
}

// Exclusive prefix sum of len counts into out (len + 1 entries: the last is
// the total).  Three launches over
// tiles of 4096 entries: tile sums, a scan of the tile sums, tile scans.  With
// HALVE the counts are those of the offsets in[0 .. len], halved and rounded up.
constexpr int kScanThreads = 256, kScanItems = 16;
constexpr uint32_t kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *total) {
  __shared__ uint32_t warp_sum[kScanThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) warp_sum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < kScanThreads / 32 ? warp_sum[lane] : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, d);
      if (lane >= d) w += y;
    }
    if (lane < kScanThreads / 32) warp_sum[lane] = w;
  }
  __syncthreads();
  const uint32_t before = (warp ? warp_sum[warp - 1] : 0) + x - v;
  *total = warp_sum[kScanThreads / 32 - 1];
  __syncthreads();
  return before;
}

template <bool HALVE>
__device__ __forceinline__ uint32_t scan_count(const uint32_t *in, uint64_t i) {
  return HALVE ? (in[i + 1] - in[i] + 1) >> 1 : in[i];
}

template <bool HALVE>
__global__ void __launch_bounds__(kScanThreads)
    k_scan_tiles(const uint32_t *__restrict__ in, uint64_t len, uint32_t *__restrict__ tile_sum) {
  const uint64_t base = (uint64_t)blockIdx.x * kScanTile;
  uint32_t v = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const uint64_t i = base + (uint64_t)k * kScanThreads + threadIdx.x;
    if (i < len) v += scan_count<HALVE>(in, i);
  }
  uint32_t total;
  block_excl_scan(v, &total);
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = total;
}

// exclusive scan of the tile sums in place, total at [ntiles]
__global__ void __launch_bounds__(kScanThreads) k_scan_top(uint32_t *tile_sum, uint32_t ntiles) {
  const uint32_t per = (ntiles + kScanThreads - 1) / kScanThreads;
  const uint32_t lo = threadIdx.x * per, hi = lo + per < ntiles ? lo + per : ntiles;
  uint32_t v = 0;
  for (uint32_t k = lo; k < hi; ++k) v += tile_sum[k];
  uint32_t total;
  uint32_t run = block_excl_scan(v, &total);
  for (uint32_t k = lo; k < hi; ++k) {
    const uint32_t t = tile_sum[k];
    tile_sum[k] = run;
    run += t;
  }
  if (threadIdx.x == 0) tile_sum[ntiles] = total;
}

template <bool HALVE>
__global__ void __launch_bounds__(kScanThreads)
    k_scan_down(const uint32_t *__restrict__ in, uint64_t len, const uint32_t *__restrict__ tile_off,
                uint32_t ntiles, uint32_t *__restrict__ out) {
  const uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems], sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = base + k < len ? scan_count<HALVE>(in, base + k) : 0;
    sum += v[k];
  }
  uint32_t total;
  uint32_t run = tile_off[blockIdx.x] + block_excl_scan(sum, &total);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < len) {
      out[base + k] = run;
    }
    run += v[k];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) out[len] = tile_off[ntiles];
}

template <bool HALVE>
int scan_u32(const uint32_t *in, uint64_t len, uint32_t *out, uint32_t *tiles, cudaStream_t s) {
  const uint32_t ntiles = (uint32_t)((len + kScanTile - 1) / kScanTile);
  k_scan_tiles<HALVE><<<ntiles, kScanThreads, 0, s>>>(in, len, tiles);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  k_scan_top<<<1, kScanThreads, 0, s>>>(tiles, ntiles);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  k_scan_down<HALVE><<<ntiles, kScanThreads, 0, s>>>(in, len, tiles, ntiles, out);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}

// The digits kernel left each entry's place in its bucket (its atomic's result), so
// this one needs no atomics: 200003 points 113 -> 33 us.
// With one bucket set per window an entry names its point i; with window
// tables (one bucket set) it names the table entry w n + i = 2^(c w) P_i.
__global__ void k_msm_scatter(const uint32_t *__restrict__ digits, uint64_t n, MsmPlan p,
                              const uint32_t *__restrict__ rank, const uint32_t *__restrict__ off,
                              uint32_t *__restrict__ list) {
  const uint64_t total = (uint64_t)p.W * n;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t e = digits[t];
    if (e == kNone) continue;
    const uint64_t w = t / n, i = t - w * n;
    const bool per_window = p.nsets > 1;
    list[off[(per_window ? (uint32_t)(w * p.B) : 0u) + (e >> 1)] + rank[t]] = (uint32_t)(per_window ? i : t) | ((e & 1u) << 31);
  }
}

constexpr int kPointThreads = 128;
constexpr int kAccumulateBlocks = 3;       // resident blocks per SM (168 registers)
constexpr uint32_t kRunMin = 4, kRunMax = 64;
constexpr uint32_t kJoinMin = 3;           // partial sums one thread adds up (3 / 5 / 8:
                                           // 200003 points 2.42 / 2.45 / 2.47 ms)
constexpr uint32_t kJoinChunk = 1024;      // partial sums one block adds up

// Entries per run for a list of that many: as many runs as threads are resident
// at once (3 blocks of 128 per SM), or a multiple, so that all waves are full.
// Fixed-base 2^20 points (17.8 M entries): 7.85 ms as one wave of 306 entries,
// 7.33 / 6.98 / 7.05 / 7.03 with runs of at most 128 / 64 / 48 / 32: the SMs do
// not keep step, and shorter waves even that out.  4 blocks per SM (128
// registers, spills): no faster.  Lists too short to fill the chip take runs of
// kRunMin, whose additions follow one another (10 us each); 4 / 6 / 10: 2000 points
// 835 / 852 / 876 us, window tables 1000 points 420 / 430 / 470, 2^13 473 / 500 /
// 512, but 8000 points 932 / 905 / 934.  The kernels take it from the list's real
// length (zero digits have no entry): half of 2^18 scalars zero and the rest one
// took 1638 us with runs sized for a full list.
__host__ __device__ __forceinline__ uint32_t equal_run(uint64_t items, uint32_t resident, uint32_t least,
                                                       uint32_t most) {
  const uint64_t span = (uint64_t)resident * most;
  const uint64_t waves = items ? (items + span - 1) / span : 1;
  const uint64_t K = (items + resident * waves - 1) / (resident * waves);
  return (uint32_t)(K < least ? least : K);
}
__host__ __device__ __forceinline__ uint32_t run_length(uint64_t entries, uint32_t resident) {
  return equal_run(entries, resident, kRunMin, kRunMax);
}
// Outputs per thread of a round of pair sums: longer runs spread the inversion
// over more sums, shorter ones even out the SMs.  Fixed-base 2^20 points, three
// rounds, with at most 80 / 160 / 320: 6.27 / 6.23 / 6.23 ms; 2^22 points 23.6 /
// 23.3 / 23.4 ms.
constexpr uint32_t kPairMin = 16, kPairMax = 160;
__host__ __device__ __forceinline__ uint32_t pair_run(uint64_t outputs, uint32_t resident) {
  return equal_run(outputs, resident, kPairMin, kPairMax);
}
// runs of a list of at most that many items, at most: their length is least or
// more, and a shorter list makes no more waves
inline uint32_t most_runs(uint64_t items, uint32_t resident, uint32_t least, uint32_t most) {
  const uint64_t span = (uint64_t)resident * most;
  const uint64_t by_waves = (uint64_t)resident * ((items + span - 1) / span);
  const uint64_t by_least = items / least + 1;
  return (uint32_t)(by_least < by_waves ? by_least : by_waves);
}
// partial sums of a bucket that one thread joins: twice an average bucket's
__device__ __forceinline__ uint32_t join_few(uint32_t entries, uint32_t nb, uint32_t K) {
  const uint32_t twice = 2 * (entries / ((uint64_t)nb * K) + 1);
  return twice > kJoinMin ? twice : kJoinMin;
}

// the bucket whose range [off[b], off[b+1]) holds entry t
__device__ __forceinline__ uint32_t bucket_of(const uint32_t *off, uint32_t nb, uint32_t t) {
  uint32_t lo = 0, hi = nb;  // off[lo] <= t < off[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (off[mid] <= t) lo = mid;
    else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ fq ld_fq(const fq *p) {
  const uint4 *q = reinterpret_cast<const uint4 *>(p);
  fq r;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint4 u = q[k];
    r.v[4 * k] = u.x, r.v[4 * k + 1] = u.y, r.v[4 * k + 2] = u.z, r.v[4 * k + 3] = u.w;
  }
  return r;
}
__device__ __forceinline__ void st_fq(fq *p, const fq &a) {
  uint4 *q = reinterpret_cast<uint4 *>(p);
#pragma unroll
  for (int k = 0; k < 3; ++k) q[k] = make_uint4(a.v[4 * k], a.v[4 * k + 1], a.v[4 * k + 2], a.v[4 * k + 3]);
}

// Entry k of a sorted list: point list[k] & 0x7fffffff, negated when bit 31 is
// set, or (without a list) points[k].
struct EntryPoints {
  const g1a *points;
  const uint32_t *list;
  __device__ __forceinline__ uint32_t key(uint32_t k) const { return list ? list[k] : k; }
  __device__ __forceinline__ fq x(uint32_t key) const { return ld_fq(&points[key & 0x7fffffffu].x); }
  __device__ __forceinline__ fq y(uint32_t key) const {
    const fq v = ld_fq(&points[key & 0x7fffffffu].y);
    return list && key >> 31 ? fq_neg(v) : v;  // fq_neg(0) = 0: infinity stays all zero
  }
};

// What an output of a round of pair sums is: a copy of the point with key k1, the
// point at infinity, or a sum that takes a division.
enum PairKind : uint32_t { kPairCopy, kPairNone, kPairDouble, kPairAdd };

// 16-byte units of a thread's operands in shared memory, [unit][thread]: two
// slots of x1, x2, y1, y2 and the parked product
constexpr uint32_t kPairUnits = 15, kPairSmem = 2 * kPairUnits * kPointThreads * 16;
__device__ __forceinline__ void fetch_fq(uint4 *dst, const fq *p) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + k * kPointThreads);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d),
                 "l"(reinterpret_cast<const uint4 *>(p) + k)
                 : "memory");
  }
}
__device__ __forceinline__ fq take_fq(const uint4 *src) {
  fq r;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint4 u = src[k * kPointThreads];
    r.v[4 * k] = u.x, r.v[4 * k + 1] = u.y, r.v[4 * k + 2] = u.z, r.v[4 * k + 3] = u.w;
  }
  return r;
}

// One round of pair sums: the entries off[b] .. off[b+1] of each bucket become
// half as many, out[next[b] + j] = entry 2j + entry 2j + 1 in affine form.  An
// affine sum costs a division, y' = l (x1 - x') - y1 with l = (y2 - y1) / (x2 - x1),
// and a thread's divisions share one inversion (Montgomery's simultaneous
// inversion): five multiplies and a square a sum, plus the share of the
// inversion, against eight and two squares of a sum into an XYZZ accumulator.
// A warp takes 32 K outputs in a row, neighbouring lanes neighbouring ones.  The
// forward pass leaves each output's keys and kind in its y and the product of
// the divisors before it in its x, for the backward pass.  Operands are copied
// to shared memory one step ahead, keys loaded two steps ahead (with plain loads
// the gathers' latency took the whole gain: 1.55 against 1.27 ms for 4.5 M sums).
// All lanes make K steps and meet at each multiply: left to themselves, the
// lanes of a warp drift apart at the branches and 18 of 32 work.  One warp
// inverts for its block, an inversion for 128 K sums: each thread inverting for
// itself took 6.35 instead of 6.23 ms.  Bound by the multiply pipe (69 % busy)
// and by the one inversion's latency, per round.  Bucket sums in all, fixed-base
// 2^20 points: 6.98 -> 6.23 ms; 2^20 points 8.42 -> 7.87 ms, 2^22 26.7 -> 22.5.
__global__ void __launch_bounds__(kPointThreads, kAccumulateBlocks)
    k_msm_pairs(EntryPoints in, const uint32_t *__restrict__ off, const uint32_t *__restrict__ next,
                uint32_t nb, uint32_t resident, g1a *out) {
  extern __shared__ uint4 pair_sm[];
  const uint32_t total = next[nb], K = pair_run(total, resident);
  const uint64_t block0 = (uint64_t)blockIdx.x * kPointThreads * K;
  if (block0 >= total) return;
  // this lane's outputs: lo + 32 i, i < m
  const uint64_t lo64 = block0 + (uint64_t)(threadIdx.x & ~31u) * K + (threadIdx.x & 31);
  const uint32_t lo = lo64 < total ? (uint32_t)lo64 : total;
  const uint32_t left = (total - lo + 31) / 32, m = left < K ? left : K;
  uint4 *const sm = pair_sm + threadIdx.x;
  const auto slot = [&](uint32_t i) { return sm + (i & 1) * kPairUnits * kPointThreads; };
  constexpr uint32_t U = 3 * kPointThreads;  // x1, x2, y1, y2, product: U apart

  uint32_t b = m ? bucket_of(next, nb, lo) : 0, begin = next[b], end = next[b + 1];
  // keys of output i of this lane; k2 = k1 for a bucket's odd entry
  const auto keys = [&](uint32_t i, uint32_t &k1, uint32_t &k2) {
    k1 = k2 = 0;
    if (i >= m) return;
    const uint32_t o = lo + 32 * i;
    for (int k = 0; o >= end && k < 8; ++k) ++b, begin = end, end = next[b + 1];
    if (o >= end) b = bucket_of(next, nb, o), begin = next[b], end = next[b + 1];
    const uint32_t src = off[b] + 2 * (o - begin);
    const bool two = src + 1 < off[b + 1];
    k1 = in.key(src);
    k2 = two ? in.key(src + 1) : kNone;
  };
  const auto fetch_x = [&](uint32_t i, uint32_t k1, uint32_t k2) {
    if (i < m && k2 != kNone) {
      fetch_fq(slot(i), &in.points[k1 & 0x7fffffffu].x);
      fetch_fq(slot(i) + U, &in.points[k2 & 0x7fffffffu].x);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint32_t a1, a2, b1, b2;  // keys of steps i and i + 1
  keys(0, a1, a2);
  keys(1, b1, b2);
  fetch_x(0, a1, a2);
  fq prod = fq_one();
#pragma unroll 1
  for (uint32_t i = 0; i < K; ++i) {
    fetch_x(i + 1, b1, b2);
    uint32_t c1, c2;
    keys(i + 2, c1, c2);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    fq d = fq_one();
    if (i < m) {
      g1a *dst = out + lo + 32 * (uint64_t)i;
      PairKind kind = kPairCopy;
      if (a2 != kNone) {
        const fq x1 = take_fq(slot(i)), x2 = take_fq(slot(i) + U);
        d = fq_sub(x2, x1);
        const bool z1 = fq_is_zero(x1), z2 = fq_is_zero(x2), same = fq_is_zero(d);
        kind = kPairAdd;
        if (z1 | z2 | same) {  // infinity, or equal abscissae: the ordinates decide
          const fq y1 = in.y(a1), y2 = in.y(a2);
          if (z2 && fq_is_zero(y2)) {
            kind = kPairCopy;
          } else if (z1 && fq_is_zero(y1)) {
            kind = kPairCopy, a1 = a2;
          } else if (same) {
            kind = fq_is_zero(fq_sub(y1, y2)) && !fq_is_zero(y1) ? kPairDouble : kPairNone;
          }
          if (kind == kPairDouble) d = fq_dbl(y1);
          else if (kind != kPairAdd) d = fq_one();
        }
        if (kind >= kPairDouble) st_fq(&dst->x, prod);
      }
      *reinterpret_cast<uint4 *>(&dst->y) = make_uint4(a1, a2, kind, 0);
    }
    a1 = b1, a2 = b2, b1 = c1, b2 = c2;
    __syncwarp();
    prod = fq_mul(prod, d);
  }
  // 1 / prod (a product of non-zero values): the first warp inverts for the
  // block, lane l the product of threads l, l + 32, l + 64 and l + 96
  fq *const shared = reinterpret_cast<fq *>(pair_sm);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  st_fq(shared + threadIdx.x, prod);
  __syncthreads();
  if (threadIdx.x < 32) {
    fq *q = shared + threadIdx.x;
    fq before[kPointThreads / 32 - 1];  // products of the first 1, 2, 3
    fq all = ld_fq(q);
#pragma unroll
    for (int k = 1; k < kPointThreads / 32; ++k) {
      before[k - 1] = all;
      all = fq_mul(all, ld_fq(q + 32 * k));
    }
    all = fq_inv_fast(all);
#pragma unroll
    for (int k = kPointThreads / 32 - 1; k > 0; --k) {
      const fq p = ld_fq(q + 32 * k);
      st_fq(q + 32 * k, fq_mul(all, before[k - 1]));
      all = fq_mul(all, p);
    }
    st_fq(q, all);
  }
  __syncthreads();
  fq inv = ld_fq(shared + threadIdx.x);
  __syncthreads();

  const auto load_info = [&](uint32_t i) {  // i may have wrapped below zero
    uint4 r = make_uint4(0, 0, kPairNone, 0);
    if (i < m) r = *reinterpret_cast<const uint4 *>(&out[lo + 32 * (uint64_t)i].y);
    return r;
  };
  const auto fetch_all = [&](uint32_t i, const uint4 &f) {
    if (f.z != kPairNone) {
      const g1a *p1 = in.points + (f.x & 0x7fffffffu), *p2 = in.points + (f.y & 0x7fffffffu);
      fetch_fq(slot(i), &p1->x);
      fetch_fq(slot(i) + 2 * U, &p1->y);
      if (f.z == kPairAdd) {
        fetch_fq(slot(i) + U, &p2->x);
        fetch_fq(slot(i) + 3 * U, &p2->y);
      }
      if (f.z >= kPairDouble) fetch_fq(slot(i) + 4 * U, &out[lo + 32 * (uint64_t)i].x);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint4 f0 = load_info(K - 1), f1 = load_info(K - 2);
  fetch_all(K - 1, f0);
#pragma unroll 1
  for (uint32_t i = K; i-- > 0;) {
    fetch_all(i - 1, f1);
    const uint4 f2 = load_info(i - 2);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    fq x = fq_zero(), y = x, x2 = x, num = x, before = x, d = fq_one();
    if (f0.z != kPairNone) {
      x = take_fq(slot(i));
      y = take_fq(slot(i) + 2 * U);
      if (in.list && f0.x >> 31) y = fq_neg(y);
      if (f0.z >= kPairDouble) before = take_fq(slot(i) + 4 * U);
      if (f0.z == kPairAdd) {
        x2 = take_fq(slot(i) + U);
        num = take_fq(slot(i) + 3 * U);
        if (in.list && f0.y >> 31) num = fq_neg(num);
        num = fq_sub(num, y);
        d = fq_sub(x2, x);
      } else if (f0.z == kPairDouble) {
        const fq xx = fq_sqr(x);
        num = fq_add(fq_dbl(xx), xx);
        x2 = x;
        d = fq_dbl(y);
      }
    }
    __syncwarp();
    const fq l = fq_mul(num, fq_mul(inv, before));
    inv = fq_mul(inv, d);
    const fq x3 = fq_sub(fq_sub(fq_sqr(l), x), x2);
    const fq y3 = fq_sub(fq_mul(l, fq_sub(x, x3)), y);
    if (i < m) {
      g1a *dst = out + lo + 32 * (uint64_t)i;
      st_fq(&dst->x, f0.z >= kPairDouble ? x3 : x);
      st_fq(&dst->y, f0.z >= kPairDouble ? y3 : y);
    }
    f0 = f1, f1 = f2;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Bucket sums.  Thread t adds the signed affine points of entries [t K, (t+1) K)
// of the sorted list, starting a new sum at each bucket boundary.  Every lane
// does the same number of additions, so the warps are full whatever the buckets
// hold; with one thread per 16 entries of a bucket, and a level of partial sums
// after it, a quarter of the lanes waited.  GB300: 200003 points 3.63 -> 3.13 ms,
// 2^20 9.84 -> 8.48 ms, fixed-base 2^20 7.65 -> 6.98 ms.  Inlining the ten
// multiplies instead of calling them: 3.17 -> 3.29 ms.
// A bucket that lies inside the run goes to buckets[]; the sum shared with the
// run before goes to part[2 t], the one shared only with the run after to
// part[2 t + 1].  Bound by the multiply pipe.
__global__ void __launch_bounds__(kPointThreads, kAccumulateBlocks)
    k_msm_accumulate(EntryPoints in, const uint32_t *__restrict__ off, uint32_t nb, uint32_t resident,
                     g1x *__restrict__ part, g1x *__restrict__ buckets) {
  const uint32_t total = off[nb], K = run_length(total, resident);
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t lo64 = (uint64_t)t * K;
  if (lo64 >= total) return;
  const uint32_t lo = (uint32_t)lo64, hi = total - lo < K ? total : lo + K;
  uint32_t b = bucket_of(off, nb, lo);
  uint32_t start = off[b], end = off[b + 1];
  g1x acc = g1x_inf();
  for (uint32_t k = lo;; ++k) {
    if (k == end || k == hi) {  // the sum of bucket b ends here
      g1x *dst = start < lo ? part + 2 * (uint64_t)t : end > hi ? part + 2 * (uint64_t)t + 1 : buckets + b;
      *dst = acc;
      if (k == hi) break;
      do {
        ++b;
        start = end;
        end = off[b + 1];
      } while (end == k);  // skips empty buckets
      acc = g1x_inf();
    }
    const uint32_t e = in.key(k);
    acc = g1x_add_affine(acc, g1a{in.x(e), in.y(e)});
  }
}

// A bucket of entries [start, end) is shared by runs start / K .. (end - 1) / K:
// the first left its sum in its second slot, the others in their first.
struct BucketSpan {
  uint32_t first, m;  // first run, number of partial sums (1: complete, 0: empty)
};
__device__ __forceinline__ BucketSpan bucket_span(const uint32_t *off, uint32_t b, uint32_t K) {
  const uint32_t start = off[b], end = off[b + 1];
  if (start == end) return {0, 0};
  return {start / K, (end - 1) / K - start / K + 1};
}
__device__ __forceinline__ uint64_t partial_index(const BucketSpan &s, uint32_t j) {
  return 2 * (uint64_t)(s.first + j) + (j == 0 ? 1 : 0);
}

// Lists the buckets of more partial sums than one thread joins: items[i] = (bucket, chunk)
// for every kJoinChunk of them, multi[] = (bucket, first item) for buckets of
// several chunks; counts in n_items[0] and n_items[1].
__global__ void k_msm_spans(const uint32_t *__restrict__ off, uint32_t nb, uint32_t resident, uint2 *__restrict__ items, uint2 *__restrict__ multi,
                            uint32_t *__restrict__ n_items) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  const uint32_t K = run_length(off[nb], resident);
  const BucketSpan sp = bucket_span(off, b, K);
  if (sp.m <= join_few(off[nb], nb, K)) return;
  const uint32_t chunks = (sp.m + kJoinChunk - 1) / kJoinChunk;
  const uint32_t first = atomicAdd(n_items, chunks);
  for (uint32_t c = 0; c < chunks; ++c) items[first + c] = make_uint2(b, c);
  if (chunks > 1) multi[atomicAdd(n_items + 1, 1u)] = make_uint2(b, first);
}

// ---- Points spread over a warp (fq_lanes.cuh): Y with element 0, X with 1, ZZ with
// 3, ZZZ with 4; element 2 is scratch.  X and Y are below 1.04 q, ZZ below 1.9 q and
// ZZZ below 1.5 q; ZZ = 0 or q is infinity.  For chains and trees that are
// bound by the latency of dependent additions: a doubling 1.46 us, an addition 2.2 us, against
// 3.56 (its multiplies on four lanes) and 13 us (one lane).
__device__ __forceinline__ digit point_load(const Spread &S, const g1x *p) {
  const uint32_t c = S.el == 0 ? 12 : S.el == 3 ? 24 : S.el == 4 ? 36 : 0;
  const uint2 w = *reinterpret_cast<const uint2 *>(reinterpret_cast<const uint32_t *>(p) + c + 2 * S.k);
  return {w.x, w.y, 0};
}
// as it is
__device__ __forceinline__ void point_park(const Spread &S, const digit &P, g1x *p) {
  const uint32_t c = S.el == 0 ? 12 : S.el == 1 ? 0 : S.el == 3 ? 24 : 36;
  if (S.el < 5 && S.el != 2)
    *reinterpret_cast<uint2 *>(reinterpret_cast<uint32_t *>(p) + c + 2 * S.k) = make_uint2(P.l, P.h);
}
// with reduced coordinates
__device__ __forceinline__ void point_store(const Spread &S, const digit &P, g1x *p) {
  const uint32_t c = S.lane & 3;  // X, Y, ZZ, ZZZ
  const uint32_t from = c == 0 ? 1 : c == 1 ? 0 : c + 1;
  fq v;
#pragma unroll
  for (uint32_t k = 0; k < kSpread; ++k) {
    v.v[2 * k] = __shfl_sync(0xffffffffu, P.l, from * kSpread + k);
    v.v[2 * k + 1] = __shfl_sync(0xffffffffu, P.h, from * kSpread + k);
  }
  v = fq_mul(v, fq_one());
  if (S.lane < 4) st_fq(&p->x + c, v);
}
// (the same for all lanes)
__device__ __forceinline__ bool point_is_inf(const Spread &S, const digit &P) {
  return element_all(__ballot_sync(0xffffffffu, (P.l | P.h) == 0), 3) ||
         element_all(__ballot_sync(0xffffffffu, P.l == S.q[0][0] && P.h == S.q[0][1]), 3);
}

// dbl-2008-s-1; Y = 0 gives ZZ = 0.  Bounds in units of q: V < 4.5, M < 3.4, S < 1.5,
// W < 3, M (S - X') < 2.3.
__device__ __forceinline__ digit point_dbl(const Spread &S, const digit &P) {
  const uint32_t el = S.el;
  digit r = S.mul(P, P);                    // Y^2 (0), X^2 (1)
  digit g = S.from(r, el == 2 ? 1 : 0);     // Y^2 (0, 1, 3), X^2 (2)
  const digit g2 = Spread::add(g, g);
  const digit m = S.norm(Spread::add(g2, sel_digit(el == 2, g, g2)));  // V = 4 Y^2, M = 3 X^2 (2)
  // W / 2 = Y V (0), S = X V (1), M^2 (2), ZZ' = ZZ V (3)
  r = S.mul(sel_digit(el == 2, m, P), m);
  r = sel_digit(el == 0, Spread::add(r, r), r);
  g = S.from(r, el == 1 ? 2 : el == 2 ? 1 : 0);  // M^2 (1), S (2), W (4)
  const digit s = sel_digit(el == 2, g, r), mm = sel_digit(el == 2, r, g);
  // X' = M^2 - 2 S (1, 2); W (0, 4), ZZ' (3)
  digit x = S.reduce(Spread::sub(Spread::sub(Spread::add(mm, S.multiple(3)), s), s));
  x = S.norm(sel_digit(el == 1 || el == 2, x, sel_digit(el == 4, g, r)));
  // W Y (0), M (S - X') (2), ZZZ' = W ZZZ (4)
  const digit d = S.norm(sel_digit(el == 2, Spread::sub(Spread::add(s, S.multiple(2)), x), x));
  r = S.mul(sel_digit(el == 2, m, P), d);
  // Y' = M (S - X') - W Y (0), ZZZ' (4)
  const digit y = S.reduce(Spread::sub(Spread::add(S.from(r, 2), S.multiple(2)), r));
  r = S.norm(sel_digit(el == 0, y, r));
  return sel_digit(el == 0 || el == 4, r, x);
}

// add-2008-s.  Bounds in units of q: products of coordinates < 1.4, P, R < 3.2,
// P^2, R^2 < 2.1, P^3 < 1.7, Q < 1.3, R (Q - X') < 2.1.
__device__ __forceinline__ digit point_add(const Spread &S, const digit &A, const digit &B) {
  if (point_is_inf(S, B)) return A;
  if (point_is_inf(S, A)) return B;
  const uint32_t el = S.el;
  // s1 = Y1 ZZZ2 (0), u1 = X1 ZZ2 (1), u2 = X2 ZZ1 (2), ZZ1 ZZ2 (3), s2 = Y2 ZZZ1 (4)
  const digit b1 = S.from(B, el == 2 ? 1 : 0), b2 = S.from(B, el == 0 ? 4 : 3), a1 = S.from(A, 3);
  digit r = S.mul(sel_digit(el == 2 || el == 4, b1, A), sel_digit(el == 2, a1, sel_digit(el == 4, A, b2)));
  // R = s2 - s1 (0), P = u2 - u1 (1), u1 (2), ZZ1 ZZ2 (3), s1 (4)
  digit g = S.from(r, el == 0 ? 4 : el == 1 ? 2 : el == 2 ? 1 : 0);
  const digit diff = Spread::sub(Spread::add(g, S.multiple(2)), r);
  const digit d = S.norm(sel_digit(el < 2, diff, sel_digit(el == 3, r, g)));
  const digit z = S.norm(S.reduce(d));
  const uint32_t zero = __ballot_sync(0xffffffffu, (z.l | z.h) == 0);
  const uint32_t isq = __ballot_sync(0xffffffffu, z.l == S.q[0][0] && z.h == S.q[0][1]);
  if (element_all(zero, 1) || element_all(isq, 1)) {  // equal x: the same point or opposite ones
    if (element_all(zero, 0) || element_all(isq, 0)) return point_dbl(S, A);
    return {0, 0, 0};
  }
  // R^2 (0), P^2 (1), ZZZ1 ZZZ2 (2)
  const digit a4 = S.from(A, 4), b4 = S.from(B, 4);
  const digit r2 = S.mul(sel_digit(el == 2, a4, d), sel_digit(el == 2, b4, d));
  const digit pp = S.norm(S.from(r2, 1));
  // P^3 (1), Q = u1 P^2 (2), ZZ' = ZZ1 ZZ2 P^2 (3)
  const digit r3 = S.mul(d, pp);
  const digit ppp = S.norm(S.from(r3, 1)), q = S.from(r3, 2);
  // X' = R^2 - P^3 - 2 Q (all)
  digit x = Spread::add(Spread::add(S.from(r2, 0), S.multiple(2)), S.multiple(3));
  x = S.norm(S.reduce(Spread::sub(Spread::sub(Spread::sub(x, ppp), q), q)));
  const digit e = S.norm(Spread::sub(Spread::add(q, S.multiple(2)), x));
  // R (Q - X') (0), ZZZ' = ZZZ1 ZZZ2 P^3 (2), s1 P^3 (4)
  r = S.mul(S.norm(sel_digit(el == 2, r2, d)), sel_digit(el == 0, e, ppp));
  g = S.from(r, el == 0 ? 4 : 2);
  const digit y = S.reduce(Spread::sub(Spread::add(r, S.multiple(2)), g));
  return S.norm(sel_digit(el == 0, y, sel_digit(el == 3, r3, sel_digit(el == 4, g, x))));
}

// sum of val(j), lo <= j < hi, by a block of kPointThreads (the result in
// red[0] for all): strided sums, then a tree in shared memory, its lower levels
// with a warp to each addition (128 values in 220 blocks: 106 -> 71 us)
constexpr uint32_t kWarpAdds = 16;
template <typename F>
__device__ __forceinline__ g1x block_sum(uint32_t lo, uint32_t hi, g1x *red, F val) {
  g1x acc = g1x_inf();
  for (uint32_t j = lo + threadIdx.x; j < hi; j += kPointThreads) acc = g1x_add(acc, val(j));
  red[threadIdx.x] = acc;
  __syncthreads();
  for (uint32_t h = kPointThreads / 2; h > kWarpAdds; h >>= 1) {
    if (threadIdx.x < h) red[threadIdx.x] = g1x_add(red[threadIdx.x], red[threadIdx.x + h]);
    __syncthreads();
  }
  const Spread S;
  for (uint32_t h = kWarpAdds; h > 0; h >>= 1) {
    for (uint32_t i = threadIdx.x / 32; i < h; i += kPointThreads / 32) {
      const digit a = point_load(S, red + i), b = point_load(S, red + i + h);
      if (point_is_inf(S, b)) continue;
      point_park(S, point_add(S, a, b), red + i);
    }
    __syncthreads();
  }
  if (threadIdx.x < 32) {
    const digit a = point_load(S, red);
    point_store(S, a, red);
  }
  __syncthreads();
  const g1x r = red[0];
  __syncthreads();  // red may be used again
  return r;
}

// Joins the shared buckets: the first `small_blocks` blocks take one bucket per
// thread, the others (128 threads each) the listed chunks of the larger ones,
// whose sums go to buckets[] or, with several chunks, to chunk_sum[item].
__global__ void __launch_bounds__(kPointThreads)
    k_msm_join(const g1x *__restrict__ part, const uint32_t *__restrict__ off, uint32_t nb,
               uint32_t resident, uint32_t small_blocks, const uint2 *__restrict__ items,
               const uint32_t *__restrict__ n_items, g1x *__restrict__ chunk_sum,
               g1x *__restrict__ buckets) {
  __shared__ __align__(16) g1x red[kPointThreads];
  const uint32_t K = run_length(off[nb], resident);
  if (blockIdx.x < small_blocks) {
    const uint32_t few = join_few(off[nb], nb, K);
    const uint32_t b = blockIdx.x * kPointThreads + threadIdx.x;
    if (b >= nb) return;
    const BucketSpan sp = bucket_span(off, b, K);
    if (sp.m < 2 || sp.m > few) return;
    g1x acc = part[partial_index(sp, 0)];
    for (uint32_t j = 1; j < sp.m; ++j) acc = g1x_add(acc, part[partial_index(sp, j)]);
    buckets[b] = acc;
    return;
  }
  const uint32_t n = n_items[0];
  for (uint32_t it = blockIdx.x - small_blocks; it < n; it += gridDim.x - small_blocks) {
    const uint2 item = items[it];
    const BucketSpan sp = bucket_span(off, item.x, K);
    const uint32_t lo = item.y * kJoinChunk, hi = sp.m - lo < kJoinChunk ? sp.m : lo + kJoinChunk;
    const g1x sum = block_sum(lo, hi, red, [&](uint32_t j) { return part[partial_index(sp, j)]; });
    if (threadIdx.x == 0) (sp.m <= kJoinChunk ? buckets[item.x] : chunk_sum[it]) = sum;
  }
}

// the chunks of the buckets that have several
__global__ void __launch_bounds__(kPointThreads)
    k_msm_join_chunks(const uint32_t *__restrict__ off, uint32_t nb, uint32_t resident,
                      const uint2 *__restrict__ multi,
                      const uint32_t *__restrict__ n_items, const g1x *__restrict__ chunk_sum,
                      g1x *__restrict__ buckets) {
  __shared__ __align__(16) g1x red[kPointThreads];
  const uint32_t n = n_items[1], K = run_length(off[nb], resident);
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const uint2 mb = multi[i];
    const BucketSpan sp = bucket_span(off, mb.x, K);
    const uint32_t chunks = (sp.m + kJoinChunk - 1) / kJoinChunk;
    const g1x sum = block_sum(0, chunks, red, [&](uint32_t j) { return chunk_sum[mb.y + j]; });
    if (threadIdx.x == 0) buckets[mb.x] = sum;
  }
}

// Segment s of window w holds buckets b = s G + j, j < G.  Its thread leaves
// R_s = sum_j B_b and T_s = sum_j (j + 1) B_b (running sums from the top), so
// that the window sum sum_b (b + 1) B_b = sum_s T_s + G sum_s s R_s.
__global__ void __launch_bounds__(kPointThreads)
    k_msm_segments(const g1x *__restrict__ buckets, MsmPlan p, g1x *__restrict__ seg_t,
                   g1x *__restrict__ seg_r) {
  const uint64_t total = (uint64_t)p.nsets * p.S;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const g1x *row = buckets + t * p.G;  // segments are consecutive in each window
    g1x run = g1x_inf(), sum = g1x_inf();
    for (int j = (int)p.G - 1; j >= 0; --j) {
      run = g1x_add(run, row[j]);
      __syncwarp();  // lanes that met an empty bucket wait for the others
      sum = g1x_add(sum, run);
      __syncwarp();
    }
    seg_t[t] = sum;
    seg_r[t] = run;
  }
}

// The same for segments of four buckets, two lanes each: four dependent additions
// instead of six.  R = (B0 + B1) + (B2 + B3) and T = (R + B1) + ((B2 + B3) + B3 +
// (B2 + B3)).  Bound by the additions' latency; kPairedLanes says when.
__device__ __forceinline__ g1x neighbour(const g1x &a) {  // the other lane's
  g1x r;
  const uint32_t *u = reinterpret_cast<const uint32_t *>(&a);
  uint32_t *v = reinterpret_cast<uint32_t *>(&r);
#pragma unroll
  for (uint32_t k = 0; k < sizeof(g1x) / 4; ++k) v[k] = __shfl_xor_sync(0xffffffffu, u[k], 1);
  return r;
}
__global__ void __launch_bounds__(kPointThreads)
    k_msm_segments4(const g1x *__restrict__ buckets, uint64_t total, g1x *__restrict__ seg_t,
                    g1x *__restrict__ seg_r) {
  const uint64_t i = (uint64_t)blockIdx.x * kPointThreads + threadIdx.x;
  const uint64_t t = i / 2 < total ? i / 2 : total - 1;  // all lanes stay for the exchanges
  const uint32_t up = (uint32_t)i & 1;                   // buckets 2 and 3
  const g1x *row = buckets + 4 * t + 2 * up;
  const g1x odd = row[1];
  const g1x s = g1x_add(row[0], odd);
  __syncwarp();
  // R (down), B2 + 2 B3 (up)
  const g1x other = neighbour(s);
  g1x a = g1x_add(s, up ? odd : other);
  if (!up && i / 2 < total) seg_r[t] = a;
  // R + B1, 2 B2 + 3 B3
  a = g1x_add(a, up ? s : odd);
  const g1x b = neighbour(a);
  if (!up && i / 2 < total) seg_t[t] = g1x_add(a, b);
}

// Window sums from the segments: sum_b (b + 1) B_b = sum_s T_s + G sum_s s R_s,
// and sum_s s R_s = sum_k 2^k Q_k, where Q_k adds the R_s of the segments whose
// index s has bit k set.  So a window needs 1 + lg S plain sums (sum j = 0 is
// sum_s T_s, sum j = 1 + k is Q_k) and one short Horner chain; no sum weights
// a point by more than one doubling at a time.
//
// Each sum is cut into chunks of p.chunk terms; one thread adds one chunk (8
// instead of 16 terms: 303 -> 118 us of dependent additions).  All lanes make the
// same steps and meet after each: left to themselves they drift apart at empty
// segments and at the sums' ends, and the warp repeats the addition for each group
// (1000 points, 26 sets of 2^9 buckets: 96 -> 55 us).
// Window w's chunks are part[w ncw + u]: u < nc0 for sum 0, then nc1 chunks
// for each Q_k in order of k.
struct ChunkCounts {
  uint32_t nc0, nc1, ncw;
};

__host__ __device__ __forceinline__ ChunkCounts chunk_counts(const MsmPlan &p) {
  ChunkCounts c;
  c.nc0 = (p.S + p.chunk - 1) / p.chunk;
  c.nc1 = (p.S / 2 + p.chunk - 1) / p.chunk;
  c.ncw = c.nc0 + p.lgS * c.nc1;
  return c;
}

__global__ void __launch_bounds__(kPointThreads)
    k_msm_bitsums(const g1x *__restrict__ seg_t, const g1x *__restrict__ seg_r, MsmPlan p,
                  g1x *__restrict__ part) {
  const ChunkCounts cc = chunk_counts(p);
  const uint64_t total = (uint64_t)p.nsets * cc.ncw;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t w = (uint32_t)(t / cc.ncw), u = (uint32_t)(t - (uint64_t)w * cc.ncw);
    const bool t_sum = u < cc.nc0;
    const uint32_t k = t_sum ? 0 : (u - cc.nc0) / cc.nc1;
    const uint32_t ch = t_sum ? u : u - cc.nc0 - k * cc.nc1, terms = t_sum ? p.S : p.S >> 1;
    const g1x *row = (t_sum ? seg_t : seg_r) + (uint64_t)w * p.S;
    g1x acc = g1x_inf();
    for (uint32_t i = ch * p.chunk, j = 0; j < p.chunk; ++i, ++j) {
      // the i-th segment index with bit k set
      const uint32_t s = t_sum ? i : ((i >> k) << (k + 1)) | (1u << k) | (i & ((1u << k) - 1));
      if (i < terms) acc = j ? g1x_add(acc, row[s]) : row[s];
      __syncwarp();
    }
    part[t] = acc;
  }
}

// Sums of every (window, sum)'s chunks, in blocks of at most kReduceSpan: a warp
// adds up to 8 of them, each addition spread over it, then the warps' sums meet in
// a tree.  in and out are the numbers of inputs and of blocks per sum; where a sum
// takes several blocks a second launch adds those.  Bound by the latency of the
// additions (2.2 us alone, 4.3 with four warps to a sub-partition).  One block of
// 128 threads per sum, a lane to an addition down to 16 of them, took 170 us for
// one bucket set of 2^15 buckets against 68 us for both launches (16 to a warp: 80),
// and 91 us for 20 sets of 2^12 against 92.
constexpr uint32_t kReduceWarps = 8, kReduceSpan = 8 * kReduceWarps;
__host__ __device__ __forceinline__ ChunkCounts reduced_counts(const ChunkCounts &in, uint32_t lgS) {
  ChunkCounts c;
  c.nc0 = (in.nc0 + kReduceSpan - 1) / kReduceSpan;
  c.nc1 = (in.nc1 + kReduceSpan - 1) / kReduceSpan;
  c.ncw = c.nc0 + lgS * c.nc1;
  return c;
}
__global__ void __launch_bounds__(32 * kReduceWarps)
    k_msm_bitreduce(const g1x *__restrict__ part, ChunkCounts in, ChunkCounts out, g1x *__restrict__ sums) {
  __shared__ __align__(16) g1x red[kReduceWarps];
  const uint32_t w = blockIdx.x / out.ncw, u = blockIdx.x - w * out.ncw;
  const bool t_sum = u < out.nc0;
  const uint32_t v = t_sum ? u : u - out.nc0, blocks = t_sum ? out.nc0 : out.nc1;
  const uint32_t k = v / blocks, count = t_sum ? in.nc0 : in.nc1;
  const uint32_t span = (count + blocks - 1) / blocks, lo = (v - k * blocks) * span;
  const uint32_t hi = lo + span < count ? lo + span : count;
  const g1x *row = part + (uint64_t)w * in.ncw + (t_sum ? 0 : in.nc0 + k * in.nc1);
  const uint32_t warp = threadIdx.x / 32;
  const Spread S;
  digit acc = {0, 0, 0}, next = {0, 0, 0};
  uint32_t i = lo + warp;
  if (i < hi) next = point_load(S, row + i);
#pragma unroll 1
  for (; i < hi; i += kReduceWarps) {
    const digit p = next;
    if (i + kReduceWarps < hi) next = point_load(S, row + i + kReduceWarps);
    acc = point_add(S, acc, p);
  }
  point_park(S, acc, red + warp);
  __syncthreads();
#pragma unroll 1
  for (uint32_t h = kReduceWarps / 2; h > 0; h >>= 1) {
    if (warp < h) {
      acc = point_add(S, acc, point_load(S, red + warp + h));
      point_park(S, acc, red + warp);
    }
    __syncthreads();
  }
  if (warp == 0) point_store(S, acc, sums + blockIdx.x);
}

// One warp per window: win[w] = sum_s T_s + G sum_k 2^k Q_k (Horner over k)
__global__ void __launch_bounds__(32) k_msm_wincombine(const g1x *__restrict__ sums, MsmPlan p,
                                                       g1x *__restrict__ win) {
  const Spread S;
  const g1x *q = sums + (uint64_t)blockIdx.x * (1 + p.lgS);  // q[0] = sum T, q[1 + k] = Q_k
  digit acc = {0, 0, 0};
#pragma unroll 1
  for (int k = (int)p.lgS - 1; k >= -1; --k) {
    // Q_k after one doubling, then (k = -1) sum_s T_s after lg G
    for (uint32_t j = k >= 0 ? 1 : p.lgG; j > 0; --j) acc = point_dbl(S, acc);
    acc = point_add(S, acc, point_load(S, q + 1 + k));
  }
  point_store(S, acc, win + blockIdx.x);
}

// Horner over the windows (one warp), then affine; out = Jacobian (x, y, 1),
// or all zero for the point at infinity
__global__ void __launch_bounds__(32) k_msm_final(const g1x *__restrict__ win, MsmPlan p,
                                                  fq *__restrict__ out) {
  __shared__ __align__(16) g1x sum;
  const Spread S;
  digit acc = {0, 0, 0};
#pragma unroll 1
  for (int w = (int)p.nsets - 1; w >= 0; --w) {
    if (!point_is_inf(S, acc))  // the upper windows of short scalars are empty
      for (uint32_t j = 0; j < p.c; ++j) acc = point_dbl(S, acc);
    acc = point_add(S, acc, point_load(S, win + w));
  }
  point_store(S, acc, &sum);
  __syncwarp();
  if (threadIdx.x != 0) return;
  const g1a a = g1x_to_affine(sum);
  const bool inf = g1x_is_inf(sum);
  out[0] = a.x;
  out[1] = a.y;
  out[2] = inf ? fq_zero() : fq_one();
}

struct MsmLayout {
  size_t digits, counts, n_items, offsets, list, part, items, multi, chunk_sum, buckets, seg_t,
      seg_r, chunks, chunks2, sums, win, tiles, pairs[2], pair_off, total;
  uint32_t resident; // threads of k_msm_accumulate resident at once
  uint32_t runs;     // runs of the list at most
};

// Rounds of pair sums before the buckets are accumulated: while a round has 14
// outputs per resident thread (28 with window tables), over which an inversion and
// the round's launches spread, and 8 per bucket, below which unpaired entries and steps between buckets
// take the gain.  Milliseconds with 0, 1, 2, 3 and 4 rounds (rule's choice marked):
//   200003 points  3.13 3.08* 3.12 3.30 3.55   window tables 2.03 2.00* 2.07 2.25
//   2^20 points    8.42 7.97 7.87* 7.94 8.10   window tables 6.97 6.46 6.29 6.23* 6.26
//   2^22 points    26.7 24.4 23.1 22.6 22.5*
//   2^16 points    2.05* 2.18 2.47             window tables 1.16* 1.35 1.53
// Since inversions take 32 instead of 57 us the bound is 14 instead of 28: 2^17 points
// 1937 -> 1893 us, 2^18 2792 -> 2719, 200003 2368 -> 2350; with window tables 2^17
// 1236 -> 1250, 200003 1605 -> 1623, so it stays 28 there.
// The bound on the entries keeps the rounds' buffers below 20 GB.
uint32_t pair_rounds(uint64_t n, const MsmPlan &p) {
  const uint64_t entries = (uint64_t)p.W * n, nb = (uint64_t)p.nsets * p.B;
  const uint64_t resident = (uint64_t)device_sm_count() * kAccumulateBlocks * kPointThreads;
  const uint64_t per_thread = p.nsets > 1 ? 14 : 28;
  uint32_t r = 0;
  if (entries <= 1ull << 28)
    while ((entries >> (r + 1)) >= per_thread * resident && (entries >> (r + 1)) >= 8 * nb) ++r;
  return r;
}
// outputs of a round over that many inputs, at most: every bucket rounds up
inline uint64_t pair_outputs(uint64_t inputs, uint64_t nb) { return (inputs + nb) / 2; }

MsmLayout msm_layout(uint64_t n, const MsmPlan &p, uint32_t rounds) {
  MsmLayout L{};
  auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const uint64_t nb = (uint64_t)p.nsets * p.B;
  const uint64_t entries = (uint64_t)p.W * n;
  L.resident = (uint32_t)device_sm_count() * kAccumulateBlocks * kPointThreads;
  L.runs = most_runs(entries, L.resident, kRunMin, kRunMax);
  // each run leaves at most two partial sums, and a listed bucket has more than
  // kJoinMin of them: at most 2 runs / 4 buckets, plus one item per full chunk
  const uint64_t items = L.runs / 2 + 2 * (uint64_t)L.runs / kJoinChunk + 64, multi = 2 * (uint64_t)L.runs / kJoinChunk + 1;
  size_t o = 0;
  L.digits = o, o += up(entries * 4);
  L.counts = o, o += nb * 4;
  L.n_items = o, o = up(o + 8);  // cleared with the counts
  L.offsets = o, o += up((nb + 1) * 4);
  L.list = o, o += up(entries * 4);
  // the entries' ranks first: 384 bytes per run of at most kRunMax entries
  L.part = o, o += up(2 * (size_t)L.runs * sizeof(g1x));
  L.items = o, o += up(items * sizeof(uint2));
  L.multi = o, o += up(multi * sizeof(uint2));
  L.chunk_sum = o, o += up(items * sizeof(g1x));
  L.buckets = o, o += up(nb * sizeof(g1x));
  L.seg_t = o, o += up((size_t)p.nsets * p.S * sizeof(g1x));
  L.seg_r = o, o += up((size_t)p.nsets * p.S * sizeof(g1x));
  const ChunkCounts chunks = chunk_counts(p);
  L.chunks = o, o += up((size_t)p.nsets * chunks.ncw * sizeof(g1x));
  L.chunks2 = o, o += up((size_t)p.nsets * reduced_counts(chunks, p.lgS).ncw * sizeof(g1x));
  L.sums = o, o += up((size_t)p.nsets * (1 + p.lgS) * sizeof(g1x));
  L.win = o, o += up((size_t)p.nsets * sizeof(g1x));
  L.tiles = o, o += up(((nb + kScanTile - 1) / kScanTile + 1) * 4);
  if (rounds > 0) {  // the rounds write two buffers in turn
    const uint64_t first = pair_outputs(entries, nb);
    L.pairs[0] = o, o += up(first * sizeof(g1a));
    if (rounds > 1) L.pairs[1] = o, o += up(pair_outputs(first, nb) * sizeof(g1a));
  }
  L.pair_off = o, o += rounds ? up((nb + 1) * 4) : 0;
  L.total = o;
  return L;
}

// one thread per unit of work (loops stride only past 2^31 - 1 blocks): 2^20
// points took 13.77 ms, against 14.09 ms with grids capped at 8-16 blocks
// per SM
unsigned grid_for(uint64_t work, int threads) {
  const uint64_t want = (work + threads - 1) / threads;
  const uint64_t cap = 0x7fffffffull;
  return (unsigned)(want < cap ? (want ? want : 1) : cap);
}

// ---- window tables of a fixed point set: table[w n + i] = 2^(c w) P_i in
// affine form.  Window w + 1 comes from window w by c doublings in XYZZ and a
// batched conversion back to affine: Montgomery's simultaneous inversion over
// runs of kTableRun points, one field inversion per run.
constexpr uint32_t kTableRun = 32;

__global__ void __launch_bounds__(kPointThreads)
    k_msm_table_double(const g1a *__restrict__ prev, uint64_t n, uint32_t c, g1x *__restrict__ out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    g1x q = g1x_dbl_affine(ld_g1a(prev + i));
    for (uint32_t k = 1; k < c; ++k) q = g1x_dbl(q);
    out[i] = q;
  }
}

// x = X / ZZ, y = Y / ZZZ with 1 / (ZZ ZZZ) from the run's one inversion; the
// forward pass parks the running products in out[].x, the backward pass reads
// each one before it overwrites it.  Infinity (ZZ = 0) becomes all zero.
__global__ void __launch_bounds__(kPointThreads)
    k_msm_table_affine(const g1x *__restrict__ q, uint64_t n, g1a *__restrict__ out) {
  const uint64_t runs = (n + kTableRun - 1) / kTableRun;
  for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < runs;
       r += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t lo = r * kTableRun, hi = lo + kTableRun < n ? lo + kTableRun : n;
    fq acc = fq_one();
    for (uint64_t j = lo; j < hi; ++j) {
      const g1x p = q[j];
      if (!g1x_is_inf(p)) acc = fq_mul(acc, fq_mul(p.zz, p.zzz));
      out[j].x = acc;
    }
    fq inv = fq_inv_fast(acc);  // acc is a product of non-zero values
    for (uint64_t j = hi; j > lo; --j) {
      const g1x p = q[j - 1];
      g1a a;
      if (g1x_is_inf(p)) {
        a.x = fq_zero();
        a.y = fq_zero();
      } else {
        const fq before = j - 1 > lo ? out[j - 2].x : fq_one();
        const fq inv_d = fq_mul(inv, before);  // 1 / (ZZ ZZZ) of this point
        inv = fq_mul(inv, fq_mul(p.zz, p.zzz));
        a.x = fq_mul(p.x, fq_mul(inv_d, p.zzz));
        a.y = fq_mul(p.y, fq_mul(inv_d, p.zz));
      }
      out[j - 1] = a;
    }
  }
}

// Window bits for a fixed point set, from the same kind of sweep (c = 10..20,
// 2^8..2^24 points on GB300) and the same top-window effect: 13 up to 2^11
// points, 16 up to 2^21 (2^20: 10.72 ms against 10.98 for 17 and 11.83 for
// 15), 20 beyond (2^22: 33.8 against 35.8 for 19).  One bucket set serves all
// windows, so a large c costs little aggregation, and a bucket of many entries is
// joined from many runs.  Microseconds with 13 / 16: 4096 points 511 / 454, 8000
// 688 / 473, 2^14 854 / 528.
uint32_t fixed_window_bits(uint64_t n) {
  const uint32_t lg = ceil_lg(n);
  return lg <= 11 ? 13 : lg <= 21 ? 16 : 20;
}

// The pipeline behind both entry points.  points holds n affine points (one
// bucket set per window) or the W n window-table entries (one bucket set);
// scalars n plain 256-bit integers; out receives (x, y, 1), or zeros.
int msm_run(const g1a *points, const uint32_t *scalars, uint64_t n, const MsmPlan &p, fq *out,
            cudaStream_t s) {
  uint32_t rounds = pair_rounds(n, p);
  MsmLayout L = msm_layout(n, p, rounds);
  const MsmLayout least = msm_layout(n, p, 0);
  size_t got = 0;
  int st = PP_OK;
  char *ws = static_cast<char *>(workspace_get_most(L.total, least.total, s, 3, &got, &st));
  if (st) return st;
  if (got < L.total) L = least, rounds = 0;  // no room for the rounds' buffers
  auto u32 = [&](size_t off) { return reinterpret_cast<uint32_t *>(ws + off); };
  auto pts = [&](size_t off) { return reinterpret_cast<g1x *>(ws + off); };
  uint32_t *digits = u32(L.digits), *counts = u32(L.counts), *offsets = u32(L.offsets);
  uint32_t *rank = u32(L.part), *list = u32(L.list), *n_items = u32(L.n_items);
  uint32_t *tiles = u32(L.tiles);
  uint2 *items = reinterpret_cast<uint2 *>(ws + L.items), *multi = reinterpret_cast<uint2 *>(ws + L.multi);
  g1x *buckets = pts(L.buckets), *seg_t = pts(L.seg_t), *seg_r = pts(L.seg_r), *win = pts(L.win);
  g1x *chunks = pts(L.chunks), *chunks2 = pts(L.chunks2), *sums = pts(L.sums), *part = pts(L.part), *chunk_sum = pts(L.chunk_sum);
  const uint64_t nb = (uint64_t)p.nsets * p.B;

  // 1-3: signed digits, bucket sizes, counting sort of (point, sign) by bucket
  PP_CUDA_TRY(cudaMemsetAsync(counts, 0, nb * 4 + 8, s));  // and n_items
  k_msm_digits<<<grid_for(n, 256), 256, 0, s>>>(scalars, n, p, digits, rank, counts);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  if ((st = scan_u32<false>(counts, nb, offsets, tiles, s))) return st;
  k_msm_scatter<<<grid_for((uint64_t)p.W * n, 256), 256, 0, s>>>(digits, n, p, rank, offsets, list);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();

  // 4: rounds of pair sums, each halving every bucket's entries
  EntryPoints in{points, list};
  uint32_t *spare = u32(L.pair_off);
  if (rounds)
    PP_CUDA_TRY(cudaFuncSetAttribute(k_msm_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairSmem));
  uint64_t left = (uint64_t)p.W * n;
  for (uint32_t r = 0; r < rounds; ++r) {
    if ((st = scan_u32<true>(offsets, nb, spare, tiles, s))) return st;
    left = pair_outputs(left, nb);
    g1a *pair_sums = reinterpret_cast<g1a *>(ws + L.pairs[r & 1]);
    k_msm_pairs<<<grid_for(most_runs(left, L.resident, kPairMin, kPairMax), kPointThreads),
                  kPointThreads, kPairSmem, s>>>(in, offsets, spare, (uint32_t)nb, L.resident, pair_sums);
    PP_COUNT_LAUNCH();
    PP_LAUNCH_CHECK();
    in = EntryPoints{pair_sums, nullptr};
    uint32_t *const t = offsets;
    offsets = spare;
    spare = t;
  }

  // 5: bucket sums over equal runs of the list, then the shared buckets
  PP_CUDA_TRY(cudaMemsetAsync(buckets, 0, nb * sizeof(g1x), s));  // all zero = infinity
  k_msm_accumulate<<<grid_for(L.runs, kPointThreads), kPointThreads, 0, s>>>(
      in, offsets, (uint32_t)nb, L.resident, part, buckets);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  k_msm_spans<<<grid_for(nb, 256), 256, 0, s>>>(offsets, (uint32_t)nb, L.resident, items, multi,
                                                   n_items);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  const unsigned small_blocks = grid_for(nb, kPointThreads), big_blocks = 2 * (unsigned)device_sm_count();
  k_msm_join<<<small_blocks + big_blocks, kPointThreads, 0, s>>>(
      part, offsets, (uint32_t)nb, L.resident, small_blocks, items, n_items, chunk_sum, buckets);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  k_msm_join_chunks<<<(unsigned)device_sm_count(), kPointThreads, 0, s>>>(
      offsets, (uint32_t)nb, L.resident, multi, n_items, chunk_sum, buckets);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();

  // 6-8: weighted bucket sums per bucket set, sets combined, affine result
  const uint64_t segments = (uint64_t)p.nsets * p.S;
  if (p.G == 4 && 2 * segments <= kPairedLanes)
    k_msm_segments4<<<grid_for(2 * segments, kPointThreads), kPointThreads, 0, s>>>(buckets, segments, seg_t, seg_r);
  else
    k_msm_segments<<<grid_for(segments, kPointThreads), kPointThreads, 0, s>>>(buckets, p, seg_t, seg_r);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  const ChunkCounts cc = chunk_counts(p), some = reduced_counts(cc, p.lgS), one{1, 1, 1 + p.lgS};
  k_msm_bitsums<<<grid_for((uint64_t)p.nsets * cc.ncw, kPointThreads), kPointThreads, 0, s>>>(seg_t, seg_r, p, chunks);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  const bool twice = some.nc0 > 1;
  k_msm_bitreduce<<<p.nsets * some.ncw, 32 * kReduceWarps, 0, s>>>(chunks, cc, some, twice ? chunks2 : sums);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  if (twice) {
    k_msm_bitreduce<<<p.nsets * one.ncw, 32 * kReduceWarps, 0, s>>>(chunks2, some, one, sums);
    PP_COUNT_LAUNCH();
    PP_LAUNCH_CHECK();
  }
  k_msm_wincombine<<<p.nsets, 32, 0, s>>>(sums, p, win);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  k_msm_final<<<1, 32, 0, s>>>(win, p, out);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}

}  // namespace
}  // namespace pp

extern "C" int pp_msm_g1(const void *d_points, const void *d_scalars, uint64_t n, void *d_out,
                         void *stream) {
  using namespace pp;
  auto aligned16 = [](const void *q) { return q && (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (!aligned16(d_out) || (n && (!aligned16(d_points) || !aligned16(d_scalars)))) {
    set_error("pp_msm_g1: buffers must be 16-byte aligned device pointers");
    return PP_E_INVAL;
  }
  if (n >= (1ull << 31)) {
    set_error("pp_msm_g1: n = %llu points; at most 2^31 - 1", (unsigned long long)n);
    return PP_E_UNSUPPORTED;
  }
  cudaStream_t s = (cudaStream_t)stream;
  if (n == 0) {
    PP_CUDA_TRY(cudaMemsetAsync(d_out, 0, 3 * sizeof(fq), s));
    return PP_OK;
  }
  const MsmPlan p = msm_plan(n);
  if ((uint64_t)p.W * n >= (1ull << 32)) {
    set_error("pp_msm_g1: n = %llu points is too many for 32-bit bucket offsets",
              (unsigned long long)n);
    return PP_E_UNSUPPORTED;
  }
  return msm_run(static_cast<const g1a *>(d_points), static_cast<const uint32_t *>(d_scalars), n, p,
                 static_cast<fq *>(d_out), s);
}

extern "C" int pp_msm_g1_window_bits(uint64_t n) { return (int)pp::msm_plan(n).c; }

extern "C" int pp_msm_g1_set_window_bits(uint32_t lg_n, uint32_t window_bits) {
  if (lg_n > 32 || (window_bits && (window_bits < 6 || window_bits > 20))) {
    pp::set_error("pp_msm_g1_set_window_bits: lg_n <= 32 and window_bits 0 or 6..20");
    return PP_E_INVAL;
  }
  pp::g_window_bits[lg_n].store(window_bits, std::memory_order_relaxed);
  return PP_OK;
}

// ---- fixed-base form: the window tables of one point set stay in HBM ----
struct pp_msm_bases {
  int device;
  uint64_t n;
  uint32_t c;
  pp::g1a *table;  // W n affine points, table[w n + i] = 2^(c w) P_i
};

extern "C" int pp_msm_g1_bases_create(const void *d_points, uint64_t n, uint32_t window_bits,
                                      pp_msm_bases **bases, void *stream) {
  using namespace pp;
  if (!bases) {
    set_error("pp_msm_g1_bases_create: null handle pointer");
    return PP_E_INVAL;
  }
  *bases = nullptr;
  if (!d_points || (reinterpret_cast<uintptr_t>(d_points) & 15)) {
    set_error("pp_msm_g1_bases_create: points must be a 16-byte aligned device pointer");
    return PP_E_INVAL;
  }
  if (n == 0 || (window_bits && (window_bits < 6 || window_bits > 20))) {
    set_error("pp_msm_g1_bases_create: need n >= 1 and window_bits 0 (automatic) or 6..20");
    return PP_E_INVAL;
  }
  const uint32_t c = window_bits ? window_bits : fixed_window_bits(n);
  const uint64_t W = 256 / c + 1;
  if (W * n >= (1ull << 31)) {
    set_error("pp_msm_g1_bases_create: %llu windows x %llu points exceed 2^31 table entries",
              (unsigned long long)W, (unsigned long long)n);
    return PP_E_UNSUPPORTED;
  }
  cudaStream_t s = (cudaStream_t)stream;
  int dev = 0;
  PP_CUDA_TRY(cudaGetDevice(&dev));
  g1a *table = nullptr;
  PP_COUNT_ALLOC(W * n * sizeof(g1a));
  if (cudaMalloc(&table, W * n * sizeof(g1a)) != cudaSuccess) {
    cudaGetLastError();
    set_error("pp_msm_g1_bases_create: cannot allocate %llu bytes of window tables",
              (unsigned long long)(W * n * sizeof(g1a)));
    return PP_E_NOMEM;
  }
  g1x *tmp = nullptr;
  PP_COUNT_ALLOC(n * sizeof(g1x));
  if (cudaMallocAsync(&tmp, n * sizeof(g1x), s) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(table);
    set_error("pp_msm_g1_bases_create: cannot allocate %llu bytes of scratch",
              (unsigned long long)(n * sizeof(g1x)));
    return PP_E_NOMEM;
  }
  int st = PP_OK;
  if (cudaMemcpyAsync(table, d_points, n * sizeof(g1a), cudaMemcpyDeviceToDevice, s) != cudaSuccess) {
    st = PP_E_CUDA;
    set_error("pp_msm_g1_bases_create: copying the points failed: %s",
              cudaGetErrorString(cudaGetLastError()));
  }
  for (uint64_t w = 1; st == PP_OK && w < W; ++w) {
    k_msm_table_double<<<grid_for(n, kPointThreads), kPointThreads, 0, s>>>(table + (w - 1) * n,
                                                                               n, c, tmp);
    PP_COUNT_LAUNCH();
    k_msm_table_affine<<<grid_for((n + kTableRun - 1) / kTableRun, kPointThreads), kPointThreads,
                         0, s>>>(tmp, n, table + w * n);
    PP_COUNT_LAUNCH();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      st = PP_E_CUDA;
      set_error("pp_msm_g1_bases_create: kernel launch failed: %s", cudaGetErrorString(e));
    }
  }
  cudaFreeAsync(tmp, s);
  if (st) {
    cudaFree(table);
    return st;
  }
  *bases = new pp_msm_bases{dev, n, c, table};
  return PP_OK;
}

extern "C" int pp_msm_g1_bases_destroy(pp_msm_bases *bases) {
  if (!bases) return PP_OK;
  int cur = 0;
  cudaGetDevice(&cur);
  cudaSetDevice(bases->device);
  const cudaError_t e = cudaFree(bases->table);
  cudaSetDevice(cur);
  delete bases;
  if (e != cudaSuccess) {
    pp::set_error("pp_msm_g1_bases_destroy: cudaFree failed: %s", cudaGetErrorString(e));
    return PP_E_CUDA;
  }
  return PP_OK;
}

extern "C" int pp_msm_g1_bases_info(const pp_msm_bases *bases, uint64_t *n, uint32_t *window_bits,
                                    uint64_t *table_bytes) {
  if (!bases) {
    pp::set_error("pp_msm_g1_bases_info: null handle");
    return PP_E_INVAL;
  }
  const uint64_t W = 256 / bases->c + 1;
  if (n) *n = bases->n;
  if (window_bits) *window_bits = bases->c;
  if (table_bytes) *table_bytes = W * bases->n * sizeof(pp::g1a);
  return PP_OK;
}

extern "C" int pp_msm_g1_fixed(const pp_msm_bases *bases, const void *d_scalars, void *d_out,
                               void *stream) {
  using namespace pp;
  auto aligned16 = [](const void *q) { return q && (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (!bases || !aligned16(d_scalars) || !aligned16(d_out)) {
    set_error("pp_msm_g1_fixed: need a handle and 16-byte aligned device buffers");
    return PP_E_INVAL;
  }
  int dev = 0;
  PP_CUDA_TRY(cudaGetDevice(&dev));
  if (dev != bases->device) {
    set_error("pp_msm_g1_fixed: the tables live on device %d, the current device is %d",
              bases->device, dev);
    return PP_E_INVAL;
  }
  return msm_run(bases->table, static_cast<const uint32_t *>(d_scalars), bases->n,
                 msm_plan_for(bases->c, 1), static_cast<fq *>(d_out), (cudaStream_t)stream);
}

// ---- s_i G for the generator: test and benchmark points, commitments to
// known constants.  One thread per scalar, double-and-add from bit 255.
namespace pp {
namespace {

__global__ void __launch_bounds__(kPointThreads)
    k_g1_mul_gen(const uint32_t *__restrict__ scalars, uint64_t n, g1a *__restrict__ out) {
  const g1a G = g1_generator();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t s[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) s[k] = scalars[8 * i + k];
    g1x acc = g1x_inf();
    for (int b = 255; b >= 0; --b) {
      acc = g1x_dbl(acc);
      if ((s[b >> 5] >> (b & 31)) & 1u) acc = g1x_add_affine(acc, G);
    }
    out[i] = g1x_to_affine(acc);
  }
}

}  // namespace
}  // namespace pp

extern "C" int pp_g1_mul_gen(const void *d_scalars, uint64_t n, void *d_out, void *stream) {
  using namespace pp;
  auto aligned16 = [](const void *q) { return q && (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (n == 0) return PP_OK;
  if (!aligned16(d_scalars) || !aligned16(d_out)) {
    set_error("pp_g1_mul_gen: buffers must be 16-byte aligned device pointers");
    return PP_E_INVAL;
  }
  k_g1_mul_gen<<<grid_for(n, kPointThreads), kPointThreads, 0, (cudaStream_t)stream>>>(
      static_cast<const uint32_t *>(d_scalars), n, static_cast<g1a *>(d_out));
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}
