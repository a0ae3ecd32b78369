// ntt.cu -- in-HBM multi-pass NTT over Fr for sm_103a.
//
// Structure (GB300-first, not the reference's 3-kernel CT layout):
//  * A transform of 2^L points is split into P passes of 2^k_p-point
//    sub-transforms (k_p <= 11), the four-step / Stockham factorisation
//    N = R_1 * R_2 * ... * R_P.  Pass p runs, for every prefix of already
//    transformed digits and every column c < S_p = R_{p+1}..R_P, an R_p-point
//    DFT over the elements at stride S_p, multiplies output k by the layer
//    twiddle w_{R_p S_p}^(c k) and stores it in place; the last pass writes
//    the digit-reversed (natural) output order directly, so no bit-reversal
//    kernel and no uncoalesced swap pass is needed.
//  * A thread block owns a tile of R_p x T_p elements (R_p * T_p <= 2048,
//    64 KiB of shared memory, XOR-swizzled 16-byte units); T_p adjacent
//    columns give >= 128-byte contiguous row segments for coalesced HBM
//    access.  Each column's DFT runs as radix-8 rounds held in registers (8
//    elements per thread), with a final radix-4/2 round; the first round reads
//    its elements straight from global memory and the last one writes them
//    there, so shared memory only carries the exchanges in between.
//  * Every multiply is on the integer pipe; the transform is compute-bound
//    (~11 multiplies per element at 2^24 against 3 HBM passes), so the
//    inter-pass twiddles are read from HBM tables (one load instead of a
//    multiply), and inverse transforms fold 2^-L into the first layer table.
//    The twiddles inside a pass are few, so they are kept in the four-part
//    form of fr_mul_const4 (82 wide products instead of 112): per-round tables
//    read through L1, and the 8-point DFT's three roots in constant memory.
//
// Reference behaviour restated: natural order in and out, w_N =
// forward_roots_of_unity[lg N] = 7^((r-1)/N) (PLONK/utils/zkp/cuda/
// zksnark_ntt/parameters/bls12_381.h:29-83), inverse scaled by N^-1
// (ct_mixed_radix_wide.cuh:173-176).
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "ntt.cuh"

namespace pp {

// ------------------------------------------------------------------ host math
static fr host_pow_limbs(const fr &a, const uint32_t e[8]) {
  fr acc = fr_one();
  bool started = false;
  for (int w = 7; w >= 0; --w)
    for (int b = 31; b >= 0; --b) {
      if (started) acc = fr_sqr(acc);
      if ((e[w] >> b) & 1) {
        acc = started ? fr_mul(acc, a) : a;
        started = true;
      }
    }
  return acc;
}

fr host_mont_small(uint64_t x) {
  fr t = fr_zero();
  t.v[0] = (uint32_t)x;
  t.v[1] = (uint32_t)(x >> 32);
  return fr_mul(t, fr_rr());
}
fr host_pow(const fr &a, uint64_t e) { return fr_pow_u64(a, e); }
fr host_inv(const fr &a) { return fr_inv(a); }

fr host_root_of_unity(int lg, bool inverse) {
  static std::once_flag once;
  static fr fwd[33], inv[33];
  std::call_once(once, [] {
    // (r - 1) >> 32, 32-bit limbs
    const uint32_t e[8] = {0xffffffffu, PP_R2, PP_R3, PP_R4, PP_R5, PP_R6, PP_R7, 0u};
    fwd[32] = host_pow_limbs(host_mont_small(7), e);
    for (int k = 31; k >= 0; --k) fwd[k] = fr_sqr(fwd[k + 1]);
    for (int k = 0; k <= 32; ++k) inv[k] = fr_inv(fwd[k]);
  });
  return inverse ? inv[lg] : fwd[lg];
}

// ------------------------------------------------------------- device code
// Place of element e = row T + col of a tile among its 16-byte units.  Linear
// over XOR: a thread's 8 elements differ in bits that its first one has clear,
// so their places are the first one's XOR a value that the whole warp shares.
__host__ __device__ __forceinline__ uint32_t swz(uint32_t e) {
  return e ^ (((e >> 3) ^ (e >> 6) ^ (e >> 9)) & 7u);
}

// A tile's elements as two planes of 16-byte units, low halves then high halves
// at a fixed distance (an immediate of the access).  The kernel's bound is the
// pipe that the wide products and the address arithmetic share: with places and
// strides as here instead of an address worked out per access, a transform of
// 2^18 takes 49.3 us instead of 55.3, 2^20 174 instead of 183, 2^24 2606
// instead of 2751.  The bank conflicts are the same as before, none.
constexpr uint32_t kTileElems = 2048, kTileBytes = kTileElems * sizeof(fr);
struct SmemTile {
  uint4 *s;
  __device__ __forceinline__ fr get(uint32_t place) const {
    const uint4 a = s[place], b = s[place + kTileElems];
    return fr{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
  }
  __device__ __forceinline__ void put(uint32_t place, const fr &v) const {
    s[place] = make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]);
    s[place + kTileElems] = make_uint4(v.v[4], v.v[5], v.v[6], v.v[7]);
  }
  // asynchronous copy of *p into the place (cp.async, 16 bytes each)
  __device__ __forceinline__ void fetch(uint32_t place, const fr *p) const {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(s + place);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(p) : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + kTileElems * 16),
                 "l"(reinterpret_cast<const uint4 *>(p) + 1)
                 : "memory");
  }
};

// Inside a transform values are kept below 2r (fr_*_lazy); the last round of
// the last pass makes them canonical before they leave the kernel.
__device__ __forceinline__ void bfly(fr &a, fr &b) {
  const fr t = a;
  a = fr_add_lazy(t, b);
  b = fr_sub_lazy(t, b);
}

// g, g^2, g^3 for g = 7^((r - 1) / 8), the forward 8-point DFT's root, each as
// the four products of fr_mul_const4
__constant__ fr c_root8[3][4] = {
    {
        {{0xcef49ea0u, 0xdcd5caa8u, 0xbd6d1816u, 0x69201e87u,
          0xcf28faf2u, 0x783ec6b6u, 0x87a05b34u, 0x1e0586d8u}},
        {{0xde0a24a3u, 0xdfaa358fu, 0x8f1ab3c9u, 0x3a13d616u,
          0x407da03fu, 0xd862d68du, 0x17ac7fefu, 0x0b97f08eu}},
        {{0x9b12398eu, 0x4b53ca4eu, 0x7624ef38u, 0xa0d9e7f3u,
          0x9524919bu, 0x47e4ef53u, 0xe24cf722u, 0x5fe27ea0u}},
        {{0x44eb37e9u, 0xe757b80eu, 0x4229cdacu, 0x9df71901u,
          0x5bdd56fdu, 0xcbb407acu, 0xf1dfe463u, 0x3ba5b74du}},
    },
    {
        {{0xc7edfb36u, 0x381204c8u, 0xc7ed6ccbu, 0xc59889a0u,
          0x307d7343u, 0x26b07cdau, 0xd246eae2u, 0x274ed2c8u}},
        {{0xcc3033f3u, 0xdd027557u, 0x3d5071f7u, 0xda5fec58u,
          0x53ff4e10u, 0xd6b1d7c9u, 0x8bee15e0u, 0x1c496903u}},
        {{0x9e3a2626u, 0x234eedafu, 0x05d6a1f7u, 0xce1bb45du,
          0xb4dc675bu, 0x44ba87bbu, 0x600997adu, 0x26b36dfau}},
        {{0x5593a1d4u, 0x54f62ddcu, 0x689ce4a1u, 0x29f28715u,
          0x4630a8abu, 0xa058db80u, 0x070dfcaau, 0x2c58143fu}},
    },
    {
        {{0x2fb113e9u, 0x11d87474u, 0xdfb3fc26u, 0x319788e0u,
          0x92036cf2u, 0xf41937d2u, 0x80f69024u, 0x4d0272cbu}},
        {{0xfa7a5327u, 0x5b7707ecu, 0x2ed969adu, 0x17f947e5u,
          0xfceb0de1u, 0x9a8fc772u, 0x8d46ac2cu, 0x67ccda1au}},
        {{0x4fd24120u, 0xcaf5f51cu, 0x9d075bc9u, 0xdd83221cu,
          0x6588868cu, 0x410bf77cu, 0xfd335d4du, 0x57893116u}},
        {{0x3a74abb7u, 0x043dfd25u, 0x6cf2b08cu, 0xf7b43b7eu,
          0xe1196756u, 0x7c149dabu, 0x91e39a97u, 0x0ac07ea6u}},
    },
};

// 8-point forward DFT, natural order in and out (decimation in frequency; the
// output permutation is a renaming).  The inverse DFT is the same values with
// output k at (8 - k) mod 8, so one set of roots serves both directions.
// inputs_used() is called once every input has been read.
template <typename F>
__device__ __forceinline__ void dft8(fr x[8], F inputs_used) {
  bfly(x[0], x[4]);
  bfly(x[1], x[5]);
  bfly(x[2], x[6]);
  bfly(x[3], x[7]);
  inputs_used();
  x[5] = fr_mul_const4(x[5], c_root8[0]);
  x[6] = fr_mul_const4(x[6], c_root8[1]);
  x[7] = fr_mul_const4(x[7], c_root8[2]);
  bfly(x[0], x[2]);
  bfly(x[1], x[3]);
  bfly(x[4], x[6]);
  bfly(x[5], x[7]);
  x[3] = fr_mul_const4(x[3], c_root8[1]);
  x[7] = fr_mul_const4(x[7], c_root8[1]);
  bfly(x[0], x[1]);
  bfly(x[2], x[3]);
  bfly(x[4], x[5]);
  bfly(x[6], x[7]);
  fr t = x[1];
  x[1] = x[4];
  x[4] = t;
  t = x[3];
  x[3] = x[6];
  x[6] = t;
}

// Round twiddles.  A round of 8-point DFTs with 2^lgSj columns (lgSj = 1 .. 8)
// multiplies output k of column c by w_R^(c k), R = 2^(lgSj + 3).  Each twiddle
// is eight 16-byte units (two per part of fr_mul_const4's four), unit h of
// output k at [k - 1][h][round_column(lgSj) + c]: the lanes of a warp, on
// neighbouring columns, read contiguous bytes, and all units lie at constant
// distances from the first (kRoundStride units, not a multiple of a power of
// two of cache lines).
constexpr uint32_t kRoundStride = 520;  // 510 columns of all lgSj, padded
constexpr uint32_t kRoundUnits = 56 * kRoundStride;
__host__ __device__ __forceinline__ uint32_t round_column(uint32_t lgSj) { return (1u << lgSj) - 2; }
__device__ __forceinline__ fr mul_round_twiddle(const fr &x, const uint4 *t) {
  fr w[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const uint4 a = __ldg(t + 2 * p * kRoundStride), b = __ldg(t + (2 * p + 1) * kRoundStride);
    w[p] = fr{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
  }
  return fr_mul_const4(x, w);
}

__device__ __forceinline__ uint32_t digit_reverse(uint32_t o, uint32_t lgR) {
  uint32_t rem = lgR, p = 0, t = o;
  while (rem > 0) {
    const uint32_t lgr = rem >= 3 ? 3 : rem;
    const uint32_t k = t & ((1u << lgr) - 1);
    t >>= lgr;
    rem -= lgr;
    p += k << rem;
  }
  return p;
}

// the output index held at position p of a finished column (the inverse of
// digit_reverse; additive over disjoint bits of p)
__device__ __forceinline__ uint32_t digit_index(uint32_t p, uint32_t lgR) {
  uint32_t rem = lgR, o = 0, sh = 0;
  while (rem > 0) {
    const uint32_t lgr = rem >= 3 ? 3 : rem;
    rem -= lgr;
    o += ((p >> rem) & ((1u << lgr) - 1)) << sh;
    sh += lgr;
  }
  return o;
}

// w_{R S}^(o c) from the split tables (both canonical, so the product is)
__device__ __forceinline__ fr split_layer_twiddle(const PassArgs &a, uint32_t o, uint64_t c) {
  const uint64_t e = (uint64_t)o * c;
  return fr_mul(ldg_fr(a.tw_hi + (e >> a.tw_lgh)), ldg_fr(a.tw_lo + (e & ((1ull << a.tw_lgh) - 1))));
}

// The layer multiply as a call: inlined eight times per thread it is 24 KB of
// code that every tile walks through (2^22: 714 us inlined, 702 called; 2^24:
// 2760 and 2738).  The round twiddles, in the loop, are faster inlined.
__device__ __noinline__ fr mul_layer(fr a, fr b) { return fr_mul_lazy(a, b); }

// where a tile's elements lie
struct TileGeom {
  uint64_t base = 0, col0 = 0;         // intermediate pass: first element, first column
  uint64_t in_base = 0, out_base = 0;  // last pass: first input and output element
  uint32_t lgS1 = 0;
  __device__ __forceinline__ uint64_t src(const PassArgs &a, uint32_t n, uint32_t col) const {
    if (!a.last) return base + ((uint64_t)n << a.lgS) + col;
    return in_base + ((uint64_t)col << lgS1) + n;  // one pass: in_base = col = 0
  }
};

__device__ __forceinline__ TileGeom tile_geom(const PassArgs &a, const uint64_t tileid) {
  TileGeom t;
  if (!a.last) {
    const uint32_t lgtpq = a.lgS - a.lgT;
    const uint64_t q = tileid >> lgtpq, ct = tileid & ((1ull << lgtpq) - 1);
    t.col0 = ct << a.lgT;
    t.base = (q << (a.lgR + a.lgS)) + t.col0;
  } else if (a.P > 1) {
    const uint32_t lgR1 = a.lgRp[0];
    t.lgS1 = a.lgN - lgR1;
    const uint32_t lgkb = lgR1 - a.lgT;
    const uint64_t kb = tileid & ((1ull << lgkb) - 1), rest = tileid >> lgkb;
    uint64_t rin = 0, r = rest;
    uint32_t acc = lgR1;
    for (uint32_t j = 1; j + 1 < a.P; ++j) {
      const uint32_t bits = a.lgRp[j];
      acc += bits;
      rin += (r & ((1ull << bits) - 1)) << (a.lgN - acc);
      r >>= bits;
    }
    t.in_base = ((kb << a.lgT) << t.lgS1) + rin;
    t.out_base = (kb << a.lgT) + (rest << lgR1);
  }
  return t;
}

// One tile of one pass: load (+ input multiply), column DFTs, layer twiddle or
// scale, store.  Bound by the integer-multiply pipe (68 % busy: 16 warps per SM
// at 128 registers) and by the loads' latency around it.  GB300, 2^24 points:
// 3.32 ms with general multiplies and every round through shared memory, 2.87
// with the four-part twiddles and the first and last round on global memory,
// 2.74 with the layer twiddles fetched during the last round and multiplied by
// a called function (pieces left out, for scale: layer multiplies 370 us, their
// loads 220 before the asynchronous fetch, input loads 250, round-twiddle loads
// 224).  Asking L2 for the next wave's tiles made it 1.4 % slower, 1024-element
// tiles with four blocks per SM 7 %.
// The block may be wider than the tile needs (batched
// launches use 256 threads for every job); surplus threads only join the
// barriers.
template <bool HOSTIO>
__device__ __forceinline__ void ntt_tile(const PassArgs &a, const uint64_t tileid, uint4 *sm) {
  // HOSTIO = false compiles out the host-endpoint paths (unit_in, unit_out);
  // every pass is still correct without them, with element-wise accesses
  const bool unit_in = HOSTIO && a.unit_in, unit_out = HOSTIO && a.unit_out;
  const SmemTile tile{sm};
  const uint32_t R = 1u << a.lgR, T = 1u << a.lgT, E = R << a.lgT;
  const uint32_t nthr = E >> 3;
  const uint32_t tid = threadIdx.x;
  const bool active = tid < nthr;

  const TileGeom geo = tile_geom(a, tileid);
  const uint64_t base = geo.base, col0 = geo.col0, out_base = geo.out_base;

  // ---- a host-memory input without a multiply on the way in goes through
  // shared memory in 16-byte halves, so one warp instruction reads whole
  // 128-byte lines; a thread's 16 loads issue in two groups of eight before
  // their shared-memory stores, so it waits on host memory twice per tile
  // instead of sixteen times.
  const bool stage_in = unit_in && !(a.first && a.in_kind == NTT_IN_DIAG);
  // a host-memory output without a scale leaves the tile the same way
  const bool stage_out = unit_out && !(a.last && a.has_post_scale);
  auto tile_src = [&](uint32_t n, uint32_t col) -> uint64_t { return geo.src(a, n, col); };
  if (stage_in) {
    const uint4 zero4 = make_uint4(0, 0, 0, 0);
    if (active) {
#pragma unroll
      for (uint32_t k0 = 0; k0 < 16; k0 += 8) {
        uint4 v[8];
        uint32_t dst[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
          const uint32_t u = tid + (k0 + i) * nthr;
          const uint32_t e = u >> 1, h = u & 1;
          const uint32_t n = a.last ? e & (R - 1) : e >> a.lgT, col = a.last ? e >> a.lgR : e & (T - 1);
          const uint64_t g = tile_src(n, col);
          dst[i] = swz((n << a.lgT) + col) + h * kTileElems;
          v[i] = zero4;
          if (!a.first) {
            v[i] = __ldcs(reinterpret_cast<const uint4 *>(a.in + g) + h);
          } else if (a.in_kind == NTT_IN_SPREAD) {
            if ((g & ((1ull << a.spread) - 1)) == 0)
              v[i] = __ldcs(reinterpret_cast<const uint4 *>(a.in + (g >> a.spread)) + h);
          } else if (g < a.n_valid) {
            v[i] = __ldcs(reinterpret_cast<const uint4 *>(a.in + g) + h);
          }
        }
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) tile.s[dst[i]] = v[i];
      }
    }
    __syncthreads();
  }
  auto load = [&](uint32_t n, uint32_t col) -> fr {
    const uint64_t g = tile_src(n, col);
    if (!a.first) return ldcs_fr(a.in + g);
    if (a.in_kind == NTT_IN_SPREAD)
      return (g & ((1ull << a.spread) - 1)) == 0 ? ldcs_fr(a.in + (g >> a.spread)) : fr_zero();
    if (g >= a.n_valid) return fr_zero();
    const fr v = ldcs_fr(a.in + g);
    if (a.in_kind != NTT_IN_DIAG) return v;
    const fr d = a.diag_hi ? fr_mul(ldg_fr(a.diag + (g & ((1ull << a.diag_lgh) - 1))),
                                    ldg_fr(a.diag_hi + (g >> a.diag_lgh)))
                           : ldcs_fr(a.diag + g);
    return fr_mul_lazy(v, d);
  };

  // ---- column DFTs: radix-8 rounds, final radix-4/2 round.  A thread holds
  // the 8 positions pb + (j << lgs) of one column.  Neighbouring lanes take
  // neighbouring columns (contiguous in global memory, and few distinct
  // twiddles per warp), except where the last pass reads: there a column is
  // contiguous.
  {
    const uint32_t lgcpt = a.lgR - 3;
    uint32_t lgP = 0, rem = a.lgR;
#pragma unroll 1
    for (;;) {
      const uint32_t lgr = rem >= 3 ? 3 : rem;
      const uint32_t lgSj = rem - lgr;
      if (active) {  // surplus threads of a wider block: barriers only
        const bool by_row = a.last && lgP == 0;
        const uint32_t col = by_row ? tid >> lgcpt : tid & (T - 1);
        const uint32_t d = by_row ? tid & ((1u << lgcpt) - 1) : tid >> a.lgT;
        const uint32_t lgs = lgr == 3 ? lgSj : 0;
        const uint32_t c = d & ((1u << lgs) - 1);
        const uint32_t pb = ((d >> lgs) << (lgs + 3)) + c;
        // the thread's element i sits at place0 ^ place(i)
        const uint32_t place0 = swz((pb << a.lgT) + col);
        const auto place = [&](uint32_t i) { return swz(i << (lgs + a.lgT)); };
        // over zero padding only the first 8 >> zero_lg inputs can be non-zero
        const uint32_t zlg = lgP == 0 ? a.zero_lg : 0;
        fr x[8];
        if (lgP > 0 || stage_in) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (i > 0 && zlg >= 3) break;
            if (i > 1 && zlg == 2) break;
            x[i] = tile.get(place0 ^ place(i));
          }
        } else if (!a.first || (a.in_kind == NTT_IN_PLAIN && zlg == 0 && a.n_valid >> a.lgN)) {
          const fr *p = a.in + geo.src(a, pb, col);
          const uint64_t step = 1ull << (lgs + (a.last ? 0 : a.lgS));
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = ldcs_fr(p + i * step);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (i > 0 && zlg >= 3) break;
            if (i > 1 && zlg == 2) break;
            x[i] = load(pb + ((uint32_t)i << lgs), col);
          }
        }
        // output j of the round goes to position pb + (at(j) << lgs): the
        // inverse transform takes the forward DFT's outputs in reverse
        const auto at = [&](uint32_t j) -> uint32_t {
          if (!a.inverse || lgr == 1) return j;
          return lgr == 3 ? (8 - j) & 7 : (j & 4) | ((4 - (j & 3)) & 3);
        };
        // in the last round position pb + j holds output o0 + index(j): the
        // last digit, and the low bits of the one before it (radix 4 and 2)
        const uint32_t osh = a.last ? a.lgN - a.lgR : a.lgS;
        const uint64_t o0 = (uint64_t)digit_index(pb, a.lgR) << osh;
        const auto index = [&](uint32_t j) -> uint64_t {
          const uint32_t lowd = (j & ((1u << lgr) - 1)) << (a.lgR - lgr);
          return (uint64_t)(lgr == 3 ? lowd : lowd + ((j >> lgr) << (a.lgR - lgr - 3))) << osh;
        };
        // the last round of an intermediate pass fetches its layer twiddles
        // into the tile slots it has just read (nobody else uses them), so
        // they arrive while the round computes
        const bool fetch = lgSj == 0 && !stage_out && a.tw_layer;
        const auto fetch_layer = [&] {
          if (!fetch) return;
          const fr *t = a.tw_layer + o0 + col0 + col;
#pragma unroll
          for (uint32_t j = 0; j < 8; ++j) tile.fetch(place0 ^ place(j), t + index(j));
          asm volatile("cp.async.commit_group;" ::: "memory");
        };
        if (lgr == 3) {
          if (zlg >= 3) {
            fetch_layer();
            // the 8-point DFT of (x0, 0, ..., 0) is x0 in every output
#pragma unroll
            for (int i = 1; i < 8; ++i) x[i] = x[0];
          } else if (zlg == 2) {
            // X[k] = x0 + x1 g^k, g^4 = -1
            const fr x0 = x[0], x1 = x[1];
            fetch_layer();
            const fr t1 = fr_mul_const4(x1, c_root8[0]), t2 = fr_mul_const4(x1, c_root8[1]);
            const fr t3 = fr_mul_const4(x1, c_root8[2]);
            x[0] = fr_add_lazy(x0, x1);
            x[4] = fr_sub_lazy(x0, x1);
            x[1] = fr_add_lazy(x0, t1);
            x[5] = fr_sub_lazy(x0, t1);
            x[2] = fr_add_lazy(x0, t2);
            x[6] = fr_sub_lazy(x0, t2);
            x[3] = fr_add_lazy(x0, t3);
            x[7] = fr_sub_lazy(x0, t3);
          } else {
            dft8(x, fetch_layer);
          }
          if (lgSj > 0) {
            const uint4 *tw = a.tw_round + round_column(lgSj) + c;
#pragma unroll
            for (uint32_t j = 1; j < 8; ++j)
              x[j] = mul_round_twiddle(x[j], tw + (at(j) - 1) * 8 * kRoundStride);
          }
        } else if (lgr == 2) {
#pragma unroll
          for (int h = 0; h < 8; h += 4) {
            bfly(x[h + 0], x[h + 2]);
            bfly(x[h + 1], x[h + 3]);
          }
          fetch_layer();
#pragma unroll
          for (int h = 0; h < 8; h += 4) {
            x[h + 3] = fr_mul_const4(x[h + 3], c_root8[1]);
            bfly(x[h + 0], x[h + 1]);
            bfly(x[h + 2], x[h + 3]);
            const fr t = x[h + 1];  // bit-reversed -> natural
            x[h + 1] = x[h + 2];
            x[h + 2] = t;
          }
        } else {
#pragma unroll
          for (int h = 0; h < 8; h += 2) bfly(x[h], x[h + 1]);
          fetch_layer();
        }
        if (lgSj > 0 || stage_out) {
          // the 16-byte output path copies tile words: canonical here
          if (lgSj == 0 && a.last) {
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = fr_canon(x[i]);
          }
#pragma unroll
          for (uint32_t j = 0; j < 8; ++j) tile.put(place0 ^ place(at(j)), x[j]);
        } else {
          // ---- the last round stores (coalesced), with the layer twiddle or
          // the final scale
          if (fetch) asm volatile("cp.async.wait_group 0;" ::: "memory");
          fr *dst = a.out + (a.last ? out_base : base) + col + o0;
#pragma unroll
          for (uint32_t j = 0; j < 8; ++j) {
            fr v = x[j];
            if (a.last) {
              v = fr_canon(v);
              if (a.has_post_scale) v = fr_mul(v, a.post_scale);
            } else if (fetch) {
              v = mul_layer(v, tile.get(place0 ^ place(at(j))));
            }
            st_fr(dst + index(at(j)), v);
          }
        }
      }
      if (lgSj == 0) break;
      // the next round exchanges among 2^lgSj threads of a column, and with
      // neighbouring lanes on neighbouring columns those T 2^lgSj threads are
      // one warp in the later rounds
      if ((T << lgSj) <= 32 && !(a.last && lgP == 0)) __syncwarp();
      else __syncthreads();
      lgP += lgr;
      rem -= lgr;
    }
  }
  if (!stage_out) return;
  __syncthreads();

  // ---- host output through the tile: whole 128-byte lines leave it (partial
  // lines cost C2C bandwidth)
  if (!a.last && (a.tw_layer || a.tw_lo)) {
    // an intermediate pass: the layer twiddles go into the tile first
    for (uint32_t e = tid; active && e < E; e += nthr) {
      const uint32_t o = e >> a.lgT, col = e & (T - 1);
      const uint32_t at = swz((digit_reverse(o, a.lgR) << a.lgT) + col);
      const fr w = a.tw_layer ? ldcs_fr(a.tw_layer + ((uint64_t)o << a.lgS) + col0 + col)
                              : split_layer_twiddle(a, o, col0 + col);
      tile.put(at, fr_mul_lazy(tile.get(at), w));
    }
    __syncthreads();
  }
  for (uint32_t u = tid; active && u < 2 * E; u += nthr) {
    const uint32_t e = u >> 1, h = u & 1;
    const uint32_t o = e >> a.lgT, col = e & (T - 1);
    const uint4 v = tile.s[swz((digit_reverse(o, a.lgR) << a.lgT) + col) + h * kTileElems];
    const uint64_t g = a.last ? out_base + col + ((uint64_t)o << (a.lgN - a.lgR))
                              : base + ((uint64_t)o << a.lgS) + col;
    reinterpret_cast<uint4 *>(a.out + g)[h] = v;
  }
}

#ifndef PP_NTT_MINB
#define PP_NTT_MINB 2  // blocks per SM the pass kernels are compiled for
#endif
template <bool HOSTIO>
__global__ void __launch_bounds__(256, PP_NTT_MINB) k_ntt_pass(const PassArgs a) {
  extern __shared__ uint4 sm[];
  // a dependent pass's blocks may be placed while the one before it drains
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  ntt_tile<HOSTIO>(a, blockIdx.x, sm);
}

// One batch level: the tiles of every job pass at this level are numbered
// consecutively (tile_start = prefix sums over the jobs), one block per tile
// as in k_ntt_pass; a block finds its job by a binary search over the starts.
__global__ void __launch_bounds__(256, PP_NTT_MINB) k_ntt_batch_level(const __grid_constant__ LevelParams p) {
  extern __shared__ uint4 sm[];
  const uint64_t t = blockIdx.x;
  uint32_t lo = 0, hi = p.count;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (p.tile_start[mid] <= t) lo = mid;
    else hi = mid;
  }
  ntt_tile<false>(p.args[lo], t - p.tile_start[lo], sm);  // device endpoints
}

// Latency form (single calls of 2^3 .. 2^17 points): one column of R points per
// block, R / 2 threads (at least a warp), one pass up to 2^8 points and two
// above.  Transforms this small are bound by the length of the dependent chain,
// not by the multiply pipe, and the tile kernel's unrolled rounds (60 KB of
// code) by instruction fetch.  So each thread holds one butterfly of a radix-2
// decimation-in-time layer:
//  * the first layer reads its two rows straight from global memory (bit
//    reversal is the address) and has no multiply; the last one stores its two
//    outputs, in natural order, from registers;
//  * a layer's twiddle, in the four-part form (557 cycles a multiply for a lone
//    warp, the general one takes 765), is loaded before the barrier that the
//    layer waits on;
//  * the first six layers' exchanges stay inside a warp (__syncwarp);
//  * the second pass's blocks are placed while the first pass drains.
// GB300, us per call, against the form before it (general multiply, canonical
// additions, a barrier and a dependent twiddle load per layer): 2^9 11.0 (14.4),
// 2^12 12.3 (18.4), 2^14 14.3 (20.5), 2^16 18.5 (30.7), 2^17 34.8 (49.0); up to
// 2^8 the host's call takes longer than the kernel.  2^18: 54.9 here, 55.3 with
// the tile kernel; 2^19: 109 and 94.
// Values are lazy (below 2r) until the last pass stores them.  Every input of
// the block is read before the first barrier, so one pass may run in place
// (with one warp: before the first __syncwarp).
__device__ __forceinline__ uint32_t small_swz(uint32_t i) {
  return i ^ (((i >> 3) ^ (i >> 6) ^ (i >> 9)) & 7u);
}
// twiddles of layer s >= 1 (w_{2^(s+1)}^j, j < 2^s), eight planes of 2^s units
__host__ __device__ __forceinline__ uint32_t layer_offset(uint32_t s) { return 8 * ((1u << s) - 1); }
constexpr uint32_t kLayerUnits = 8 * 1023;  // layers 0 .. 9

__global__ void __launch_bounds__(512) k_ntt_small_pass(const PassArgs a) {
  extern __shared__ uint4 sm[];
  const uint32_t lgR = a.lgR, R = 1u << lgR, half = R >> 1, b = threadIdx.x;
  uint4 *lo = sm, *hi = sm + R;  // element i: words 0..3 at lo[swz(i)], 4..7 at hi
  const auto put = [&](uint32_t i, const fr &v) {
    lo[small_swz(i)] = make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]);
    hi[small_swz(i)] = make_uint4(v.v[4], v.v[5], v.v[6], v.v[7]);
  };
  const auto get = [&](uint32_t i) {
    const uint4 u = lo[small_swz(i)], v = hi[small_swz(i)];
    return fr{{u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w}};
  };
  const TileGeom geo = tile_geom(a, blockIdx.x);
  const bool active = b < half;
  const uint32_t bn = __brev(b) >> (33 - lgR);  // row of the thread's first input
  // a dependent pass may start while the one before it drains
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  fr x[2];
  if (active) {
#pragma unroll
    for (uint32_t i = 0; i < 2; ++i) {
      const uint64_t g = geo.src(a, bn + i * half, 0);
      if (!a.first) {
        x[i] = ldcs_fr(a.in + g);
      } else if (a.in_kind == NTT_IN_SPREAD) {
        x[i] = (g & ((1ull << a.spread) - 1)) == 0 ? ldcs_fr(a.in + (g >> a.spread)) : fr_zero();
      } else {
        x[i] = g < a.n_valid ? ldcs_fr(a.in + g) : fr_zero();
      }
    }
    if (a.first && a.in_kind == NTT_IN_DIAG) {
#pragma unroll 1
      for (uint32_t i = 0; i < 2; ++i) {
        const uint64_t g = geo.src(a, bn + i * half, 0);
        const fr d = g < a.n_valid ? ldcs_fr(a.diag + g) : fr_zero();
        const fr v = fr_mul_lazy(i ? x[1] : x[0], d);
        if (i) x[1] = v;
        else x[0] = v;
      }
    }
    bfly(x[0], x[1]);
    put(2 * b, x[0]);
    put(2 * b + 1, x[1]);
  }
  uint32_t p = 2 * b, q = 2 * b + 1;
#pragma unroll 1
  for (uint32_t s = 1; s < lgR; ++s) {
    const uint32_t j = b & ((1u << s) - 1);
    uint4 w[8];
    if (active) {
      const uint4 *t = a.tw_dit + layer_offset(s) + j;
#pragma unroll
      for (int k = 0; k < 8; ++k) w[k] = __ldg(t + (k << s));
    }
    // layers 0 .. 5 stay within the 64 elements of a warp
    if (s <= 5) __syncwarp();
    else __syncthreads();
    p = ((b >> s) << (s + 1)) + j;
    q = p + (1u << s);
    if (active) {
      fr wp[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        wp[k] = fr{{w[2 * k].x, w[2 * k].y, w[2 * k].z, w[2 * k].w, w[2 * k + 1].x, w[2 * k + 1].y,
                    w[2 * k + 1].z, w[2 * k + 1].w}};
      x[0] = get(p);
      x[1] = fr_mul_const4(get(q), wp);
      bfly(x[0], x[1]);
      if (s + 1 < lgR) {
        put(p, x[0]);
        put(q, x[1]);
      }
    }
  }
  if (!active) return;
#pragma unroll 1
  for (uint32_t i = 0; i < 2; ++i) {
    const uint64_t o = i ? q : p;
    fr v = i ? x[1] : x[0];
    if (!a.last) {
      v = fr_mul_lazy(v, ldcs_fr(a.tw_layer + (o << a.lgS) + geo.col0));
      st_fr(a.out + geo.base + (o << a.lgS), v);
    } else {
      v = fr_canon(v);
      if (a.has_post_scale) v = fr_mul(v, a.post_scale);
      st_fr(a.out + geo.out_base + (o << (a.lgN - a.lgR)), v);
    }
  }
}

// transforms of 1, 2 or 4 points (one thread, direct evaluation)
__global__ void k_ntt_tiny(const fr *in, fr *out, uint32_t lgN, fr w, fr scale, int has_scale,
                           uint32_t in_kind, const fr *diag, uint64_t n_valid, uint32_t spread) {
  const uint32_t n = 1u << lgN;
  fr x[4], y[4];
  for (uint32_t i = 0; i < n; ++i) {
    if (in_kind == NTT_IN_SPREAD)
      x[i] = (i & ((1u << spread) - 1)) == 0 ? in[i >> spread] : fr_zero();
    else if (i < n_valid)
      x[i] = in_kind == NTT_IN_DIAG ? fr_mul(in[i], diag[i]) : in[i];
    else
      x[i] = fr_zero();
  }
  for (uint32_t k = 0; k < n; ++k) {
    fr acc = fr_zero(), wk = fr_one(), wkj = fr_one();
    for (uint32_t t = 0; t < k; ++t) wk = fr_mul(wk, w);
    for (uint32_t j = 0; j < n; ++j) {
      acc = fr_add(acc, fr_mul(x[j], wkj));
      wkj = fr_mul(wkj, wk);
    }
    y[k] = has_scale ? fr_mul(acc, scale) : acc;
  }
  for (uint32_t k = 0; k < n; ++k) out[k] = y[k];
}

// out[i] = base^e(i) via three 10-bit windows; e(i) = i (kind 0) or
// (i >> lgS) * (i & (2^lgS - 1)) (kind 1, layer tables); optional scale.
__global__ void k_pow_table(fr *out, uint64_t count, const fr *__restrict__ win, uint32_t kind,
                            uint32_t lgS, fr scale, int has_scale) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < count;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t e = kind == 0 ? i : (i >> lgS) * (i & ((1ull << lgS) - 1));
    fr v = ldg_fr(win + (e & 1023));
    if ((e >> 10) & 1023) v = fr_mul(v, ldg_fr(win + 1024 + ((e >> 10) & 1023)));
    if ((e >> 20) & 1023) v = fr_mul(v, ldg_fr(win + 2048 + ((e >> 20) & 1023)));
    if (has_scale) v = fr_mul(v, scale);
    st_fr(out + i, v);
  }
}

// the round tables (round_column, mul_round_twiddle) from inner[e] = w_2048^e:
// block 7 (lgSj - 1) + k - 1, one thread per column
struct Fr4 {
  fr v[4];
};
__global__ void k_round_table(uint4 *out, const fr *__restrict__ inner, const Fr4 f) {
  const uint32_t lgSj = blockIdx.x / 7 + 1, k = blockIdx.x % 7 + 1, c = threadIdx.x;
  if (c >> lgSj) return;
  const fr w = ldg_fr(inner + ((c * k) << (8 - lgSj)));
  uint4 *t = out + (k - 1) * 8 * kRoundStride + round_column(lgSj) + c;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const fr v = fr_mul(w, f.v[p]);
    t[2 * p * kRoundStride] = make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]);
    t[(2 * p + 1) * kRoundStride] = make_uint4(v.v[4], v.v[5], v.v[6], v.v[7]);
  }
}

// the latency form's layer tables from inner[e] = w_2048^e: layer blockIdx.y,
// one thread per entry
__global__ void k_layer_table(uint4 *out, const fr *__restrict__ inner, const Fr4 f) {
  const uint32_t s = blockIdx.y, j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >> s) return;
  const fr w = ldg_fr(inner + (j << (10 - s)));
  uint4 *t = out + layer_offset(s) + j;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const fr v = fr_mul(w, f.v[p]);
    t[(2 * p) << s] = make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]);
    t[(2 * p + 1) << s] = make_uint4(v.v[4], v.v[5], v.v[6], v.v[7]);
  }
}

// ------------------------------------------------------------ host side
namespace {

std::mutex g_mu;

struct RoundKey {
  int dev;
  bool inv;
  bool operator<(const RoundKey &o) const { return std::tie(dev, inv) < std::tie(o.dev, o.inv); }
};

struct Plan {
  uint32_t lgN = 0;
  bool inverse = false;
  uint32_t P = 0;
  uint32_t lgR[4] = {0, 0, 0, 0};
  uint32_t lgT[4] = {0, 0, 0, 0};
  const uint4 *tw_round = nullptr;
  fr *tw_layer[4] = {nullptr, nullptr, nullptr, nullptr};
  // host-pass plans: split layer tables instead of tw_layer
  fr *tw_lo[4] = {nullptr, nullptr, nullptr, nullptr};
  fr *tw_hi[4] = {nullptr, nullptr, nullptr, nullptr};
  uint32_t tw_lgh[4] = {0, 0, 0, 0};
  fr post_scale;
  bool has_post_scale = false;
};

void free_plan_tables(Plan *p) {
  for (int j = 0; j < 4; ++j) {
    cudaFree(p->tw_layer[j]);
    cudaFree(p->tw_lo[j]);
    cudaFree(p->tw_hi[j]);
  }
}

struct PlanKey {
  int dev;
  uint32_t lgN;
  bool inv;
  bool small;  // the latency form for single calls of 2^9 .. 2^17 points
  bool split;  // split layer tables (host-pass transforms)
  bool host;   // host endpoints that the size's own split serves badly
  bool operator<(const PlanKey &o) const {
    return std::tie(dev, lgN, inv, small, split, host) <
           std::tie(o.dev, o.lgN, o.inv, o.small, o.split, o.host);
  }
};

struct PowKey {
  int dev;
  uint32_t lg;
  uint32_t h[8];
  bool operator<(const PowKey &o) const {
    if (dev != o.dev) return dev < o.dev;
    if (lg != o.lg) return lg < o.lg;
    return std::memcmp(h, o.h, sizeof(h)) < 0;
  }
};

std::map<RoundKey, uint4 *> g_round;
std::map<PlanKey, Plan *> g_plans;
std::map<PowKey, fr *> g_pows;
std::map<uint32_t, std::vector<uint32_t>> g_split_override;

std::vector<uint32_t> default_split(uint32_t lgN) {
  std::vector<uint32_t> b;
  if (lgN <= 11) {
    b.push_back(lgN);
    return b;
  }
  const uint32_t P = (lgN + 8) / 9;
  for (uint32_t p = 0; p < P; ++p) b.push_back(lgN / P + (p < lgN % P ? 1 : 0));
  return b;
}

// The split for host endpoints (host_split_differs): the passes that touch host
// memory are bound by the link and do their multiplies beside it, so they take
// as many bits as whole 128-byte lines allow (9) and the middle pass the rest.
// 2^22 points: 9, 4, 9 bits 1626 us, 8, 7, 7 bits 1696 us.
std::vector<uint32_t> host_split(uint32_t lgN) {
  if (lgN < 19 || lgN > 27) return default_split(lgN);
  const uint32_t mid = lgN > 21 ? lgN - 18 : 3, ends = lgN - mid;
  return {ends - ends / 2, mid, ends / 2};
}

int build_windows(const fr &base, fr **d_win) {
  std::vector<fr> w(3072);
  fr step = base;
  for (int k = 0; k < 3; ++k) {
    w[1024 * k] = fr_one();
    for (int j = 1; j < 1024; ++j) w[1024 * k + j] = fr_mul(w[1024 * k + j - 1], step);
    fr s = step;
    for (int t = 0; t < 10; ++t) s = fr_sqr(s);  // step^(2^10)
    step = s;
  }
  PP_COUNT_ALLOC(3072 * sizeof(fr));
  PP_CUDA_TRY(cudaMalloc(d_win, 3072 * sizeof(fr)));
  PP_CUDA_TRY(cudaMemcpy(*d_win, w.data(), 3072 * sizeof(fr), cudaMemcpyHostToDevice));
  return PP_OK;
}

// builds base^e(i) for i < count on the device (synchronous: setup only)
int build_table(fr **out, uint64_t count, const fr &base, uint32_t kind, uint32_t lgS,
                const fr *scale) {
  fr *win = nullptr;
  int st = build_windows(base, &win);
  if (st) return st;
  PP_COUNT_ALLOC(count * sizeof(fr));
  cudaError_t e = cudaMalloc(out, count * sizeof(fr));
  if (e != cudaSuccess) {
    cudaFree(win);
    set_error("table allocation of %llu elements failed: %s", (unsigned long long)count,
              cudaGetErrorString(e));
    return PP_E_NOMEM;
  }
  const int threads = 256;
  const uint64_t blocks64 = (count + threads - 1) / threads;
  const int blocks = (int)(blocks64 < 152 * 64 ? blocks64 : 152 * 64);
  k_pow_table<<<blocks, threads>>>(*out, count, win, kind, lgS, scale ? *scale : fr_one(),
                                   scale ? 1 : 0);
  PP_COUNT_LAUNCH();
  e = cudaDeviceSynchronize();
  cudaFree(win);
  if (e != cudaSuccess) {
    set_error("table kernel failed: %s", cudaGetErrorString(e));
    return PP_E_CUDA;
  }
  return PP_OK;
}

// the round tables of a direction (kRoundUnits 16-byte units), then the layer
// tables of the latency form (kLayerUnits)
int get_round(int dev, bool inv, const uint4 **out) {
  const RoundKey k{dev, inv};
  auto it = g_round.find(k);
  if (it != g_round.end()) {
    *out = it->second;
    return PP_OK;
  }
  fr *inner = nullptr;  // w_2048^e, e < 2048
  const int st = build_table(&inner, 2048, host_root_of_unity(11, inv), 0, 0, nullptr);
  if (st) return st;
  // factors that take a Montgomery-form w to w 2^(64 p + 96)
  Fr4 f;
  std::memset(&f, 0, sizeof(f));
  for (int p = 0; p < 3; ++p) f.v[p].v[2 * p + 3] = 1;
  f.v[3] = host_mont_small(1ull << 32);  // 2^288
  uint4 *t = nullptr;
  const size_t bytes = (kRoundUnits + kLayerUnits) * sizeof(uint4);
  PP_COUNT_ALLOC(bytes);
  cudaError_t e = cudaMalloc(&t, bytes);
  if (e != cudaSuccess) {
    cudaFree(inner);
    set_error("round twiddle tables: %s", cudaGetErrorString(e));
    return PP_E_NOMEM;
  }
  k_round_table<<<7 * 8, 256>>>(t, inner, f);
  PP_COUNT_LAUNCH();
  k_layer_table<<<dim3(2, 10), 256>>>(t + kRoundUnits, inner, f);
  PP_COUNT_LAUNCH();
  e = cudaDeviceSynchronize();
  cudaFree(inner);
  if (e != cudaSuccess) {
    cudaFree(t);
    set_error("table kernel failed: %s", cudaGetErrorString(e));
    return PP_E_CUDA;
  }
  g_round[k] = t;
  *out = t;
  return PP_OK;
}

// small: two passes of about lgN / 2 bits with one column per tile, so that
// each pass of a 2^9 .. 2^17-point transform spreads over 16 .. 512 blocks
// (the throughput plan's 2048-element tiles give 1 .. 64)
// split: layer twiddles as two tables of about 2^(lgRS / 2) entries each
// (w^i and w^(i 2^h)) instead of one of 2^lgRS, for transforms whose data
// never sits in device memory
// host: host_split instead of the size's own split (host_split_differs)
int get_plan(int dev, uint32_t lgN, bool inv, Plan **out, bool small = false, bool split = false,
             bool host = false) {
  PlanKey key{dev, lgN, inv, small, split, host};
  auto it = g_plans.find(key);
  if (it != g_plans.end()) {
    *out = it->second;
    return PP_OK;
  }
  auto ov = g_split_override.find(lgN);
  std::vector<uint32_t> bits =
      host ? host_split(lgN) : ov != g_split_override.end() ? ov->second : default_split(lgN);
  if (small) bits = {lgN - lgN / 2, lgN / 2};
  Plan *p = new Plan();
  p->lgN = lgN;
  p->inverse = inv;
  p->P = (uint32_t)bits.size();
  const fr ninv = host_inv(host_mont_small(1ull << lgN));
  int st = get_round(dev, inv, &p->tw_round);
  if (st) {
    delete p;
    return st;
  }
  uint32_t acc = 0;
  for (uint32_t j = 0; j < p->P; ++j) {
    p->lgR[j] = bits[j];
    acc += bits[j];
    const uint32_t lgS = lgN - acc;
    if (p->P == 1 || small) {
      p->lgT[j] = 0;
    } else if (j + 1 < p->P) {
      const uint32_t want = 11 - bits[j];
      p->lgT[j] = want < lgS ? want : lgS;
    } else {
      const uint32_t want = 11 - bits[j];
      p->lgT[j] = want < bits[0] ? want : bits[0];
    }
    if (j + 1 < p->P) {
      // w_{R S}^(c k) with R S = 2^(lgN - (acc - bits[j]))
      const uint32_t lgRS = lgN - (acc - bits[j]);
      const bool fold = inv && j == 0;  // 2^-lgN folded into the first layer
      const fr w = host_root_of_unity((int)lgRS, inv);
      if (!split) {
        st = build_table(&p->tw_layer[j], 1ull << lgRS, w, 1, lgS, fold ? &ninv : nullptr);
      } else {
        const uint32_t h = (lgRS + 1) / 2;
        p->tw_lgh[j] = h;
        st = build_table(&p->tw_lo[j], 1ull << h, w, 0, 0, fold ? &ninv : nullptr);
        if (!st) st = build_table(&p->tw_hi[j], 1ull << (lgRS - h), host_pow(w, 1ull << h), 0, 0, nullptr);
      }
      if (st) {
        free_plan_tables(p);
        delete p;
        return st;
      }
    }
  }
  if (inv && p->P == 1) {
    p->post_scale = ninv;
    p->has_post_scale = true;
  }
  g_plans[key] = p;
  *out = p;
  return PP_OK;
}

// Whether a transform with host endpoints should leave the size's own split:
// passes of 10 or 11 bits take one or two columns per tile, so the first
// pass's reads and the last one's writes are 32- or 64-byte pieces of host
// memory.  host_split's passes move whole 128-byte lines (2^22 points: 2042 us
// with 11 + 11 bits, 1626 with 9 + 4 + 9; the link alone takes 640 in and 700
// out).  Not while the stream is being captured
// unless its tables exist: building them allocates.
bool host_split_differs(uint32_t lgN, const NttInputDesc &in) {
  if (!in.in_host && !in.out_host) return false;
  const auto ov = g_split_override.find(lgN);
  if (ov == g_split_override.end() || ov->second.size() < 2) return false;
  return (in.in_host && ov->second.front() > 9) || (in.out_host && ov->second.back() > 9);
}

bool g_attr_set[64] = {false};

}  // namespace

int ntt_prepare(uint32_t lg_m, bool inverse, bool host_endpoints) {
  if (lg_m > PP_MAX_LG_N) return PP_E_UNSUPPORTED;
  int dev = 0;
  PP_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_mu);
  if (lg_m <= 2) return PP_OK;
  Plan *p = nullptr;
  int st = get_plan(dev, lg_m, inverse, &p);
  if (!st && ntt_small_form(lg_m)) st = get_plan(dev, lg_m, inverse, &p, true);
  if (!st && host_endpoints && !ntt_small_form(lg_m)) {
    NttInputDesc both;
    both.in_host = both.out_host = true;
    if (host_split_differs(lg_m, both)) st = get_plan(dev, lg_m, inverse, &p, false, false, true);
  }
  return st;
}

int ntt_set_split(uint32_t lg_m, const uint32_t *bits) {
  std::lock_guard<std::mutex> lk(g_mu);
  if (!bits) {
    g_split_override.erase(lg_m);
  } else {
    std::vector<uint32_t> b;
    uint32_t sum = 0;
    for (int i = 0; i < 4 && bits[i]; ++i) {
      if (bits[i] < 3 || bits[i] > 11) return PP_E_INVAL;
      b.push_back(bits[i]);
      sum += bits[i];
    }
    if (sum != lg_m || b.empty() || (b.size() > 1 && lg_m <= 3)) return PP_E_INVAL;
    g_split_override[lg_m] = b;
  }
  // drop cached plans of this size so the next call rebuilds them
  for (auto it = g_plans.begin(); it != g_plans.end();) {
    if (it->first.lgN == lg_m) {
      free_plan_tables(it->second);
      delete it->second;
      it = g_plans.erase(it);
    } else {
      ++it;
    }
  }
  return PP_OK;
}

void ntt_get_split(uint32_t lg_m, uint32_t *bits, uint32_t *npass) {
  std::lock_guard<std::mutex> lk(g_mu);
  auto ov = g_split_override.find(lg_m);
  std::vector<uint32_t> b = ov != g_split_override.end() ? ov->second : default_split(lg_m);
  *npass = (uint32_t)b.size();
  for (size_t i = 0; i < b.size() && i < 4; ++i) bits[i] = b[i];
}

const fr *pow_table(const fr &h, uint32_t lg_n, int *status) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    *status = PP_E_CUDA;
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(g_mu);
  PowKey k{dev, lg_n, {}};
  std::memcpy(k.h, h.v, sizeof(k.h));
  auto it = g_pows.find(k);
  if (it != g_pows.end()) {
    *status = PP_OK;
    return it->second;
  }
  fr *t = nullptr;
  *status = build_table(&t, 1ull << lg_n, h, 0, 0, nullptr);
  if (*status) return nullptr;
  g_pows[k] = t;
  return t;
}

void ntt_release_tables() {
  std::lock_guard<std::mutex> lk(g_mu);
  for (auto &kv : g_round) cudaFree(kv.second);
  for (auto &kv : g_plans) {
    free_plan_tables(kv.second);
    delete kv.second;
  }
  for (auto &kv : g_pows) cudaFree(kv.second);
  g_round.clear();
  g_plans.clear();
  g_pows.clear();
}

namespace {
int describe_passes(const fr *d_in, fr *d_out, fr *work, uint32_t lg_m, bool inverse,
                    const NttInputDesc &in, std::vector<PassArgs> &passes,
                    std::vector<uint64_t> &tiles, bool small, bool split, bool host);
}  // namespace

int ntt_describe(const fr *d_in, fr *d_out, fr *work, uint32_t lg_m, bool inverse,
                 const NttInputDesc &in, std::vector<PassArgs> &passes,
                 std::vector<uint64_t> &tiles, bool small, bool host) {
  return describe_passes(d_in, d_out, work, lg_m, inverse, in, passes, tiles, small, false, host);
}

namespace {
int describe_passes(const fr *d_in, fr *d_out, fr *work, uint32_t lg_m, bool inverse,
                    const NttInputDesc &in, std::vector<PassArgs> &passes,
                    std::vector<uint64_t> &tiles, bool small, bool split, bool host) {
  if (lg_m > PP_MAX_LG_N || lg_m < 3) {
    set_error("batched transform of 2^%u points: supported sizes are 2^3 .. 2^%d", lg_m, PP_MAX_LG_N);
    return PP_E_UNSUPPORTED;
  }
  const uint64_t N = 1ull << lg_m;
  int dev = 0;
  PP_CUDA_TRY(cudaGetDevice(&dev));
  Plan *plan = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    int st = get_plan(dev, lg_m, inverse, &plan, small, split, host);
    if (st) return st;
    if (dev < 64 && !g_attr_set[dev]) {
      PP_CUDA_TRY(cudaFuncSetAttribute(k_ntt_pass<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kTileBytes));
      PP_CUDA_TRY(cudaFuncSetAttribute(k_ntt_pass<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kTileBytes));
      PP_CUDA_TRY(cudaFuncSetAttribute(k_ntt_batch_level,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kTileBytes));
      g_attr_set[dev] = true;
    }
  }
  if (plan->P > 1 && !work) {
    set_error("transform of 2^%u points needs a workspace", lg_m);
    return PP_E_INVAL;
  }
  PassArgs a;
  std::memset(&a, 0, sizeof(a));
  a.lgN = lg_m;
  a.P = plan->P;
  a.inverse = inverse ? 1 : 0;
  a.tw_round = plan->tw_round;
  a.tw_dit = plan->tw_round + kRoundUnits;
  for (uint32_t j = 0; j < plan->P; ++j) a.lgRp[j] = plan->lgR[j];
  a.diag = in.diag;
  a.diag_hi = in.diag_hi;
  a.diag_lgh = in.diag_lgh;
  a.n_valid = in.n_valid ? in.n_valid : N;
  a.in_kind = (uint32_t)in.kind;
  a.spread = in.spread;
  uint32_t acc = 0;
  for (uint32_t j = 0; j < plan->P; ++j) {
    acc += plan->lgR[j];
    a.lgR = plan->lgR[j];
    a.lgT = plan->lgT[j];
    a.lgS = lg_m - acc;
    a.first = j == 0;
    a.last = j + 1 == plan->P;
    a.unit_in = a.first && in.in_host;
    // zero-padded input (n_valid = N / 2^z): pass 1's rows >= R >> z are zero
    a.zero_lg = 0;
    if (a.first && !a.last && in.kind != NTT_IN_SPREAD && in.n_valid && in.n_valid < N &&
        (in.n_valid & (in.n_valid - 1)) == 0) {
      uint32_t z = 0;
      while ((in.n_valid << z) < N) ++z;
      a.zero_lg = z;
    }
    a.unit_out = a.last && in.out_host;
    a.in = j == 0 ? d_in : work;
    a.out = a.last ? d_out : work;
    a.tw_layer = plan->tw_layer[j];
    a.tw_lo = plan->tw_lo[j];
    a.tw_hi = plan->tw_hi[j];
    a.tw_lgh = plan->tw_lgh[j];
    a.has_post_scale = a.last && plan->has_post_scale;
    a.post_scale = plan->post_scale;
    passes.push_back(a);
    tiles.push_back(N >> (a.lgR + a.lgT));
  }
  return PP_OK;
}
}  // namespace

// One kernel over `blocks` tiles.  After another pass its blocks may be placed
// while that one drains; they wait for it (griddepcontrol.wait) before they read.
// On average a boundary costs 1.5 us less: 2^18 points 50.2 -> 48.6 us, 2^19 90.1 ->
// 87.3, 2^21 319 -> 315.  A batch plan's levels gained nothing by it.
static int launch_pass(void (*kernel)(const PassArgs), const PassArgs &args, uint64_t blocks, uint32_t threads, size_t smem,
                       bool follows, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = follows ? 1 : 0;
  PP_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, args));
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}

int ntt_launch_level(const LevelParams &params, cudaStream_t stream) {
  if (!params.total_tiles) return PP_OK;
  if (params.total_tiles > 0x7fffffffull) {
    set_error("batch level of %llu tiles exceeds one launch", (unsigned long long)params.total_tiles);
    return PP_E_UNSUPPORTED;
  }
  k_ntt_batch_level<<<(unsigned)params.total_tiles, 256, kTileBytes, stream>>>(params);
  PP_COUNT_LAUNCH();
  PP_LAUNCH_CHECK();
  return PP_OK;
}

int ntt_run(const fr *d_in, fr *d_out, uint32_t lg_m, bool inverse, const NttInputDesc &in,
            cudaStream_t stream) {
  if (lg_m > PP_MAX_LG_N) {
    set_error("transform of 2^%u points exceeds the supported 2^%d", lg_m, PP_MAX_LG_N);
    return PP_E_UNSUPPORTED;
  }
  const uint64_t N = 1ull << lg_m;
  const uint64_t n_valid = in.n_valid ? in.n_valid : N;
  if (lg_m <= 2) {
    const fr w = host_root_of_unity((int)lg_m, inverse);
    const fr s = host_inv(host_mont_small(N));
    k_ntt_tiny<<<1, 1, 0, stream>>>(d_in, d_out, lg_m, w, s, inverse ? 1 : 0, in.kind, in.diag,
                                    n_valid, in.spread);
    PP_COUNT_LAUNCH();
    PP_LAUNCH_CHECK();
    return PP_OK;
  }
  const bool small = ntt_small_form(lg_m);
  bool host = false;
  if (!small && (in.in_host || in.out_host)) {
    int dev = 0;
    PP_CUDA_TRY(cudaGetDevice(&dev));
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    PP_CUDA_TRY(cudaStreamIsCapturing(stream, &cap));
    std::lock_guard<std::mutex> lk(g_mu);
    host = host_split_differs(lg_m, in) &&
           (cap == cudaStreamCaptureStatusNone ||
            g_plans.count(PlanKey{dev, lg_m, inverse, false, false, true}));
  }
  uint32_t bits[4], np = 2;
  if (!small) ntt_get_split(lg_m, bits, &np);
  fr *work = nullptr;
  if (np > 1) {
    int st = PP_OK;
    work = static_cast<fr *>(workspace_get(N * sizeof(fr), stream, 0, &st));
    if (st) return st;
  }
  std::vector<PassArgs> passes;
  std::vector<uint64_t> tiles;
  int st = ntt_describe(d_in, d_out, work, lg_m, inverse, in, passes, tiles, small, host);
  if (st) return st;
  if (small || (passes.size() == 1 && lg_m <= kSmallOnePass)) {
    for (size_t j = 0; j < passes.size(); ++j) {
      const uint32_t R = 1u << passes[j].lgR;
      if ((st = launch_pass(k_ntt_small_pass, passes[j], tiles[j], R / 2 < 32 ? 32 : R / 2, R * sizeof(fr), j > 0 || in.follows, stream)))
        return st;
    }
    return PP_OK;
  }
  for (size_t j = 0; j < passes.size(); ++j) {
    const uint32_t E = 1u << (passes[j].lgR + passes[j].lgT);
    const bool host_io = passes[j].unit_in || passes[j].unit_out;
    if ((st = launch_pass(host_io ? k_ntt_pass<true> : k_ntt_pass<false>, passes[j], tiles[j], E / 8, kTileBytes, j > 0 || in.follows, stream)))
      return st;
  }
  return PP_OK;
}

int ntt_host_plan_passes(uint32_t lg_m, uint32_t *passes) {
  if (lg_m <= 11) {
    *passes = 1;
    return PP_OK;
  }
  int dev = 0;
  PP_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_mu);
  Plan *plan = nullptr;
  const int st = get_plan(dev, lg_m, false, &plan, false, true);
  if (st) return st;
  *passes = plan->P;
  return PP_OK;
}

int ntt_run_host_passes(const fr *h_in, fr *h_out, fr *h_scratch, uint32_t lg_m, bool inverse,
                        cudaStream_t stream) {
  return ntt_run_host_passes(h_in, h_out, h_scratch, lg_m, inverse, NttInputDesc(), stream);
}

int ntt_run_host_passes(const fr *h_in, fr *h_out, fr *h_scratch, uint32_t lg_m, bool inverse,
                        const NttInputDesc &desc, cudaStream_t stream) {
  NttInputDesc in = desc;
  in.in_host = in.out_host = true;
  if (lg_m <= 11) {
    // one pass (or the tiny kernel): host in, host out, no intermediate; a
    // diagonal here is a full table (at most 2^11 entries)
    if (in.diag_hi) {
      set_error("transform of 2^%u points: split diagonal tables are for more than 2^11 points", lg_m);
      return PP_E_INVAL;
    }
    return ntt_run(h_in, h_out, lg_m, inverse, in, stream);
  }
  if (lg_m > PP_MAX_LG_N) {
    set_error("transform of 2^%u points exceeds the supported 2^%d", lg_m, PP_MAX_LG_N);
    return PP_E_UNSUPPORTED;
  }
  if (in.kind == NTT_IN_DIAG && !in.diag_hi) {
    set_error("transform of 2^%u points over host memory: the diagonal must be split", lg_m);
    return PP_E_INVAL;
  }
  std::vector<PassArgs> passes;
  std::vector<uint64_t> tiles;
  int st = describe_passes(h_in, h_out, h_scratch, lg_m, inverse, in, passes, tiles, false, true, false);
  if (st) return st;
  // pass j reads X_j and writes X_(j+1): X_0 = h_in, X_P = h_out, and the
  // intermediates alternate so that X_(P-1) = h_scratch
  const size_t P = passes.size();
  std::vector<fr *> X(P + 1);
  X[0] = const_cast<fr *>(h_in);
  X[P] = h_out;
  for (size_t j = P - 1; j >= 1; --j) X[j] = ((P - 1 - j) & 1) ? h_out : h_scratch;
  for (size_t j = 0; j < P; ++j) {
    PassArgs &a = passes[j];
    a.in = X[j];
    a.out = X[j + 1];
    a.unit_in = 1;
    a.unit_out = 1;
    const uint32_t E = 1u << (a.lgR + a.lgT);
    k_ntt_pass<true><<<(unsigned)tiles[j], E / 8, kTileBytes, stream>>>(a);
    PP_COUNT_LAUNCH();
    PP_LAUNCH_CHECK();
  }
  return PP_OK;
}

}  // namespace pp
