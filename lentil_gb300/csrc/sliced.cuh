// Exact-sum GEMMs on the tensor cores: FP64-accurate products by slicing.
//
// This part's FP64 units retire two FMAs a clock per SM, its tensor cores
// 4096 bf16 ones, so each FP64 product is taken apart into bf16 products
// whose sums are exact (the error-free transformation of Ozaki, Ogita, Oishi
// and Rump, Numerical Algorithms 59, 2012; on tensor cores: Mukunoki et al.,
// ISC 2020):
//   - every vector of a contraction (a column of f, a row of E1, ...) is
//     scaled by a power of two above its largest entry and cut into signed
//     digits of 9 bits, |d| <= 256, each exact in bf16; digit i is stored as
//     d 2^(-9 i).  Data has ND = 7 digits (62 bits below the vector's largest
//     entry: with 54, fields with isolated spikes lost a factor of two against
//     FP64), a DFT matrix NE = 6 (its entries are 53-bit numbers of modulus 1);
//   - the products of digits with i + j <= 6 are kept, grouped by s = i + j.  A
//     group's sum over 64 K entries is at most (s + 1) 64 2^16 <= 2^24 units
//     for s <= 3: the FP32 accumulators hold it exactly, whatever order or
//     rounding the tensor core uses.  Groups 4 to 6 share an accumulator
//     (their rounding is below 2^-56 of the operands);
//   - every 64 K entries (256 for group 0, 128 for group 1: their sums have the
//     room) the accumulators are drained into 64-bit integers in registers, in
//     units of 2^-(16 + S): exact for groups 0-3.  Integer sums
//     do not depend on their order, so dealing K out over CTAs gives the same
//     bits.
// What is left is the rounding of the operands, the products left out, and one
// rounding per stored result; an FP64 accumulation rounds at every K step.
//
// A complex product needs no complex arithmetic on the way: operand B holds
// the row sets [-im | re | im], operand A the sets [re | im], and a tile's
// columns are 48 real and the same 48 imaginary parts,
//     A re rows x (B re, B im rows)  +  A im rows x (B -im, B re rows),
// so that the accumulators hold the complex sums.  Real operands have one set
// and a tile 96 columns.
#pragma once

#include <algorithm>
#include <cmath>
#include <mutex>

#include "common.cuh"
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace lgb {
namespace {

using namespace tc;


constexpr int ND = 7;                        // digits of a data operand (f, the intermediate)
constexpr int NE = 6;                        // digits of a DFT matrix (|E| <= 1, 53-bit entries)
constexpr int BETA = 9;                      // bits per digit
constexpr int BM = 128, BC = 48, BK = 32;    // tile: A rows, complex B rows, K per stage
constexpr int BN = 2 * BC;                   // MMA columns
constexpr int STAGES = 2;
constexpr int GROUPS = 5;                    // accumulators: s = 0, 1, 2, 3, and 4 to 6 together
constexpr uint32_t A_SLICE = BM * BK * 2, B_SLICE = BN * BK * 2;
constexpr uint32_t stage_bytes(int na, int nb) { return na * A_SLICE + nb * B_SLICE; }
constexpr int EPI_WARPS = 8;
constexpr int NUM_THREADS = 64 + 32 * EPI_WARPS;
constexpr uint32_t BAR_BYTES = 256;
constexpr uint32_t smem_bytes(int na, int nb) { return STAGES * stage_bytes(na, nb) + BAR_BYTES + 1024; }
constexpr int RUN = BC / 2;                  // tile columns per epilogue warp, of either half
constexpr unsigned long long WAIT_NS = 2000000000ull;
static_assert(smem_bytes(ND, ND) <= 232448, "shared memory per CTA");
static_assert(GROUPS * BN <= 512 && RUN == 24, "tensor memory columns; the drain loads 3 x 8 of them");

// How a launch's work is dealt out: the chains (two stages of one tile: 32
// complex K entries, or 64 real ones) of all tiles in a row, `per` of them to
// each CTA.  A tile's chains then lie in
// one CTA or in a few neighbouring ones, which write a partial sum each.
struct Deal {
  int tilesA, tilesB;        // tiles of one item: A rows (fastest), B rows
  int chains;                // per tile
  int per;                   // chains per CTA
  __host__ __device__ int first_cta(int tile) const { return tile * chains / per; }
  __host__ __device__ int parts(int tile) const {
    return ((tile + 1) * chains - 1) / per - first_cta(tile) + 1;
  }
};

// Which chains of a real contraction a column tile takes: all, or, for a
// banded operand B whose row k covers K entries around k * step, a window.
struct Band {
  int step;                  // 0: all chains
  int total, count;          // chains of the whole contraction, of a window
  __host__ __device__ int first(int tb) const {
    if (step == 0) return 0;
    const int c = (tb * BN * step - step - 34) / 64;         // rows start at most step / 2 + 33 before
    return c < 0 ? 0 : (c < total - count ? c : total - count);
  }
};

struct GemmParams {
  Deal deal;
  Band band;                 // real contractions
  int total;                 // chains of all tiles of all items
  int rowsB;                 // complex
  int ld;                    // P row pitch (entries)
  int dA, dB;                // digit planes between items (0: shared by all items)
  int S;                     // P unit: 2^-(16 + S) of the scaled operands
  void* P;                   // [item][part][rowsB][ld] longlong2 (re, im), or long long
  long long item_stride;     // entries between items
  int* err;
  unsigned long long wait_ns;
};

// One CTA's run of chains of one tile.
struct Segment {
  int item, m0, n0;          // tile origin: complex A row, B row
  int chain, count;
  int part;                  // which of the tile's partial sums
};
template <bool REAL>
__device__ __forceinline__ Segment segment_at(const GemmParams& p, int pos, int end) {
  Segment s;
  const int tile = pos / p.deal.chains;
  s.chain = pos - tile * p.deal.chains;
  s.count = min(p.deal.chains - s.chain, end - pos);
  const int tiles = p.deal.tilesA * p.deal.tilesB;
  s.item = tile / tiles;
  const int t = tile - s.item * tiles;
  const int tb = t / p.deal.tilesA;
  s.m0 = (t - tb * p.deal.tilesA) * BM;
  s.n0 = tb * (REAL ? BN : BC);
  if (REAL) s.chain += p.band.first(tb);
  s.part = (int)blockIdx.x - p.deal.first_cta(tile);
  return s;
}

// Which chains of a segment (r = 0, 1, ...) start and end a sum of group g:
// groups 0 and 1 run over four and two chains, at most 4 * 64 2^16 = 2 * 2 * 64
// 2^16 = 2^24.  (Draining every group after every chain left the MMA waiting
// 16 % of the time for the last ones of 20 drains in four chains; these are 15.)
__device__ __forceinline__ bool starts(int g, int r) {
  return g == 0 ? (r & 3) == 0 : g == 1 ? (r & 1) == 0 : true;
}
__device__ __forceinline__ bool drains(int g, int r, int count) {
  return g == 0 ? (r & 3) == 3 || r == count - 1 : g == 1 ? (r & 1) == 1 || r == count - 1 : true;
}

// The digit products A_i B_j of one sum i + j, two k-steps each, added to the
// accumulator d (started afresh when `fresh`).  The operand descriptors are
// one 64-bit base each plus constants, and the warp stays converged around
// them: with descriptors worked out per MMA, or in a loop that one lane runs
// alone, the issuing warp was the limit, at 95 to 100 clk an MMA.
template <int NA, int NB, int SUM>
__device__ __forceinline__ void mma_sum(uint32_t on, uint32_t d, uint64_t da, uint64_t db, uint32_t idesc,
                                        bool fresh) {
#pragma unroll
  for (int i = 0; i < NA; ++i) {
    const int j = SUM - i;
    if (j < 0 || j >= NB) continue;
#pragma unroll
    for (int k = 0; k < BK / 16; ++k) {
      const bool start = fresh && k == 0 && (i == 0 || SUM - i == NB - 1);   // the first one issued
      mma_f16_cta(on, d, da + ((i * A_SLICE + k * 32) >> 4), db + ((j * B_SLICE + k * 32) >> 4), idesc,
                  start ? 0u : 1u);
    }
  }
}

// P over this CTA's chains.
//
// Bound by the tensor pipe: 108 MMAs (27 digit products x 4 k-steps; 112 for
// two data operands) of 128 x 96 x 16 per chain.  96 columns is the widest tile whose five
// accumulators fit the 512 TMEM columns; the MMA then reads 7 KB of shared
// memory per 48 clocks (149 B/clk against the 128 B/clk port), so it runs at
// 56 clk at best.  Roles: warp 0 TMA (two stages of 32 K entries, all digits),
// warp 1 MMA issue, warps 2..9 drain (lane quadrant w % 4, column half
// (w - 2) / 4).  The groups are drained one by one, in the order they are
// issued, while the next ones run.  One CTA per SM takes its share of the
// chains (Deal), so the pipeline fills once per launch and no wave is partly
// empty.
template <int NA, int NB, bool REAL>
__global__ void __launch_bounds__(NUM_THREADS, 1)
sliced_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const GemmParams p) {
  constexpr uint32_t A_STAGE = NA * A_SLICE, STAGE_BYTES = stage_bytes(NA, NB);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t bars = base + STAGES * STAGE_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 16u + 8u * s; };
  auto acc_full = [&](int g) { return bars + 32u + 8u * g; };
  auto acc_empty = [&](int g) { return bars + 80u + 8u * g; };
  const uint32_t drain_bar = bars + 128u;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + (bars - raw) + 136);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int begin = blockIdx.x * p.deal.per, end = min(p.total, begin + p.deal.per);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int g = 0; g < GROUPS; ++g) {
      mbar_init(acc_full(g), 1);
      mbar_init(acc_empty(g), EPI_WARPS);
    }
    mbar_init(drain_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      prefetch_map(&tmA);
      prefetch_map(&tmB);
      int it = 0;
      bool ok = true;
      for (int pos = begin; ok && pos < end;) {
        const Segment w = segment_at<REAL>(p, pos, end);
        pos += w.count;
        for (int st = 2 * w.chain; st < 2 * (w.chain + w.count); ++st, ++it) {
          const int s = it % STAGES, im = st & 1, k = (REAL ? st : st >> 1) * BK;
          if (!mbar_wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, p.err, p.wait_ns)) { ok = false; break; }
          mbar_expect_tx(full_bar(s), STAGE_BYTES);
          const uint32_t sa = base + s * STAGE_BYTES;
          tma_load_4d_cta(sa, &tmA, full_bar(s), k, w.m0, REAL ? 0 : im, w.item * p.dA);
          tma_load_4d_cta(sa + A_STAGE, &tmB, full_bar(s), k, w.n0, REAL ? 0 : 1 - im, w.item * p.dB);
        }
      }
      for (int k = max(0, it - STAGES); k < it; ++k)       // issued copies land before exit
        mbar_wait_issued(full_bar(k % STAGES), (k / STAGES) & 1, p.wait_ns);
    }
  } else if (warp == 1) {
    const uint32_t on = elect_one();
    auto wait = [&](uint32_t bar, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, p.err, p.wait_ns)) != 0;
    };
    constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                               ((uint32_t)(BM >> 4) << 24);       // FP32 += BF16 . BF16
    int it = 0;                                // stages issued
    int n[GROUPS] = {};                        // drains asked for, by group
    bool ok = true;
    for (int pos = begin; ok && pos < end;) {
      const Segment w = segment_at<REAL>(p, pos, end);
      pos += w.count;
      for (int st = 0; ok && st < 2 * w.count; ++st, ++it) {
        const int s = it % STAGES, r = st >> 1;
        if (!wait(full_bar(s), (it / STAGES) & 1)) { ok = false; break; }
        const uint64_t da = smem_desc_sw64(base + s * STAGE_BYTES);
        const uint64_t db = smem_desc_sw64(base + s * STAGE_BYTES + A_STAGE);
#pragma unroll
        for (int g = GROUPS - 1; g >= 0; --g) {
          const bool first = (st & 1) == 0 && starts(g, r), last = (st & 1) == 1 && drains(g, r, w.count);
          // this accumulator's previous sum has been drained
          if (first && !wait(acc_empty(g), (n[g] & 1) ^ 1)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d = tmem + g * BN;
          if (g == 4) {                        // small products first
            mma_sum<NA, NB, 6>(on, d, da, db, idesc, first);
            mma_sum<NA, NB, 5>(on, d, da, db, idesc, false);
            mma_sum<NA, NB, 4>(on, d, da, db, idesc, false);
          }
          if (g == 3) mma_sum<NA, NB, 3>(on, d, da, db, idesc, first);
          if (g == 2) mma_sum<NA, NB, 2>(on, d, da, db, idesc, first);
          if (g == 1) mma_sum<NA, NB, 1>(on, d, da, db, idesc, first);
          if (g == 0) mma_sum<NA, NB, 0>(on, d, da, db, idesc, first);
          if (last) {
            mma_commit_cta(on, acc_full(g));
            ++n[g];
          }
        }
        if (ok) mma_commit_cta(on, empty_bar(s));
      }
    }
    mma_commit_cta(on, drain_bar);
    mbar_wait_issued(drain_bar, 0, p.wait_ns);
    __syncwarp();
  } else {
    const int q4 = warp & 3, ch = (warp - 2) >> 2;
    const uint32_t trow = tmem + ((uint32_t)(q4 * 32) << 16) + ch * RUN;
    const float unit4 = ldexpf(1.f, p.S);
    const int m1 = 1 << (p.S - BETA), m2 = 1 << (p.S - 2 * BETA), m3 = 1 << (p.S - 3 * BETA);
    int n[GROUPS] = {};                        // drains done, by group
    bool ok = true;
    for (int pos = begin; ok && pos < end;) {
      const Segment w = segment_at<REAL>(p, pos, end);
      pos += w.count;
      long long acc[2 * RUN];                  // RUN real parts, RUN imaginary parts (or 2 RUN columns)
#pragma unroll
      for (int j = 0; j < 2 * RUN; ++j) acc[j] = 0;
      for (int k = 0; ok && k < w.count; ++k) {
#pragma unroll
        for (int g = GROUPS - 1; g >= 0; --g) {
          if (!drains(g, k, w.count)) continue;
          ok = __all_sync(0xffffffffu, mbar_wait(acc_full(g), n[g] & 1, p.err, p.wait_ns));
          if (!ok) break;
          ++n[g];
          tc_fence_after();
          uint32_t r[2 * RUN];
#pragma unroll
          for (int h = 0; h < 6; ++h) tmem_ld8(trow + g * BN + (h / 3) * BC + (h % 3) * 8, r + h * 8);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty(g));
#pragma unroll
          for (int j = 0; j < 2 * RUN; ++j) {
            const float v = __uint_as_float(r[j]);
            if (g == 4) acc[j] += (long long)__float2int_rn(v * unit4);
            else if (g == 3) acc[j] += (long long)__float2int_rn(v * 0x1p27f) * m3;
            else if (g == 2) acc[j] += (long long)__float2int_rn(v * 0x1p18f) * m2;
            else if (g == 1) acc[j] += (long long)__float2int_rn(v * 0x1p9f) * m1;
            else acc[j] += (long long)__float2int_rn(v) << p.S;
          }
        }
      }
      if (!ok) break;
      const int n0 = w.n0 + ch * RUN;
      const size_t at = (size_t)w.item * p.item_stride + ((size_t)w.part * p.rowsB + n0) * p.ld + w.m0 +
                        q4 * 32 + lane;
      if (REAL) {
        long long* out = static_cast<long long*>(p.P) + at;
#pragma unroll
        for (int j = 0; j < 2 * RUN; ++j) {
          const int col = j < RUN ? j : BC + j - RUN;
          if (n0 + col < p.rowsB) out[(size_t)col * p.ld] = acc[j];
        }
      } else {
        longlong2* out = static_cast<longlong2*>(p.P) + at;
#pragma unroll
        for (int j = 0; j < RUN; ++j)
          if (n0 + j < p.rowsB) out[(size_t)j * p.ld] = make_longlong2(acc[j], acc[RUN + j]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// ---------------------------------------------------------------- digits ---
// The N digits of X, |X| <= 2^(9 N - 1), as bf16 bits in the high half of a
// word; digit i carries 2^(-9 i).  A bias of 256 in every place turns the
// signed digits into bit fields; a field under the exponent of 1.5 2^23 is a
// float, and one FMA takes bias and offset off and scales (exactly): three
// instructions a digit, none of them on the conversion or 64-bit paths.
template <int N>
__device__ __forceinline__ void digits_of(long long X, uint32_t (&d)[N]) {
  constexpr unsigned long long ones = 0x0040201008040201ull;          // sum of 2^(9 i), i < 7
  constexpr unsigned long long bias = 256ull * (ones & ((1ull << (BETA * (N - 1))) - 1));
  const unsigned long long Y = (unsigned long long)X + bias;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int sh = BETA * (N - 1 - i);
    const float s = 1.f / (float)(1ull << (BETA * i));
    // the leading digit is signed: 512 more keep its field positive
    const uint32_t u = (uint32_t)(Y >> sh) + (i == 0 ? 512u : 0u);
    const float f = __uint_as_float((u & (i == 0 ? 1023u : 511u)) | 0x4B400000u);
    d[i] = __float_as_uint(fmaf(f, s, -(12582912.f + (i == 0 ? 512.f : 256.f)) * s));
  }
}

// v * 2^e * scale as a double: v * 2^e, rounded to nearest even, is put together
// from its bits (a conversion from 64-bit integers holds the FP64 pipe).
__device__ __forceinline__ double scaled(long long v, int e, double scale) {
  if (v == 0) return 0.0;
  const unsigned long long m = (unsigned long long)(v < 0 ? -v : v);
  const int lz = __clzll((long long)m), exp = 63 - lz + e + 1023;
  if (exp < 1 || exp > 2045) return scalbn((double)v * scale, e);
  const unsigned long long t = m << lz;
  const uint32_t low = (uint32_t)t & 0x7FFu;
  unsigned long long q = t >> 11;                        // 53 bits, the leading one set
  q += low > 0x400u || (low == 0x400u && (q & 1));
  q += (unsigned long long)(exp - 1) << 52;              // a carry goes into the exponent
  return scale * __longlong_as_double((long long)(q | ((unsigned long long)v & 0x8000000000000000ull)));
}

constexpr int XBITS = BETA * ND - 1;         // a data entry is |X| < 2^62 of its vector's scale

// x / 2^(e - 1022) * 2^XBITS rounded to nearest, for |x| < 2^(e - 1022); e is
// a biased exponent >= 1 that is no smaller than x's.
__device__ __forceinline__ long long fixed_data(double x, int e) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  int E = (int)(u >> 52) & 0x7FF;
  long long m = (long long)(u & 0xFFFFFFFFFFFFFull);
  if (E == 0) E = 1; else m |= 1ll << 52;
  const int sh = e - E;                      // m < 2^53 has XBITS - 53 bits of room
  if (sh <= XBITS - 53) m <<= XBITS - 53 - sh;
  else m = sh > XBITS + 1 ? 0 : (m + (1ll << (sh - (XBITS - 53) - 1))) >> (sh - (XBITS - 53));
  return (long long)u < 0 ? -m : m;
}

// Digit operand of L vectors, [digit][set][L][kp] 16-bit entries: the sets of
// complex vectors are re, im (operand A, b = 0), or -im, re, im (operand B,
// b = 1); real ones have one (b = -1).
struct DigitRows {
  uint16_t* base;
  int L, kp, b;
  __host__ __device__ size_t set() const { return (size_t)L * kp; }
  __host__ __device__ size_t plane() const { return (2 + b) * set(); }
};
// Entries k, k + 1 of vector j.
template <int N>
__device__ __forceinline__ void store_digits(const DigitRows& o, int j, int k, long long re0, long long im0,
                                             long long re1, long long im1) {
  uint16_t* p = o.base + (size_t)j * o.kp + k;
  uint32_t a[N], c[N];
  digits_of(im0, a);
  digits_of(im1, c);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t w = __byte_perm(a[i], c[i], 0x7632);
    *reinterpret_cast<uint32_t*>(p + i * o.plane() + (1 + o.b) * o.set()) = w;
    if (o.b) *reinterpret_cast<uint32_t*>(p + i * o.plane()) = w ^ 0x80008000u;
  }
  digits_of(re0, a);
  digits_of(re1, c);
#pragma unroll
  for (int i = 0; i < N; ++i)
    *reinterpret_cast<uint32_t*>(p + i * o.plane() + o.b * o.set()) = __byte_perm(a[i], c[i], 0x7632);
}

constexpr int FLAG_INF = 1, FLAG_NAN = 2;

__device__ __forceinline__ void note_exponent(double x, int& e, int& flag) {
  const unsigned hi = (unsigned)__double2hiint(x) & 0x7FFFFFFFu;
  const int E = (int)(hi >> 20);
  if (E == 0x7FF)
    flag |= (hi & 0xFFFFFu) | (unsigned)__double2loint(x) ? FLAG_NAN : FLAG_INF;
  else
    e = max(e, E);
}

// A product's rows as their readers see them.
template <typename V>
struct PartialSums {
  const V* P;                // [item][part][rows][ld]
  long long item_stride;
  int ld, rows, cols;
  Deal deal;
};

constexpr int MAX_TILES_A = 256;             // 128-row tiles of the longest A operand (32768 rows)

// How many partial sums the tiles under row r of an item have, [tilesA] in
// shared memory (ends with a block barrier).
template <typename V>
__device__ __forceinline__ void count_parts(const PartialSums<V>& q, int item, int r, uint8_t* parts) {
  constexpr int width = sizeof(V) == 16 ? BC : BN;           // rows of a tile
  for (int t = threadIdx.x; t < q.deal.tilesA; t += blockDim.x)
    parts[t] = (uint8_t)q.deal.parts((item * q.deal.tilesB + r / width) * q.deal.tilesA + t);
  __syncthreads();
}

__device__ __forceinline__ void add_to(long long& a, long long b) { a += b; }
__device__ __forceinline__ void add_to(longlong2& a, longlong2 b) { a.x += b.x; a.y += b.y; }

// v[i] = the sum of n[i] parts (0: none) of the entry at offset at[i], i < COUNT.
// The parts go in the outer loop, so that COUNT loads are in flight.
template <int COUNT, typename V>
__device__ __forceinline__ void sum_parts(const V* __restrict__ P, size_t part_stride, const size_t (&at)[COUNT],
                                          const int (&n)[COUNT], V (&v)[COUNT]) {
  int most = 0;
#pragma unroll
  for (int i = 0; i < COUNT; ++i) {
    most = max(most, n[i]);
    v[i] = V{};
  }
  for (int k = 0; k < most; ++k, P += part_stride) {
    V w[COUNT];
#pragma unroll
    for (int i = 0; i < COUNT; ++i) w[i] = k < n[i] ? P[at[i]] : V{};
#pragma unroll
    for (int i = 0; i < COUNT; ++i) add_to(v[i], w[i]);
  }
}

__device__ __forceinline__ int bit_length(long long v) { return 64 - __clzll(v < 0 ? -v : v); }

// v * 2^sh, rounded when sh < 0; the result is below 2^XBITS by the caller's scale
__device__ __forceinline__ long long shift_round(long long v, int sh) {
  if (sh >= 0) return v << min(sh, 63);
  const int r = -sh;
  if (r > 62) return 0;
  const long long m = v < 0 ? -v : v;
  const long long q = (m + (1ll << (r - 1))) >> r;
  return v < 0 ? -q : q;
}

// ------------------------------------------------------------------ host ---
constexpr int GPU_SMS = 152;                 // GB300

// Chains per CTA: an even share, one CTA per SM.
inline Deal deal_of(int rowsA, int rowsB, int width, int chains, int items) {
  Deal d;
  d.tilesA = cdiv(rowsA, BM);
  d.tilesB = cdiv(rowsB, width);
  d.chains = chains;
  d.per = (int)(((long long)items * d.tilesA * d.tilesB * d.chains + GPU_SMS - 1) / GPU_SMS);
  return d;
}

// Partial sums of a tile at most, whichever chain of a CTA it starts at.
inline int max_parts(const Deal& d) { return std::min(d.chains, (d.chains + d.per - 2) / d.per + 1); }

inline int unit_shift(int K) {
  int lg = 0;
  while ((1 << lg) < K) ++lg;
  return std::min(36, 46 - lg);
}

// Tensor map of a digit operand seen as [items x digits][sets][L][kp], box
// {32, box_rows, box_sets, digits}, 64-byte swizzle.
inline int make_digit_map(CUtensorMap* map, const DigitRows& d, int digits, int items, int box_rows, int box_sets) {
  auto enc = encode_fn();
  LGB_REQUIRE(enc, LGB_ECUDA, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t row = (cuuint64_t)d.kp * 2, set = row * d.L;
  cuuint64_t dims[4] = {(cuuint64_t)d.kp, (cuuint64_t)d.L, (cuuint64_t)(2 + d.b), (cuuint64_t)digits * items};
  cuuint64_t strides[3] = {row, set, set * (2 + d.b)};
  cuuint32_t box[4] = {(cuuint32_t)BK, (cuuint32_t)box_rows, (cuuint32_t)box_sets, (cuuint32_t)digits};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult res = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, d.base, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (res != CUDA_SUCCESS)
    return set_error(LGB_ECUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)res));
  return LGB_OK;
}

// One GEMM: A's and B's digits hold itemsA and itemsB items (1: shared by all).
template <int NA, int NB, bool REAL>
int launch_gemm(const DigitRows& A, int itemsA, const DigitRows& B, int itemsB, int items, const Deal& deal,
                const Band& band, int S, void* P, long long item_stride, int ld, int* err, cudaStream_t s) {
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(sliced_gemm_kernel<NA, NB, REAL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem_bytes(NA, NB));
  });
  LGB_CUDA(attr);
  CUtensorMap a, b;
  int st;
  if ((st = make_digit_map(&a, A, NA, itemsA, BM, 1))) return st;
  if ((st = make_digit_map(&b, B, NB, itemsB, REAL ? BN : BC, REAL ? 1 : 2))) return st;
  GemmParams p{};
  p.deal = deal;
  p.band = band;
  p.total = items * deal.tilesA * deal.tilesB * deal.chains;
  p.rowsB = B.L;
  p.ld = ld;
  p.dA = itemsA > 1 ? NA : 0;
  p.dB = itemsB > 1 ? NB : 0;
  p.S = S;
  p.P = P;
  p.item_stride = item_stride;
  p.err = err;
  p.wait_ns = WAIT_NS;
  sliced_gemm_kernel<NA, NB, REAL><<<cdiv(p.total, deal.per), NUM_THREADS, smem_bytes(NA, NB), s>>>(a, b, p);
  LGB_CUDA(cudaGetLastError());
  return LGB_OK;
}

}  // namespace
}  // namespace lgb
