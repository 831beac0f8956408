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
//     d 2^(-9 i).  Seven digits hold 62 bits below the vector's largest entry
//     (with six, fields with isolated spikes lost a factor of two against FP64);
//   - the products of digits with i + j <= 6 are kept, grouped by s = i + j.  A
//     group's sum over 64 K entries is at most (s + 1) 64 2^16 <= 2^24 units
//     for s <= 3: the FP32 accumulators hold it exactly, whatever order or
//     rounding the tensor core uses.  Groups 4 to 6 share an accumulator, which
//     is cut off at its last place at every MMA: 2^-52 of the largest product
//     when every digit is at its largest and of one sign (5 x 32 products of
//     2^16 2^-36, an FP32 place of 2^-36), 2^-57 for digits at random;
//   - every 64 K entries (256 for group 0, 128 for group 1: their sums have the
//     room; 32 for groups 4 to 6) the accumulators are drained into 64-bit
//     integers in registers, in units of 2^-(16 + S): exact for groups 0-3.
//     Integer sums do not depend on their order, so dealing K out over CTAs
//     gives the same bits.
// What is left, all of it relative to the largest entries of the two vectors of
// a sum: the rounding of the operands (2^-63), the products left out (2^-60), the
// last places of groups 4 to 6 and their rounding to the unit; and one rounding
// per stored result.  An FP64 accumulation rounds at every K step.
//
// A complex product is three real ones (Gauss): operands hold the row sets re,
// im and h = (re + im) / 2, the products of like sets are
//     P0 = Ar Br,  P1 = Ai Bi,  P2 = 2 Ah Bh,
// and readers form re = P0 - P1, im = 2 P2 - P0 - P1 in integers, modulo 2^64,
// which loses nothing.  P2 counts four times and has a quarter of the unit, so that
// its roundings weigh no more than P0's and P1's.  That is 84 digit products where four real products took 108 (a DFT
// matrix had six digits then): 1019 x 941 to 1024^2 went from 337 to 300 us,
// 512^2 from 82 to 76.
#pragma once

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace lgb {
namespace {

using namespace tc;

constexpr int ND = 7;                        // digits per entry
constexpr int BETA = 9;                      // bits per digit
constexpr int BM = 128, BN = 96, BK = 32;    // tile: A rows, B rows, K per stage
constexpr int STAGES = 2;
constexpr int GROUPS = 5;                    // accumulators: s = 0, 1, 2, 3, and 4 to 6 together
constexpr uint32_t A_SLICE = BM * BK * 2, B_SLICE = BN * BK * 2;
constexpr uint32_t A_STAGE = ND * A_SLICE, STAGE_BYTES = ND * (A_SLICE + B_SLICE);
constexpr int EPI_WARPS = 16;
constexpr int NUM_THREADS = 64 + 32 * EPI_WARPS;
constexpr uint32_t BAR_BYTES = 256;
constexpr uint32_t SMEM_BYTES = STAGES * STAGE_BYTES + BAR_BYTES + 1024;
constexpr int RUN = 4 * BN / EPI_WARPS;      // tile columns per epilogue warp
constexpr int MAX_S = 40;                    // group 4's sums are ints below 2^(S - 11), S + 2 for P2
constexpr unsigned long long WAIT_NS = 2000000000ull;
static_assert(SMEM_BYTES <= 232448, "shared memory per CTA");
static_assert(GROUPS * BN <= 512 && RUN == 24, "tensor memory columns; the drain loads 3 x 8 of them");

// How a launch's work is dealt out: the chains (64 K entries of one tile) of all
// tiles of all products in a row, `per` of them to each CTA.  A tile's chains
// then lie in one CTA or in a few neighbouring ones, which write a partial sum
// each.
struct Deal {
  int tilesA, tilesB;        // tiles of one product: A rows (fastest), B rows
  int chains;                // per tile
  int per;                   // chains per CTA
  __host__ __device__ int first_cta(int tile) const { return tile * chains / per; }
  __host__ __device__ int parts(int tile) const {
    return ((tile + 1) * chains - 1) / per - first_cta(tile) + 1;
  }
};

struct GemmParams {
  Deal deal;
  int total;                 // chains of all tiles of all products
  int sets;                  // products per item
  int stages;                // of BK along K
  int rowsB;
  int ld;                    // P row pitch (entries)
  int dA, dB;                // digit planes between items (0: shared by all items)
  // P unit: 2^-(16 + S) of the scaled operands, a quarter of it for P2.  S of a tile
  // is the least of its vectors' limits (unit_limit) on one side
  const int* limits;         // [item][limit_count]
  int limit_count;
  int limit_rows;            // BM: A's vectors, BN: B's; 0: one value for all
  int* tile_S;               // out: [item][tiles of that side]
  long long* P;              // [product][part][rowsB][ld]
  long long stride;          // entries between products
  int* err;
  unsigned long long wait_ns;
  // wait-expiry test (-1: none): CTA 0 issues no loads for its stage hold_loads,
  // or does not release digits 0 to 3 of its stage hold_release
  int hold_loads, hold_release;
};

// One CTA's run of chains of one tile.
struct Segment {
  int product, m0, n0;       // tile origin: A row, B row
  int chain, count;
  int part;                  // which of the tile's partial sums
};
__device__ __forceinline__ Segment segment_at(const GemmParams& p, int pos, int end) {
  Segment s;
  const int tile = pos / p.deal.chains;
  s.chain = pos - tile * p.deal.chains;
  s.count = min(p.deal.chains - s.chain, end - pos);
  const int tiles = p.deal.tilesA * p.deal.tilesB;
  s.product = tile / tiles;
  const int t = tile - s.product * tiles;
  const int tb = t / p.deal.tilesA;
  s.m0 = (t - tb * p.deal.tilesA) * BM;
  s.n0 = tb * BN;
  s.part = (int)blockIdx.x - p.deal.first_cta(tile);
  return s;
}

// Which chains of a segment (r = 0, 1, ...) start and end a sum of group g:
// groups 0 and 1 run over four and two chains, at most 4 * 64 2^16 = 2 * 2 * 64
// 2^16 = 2^24.  (Draining every group after every chain left the MMA waiting
// 16 % of the time for the last ones of 20 drains in four chains.)  Groups 4 to 6
// start and end one every stage: drained every chain, the shared accumulator was
// cut off at group 4's last place for twice as long, and with the three groups in
// the order of A's digits too, fields of a cross of ones over 1e-3 (333 x 257)
// came out 1.27 times as far from exact as in plain FP64, amplitudes over ten
// decades 1.18 times; now 0.93 and 1.00 (1019 x 941 to 1024^2 278 -> 293 us).
__device__ __forceinline__ bool starts(int g, int r) {
  return g == 0 ? (r & 3) == 0 : g == 1 ? (r & 1) == 0 : true;
}
__device__ __forceinline__ bool drains(int g, int r, int count) {          // g < 4
  if (r == count - 1) return true;
  return g == 0 ? (r & 3) == 3 : g == 1 ? (r & 1) == 1 : true;
}

// The products of digit i of A with digits j0 >= j >= j1 of B, two k-steps, into
// the accumulators of i + j (4 to 6: the last one); the first of them starts its
// sum afresh when `fresh`.  A's tile stays in the MMA's collector for the run,
// else shared memory is read more slowly than the tensor core computes.  The
// operand descriptors are one 64-bit base each plus constants, and the warp
// stays converged around them: with descriptors worked out per MMA, or in a
// loop that one lane runs alone, the issuing warp was the limit, at 95 to 100
// clk an MMA.
__device__ __forceinline__ void mma_run(int i, int j0, int j1, uint32_t on, uint32_t tmem, uint64_t da,
                                        uint64_t db, uint32_t idesc, bool fresh) {
#pragma unroll
  for (int k = 0; k < BK / 16; ++k) {
#pragma unroll
    for (int j = j0; j >= j1; --j) {
      const int g = i + j < GROUPS ? i + j : GROUPS - 1;
      mma_f16_cta(on, tmem + g * BN, da + ((i * A_SLICE + k * 32) >> 4), db + ((j * B_SLICE + k * 32) >> 4),
                  idesc, k == 0 && j == j1 && fresh ? 0u : 1u, j != j0, j != j1);
    }
  }
}

// P over this CTA's chains.
//
// Bound by the tensor pipe: 112 MMAs (28 digit products x 4 k-steps) of
// 128 x 96 x 16 per chain, 48 clk each; 96 columns is the widest tile whose five
// accumulators fit the 512 TMEM columns.  An MMA that reads both operands from
// shared memory (7 KB) takes 56 clk, and the 98 KB that TMA writes per stage
// share the port: in the order of the sums i + j, with nothing kept, a stage
// took 3900 clk.  Runs over B's digits with A's in the collector read 4.6 KB and
// run at 49: 1019 x 941 to 1024^2 went from 121 to 110 us per GEMM (transform
// 300 -> 283), 512^2 from 76 to 71.5.  (Group 4's five products are runs of one.)
// What is left above the 81 us of MMAs: the first loads and the last sums (6 us),
// loads (12 %, by latency: L2 runs at a third of its rate) and drains that the
// MMAs wait for.
//
// Roles: warp 0 TMA (two stages of 32 K entries; digits 4 to 6 of a stage are
// done with, and loaded anew, while its sums 0 to 3 run), warp 1 MMA issue,
// warps 2..17 drain (lane quadrant w % 4, 24 columns each).  A drain takes some
// 800 clk, most of it the conversions (16 a clock).  One CTA per SM takes its
// share of the chains (Deal), so the pipeline fills once per launch and no wave
// is partly empty.
__global__ void __launch_bounds__(NUM_THREADS, 1)
sliced_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t bars = base + STAGES * STAGE_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto low_empty = [&](int s) { return bars + 16u + 8u * s; };       // digits 4 to 6
  auto high_empty = [&](int s) { return bars + 144u + 8u * s; };     // digits 0 to 3
  auto acc_full = [&](int g) { return bars + 32u + 8u * g; };
  auto acc_empty = [&](int g) { return bars + 80u + 8u * g; };
  const uint32_t drain_bar = bars + 128u;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + (bars - raw) + 160);
  volatile int* half_loaded = reinterpret_cast<volatile int*>(smem_raw + (bars - raw) + 164);

  next_may_start();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int begin = blockIdx.x * p.deal.per, end = min(p.total, begin + p.deal.per);

  if (threadIdx.x == 0) {
    *half_loaded = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 2);
      mbar_init(low_empty(s), 1);
      mbar_init(high_empty(s), 1);
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
  previous_done();

  if (warp == 0) {
    if (lane == 0) {
      prefetch_map(&tmA);
      prefetch_map(&tmB);
      int it = 0;
      bool ok = true;
      for (int pos = begin; ok && pos < end;) {
        const Segment w = segment_at(p, pos, end);
        pos += w.count;
        const int item = w.product / p.sets, set = w.product - item * p.sets;
        const int last = min(p.stages, 2 * (w.chain + w.count));
        for (int st = 2 * w.chain; st < last; ++st, ++it) {
          const int s = it % STAGES;
          const uint32_t sa = base + s * STAGE_BYTES, parity = ((it / STAGES) & 1) ^ 1;
          auto load = [&](uint32_t empty, int d0, int d1) {
            if (!mbar_wait(empty, parity, p.err, p.wait_ns)) return false;
            mbar_expect_tx(full_bar(s), (d1 - d0) * (A_SLICE + B_SLICE));
            for (int d = d0; d < d1; ++d) {
              tma_load_4d_cta(sa + d * A_SLICE, &tmA, full_bar(s), st * BK, w.m0, set, item * p.dA + d);
              tma_load_4d_cta(sa + A_STAGE + d * B_SLICE, &tmB, full_bar(s), st * BK, w.n0, set, item * p.dB + d);
            }
            return true;
          };
          if (blockIdx.x == 0 && it == p.hold_loads) continue;
          ok = load(low_empty(s), GROUPS - 1, ND);
          if (!ok) break;
          ok = load(high_empty(s), 0, GROUPS - 1);
          if (!ok) {
            // half a stage is in flight: an arrival in place of the other half's
            // lets its barrier complete when the copies land, for the wait below,
            // and the MMA warp is told to leave the stage alone
            *half_loaded = 1;
            mbar_arrive(full_bar(s));
            ++it;
            break;
          }
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
      const Segment w = segment_at(p, pos, end);
      pos += w.count;
      const int stages = min(p.stages - 2 * w.chain, 2 * w.count);
      for (int st = 0; ok && st < stages; ++st, ++it) {
        const int s = it % STAGES, r = st >> 1;
        const bool ends = (st & 1) == 1 || st == stages - 1;      // of a chain
        if (!wait(full_bar(s), (it / STAGES) & 1) || *half_loaded) { ok = false; break; }
        const uint64_t da = smem_desc_sw64(base + s * STAGE_BYTES);
        const uint64_t db = smem_desc_sw64(base + s * STAGE_BYTES + A_STAGE);
        const bool begins = (st & 1) == 0;
        auto done = [&](int g) {
          if (g == GROUPS - 1 || (ends && drains(g, r, w.count))) {
            mma_commit_cta(on, acc_full(g));
            ++n[g];
          }
        };
        // whether group g's sum starts here, once its previous one has been drained
        auto fresh = [&](int g) {
          if (g < GROUPS - 1 && (!begins || !starts(g, r))) return false;
          ok = wait(acc_empty(g), (n[g] & 1) ^ 1);
          tc_fence_after();
          return true;
        };
        tc_fence_after();
        // groups 4 to 6 first: their accumulator is drained while the others run.
        // Of them 6 and 5, then 4, whose last place the sum keeps from then on.
        const bool f4 = fresh(GROUPS - 1);
        if (!ok) break;
#pragma unroll
        for (int i = ND - 1; i >= 0; --i)
          mma_run(i, ND - 1 - i, max(GROUPS - i, 0), on, tmem, da, db, idesc, f4 && i == ND - 1);
#pragma unroll
        for (int i = GROUPS - 1; i >= 0; --i)
          mma_run(i, GROUPS - 1 - i, GROUPS - 1 - i, on, tmem, da, db, idesc, false);
        done(GROUPS - 1);
        mma_commit_cta(on, low_empty(s));
#pragma unroll
        for (int g = GROUPS - 2; g >= 0; --g) {
          const bool f = fresh(g);
          if (!ok) break;
          mma_run(g, GROUPS - 2 - g, 0, on, tmem, da, db, idesc, f);
        }
        if (!ok) break;
#pragma unroll
        for (int g = GROUPS - 2; g >= 0; --g) done(g);
        if (blockIdx.x != 0 || it != p.hold_release) mma_commit_cta(on, high_empty(s));
      }
    }
    mma_commit_cta(on, drain_bar);
    mbar_wait_issued(drain_bar, 0, p.wait_ns);
    __syncwarp();
  } else {
    const int q4 = warp & 3, ch = (warp - 2) >> 2;
    const uint32_t trow = tmem + ((uint32_t)(q4 * 32) << 16) + ch * RUN;
    int n[GROUPS] = {};                        // drains done, by group
    bool ok = true;
    for (int pos = begin; ok && pos < end;) {
      const Segment w = segment_at(p, pos, end);
      pos += w.count;
      const int item = w.product / p.sets;
      int S = MAX_S;
      if (p.limit_rows == 0) {
        S = *p.limits;
      } else {
        const int first = p.limit_rows == BM ? w.m0 : w.n0, last = min(first + p.limit_rows, p.limit_count);
        for (int i = first + lane; i < last; i += 32) S = min(S, p.limits[item * p.limit_count + i]);
        S = __reduce_min_sync(0xffffffffu, S);
        if (warp == 2 && lane == 0)
          p.tile_S[item * ((p.limit_count + p.limit_rows - 1) / p.limit_rows) + first / p.limit_rows] = S;
      }
      if (w.product - item * p.sets == 2) S += 2;
      const float unit4 = ldexpf(1.f, S);
      // sums of groups 1 to 3 are whole multiples of 2^-9, 2^-18, 2^-27 below 2^24
      // of them: three more bits leave the multipliers below 2^31
      const int m1 = 1 << (S - BETA - 3), m2 = 1 << (S - 2 * BETA - 3), m3 = 1 << (S - 3 * BETA - 3);
      unsigned long long acc[RUN];
#pragma unroll
      for (int j = 0; j < RUN; ++j) acc[j] = 0;
      for (int k = 0; ok && k < w.count; ++k) {
        auto drain = [&](int g) {
          ok = __all_sync(0xffffffffu, mbar_wait(acc_full(g), n[g] & 1, p.err, p.wait_ns));
          if (!ok) return;
          ++n[g];
          tc_fence_after();
          uint32_t r[RUN];
#pragma unroll
          for (int h = 0; h < RUN / 8; ++h) tmem_ld8(trow + g * BN + h * 8, r + h * 8);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty(g));
#pragma unroll
          for (int j = 0; j < RUN; ++j) {
            const float v = __uint_as_float(r[j]);
            if (g == 4) acc[j] += (long long)__float2int_rn(v * unit4);
            else if (g == 3) acc[j] += (long long)__float2int_rn(v * 0x1p30f) * m3;
            else if (g == 2) acc[j] += (long long)__float2int_rn(v * 0x1p21f) * m2;
            else if (g == 1) acc[j] += (long long)__float2int_rn(v * 0x1p12f) * m1;
            else acc[j] += (unsigned long long)((uint32_t)__float2int_rn(v) << (S - 32)) << 32;
          }
        };
        const int last = min(p.stages - 2 * (w.chain + k), 2);
        for (int st = 0; ok && st < last; ++st) drain(GROUPS - 1);
#pragma unroll
        for (int g = GROUPS - 2; g >= 0; --g)
          if (ok && drains(g, k, w.count)) drain(g);
      }
      if (!ok) break;
      const int n0 = w.n0 + ch * RUN;
      long long* out = p.P + (size_t)w.product * p.stride + ((size_t)w.part * p.rowsB + n0) * p.ld + w.m0 +
                       q4 * 32 + lane;
#pragma unroll
      for (int j = 0; j < RUN; ++j)
        if (n0 + j < p.rowsB) out[(size_t)j * p.ld] = (long long)acc[j];
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
// The digits of X, |X| <= 2^62, as bf16 bits in the high half of a word; digit
// i carries 2^(-9 i).  A bias of 256 in every place turns the signed digits into
// bit fields; a field under the exponent of 1.5 2^23 is a float, and one FMA
// takes bias and offset off and scales (exactly): three instructions a digit,
// none of them on the conversion or 64-bit paths.
__device__ __forceinline__ void digits_of(long long X, uint32_t (&d)[ND]) {
  constexpr unsigned long long bias = 256ull * 0x0000201008040201ull;   // 256 sum of 2^(9 i), i < 6
  const unsigned long long Y = (unsigned long long)X + bias;
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    const int sh = BETA * (ND - 1 - i);
    const float s = 1.f / (float)(1ull << (BETA * i));
    // the leading digit is signed: 512 more keep its field positive
    const uint32_t u = (uint32_t)(Y >> sh) + (i == 0 ? 512u : 0u);
    const float f = __uint_as_float((u & (i == 0 ? 1023u : 511u)) | 0x4B400000u);
    d[i] = __float_as_uint(fmaf(f, s, -(12582912.f + (i == 0 ? 512.f : 256.f)) * s));
  }
}

// v * 2^e * scale as a double
__device__ __forceinline__ double scaled(long long v, int e, double scale) {
  const unsigned long long m = (unsigned long long)(v < 0 ? -v : v);
  const int exp = 63 - __clzll((long long)m) + e + 1023;
  if (m != 0 && (exp < 1 || exp > 2045)) return scalbn((double)v * scale, e);
  const double r = scale * assembled(m, e);
  return v < 0 ? -r : r;
}

constexpr int XBITS = BETA * ND - 1;         // an entry is |X| <= 2^62 of its vector's scale

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

// Digit operand of L vectors, [digit][set][L][kp] 16-bit entries.  Complex
// vectors have three sets (re, im, (re + im) / 2), real ones one.
struct DigitRows {
  uint16_t* base;
  int L, kp, sets;
  __host__ __device__ size_t set() const { return (size_t)L * kp; }
  __host__ __device__ size_t plane() const { return sets * set(); }
};
// Entries k, k + 1 of vector j in one set.
__device__ __forceinline__ void store_digits(const DigitRows& o, int set, int j, int k, long long v0,
                                             long long v1) {
  uint16_t* p = o.base + set * o.set() + (size_t)j * o.kp + k;
  uint32_t a[ND], c[ND];
  digits_of(v0, a);
  digits_of(v1, c);
#pragma unroll
  for (int i = 0; i < ND; ++i)
    *reinterpret_cast<uint32_t*>(p + i * o.plane()) = __byte_perm(a[i], c[i], 0x7632);
}
// (a + b) / 2, to even: a rounding to one side would add up
__device__ __forceinline__ long long half_sum(long long a, long long b) {
  const long long h = (a >> 1) + (b >> 1) + (a & b & 1);
  return h + ((a ^ b) & h & 1);
}
__device__ __forceinline__ void store_digits3(const DigitRows& o, int j, int k, longlong2 z0, longlong2 z1) {
  store_digits(o, 0, j, k, z0.x, z1.x);
  store_digits(o, 1, j, k, z0.y, z1.y);
  store_digits(o, 2, j, k, half_sum(z0.x, z0.y), half_sum(z1.x, z1.y));
}

// What an entry adds to the sum of |re| + |im| of a vector, in units of 2^46 (at most
// 2^17: 16384 of them fit a word).
__device__ __forceinline__ unsigned magnitude(longlong2 z) {
  return (unsigned)(((unsigned long long)(z.x < 0 ? -z.x : z.x) + (unsigned long long)(z.y < 0 ? -z.y : z.y)) >> 46);
}

// The S that a data vector of K entries allows: its sums with entries |E| <= 1 are at
// most L 2^16, L the sum of its |re| + |im| over 2^62, below (sum + K) 2^-16, and
// L 2^(16 + S) stays below 2^63 with 2^-32 of it for the sums' roundings.
// Never less than S, which holds for any vector.  A vector with few large entries has
// a unit of up to 2^-56 of them so, where the one for K = 1040 is 2^-51: amplitudes
// over ten decades, (8 x 1040) to (8 x 260), came out 2.0 times as far from exact as in
// plain FP64 with that one, 0.9 times so (1019 x 941 to 1024^2 292 -> 296 us).
__device__ __forceinline__ int unit_limit(unsigned sum, int K, int S) {
  return min(MAX_S, max(S, 63 - (32 - __clz((int)(sum + K)))));
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

// A GEMM's products as their readers see them.
struct PartialSums {
  const long long* P;        // [product][part][rows][ld]
  long long stride;          // entries between products
  int ld, rows, cols;
  Deal deal;
  const int* tile_S;         // the tiles' S: [item][tiles along one side]
  bool by_row;               // of rows (the B side), else of columns
  __device__ __forceinline__ int S(int item, int r, int a) const {
    return by_row ? tile_S[item * deal.tilesB + r / BN] : tile_S[item * deal.tilesA + a / BM];
  }
  __device__ __forceinline__ int parts(int product, int r, int a) const {
    return deal.parts((product * deal.tilesB + r / BN) * deal.tilesA + a / BM);
  }
  __device__ __forceinline__ size_t part() const { return (size_t)rows * ld; }     // entries between parts
};

constexpr int MAX_TILES_A = 256;             // 128-row tiles of the longest A operand (32768 rows)

// How many partial sums the tiles under row r have, in COUNT products from the
// given one: [COUNT][tilesA] in shared memory (ends with a block barrier).
template <int COUNT>
__device__ __forceinline__ void count_parts(const PartialSums& q, int product, int r, uint8_t* parts) {
  for (int t = threadIdx.x; t < COUNT * q.deal.tilesA; t += blockDim.x) {
    const int c = t / q.deal.tilesA;
    parts[t] = (uint8_t)q.parts(product + c, r, (t - c * q.deal.tilesA) * BM);
  }
  __syncthreads();
}

// v[i] = the sum of n[i] parts (0: none) of the entry at offset at[i], i < COUNT.
// The parts go in the outer loop, so that COUNT loads are in flight.
template <int COUNT>
__device__ __forceinline__ void sum_parts(const long long* __restrict__ P, size_t part, const size_t (&at)[COUNT],
                                          const int (&n)[COUNT], long long (&v)[COUNT]) {
  int most = 0;
#pragma unroll
  for (int i = 0; i < COUNT; ++i) {
    most = max(most, n[i]);
    v[i] = 0;
  }
  for (int k = 0; k < most; ++k, P += part) {
    long long w[COUNT];
#pragma unroll
    for (int i = 0; i < COUNT; ++i) w[i] = k < n[i] ? P[at[i]] : 0;
#pragma unroll
    for (int i = 0; i < COUNT; ++i) v[i] += w[i];
  }
}

// The same for complex entries: n[c][i] parts of product c, 3 COUNT loads in
// flight.  4 P2, P2's sum in its units, may wrap; what is left of it does not.
template <int COUNT>
__device__ __forceinline__ void sum_parts3(const long long* __restrict__ P, size_t stride, size_t part,
                                           const size_t (&at)[COUNT], const int (&n)[3][COUNT],
                                           longlong2 (&v)[COUNT]) {
  int most = 0;
  unsigned long long re[COUNT], im[COUNT];
#pragma unroll
  for (int i = 0; i < COUNT; ++i) {
    most = max(most, max(n[0][i], max(n[1][i], n[2][i])));
    re[i] = im[i] = 0;
  }
  for (int k = 0; k < most; ++k, P += part) {
    long long w[3][COUNT];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int i = 0; i < COUNT; ++i) w[c][i] = k < n[c][i] ? P[c * stride + at[i]] : 0;
#pragma unroll
    for (int i = 0; i < COUNT; ++i) {
      re[i] += (unsigned long long)w[0][i] - (unsigned long long)w[1][i];
      im[i] += (unsigned long long)w[2][i] - (unsigned long long)w[0][i] - (unsigned long long)w[1][i];
    }
  }
#pragma unroll
  for (int i = 0; i < COUNT; ++i) v[i] = make_longlong2((long long)re[i], (long long)im[i]);
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
inline Deal deal_of(int rowsA, int rowsB, int chains, int products) {
  Deal d;
  d.tilesA = cdiv(rowsA, BM);
  d.tilesB = cdiv(rowsB, BN);
  d.chains = chains;
  d.per = (int)(((long long)products * d.tilesA * d.tilesB * d.chains + GPU_SMS - 1) / GPU_SMS);
  return d;
}

// Partial sums of a tile at most, whichever chain of a CTA it starts at.
inline int max_parts(const Deal& d) { return std::min(d.chains, (d.chains + d.per - 2) / d.per + 1); }

// S of a contraction of K entries, whatever they are: sums reach K 2^16 (times sqrt 2
// for im).  K <= 16384, so S >= 32.
inline int unit_shift(int K) {
  int lg = 0;
  while ((1 << lg) < K) ++lg;
  return std::min(MAX_S, 46 - lg);
}

// Tensor map of a digit operand seen as [items x digits][sets][L][kp], box
// {32, box_rows, 1, 1}, 64-byte swizzle.
inline int make_digit_map(CUtensorMap* map, const DigitRows& d, int items, int box_rows) {
  auto enc = encode_fn();
  LGB_REQUIRE(enc, LGB_ECUDA, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t row = (cuuint64_t)d.kp * 2, set = row * d.L;
  cuuint64_t dims[4] = {(cuuint64_t)d.kp, (cuuint64_t)d.L, (cuuint64_t)d.sets, (cuuint64_t)ND * items};
  cuuint64_t strides[3] = {row, set, set * d.sets};
  cuuint32_t box[4] = {(cuuint32_t)BK, (cuuint32_t)box_rows, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult res = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, d.base, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (res != CUDA_SUCCESS)
    return set_error(LGB_ECUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)res));
  return LGB_OK;
}

// The products of A's and B's sets over K entries, for `items` items; the
// operands hold itemsA and itemsB of them (1: shared by all).
inline int launch_gemm(const DigitRows& A, int itemsA, const DigitRows& B, int itemsB, int items, int K,
                       const Deal& deal, const int* limits, int limit_rows, int* tile_S, long long* P,
                       long long stride, int ld,
                       int* err, cudaStream_t s) {
  static OncePerDevice once;
  LGB_CUDA(allow_shared_memory(once, sliced_gemm_kernel, SMEM_BYTES));
  CUtensorMap a, b;
  int st;
  if ((st = make_digit_map(&a, A, itemsA, BM))) return st;
  if ((st = make_digit_map(&b, B, itemsB, BN))) return st;
  GemmParams p{};
  p.deal = deal;
  p.sets = A.sets;
  p.total = items * p.sets * deal.tilesA * deal.tilesB * deal.chains;
  p.stages = cdiv(K, BK);
  p.rowsB = B.L;
  p.ld = ld;
  p.dA = itemsA > 1 ? ND : 0;
  p.dB = itemsB > 1 ? ND : 0;
  p.limits = limits;
  p.limit_rows = limit_rows;
  p.limit_count = limit_rows == BM ? A.L : B.L;
  p.tile_S = tile_S;
  p.P = P;
  p.stride = stride;
  p.err = err;
  p.wait_ns = WAIT_NS;
  p.hold_loads = p.hold_release = -1;
  const SlicedStall stall = take_sliced_stall();
  if (stall.stage >= 0) {
    (stall.release ? p.hold_release : p.hold_loads) = stall.stage;
    p.wait_ns = stall.wait_ns;
  }
  LGB_CUDA(launch_next(sliced_gemm_kernel, cdiv(p.total, deal.per), NUM_THREADS, SMEM_BYTES, s, a, b, p));
  return LGB_OK;
}

}  // namespace
}  // namespace lgb
