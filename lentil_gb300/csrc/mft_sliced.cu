// K3s: complex128 matrix triple products on the tensor cores, by slicing.
//
// lentil's dft2 (lentil/fourier.py:95-101) is F = E1 . f . E2 in complex128.
// This part's FP64 units retire two FMAs a clock per SM, its tensor cores
// 4096 bf16 ones, so each FP64 product is taken apart into bf16 products
// whose sums are exact (the error-free transformation of Ozaki, Ogita, Oishi
// and Rump, Numerical Algorithms 59, 2012; on tensor cores: Mukunoki et al.,
// ISC 2020):
//   - every vector of the contraction (a column of f, a row of E1, ...) is
//     scaled by a power of two above its largest entry, rounded to 54 bits and
//     cut into NS = 6 signed digits of 9 bits, |d| <= 256, each exact in bf16;
//     digit i is stored as d 2^(-9 i);
//   - the products of digits with i + j <= 5 are kept (21 of 36; the first
//     one left out is 2^-54 of the operands), grouped by s = i + j.  A group's
//     sum over 64 K entries is at most (s + 1) 64 2^16 <= 2^24 units for
//     s <= 3: the FP32 accumulators hold it exactly, whatever order or
//     rounding the tensor core uses.  Groups 4 and 5 share an accumulator
//     (their rounding is below 2^-57 of the operands);
//   - every 64 K entries the accumulators are drained into 64-bit integers in
//     registers, in units of 2^-(16 + S): exact for groups 0-3.  Integer sums
//     do not depend on their order, so dealing K out over CTAs gives the same bits.
// What is left is the rounding of the operands to 54 bits of their vector's
// largest entry, the products left out, and one rounding per stored result;
// an FP64 accumulation rounds at every one of its K steps instead.
//
// A complex product needs no complex arithmetic on the way: operand B holds
// the row sets [-im | re | im], operand A the sets [re | im], and a tile's
// columns are 48 real and the same 48 imaginary parts,
//     A re rows x (B re, B im rows)  +  A im rows x (B -im, B re rows),
// so that the accumulators hold the complex sums.
//
// A transform is five launches:
//   slice_field   f -> digits, one exponent per vector of the contraction
//   sliced_gemm   P = E1 . f or f . E2, in integers
//   slice_rows    P's rows, scaled to their largest entry -> digits
//   sliced_gemm   P = the second product
//   finish        P -> F, scaled
// A field with a NaN gives NaN everywhere (each output sums every entry); one
// with infinities, or a device-side wait that ran out, makes `finish`
// evaluate that transform in plain FP64 instead.
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
constexpr int S_MAX = ND - 1;                // digit products with i + j <= S_MAX are kept
constexpr uint32_t A_SLICE = BM * BK * 2, B_SLICE = BN * BK * 2;
constexpr uint32_t stage_bytes(int na, int nb) { return na * A_SLICE + nb * B_SLICE; }
constexpr int EPI_WARPS = 8;
constexpr int NUM_THREADS = 64 + 32 * EPI_WARPS;
constexpr uint32_t BAR_BYTES = 256;
constexpr uint32_t smem_bytes(int na, int nb) { return STAGES * stage_bytes(na, nb) + BAR_BYTES + 1024; }
constexpr int RUN = BC / 2;                  // complex tile columns per epilogue warp
constexpr unsigned long long WAIT_NS = 2000000000ull;
static_assert(smem_bytes(ND, NE) <= 232448 && smem_bytes(NE, ND) <= 232448, "shared memory per CTA");
static_assert(GROUPS * BN <= 512 && RUN == 24, "tensor memory columns; the drain loads 3 x 8 of them");

// How a launch's work is dealt out: the chains (32 complex K entries of one
// tile: a stage of real and one of imaginary A rows) of all tiles in a row, `per` of them to each CTA.  A tile's chains then lie in
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

struct GemmParams {
  Deal deal;
  int total;                 // chains of all tiles of all items
  int rowsB;                 // complex
  int ld;                    // P row pitch (entries)
  int dA, dB;                // digit planes between items (0: shared by all items)
  int S;                     // P unit: 2^-(16 + S) of the scaled operands
  longlong2* P;              // [item][part][rowsB][ld] (re, im)
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
  s.n0 = tb * BC;
  s.part = (int)blockIdx.x - p.deal.first_cta(tile);
  return s;
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
// Bound by the tensor pipe: 108 MMAs (27 digit products x 4 k-steps) of
// 128 x 96 x 16 per chain.  96 columns is the widest tile whose five
// accumulators fit the 512 TMEM columns; the MMA then reads 7 KB of shared
// memory per 48 clocks (149 B/clk against the 128 B/clk port), so it runs at
// 56 clk at best.  Roles: warp 0 TMA (two stages of 32 K entries, all digits),
// warp 1 MMA issue, warps 2..9 drain (lane quadrant w % 4, column half
// (w - 2) / 4).  The groups are drained one by one, in the order they are
// issued, while the next ones run.  One CTA per SM takes its share of the
// chains (Deal), so the pipeline fills once per launch and no wave is partly
// empty.
template <int NA, int NB>
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
        const Segment w = segment_at(p, pos, end);
        pos += w.count;
        for (int st = 2 * w.chain; st < 2 * (w.chain + w.count); ++st, ++it) {
          const int s = it % STAGES, im = st & 1, k = (st >> 1) * BK;
          if (!mbar_wait(empty_bar(s), ((it / STAGES) & 1) ^ 1, p.err, p.wait_ns)) { ok = false; break; }
          mbar_expect_tx(full_bar(s), STAGE_BYTES);
          const uint32_t sa = base + s * STAGE_BYTES;
          tma_load_4d_cta(sa, &tmA, full_bar(s), k, w.m0, im, w.item * p.dA);
          tma_load_4d_cta(sa + A_STAGE, &tmB, full_bar(s), k, w.n0, 1 - im, w.item * p.dB);
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
    int it = 0, c = 0;                         // stages and chains issued
    bool ok = true;
    for (int pos = begin; ok && pos < end;) {
      const Segment w = segment_at(p, pos, end);
      pos += w.count;
      for (int st = 0; ok && st < 2 * w.count; ++st, ++it) {
        const int s = it % STAGES;
        const bool first = (st & 1) == 0, last = !first;
        if (!wait(full_bar(s), (it / STAGES) & 1)) { ok = false; break; }
        const uint64_t da = smem_desc_sw64(base + s * STAGE_BYTES);
        const uint64_t db = smem_desc_sw64(base + s * STAGE_BYTES + A_STAGE);
#pragma unroll
        for (int g = GROUPS - 1; g >= 0; --g) {
          // this accumulator's previous chain has been drained
          if (first && !wait(acc_empty(g), (c & 1) ^ 1)) { ok = false; break; }
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
          if (last) mma_commit_cta(on, acc_full(g));
        }
        if (ok) mma_commit_cta(on, empty_bar(s));
        if (last) ++c;
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
    int c = 0;                                 // chains drained
    bool ok = true;
    for (int pos = begin; ok && pos < end;) {
      const Segment w = segment_at(p, pos, end);
      pos += w.count;
      long long acc[2 * RUN];                  // RUN real parts, RUN imaginary parts
#pragma unroll
      for (int j = 0; j < 2 * RUN; ++j) acc[j] = 0;
      for (int k = 0; ok && k < w.count; ++k, ++c) {
#pragma unroll
        for (int g = GROUPS - 1; g >= 0; --g) {
          ok = __all_sync(0xffffffffu, mbar_wait(acc_full(g), c & 1, p.err, p.wait_ns));
          if (!ok) break;
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
      longlong2* out = p.P + (size_t)w.item * p.item_stride + ((size_t)w.part * p.rowsB + n0) * p.ld +
                       w.m0 + q4 * 32 + lane;
#pragma unroll
      for (int j = 0; j < RUN; ++j)
        if (n0 + j < p.rowsB) out[(size_t)j * p.ld] = make_longlong2(acc[j], acc[RUN + j]);
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
// A small integer as a float without the conversion pipe (16 lanes a clock)
__device__ __forceinline__ float small_float(int t) {
  return __int_as_float(0x4B400000 + t) - 12582912.f;
}

// The N digits of X, |X| <= 2^(9 N - 1), as bf16 bits in the high half of a
// word; digit i carries 2^(-9 i).
template <int N>
__device__ __forceinline__ void digits_of(long long X, uint32_t (&d)[N]) {
#pragma unroll
  for (int i = N - 1; i > 0; --i) {
    const int t = (int)((X + 256) & 511) - 256;
    X = (X - t) >> BETA;
    d[i] = __float_as_uint(small_float(t) * (1.f / (float)(1ull << (BETA * i))));
  }
  d[0] = __float_as_uint(small_float((int)X));
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

// E of modulus <= 1 as E * 2^53, rounded
__device__ __forceinline__ long long unit53(double x) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const int E = (int)(u >> 52) & 0x7FF;
  if (E == 0) return 0;
  long long m = (long long)((u & 0xFFFFFFFFFFFFFull) | (1ull << 52)) << 1;    // 54 bits
  const int sh = 1023 - E;
  if (sh > 0) m = sh > 55 ? 0 : (m + (1ll << (sh - 1))) >> sh;
  return (long long)u < 0 ? -m : m;
}

// Digit operand of L complex vectors, [digit][set][L][kp] 16-bit entries: the
// sets are re, im (operand A), or -im, re, im (operand B).
struct DigitRows {
  uint16_t* base;
  int L, kp, b;              // b: 1 for operand B
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

// DFT-matrix digits: vector j < L (output index) over the input index; matrix
// z's axis is axes[z], or ax when there is one.
__global__ void __launch_bounds__(128) matrix_digits_kernel(PhaseAxis ax, const PhaseAxis* __restrict__ axes,
                                                            int len_in, DigitRows out) {
  if (axes) ax = axes[blockIdx.z];
  out.base += (size_t)blockIdx.z * NE * out.plane();
  const int k = 2 * (blockIdx.x * blockDim.x + threadIdx.x), j = blockIdx.y;
  if (k >= out.kp) return;
  const double2 zero = make_double2(0.0, 0.0);
  const double2 e0 = k < len_in ? expm2pi_fixed_f64(phase_fixed(ax, k, j)) : zero;
  const double2 e1 = k + 1 < len_in ? expm2pi_fixed_f64(phase_fixed(ax, k + 1, j)) : zero;
  store_digits<NE>(out, j, k, unit53(e0.x), unit53(e0.y), unit53(e1.x), unit53(e1.y));
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

// f's rows (one block each) -> digits, vectors of n entries.
__global__ void __launch_bounds__(128) slice_rows_kernel(const double2* __restrict__ f, int m, int n,
                                                         DigitRows out, int* __restrict__ exps,
                                                         int* __restrict__ flags) {
  const int i = blockIdx.x, b = blockIdx.y;
  const double2* src = f + ((size_t)b * m + i) * n;
  __shared__ int se[4], sf[4];
  int e = 1, flag = 0;
  for (int k = threadIdx.x; k < n; k += 128) {
    const double2 z = src[k];
    note_exponent(z.x, e, flag);
    note_exponent(z.y, e, flag);
  }
  e = __reduce_max_sync(0xffffffffu, e);
  flag = __reduce_or_sync(0xffffffffu, flag);
  if ((threadIdx.x & 31) == 0) { se[threadIdx.x >> 5] = e; sf[threadIdx.x >> 5] = flag; }
  __syncthreads();
  e = max(max(se[0], se[1]), max(se[2], se[3]));
  flag = sf[0] | sf[1] | sf[2] | sf[3];
  if (threadIdx.x == 0) {
    exps[(size_t)b * m + i] = e - 1022;
    if (flag) atomicOr(flags + b, flag);
  }
  if (flag) return;                                       // this transform does not use its digits
  out.base += (size_t)b * ND * out.plane();
  const double2 zero = make_double2(0.0, 0.0);
  for (int k = 2 * threadIdx.x; k < out.kp; k += 256) {
    const double2 z0 = k < n ? src[k] : zero, z1 = k + 1 < n ? src[k + 1] : zero;
    store_digits<ND>(out, i, k, fixed_data(z0.x, e), fixed_data(z0.y, e), fixed_data(z1.x, e),
                     fixed_data(z1.y, e));
  }
}

constexpr int SC_COLS = 4, SC_WARPS = 16;    // columns and warps per block of slice_cols

// f's columns -> digits, vectors of m entries: SC_COLS neighbouring columns a
// block (a 64-byte piece of each row), SC_WARPS / SC_COLS warps per column.
__global__ void __launch_bounds__(32 * SC_WARPS) slice_cols_kernel(
    const double2* __restrict__ f, int m, int n, DigitRows out, int* __restrict__ exps,
    int* __restrict__ flags) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = warp % SC_COLS, part = warp / SC_COLS;
  constexpr int PARTS = SC_WARPS / SC_COLS;
  const int j = blockIdx.x * SC_COLS + c, b = blockIdx.y;
  const double2* src = f + (size_t)b * m * n + j;
  __shared__ int se[SC_WARPS], sf[SC_WARPS];
  int e = 1, flag = 0;
  if (j < n)
    for (int i = part * 32 + lane; i < m; i += 32 * PARTS) {
      const double2 z = src[(size_t)i * n];
      note_exponent(z.x, e, flag);
      note_exponent(z.y, e, flag);
    }
  e = __reduce_max_sync(0xffffffffu, e);
  flag = __reduce_or_sync(0xffffffffu, flag);
  if (lane == 0) { se[warp] = e; sf[warp] = flag; }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PARTS; ++q) { e = max(e, se[q * SC_COLS + c]); flag |= sf[q * SC_COLS + c]; }
  if (j >= n) return;
  if (part == 0 && lane == 0) {
    exps[(size_t)b * n + j] = e - 1022;
    if (flag) atomicOr(flags + b, flag);
  }
  if (flag) return;
  out.base += (size_t)b * ND * out.plane();
  const double2 zero = make_double2(0.0, 0.0);
  for (int k = 2 * (part * 32 + lane); k < out.kp; k += 64 * PARTS) {
    const double2 z0 = k < m ? src[(size_t)k * n] : zero;
    const double2 z1 = k + 1 < m ? src[(size_t)(k + 1) * n] : zero;
    store_digits<ND>(out, j, k, fixed_data(z0.x, e), fixed_data(z0.y, e), fixed_data(z1.x, e),
                     fixed_data(z1.y, e));
  }
}

// A product's rows as their readers see them.
struct PartialSums {
  const longlong2* P;        // [item][part][rows][ld]
  long long item_stride;
  int ld, rows, cols;
  Deal deal;
};

constexpr int MAX_TILES_A = 256;             // 128-row tiles of the longest A operand (32768 rows)

// How many partial sums the tiles under row r of an item have, [tilesA] in
// shared memory (ends with a block barrier).
__device__ __forceinline__ void count_parts(const PartialSums& q, int item, int r, uint8_t* parts) {
  for (int t = threadIdx.x; t < q.deal.tilesA; t += blockDim.x)
    parts[t] = (uint8_t)q.deal.parts((item * q.deal.tilesB + r / BC) * q.deal.tilesA + t);
  __syncthreads();
}

// Entry a of row r (P: the item's).
__device__ __forceinline__ longlong2 entry(const PartialSums& q, const longlong2* __restrict__ P,
                                           const uint8_t* parts, int r, int a) {
  const size_t sP = (size_t)q.rows * q.ld;
  const longlong2* p = P + (size_t)r * q.ld + a;
  longlong2 v = *p;
  for (int k = parts[a / BM] - 1; k > 0; --k) {
    const longlong2 w = *(p += sP);
    v.x += w.x;
    v.y += w.y;
  }
  return v;
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

// Row r of the first product (entry a in units of 2^(expA[a] - 16 - S)) ->
// its digits as an operand of the second.  A thread keeps its first
// 2 KEEP entries between the two passes (rows up to 2048 entries are read once).
__global__ void __launch_bounds__(256) slice_product_kernel(const PartialSums q,
                                                            const int* __restrict__ expA, int S,
                                                            DigitRows out, int* __restrict__ exps) {
  constexpr int KEEP = 4;
  constexpr int NONE = -(1 << 28);
  const int r = blockIdx.x, b = blockIdx.y;
  const longlong2* P = q.P + (size_t)b * q.item_stride;
  const int* ea = expA + (size_t)b * q.cols;
  __shared__ uint8_t parts[MAX_TILES_A];
  __shared__ int se[8];
  count_parts(q, b, r, parts);
  longlong2 kept[2 * KEEP];
  int e = NONE;
  auto look = [&](int a) {
    longlong2 v = make_longlong2(0, 0);
    if (a < q.cols) {
      v = entry(q, P, parts, r, a);
      if (v.x | v.y) e = max(e, ea[a] + max(bit_length(v.x), bit_length(v.y)));
    }
    return v;
  };
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    const int k = 2 * threadIdx.x + 512 * i;
    kept[2 * i] = look(k);
    kept[2 * i + 1] = look(k + 1);
  }
  for (int k = 512 * KEEP + threadIdx.x; k < q.cols; k += 256) look(k);
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) se[threadIdx.x >> 5] = e;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) e = max(e, se[w]);
  if (threadIdx.x == 0) exps[(size_t)b * q.rows + r] = e == NONE ? 0 : e - 16 - S;
  out.base += (size_t)b * ND * out.plane();
  auto put = [&](int k, longlong2 v0, longlong2 v1) {
    const int s0 = k < q.cols ? ea[k] - e + XBITS : 0, s1 = k + 1 < q.cols ? ea[k + 1] - e + XBITS : 0;
    store_digits<ND>(out, r, k, shift_round(v0.x, s0), shift_round(v0.y, s0), shift_round(v1.x, s1),
                     shift_round(v1.y, s1));
  };
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    const int k = 2 * threadIdx.x + 512 * i;
    if (k < out.kp) put(k, kept[2 * i], kept[2 * i + 1]);
  }
  for (int k = 512 * KEEP + 2 * threadIdx.x; k < out.kp; k += 512) {
    const longlong2 z = make_longlong2(0, 0);
    put(k, k < q.cols ? entry(q, P, parts, r, k) : z, k + 1 < q.cols ? entry(q, P, parts, r, k + 1) : z);
  }
}

// ---------------------------------------------------------------- finish ---
struct FinishParams {
  PartialSums q;             // rows M, cols N
  int M, N, S;
  const int* exps;           // [item][M] (left) or [item][N]: exponent of the sliced product
  int left;                  // (E1 f) E2, else E1 (f E2)
  double scale;
  double2* F;                // [item][M][N]
  // plain FP64 evaluation
  const double2* f;          // [item][m][n]
  int m, n;
  PhaseAxis ar, ac;
  const PhaseAxis* axes;     // per item, or null: ar, ac
  int cols;
  longlong2* scratch;        // P again: the item's intermediate rows
  const int* flags;
  const int* err;
};

__device__ __forceinline__ void cfma(double2& c, double2 a, double2 b) {
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(-a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(a.y, b.x, c.y);
}

// One output row u (left) or column v of a transform in plain FP64, by one
// block: the intermediate row, then the output from it.
__device__ __noinline__ void plain_line(const FinishParams& p, int b, int q) {
  const PhaseAxis ar = p.axes ? p.axes[b] : p.ar, ac = p.axes ? p.axes[p.cols + b] : p.ac;
  const double2* f = p.f + (size_t)b * p.m * p.n;
  double2* F = p.F + (size_t)b * p.M * p.N;
  const int len = p.left ? p.n : p.m, inner = p.left ? p.m : p.n;
  double2* T = reinterpret_cast<double2*>(p.scratch + (size_t)b * p.q.item_stride) + (size_t)q * len;
  for (int a = threadIdx.x; a < len; a += blockDim.x) {
    double2 t = make_double2(0.0, 0.0);
    for (int k = 0; k < inner; ++k) {
      if (p.left) cfma(t, expm2pi_fixed_f64(phase_fixed(ar, k, q)), f[(size_t)k * p.n + a]);
      else cfma(t, f[(size_t)a * p.n + k], expm2pi_fixed_f64(phase_fixed(ac, k, q)));
    }
    T[a] = t;
  }
  __syncthreads();
  const int outs = p.left ? p.N : p.M;
  for (int o = threadIdx.x; o < outs; o += blockDim.x) {
    double2 t = make_double2(0.0, 0.0);
    for (int k = 0; k < len; ++k) {
      if (p.left) cfma(t, T[k], expm2pi_fixed_f64(phase_fixed(ac, k, o)));
      else cfma(t, expm2pi_fixed_f64(phase_fixed(ar, k, o)), T[k]);
    }
    F[p.left ? (size_t)q * p.N + o : (size_t)o * p.N + q] = make_double2(p.scale * t.x, p.scale * t.y);
  }
  __syncthreads();
}

// F = P's entries, scaled.  Bound by reading P from L2 and by the
// FP64 pipe's two conversions and two multiplications an entry.
__global__ void __launch_bounds__(256) finish_kernel(const FinishParams p) {
  const int u = blockIdx.y, b = blockIdx.z;
  const int flag = p.flags[b];
  if (*p.err != 0 || (flag & FLAG_INF && !(flag & FLAG_NAN))) {
    if (blockIdx.x != 0) return;
    for (int q = u; q < (p.left ? p.M : p.N); q += p.M) plain_line(p, b, q);
    return;
  }
  __shared__ uint8_t parts[MAX_TILES_A];
  count_parts(p.q, b, u, parts);
  const int v = blockIdx.x * 256 + threadIdx.x;
  if (v >= p.N) return;
  double2* F = p.F + ((size_t)b * p.M + u) * p.N + v;
  if (flag) {
    const double nan = __longlong_as_double(0x7FF8000000000000ll);
    *F = make_double2(nan, nan);
    return;
  }
  const longlong2 z = entry(p.q, p.q.P + (size_t)b * p.q.item_stride, parts, u, v);
  const int e = (p.left ? p.exps[(size_t)b * p.M + u] : p.exps[(size_t)b * p.N + v]) - 16 - p.S;
  const double x = (double)z.x * p.scale, y = (double)z.y * p.scale;
  if (e > -960 && e < 960) {                    // 2^e is a normal number
    const double c = __longlong_as_double((long long)(e + 1023) << 52);
    *F = make_double2(x * c, y * c);
  } else {
    *F = make_double2(scalbn(x, e), scalbn(y, e));
  }
}

// ------------------------------------------------------------------ host ---
constexpr int GPU_SMS = 152;                 // GB300

int chains_of(int K) { return cdiv(K, BK); }

// Chains per CTA: an even share, one CTA per SM.
Deal deal_of(int rowsA, int rowsB, int K, int items) {
  Deal d;
  d.tilesA = cdiv(rowsA, BM);
  d.tilesB = cdiv(rowsB, BC);
  d.chains = chains_of(K);
  d.per = (int)(((long long)items * d.tilesA * d.tilesB * d.chains + GPU_SMS - 1) / GPU_SMS);
  return d;
}

// Partial sums of a tile at most, whichever chain of a CTA it starts at.
int max_parts(const Deal& d) { return std::min(d.chains, (d.chains + d.per - 2) / d.per + 1); }

int unit_shift(int K) {
  int lg = 0;
  while ((1 << lg) < K) ++lg;
  return std::min(36, 46 - lg);
}

// Tensor map of a digit operand seen as [items x digits][sets][L][kp], box
// {32, box_rows, box_sets, digits}, 64-byte swizzle.
int make_digit_map(CUtensorMap* map, const DigitRows& d, int digits, int items, int box_rows, int box_sets) {
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

// The data operand has ND digits and its own rows for every item, the matrix
// NE digits, shared by the items unless `own`; A is the data when DATA_A.
template <bool DATA_A>
int launch_gemm(const DigitRows& A, const DigitRows& B, bool own, int items, const Deal& deal, int S,
                longlong2* P, long long item_stride, int ld, int* err, cudaStream_t s) {
  constexpr int NA = DATA_A ? ND : NE, NB = DATA_A ? NE : ND;
  static std::once_flag once;
  static cudaError_t attr = cudaSuccess;
  std::call_once(once, [] {
    attr = cudaFuncSetAttribute(sliced_gemm_kernel<NA, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)smem_bytes(NA, NB));
  });
  LGB_CUDA(attr);
  CUtensorMap a, b;
  int st;
  if ((st = make_digit_map(&a, A, NA, DATA_A || own ? items : 1, BM, 1))) return st;
  if ((st = make_digit_map(&b, B, NB, !DATA_A || own ? items : 1, BC, 2))) return st;
  GemmParams p{};
  p.deal = deal;
  p.total = items * deal.tilesA * deal.tilesB * deal.chains;
  p.rowsB = B.L;
  p.ld = ld;
  p.dA = DATA_A || own ? NA : 0;
  p.dB = !DATA_A || own ? NB : 0;
  p.S = S;
  p.P = P;
  p.item_stride = item_stride;
  p.err = err;
  p.wait_ns = WAIT_NS;
  sliced_gemm_kernel<NA, NB><<<cdiv(p.total, deal.per), NUM_THREADS, smem_bytes(NA, NB), s>>>(a, b, p);
  LGB_CUDA(cudaGetLastError());
  return LGB_OK;
}

// Shapes of one sliced transform and its workspace.
struct Layout {
  bool left;
  int K1, K2;                // contraction lengths
  int vecs1;                 // vectors of f (K1 entries each): A rows of the first GEMM
  int rows1;                 // rows of the intermediate (K2 entries each)
  int chunk, ld1, ld2;
  Deal deal1, deal2;
  long long item_stride;     // P entries per item
  int *err, *flags, *exp1, *exp2;
  DigitRows d1, d2;          // digits of f (operand A) and of the intermediate
  longlong2* P;
  size_t bytes;
};

constexpr size_t CHUNK_BYTES = (size_t)512 << 20;

Layout layout(int count, int m, int n, int M, int N, bool left, void* ws) {
  Layout t{};
  t.left = left;
  t.K1 = t.left ? m : n;
  t.K2 = t.left ? n : m;
  t.vecs1 = t.left ? n : m;
  t.rows1 = t.left ? M : N;
  t.d1 = DigitRows{nullptr, t.vecs1, round_up(t.K1, BK), 0};
  t.d2 = DigitRows{nullptr, t.rows1, round_up(t.K2, BK), t.left ? 1 : 0};
  // first GEMM: A = vectors of f, B = the first matrix; second: P's rows are
  // F's rows, its contiguous index F's columns
  t.ld1 = round_up(t.vecs1, BM);
  t.ld2 = round_up(N, BM);
  const size_t p1 = (size_t)t.rows1 * t.ld1, p2 = (size_t)M * t.ld2;              // one partial sum
  const size_t b1 = 2 * ND * t.d1.plane(), b2 = 2 * ND * t.d2.plane();
  t.chunk = (int)std::min<long long>(
      count, std::max<long long>(1, (long long)(CHUNK_BYTES / (b1 + b2 + sizeof(longlong2) * std::max(p1, p2)))));
  t.chunk = cdiv(count, cdiv(count, t.chunk));                                    // even chunks
  t.deal1 = deal_of(t.vecs1, t.rows1, t.K1, t.chunk);
  t.deal2 = deal_of(N, M, t.K2, t.chunk);
  t.item_stride = (long long)std::max(p1 * max_parts(t.deal1), p2 * max_parts(t.deal2));
  size_t off = 0;
  auto take = [&](size_t bytes) {
    off = align_up(off, 256);
    char* q = ws ? static_cast<char*>(ws) + off : nullptr;
    off += bytes;
    return q;
  };
  t.err = reinterpret_cast<int*>(take(16 + sizeof(int) * t.chunk));
  t.flags = t.err ? t.err + 4 : nullptr;
  t.exp1 = reinterpret_cast<int*>(take(sizeof(int) * (size_t)t.chunk * t.vecs1));
  t.exp2 = reinterpret_cast<int*>(take(sizeof(int) * (size_t)t.chunk * t.rows1));
  t.d1.base = reinterpret_cast<uint16_t*>(take(b1 * t.chunk));
  t.d2.base = reinterpret_cast<uint16_t*>(take(b2 * t.chunk));
  t.P = reinterpret_cast<longlong2*>(take(sizeof(longlong2) * (size_t)t.item_stride * t.chunk));
  t.bytes = off;
  return t;
}

}  // namespace

bool sliced_left(int m, int n, int M, int N) {
  return (double)M * m * n + (double)M * n * N <= (double)m * n * N + (double)M * m * N;
}

// Where the sliced form is taken: both contractions at least 32 long, and work
// beyond which its launches cost less than the plain GEMMs.  Device time of one
// transform from a plan, plain -> sliced: 96^2 to 96^2 273 -> 35 us, 256^2
// 278 -> 39, 512^2 2330 -> 90, 1019 x 941 to 1024^2 15800 -> 373, (32 x 1024)
// to (1024 x 32) 399 -> 37.  Operands longer than 16384 would leave the 64-bit
// sums too few fraction bits.
bool sliced_applies(int m, int n, int M, int N) {
  if (std::min(std::min(m, n), std::min(M, N)) < 32 || std::max(m, n) > 16384 ||
      std::max(M, N) > 32768)
    return false;
  const double left = (double)M * m * n + (double)M * n * N, right = (double)m * n * N + (double)M * m * N;
  return std::min(left, right) >= 2.0 * 96 * 96 * 96;
}

size_t sliced_matrix_entries(int len_in, int len_out, bool operand_b) {
  return NE * DigitRows{nullptr, len_out, round_up(len_in, BK), operand_b ? 1 : 0}.plane();
}

int launch_matrix_digits(const PhaseAxis& ax, const PhaseAxis* axes, int count, int len_in, int len_out,
                         bool operand_b, uint16_t* out, cudaStream_t s) {
  const DigitRows d{out, len_out, round_up(len_in, BK), operand_b ? 1 : 0};
  matrix_digits_kernel<<<dim3(cdiv(d.kp, 256), len_out, count), 128, 0, s>>>(ax, axes, len_in, d);
  LGB_CUDA(cudaGetLastError());
  return LGB_OK;
}

size_t sliced_dft2_workspace(int count, int m, int n, int M, int N, bool left) {
  return layout(count, m, n, M, N, left, nullptr).bytes;
}

int launch_sliced_dft2(const SlicedDft2& q, void* ws, cudaStream_t s) {
  const Layout t = layout(q.count, q.m, q.n, q.M, q.N, q.left, ws);
  const bool own = q.axes != nullptr;
  DigitRows e1{const_cast<uint16_t*>(q.e1), q.M, round_up(q.m, BK), 1};
  DigitRows e2{const_cast<uint16_t*>(q.e2), q.N, round_up(q.n, BK), t.left ? 0 : 1};
  const int S1 = unit_shift(t.K1), S2 = unit_shift(t.K2);
  int st;
  for (int b0 = 0; b0 < q.count; b0 += t.chunk) {
    const int items = std::min(t.chunk, q.count - b0);
    const double2* f = q.f + (size_t)b0 * q.m * q.n;
    LGB_CUDA(cudaMemsetAsync(t.err, 0, 16 + sizeof(int) * items, s));
    if (t.left)
      slice_cols_kernel<<<dim3(cdiv(q.n, SC_COLS), items), 32 * SC_WARPS, 0, s>>>(f, q.m, q.n, t.d1, t.exp1,
                                                                                 t.flags);
    else
      slice_rows_kernel<<<dim3(q.m, items), 128, 0, s>>>(f, q.m, q.n, t.d1, t.exp1, t.flags);
    LGB_CUDA(cudaGetLastError());
    if ((st = launch_gemm<true>(t.d1, t.left ? e1 : e2, own, items, t.deal1, S1, t.P, t.item_stride, t.ld1, t.err, s)))
      return st;
    slice_product_kernel<<<dim3(t.rows1, items), 256, 0, s>>>(
        PartialSums{t.P, t.item_stride, t.ld1, t.rows1, t.vecs1, t.deal1}, t.exp1, S1, t.d2, t.exp2);
    LGB_CUDA(cudaGetLastError());
    st = t.left ? launch_gemm<false>(e2, t.d2, own, items, t.deal2, S2, t.P, t.item_stride, t.ld2, t.err, s)
                : launch_gemm<true>(t.d2, e1, own, items, t.deal2, S2, t.P, t.item_stride, t.ld2, t.err, s);
    if (st) return st;
    FinishParams p{};
    p.q = PartialSums{t.P, t.item_stride, t.ld2, q.M, q.N, t.deal2};
    p.M = q.M;
    p.N = q.N;
    p.S = S2;
    p.exps = t.exp2;
    p.left = t.left;
    p.scale = q.scale;
    p.F = q.F + (size_t)b0 * q.M * q.N;
    p.f = f;
    p.m = q.m;
    p.n = q.n;
    p.ar = q.ar;
    p.ac = q.ac;
    p.axes = own ? q.axes + b0 : nullptr;
    p.cols = q.cols;
    p.scratch = t.P;
    p.flags = t.flags;
    p.err = t.err;
    finish_kernel<<<dim3(cdiv(q.N, 256), q.M, items), 256, 0, s>>>(p);
    LGB_CUDA(cudaGetLastError());
    if (own) {
      e1.base += (size_t)items * NE * e1.plane();
      e2.base += (size_t)items * NE * e2.plane();
    }
  }
  return LGB_OK;
}

}  // namespace lgb
