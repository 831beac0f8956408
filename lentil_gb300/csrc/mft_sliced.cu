// K3s: complex128 matrix triple products on the tensor cores, by slicing
// (sliced.cuh).  lentil's dft2 (lentil/fourier.py:95-101) is F = E1 . f . E2.
//
// A transform is five launches:
//   slice_field   f -> digits, one exponent per vector of the contraction
//   sliced_gemm   P = E1 . f or f . E2, in integers
//   slice_rows    P's rows, scaled to their largest entry -> digits
//   sliced_gemm   P = the second product
//   finish        P -> F, scaled
// chained (launch_next): 512^2 took 71.5 us launched one by one with the flags
// cleared beforehand, 61.5 so (65.2 with the later changes to its sums).
// A field with a NaN gives NaN everywhere (each output sums every entry); one
// with infinities, or a device-side wait that ran out, makes `finish`
// evaluate that transform in plain FP64 instead.
#include <atomic>
#include <mutex>

#include "cossin.cuh"
#include "sliced.cuh"

namespace lgb {
namespace {

// DFT-matrix digits: vector j < L (output index) over the input index; matrix
// z's axis is axes[z], or ax when there is one.  Bound by the 42 bytes written
// per entry (17.5 us for 1019 x 1024, cold caches); the cosines are integer arithmetic because
// sincospi alone would take the FP64 pipe longer than that.
__global__ void __launch_bounds__(128) matrix_digits_kernel(PhaseAxis ax, const PhaseAxis* __restrict__ axes,
                                                            int len_in, DigitRows out) {
  __shared__ unsigned long long table[129];
  for (int i = threadIdx.x; i < 129; i += 128) table[i] = COS_TABLE[i];
  __syncthreads();
  if (axes) ax = axes[blockIdx.z];
  out.base += (size_t)blockIdx.z * ND * out.plane();
  const int k = 2 * (blockIdx.x * blockDim.x + threadIdx.x), j = blockIdx.y;
  if (k >= out.kp) return;
  const uint64_t ph = phase_fixed(ax, k, j);
  longlong2 e0 = make_longlong2(0, 0), e1 = e0;                 // (cos, sin): E = cos - i sin
  if (k < len_in) e0 = cossin_q62(ph, table);
  if (k + 1 < len_in) e1 = cossin_q62(ph + phase_step_in(ax, j), table);
  store_digits3(out, j, k, make_longlong2(e0.x, -e0.y), make_longlong2(e1.x, -e1.y));
}

// in place of a vector's exponent: it has infinities, or NaN
constexpr int EXP_INF = 1 << 20, EXP_NAN = 1 << 21;

__device__ __forceinline__ int exponent_or_flag(int e, int flag) {
  return flag & FLAG_NAN ? EXP_NAN : flag ? EXP_INF : e - 1022;
}

__device__ __forceinline__ longlong2 fixed_entry(double2 z, int e) {
  return make_longlong2(fixed_data(z.x, e), fixed_data(z.y, e));
}

// f's rows (one block each) -> digits, vectors of n entries.
__global__ void __launch_bounds__(128) slice_rows_kernel(const double2* __restrict__ f, int m, int n,
                                                         DigitRows out, int* __restrict__ exps, int S,
                                                         int* __restrict__ limits, int* __restrict__ err) {
  next_may_start();
  const int i = blockIdx.x, b = blockIdx.y;
  if (i == 0 && b == 0 && threadIdx.x == 0) *err = 0;
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
    exps[(size_t)b * m + i] = exponent_or_flag(e, flag);
    limits[(size_t)b * m + i] = S;
  }
  if (flag) return;                                       // this transform does not use its digits
  out.base += (size_t)b * ND * out.plane();
  const double2 zero = make_double2(0.0, 0.0);
  unsigned sum = 0;
  for (int k = 2 * threadIdx.x; k < out.kp; k += 256) {
    const longlong2 x0 = fixed_entry(k < n ? src[k] : zero, e), x1 = fixed_entry(k + 1 < n ? src[k + 1] : zero, e);
    sum += magnitude(x0) + magnitude(x1);
    store_digits3(out, i, k, x0, x1);
  }
  __shared__ unsigned sums[4];
  sum = __reduce_add_sync(0xffffffffu, sum);
  if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) limits[(size_t)b * m + i] = unit_limit(sums[0] + sums[1] + sums[2] + sums[3], n, S);
}

constexpr int SC_COLS = 4, SC_WARPS = 16;    // columns and warps per block of slice_cols

// f's columns -> digits, vectors of m entries: SC_COLS neighbouring columns a
// block (a 64-byte piece of each row), SC_WARPS / SC_COLS warps per column.
__global__ void __launch_bounds__(32 * SC_WARPS) slice_cols_kernel(
    const double2* __restrict__ f, int m, int n, DigitRows out, int* __restrict__ exps, int S,
    int* __restrict__ limits, int* __restrict__ err) {
  next_may_start();
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *err = 0;
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
  unsigned sum = 0;
  if (j < n && !flag) {
    out.base += (size_t)b * ND * out.plane();
    const double2 zero = make_double2(0.0, 0.0);
    for (int k = 2 * (part * 32 + lane); k < out.kp; k += 64 * PARTS) {
      const longlong2 x0 = fixed_entry(k < m ? src[(size_t)k * n] : zero, e);
      const longlong2 x1 = fixed_entry(k + 1 < m ? src[(size_t)(k + 1) * n] : zero, e);
      sum += magnitude(x0) + magnitude(x1);
      store_digits3(out, j, k, x0, x1);
    }
  }
  __shared__ unsigned sums[SC_WARPS];
  sum = __reduce_add_sync(0xffffffffu, sum);
  if (lane == 0) sums[warp] = sum;
  __syncthreads();
  if (j < n && part == 0 && lane == 0) {
    for (int q = 1; q < PARTS; ++q) sum += sums[q * SC_COLS + c];
    exps[(size_t)b * n + j] = exponent_or_flag(e, flag);
    limits[(size_t)b * n + j] = flag ? S : unit_limit(sum, m, S);
  }
}

// Row r of the first product (entry a in units of 2^(expA[a] - 16 - S), S of its
// tile) -> its digits as an operand of the second.  The first 2 KEEP entries of a thread
// stay in registers between the two passes (rows of up to 1024 are read once).
// A vector of f that is not finite marks every row.
__global__ void __launch_bounds__(256) slice_product_kernel(const PartialSums q,
                                                            const int* expA, DigitRows out,
                                                            int* __restrict__ exps, int S2,
                                                            int* __restrict__ limits) {
  next_may_start();
  constexpr int KEEP = 2, NONE = -(1 << 28);
  const int r = blockIdx.x, b = blockIdx.y;
  const long long* P = q.P + (size_t)b * 3 * q.stride + (size_t)r * q.ld;
  const int tiles = q.deal.tilesA;
  const int* ea = expA + (size_t)b * q.cols;
  __shared__ uint8_t parts[3 * MAX_TILES_A];
  __shared__ int se[8];
  __shared__ unsigned sums[8];
  count_parts<3>(q, 3 * b, r, parts);
  previous_done();
  // of entry a's units, less 16, or that its vector is not finite
  auto exponent = [&](int a) {
    const int x = a < q.cols ? ea[a] : NONE;
    return a < q.cols && x < EXP_INF ? x - q.S(b, r, a) : x;
  };
  longlong2 kept[2 * KEEP], rest[2];
  int x[2 * KEEP], y[2];
  int e = NONE;
  auto note = [&](int x, longlong2 v) {
    if (x >= EXP_INF) e = max(e, x);
    else if (v.x | v.y) e = max(e, x + max(bit_length(v.x), bit_length(v.y)));
  };
  {
    size_t at[2 * KEEP];
    int n[3][2 * KEEP];
#pragma unroll
    for (int i = 0; i < 2 * KEEP; ++i) {
      const int k = 2 * threadIdx.x + 512 * (i >> 1) + (i & 1);
      at[i] = k;
      x[i] = exponent(k);
#pragma unroll
      for (int c = 0; c < 3; ++c) n[c][i] = k < q.cols ? parts[c * tiles + k / BM] : 0;
    }
    sum_parts3<2 * KEEP>(P, q.stride, q.part(), at, n, kept);
#pragma unroll
    for (int i = 0; i < 2 * KEEP; ++i) note(x[i], kept[i]);
  }
  auto fetch = [&](int k) {                     // entries k, k + 1 -> rest
    const size_t at[2] = {(size_t)k, (size_t)k + 1};
    int n[3][2];
    y[0] = exponent(k);
    y[1] = exponent(k + 1);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      n[c][0] = k < q.cols ? parts[c * tiles + k / BM] : 0;
      n[c][1] = k + 1 < q.cols ? parts[c * tiles + (k + 1) / BM] : 0;
    }
    sum_parts3<2>(P, q.stride, q.part(), at, n, rest);
  };
  for (int k = 512 * KEEP + 2 * threadIdx.x; k < q.cols; k += 512) {
    fetch(k);
    note(y[0], rest[0]);
    note(y[1], rest[1]);
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) se[threadIdx.x >> 5] = e;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) e = max(e, se[w]);
  const int bad = e >= EXP_NAN ? EXP_NAN : e >= EXP_INF ? EXP_INF : 0;
  if (threadIdx.x == 0) {
    exps[(size_t)b * q.rows + r] = bad ? bad : e == NONE ? 0 : e - 16;
    limits[(size_t)b * q.rows + r] = S2;
  }
  if (bad) return;
  out.base += (size_t)b * ND * out.plane();
  unsigned sum = 0;
  auto put = [&](int k, int e0, int e1, longlong2 v0, longlong2 v1) {
    const int s0 = max(e0 - e + XBITS, -64), s1 = max(e1 - e + XBITS, -64);      // (beyond the row: zeros)
    const longlong2 x0 = make_longlong2(shift_round(v0.x, s0), shift_round(v0.y, s0));
    const longlong2 x1 = make_longlong2(shift_round(v1.x, s1), shift_round(v1.y, s1));
    sum += magnitude(x0) + magnitude(x1);
    store_digits3(out, r, k, x0, x1);
  };
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    const int k = 2 * threadIdx.x + 512 * i;
    if (k < out.kp) put(k, x[2 * i], x[2 * i + 1], kept[2 * i], kept[2 * i + 1]);
  }
  for (int k = 512 * KEEP + 2 * threadIdx.x; k < out.kp; k += 512) {
    fetch(k);
    put(k, y[0], y[1], rest[0], rest[1]);
  }
  sum = __reduce_add_sync(0xffffffffu, sum);
  if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) sum += sums[w];
    limits[(size_t)b * q.rows + r] = unit_limit(sum, q.cols, S2);
  }
}

// ---------------------------------------------------------------- finish ---
struct FinishParams {
  PartialSums q;             // rows M, cols N
  int M, N;
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
  const int* vec_exps;       // [item][vectors of f]: exponents, or that it has infinities
  long long* scratch;        // P again: the item's intermediate rows
  const int* err;
};

__device__ __forceinline__ void cfma(double2& c, double2 a, double2 b) {
  c.x = fma(a.x, b.x, c.x);
  c.x = fma(-a.y, b.y, c.x);
  c.y = fma(a.x, b.y, c.y);
  c.y = fma(a.y, b.x, c.y);
}

constexpr int LINES = 4;                     // output rows or columns at once
constexpr int LINE_K = 64;                   // entries of a sum staged at once

__device__ __forceinline__ double2 matrix_entry(const PhaseAxis& ax, int i, int j) {
  const longlong2 z = cossin_q62(phase_fixed(ax, i, j), COS_TABLE);
  const double c = assembled((uint64_t)(z.x < 0 ? -z.x : z.x), -62), s = assembled((uint64_t)(z.y < 0 ? -z.y : z.y), -62);
  return make_double2(z.x < 0 ? -c : c, z.y > 0 ? -s : s);
}

// Output rows (left) or columns q0 .. q0 + LINES - 1 of a transform in plain FP64,
// by one block: their intermediate rows, then the output from those.  Of a field
// with infinities (`some`) only the vectors that hold one count: what they add to
// an output is not finite, and what the others add does not change it.  An entry
// of the first matrix serves the whole block, one of the second LINES outputs.
// One infinity in 1019 x 941, to 1024^2: 136 ms with every vector and a sincospi
// for every multiply-add, 1.2 so; all of it, after an expired wait, 18 (the FP64
// GEMMs: 15.8).
__device__ __noinline__ void plain_lines(const FinishParams& p, int b, int q0, bool some) {
  __shared__ double2 e[LINE_K][LINES];
  const PhaseAxis ar = p.axes ? p.axes[b] : p.ar, ac = p.axes ? p.axes[p.cols + b] : p.ac;
  const PhaseAxis &ax1 = p.left ? ar : ac, &ax2 = p.left ? ac : ar;
  const int len = p.left ? p.n : p.m, inner = p.left ? p.m : p.n;
  const double2* f = p.f + (size_t)b * p.m * p.n;
  const size_t along = p.left ? p.n : 1, across = p.left ? 1 : p.n;      // strides of a vector, of the vectors
  double2* F = p.F + (size_t)b * p.M * p.N;
  const int lines = min(LINES, (p.left ? p.M : p.N) - q0), outs = p.left ? p.N : p.M;
  double2* T = reinterpret_cast<double2*>(p.scratch + (size_t)b * 3 * p.q.stride) + (size_t)q0 * len;
  const int* vec = p.vec_exps + (size_t)b * len;
  auto counts = [&](int k) { return !some || vec[k] >= EXP_INF; };
  for (int a0 = 0; a0 < len; a0 += blockDim.x) {
    const int a = a0 + threadIdx.x;
    const bool mine = a < len && counts(a);
    if (!__syncthreads_or(mine)) continue;
    double2 t[LINES] = {};
    for (int k0 = 0; k0 < inner; k0 += LINE_K) {
      const int ks = min(LINE_K, inner - k0);
      __syncthreads();
      for (int i = threadIdx.x; i < LINES * LINE_K; i += blockDim.x) {
        const int l = i % LINES, k = i / LINES;
        if (k < ks) e[k][l] = matrix_entry(ax1, k0 + k, q0 + min(l, lines - 1));
      }
      __syncthreads();
      if (mine) {
        const double2* x = f + a * across + k0 * along;
        for (int k = 0; k < ks; ++k, x += along) {
          const double2 z = *x;
#pragma unroll
          for (int l = 0; l < LINES; ++l) cfma(t[l], e[k][l], z);
        }
      }
    }
#pragma unroll
    for (int l = 0; l < LINES; ++l)
      if (l < lines && mine) T[(size_t)l * len + a] = t[l];
  }
  for (int o0 = 0; o0 < outs; o0 += blockDim.x) {
    const int o = o0 + threadIdx.x;
    double2 t[LINES] = {};
    for (int k0 = 0; k0 < len; k0 += LINE_K) {
      const int ks = min(LINE_K, len - k0);
      __syncthreads();                                   // T is written, e no longer read
      for (int i = threadIdx.x; i < LINES * LINE_K; i += blockDim.x) {
        const int l = i / LINE_K, k = i % LINE_K;
        if (k < ks && counts(k0 + k)) e[k][l] = T[(size_t)min(l, lines - 1) * len + k0 + k];
      }
      __syncthreads();
      for (int k = 0; k < ks; ++k) {
        if (!counts(k0 + k)) continue;
        const double2 w = matrix_entry(ax2, k0 + k, min(o, outs - 1));
#pragma unroll
        for (int l = 0; l < LINES; ++l) cfma(t[l], e[k][l], w);
      }
    }
    if (o >= outs) continue;
#pragma unroll
    for (int l = 0; l < LINES; ++l)
      if (l < lines)
        F[p.left ? (size_t)(q0 + l) * p.N + o : (size_t)o * p.N + q0 + l] =
            make_double2(p.scale * t[l].x, p.scale * t[l].y);
  }
  __syncthreads();
}

constexpr int FIN_ROWS = 4;                  // rows per finish block, of launches that fill the GPU

// F = P's entries, scaled.  Bound by reading P from L2 and writing F (40 bytes
// an entry and a part; 21 us at 1024^2, cold caches).  Results are put together
// from bits and four rows' parts are in flight at once: with conversions and
// both scalings on the FP64 pipe and a row per block it took half as long again.
template <int ROWS>
__global__ void __launch_bounds__(256) finish_kernel(const FinishParams p) {
  previous_done();
  const int b = blockIdx.z, flag = p.exps[(size_t)b * (p.left ? p.M : p.N)];      // all of them, if one is
  if (*p.err != 0 || flag == EXP_INF) {
    const int first = LINES * (blockIdx.y * gridDim.x + blockIdx.x), step = LINES * gridDim.y * gridDim.x;
    for (int q = first; q < (p.left ? p.M : p.N); q += step) plain_lines(p, b, q, *p.err == 0);
    return;
  }
  const int v = blockIdx.x * 256 + threadIdx.x, u0 = blockIdx.y * ROWS;
  if (v >= p.N) return;
  double2* F = p.F + ((size_t)b * p.M + u0) * p.N + v;
  const int rows = min(ROWS, p.M - u0);
  if (flag == EXP_NAN) {
    const double nan = __longlong_as_double(0x7FF8000000000000ll);
    for (int i = 0; i < rows; ++i) F[(size_t)i * p.N] = make_double2(nan, nan);
    return;
  }
  const int* exps = p.exps + (p.left ? (size_t)b * p.M + u0 : (size_t)b * p.N + v);
  const int unit = 16 + p.q.S(b, u0, v);
  longlong2 z[ROWS];
  size_t at[ROWS];
  int n[3][ROWS], e[ROWS];
  static_assert(BN % ROWS == 0, "the rows lie in one tile");
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const int parts = p.q.parts(3 * b + c, u0, v);
#pragma unroll
    for (int i = 0; i < ROWS; ++i) n[c][i] = i < rows ? parts : 0;
  }
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    at[i] = (size_t)(u0 + i) * p.q.ld + v;
    e[i] = i < rows ? exps[p.left ? i : 0] - unit : 0;
  }
  sum_parts3<ROWS>(p.q.P + (size_t)b * 3 * p.q.stride, p.q.stride, p.q.part(), at, n, z);
#pragma unroll
  for (int i = 0; i < ROWS; ++i)
    if (i < rows)
      F[(size_t)i * p.N] = make_double2(scaled(z[i].x, e[i], p.scale), scaled(z[i].y, e[i], p.scale));
}

// Shapes of one sliced transform and its workspace.
struct Layout {
  bool left;
  int K1, K2;                // contraction lengths
  int vecs1;                 // vectors of f (K1 entries each): A rows of the first GEMM
  int rows1;                 // rows of the intermediate (K2 entries each)
  int chunk, ld1, ld2;
  Deal deal1, deal2;
  long long stride;          // P entries per product
  int *err, *exp1, *exp2;
  int *lim1, *lim2, *tile1, *tile2;            // units: limits of the data's vectors, S of the tiles
  DigitRows d1, d2;          // digits of f (operand A) and of the intermediate
  long long* P;
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
  t.d1 = DigitRows{nullptr, t.vecs1, round_up(t.K1, BK), 3};
  t.d2 = DigitRows{nullptr, t.rows1, round_up(t.K2, BK), 3};
  // first GEMM: A = vectors of f, B = the first matrix; second: P's rows are
  // F's rows, its contiguous index F's columns
  t.ld1 = round_up(t.vecs1, BM);
  t.ld2 = round_up(N, BM);
  const size_t p1 = (size_t)t.rows1 * t.ld1, p2 = (size_t)M * t.ld2;              // one partial sum
  const size_t b1 = 2 * ND * t.d1.plane(), b2 = 2 * ND * t.d2.plane();
  t.chunk = (int)std::min<long long>(
      count, std::max<long long>(1, (long long)(CHUNK_BYTES / (b1 + b2 + 3 * sizeof(long long) * std::max(p1, p2)))));
  t.chunk = cdiv(count, cdiv(count, t.chunk));                                    // even chunks
  t.deal1 = deal_of(t.vecs1, t.rows1, cdiv(t.K1, 2 * BK), 3 * t.chunk);
  t.deal2 = deal_of(N, M, cdiv(t.K2, 2 * BK), 3 * t.chunk);
  t.stride = (long long)std::max(p1 * max_parts(t.deal1), p2 * max_parts(t.deal2));
  size_t off = 0;
  auto take = [&](size_t bytes) {
    off = align_up(off, 256);
    char* q = ws ? static_cast<char*>(ws) + off : nullptr;
    off += bytes;
    return q;
  };
  t.err = reinterpret_cast<int*>(take(16));
  t.exp1 = reinterpret_cast<int*>(take(sizeof(int) * (size_t)t.chunk * t.vecs1));
  t.exp2 = reinterpret_cast<int*>(take(sizeof(int) * (size_t)t.chunk * t.rows1));
  t.lim1 = reinterpret_cast<int*>(take(sizeof(int) * (size_t)t.chunk * t.vecs1));
  t.lim2 = reinterpret_cast<int*>(take(sizeof(int) * (size_t)t.chunk * t.rows1));
  t.tile1 = reinterpret_cast<int*>(take(sizeof(int) * (size_t)t.chunk * t.deal1.tilesA));
  t.tile2 = reinterpret_cast<int*>(take(sizeof(int) * (size_t)t.chunk * (t.left ? t.deal2.tilesB : t.deal2.tilesA)));
  t.d1.base = reinterpret_cast<uint16_t*>(take(b1 * t.chunk));
  t.d2.base = reinterpret_cast<uint16_t*>(take(b2 * t.chunk));
  t.P = reinterpret_cast<long long*>(take(sizeof(long long) * (size_t)t.stride * 3 * t.chunk));
  t.bytes = off;
  return t;
}

}  // namespace

bool sliced_left(int m, int n, int M, int N) {
  return (double)M * m * n + (double)M * n * N <= (double)m * n * N + (double)M * m * N;
}

// Where the sliced form is taken: where its five launches cost less than the
// plain GEMMs' two to four.  Device time of one transform from a plan, plain and
// sliced (us): 64^2 to 64^2 16.8 and 25.5, 88^2 26.2 and 27.1, 96^2 26.3 and 27.4,
// 104^2 35.1 and 27.5, 128^2 42.7 and 27.7, 256^2 267 and 30.8; (8 x 8) to 512^2 23.9
// and 27.8, (8 x 9) to 600^2 31.8 and 31.4, (16 x 512) to (16 x 512) 57.7 and 24.8,
// (32 x 800) to (400 x 49) 46.9 and 31.1.  The line is one of multiply-adds, near the
// crossing: beside it the plain form is up to 4 us ahead or 16 behind, by shape.
// Operands longer than 16384 would leave the 64-bit sums too few fraction bits.
bool sliced_applies(int m, int n, int M, int N) {
  if (std::min(std::min(m, n), std::min(M, N)) < 8 || std::max(m, n) > 16384 ||
      std::max(M, N) > 32768)
    return false;
  const double left = (double)M * m * n + (double)M * n * N, right = (double)m * n * N + (double)M * m * N;
  return std::min(left, right) >= 2.0 * 96 * 96 * 96;
}

static DigitRows matrix_rows(const uint16_t* digits, int len_in, int len_out) {
  return DigitRows{const_cast<uint16_t*>(digits), len_out, round_up(len_in, BK), 3};
}

size_t sliced_matrix_entries(int len_in, int len_out) { return ND * matrix_rows(nullptr, len_in, len_out).plane(); }

int launch_matrix_digits(const PhaseAxis& ax, const PhaseAxis* axes, int count, int len_in, int len_out,
                         uint16_t* out, cudaStream_t s) {
  const DigitRows d = matrix_rows(out, len_in, len_out);
  matrix_digits_kernel<<<dim3(cdiv(d.kp, 256), len_out, count), 128, 0, s>>>(ax, axes, len_in, d);
  LGB_CUDA(cudaGetLastError());
  return LGB_OK;
}

size_t sliced_dft2_workspace(int count, int m, int n, int M, int N, bool left) {
  return layout(count, m, n, M, N, left, nullptr).bytes;
}

int sliced_dft2_chunk(int count, int m, int n, int M, int N, bool left) {
  return layout(count, m, n, M, N, left, nullptr).chunk;
}

int launch_sliced_dft2(const SlicedDft2& q, void* ws, cudaStream_t s) {
  const Layout t = layout(q.count, q.m, q.n, q.M, q.N, q.left, ws);
  const bool own = q.axes != nullptr;
  DigitRows e1 = matrix_rows(q.e1, q.m, q.M), e2 = matrix_rows(q.e2, q.n, q.N);
  const int S1 = unit_shift(t.K1), S2 = unit_shift(t.K2);
  int st;
  for (int b0 = 0; b0 < q.count; b0 += t.chunk) {
    const int items = std::min(t.chunk, q.count - b0);
    const double2* f = q.f + (size_t)b0 * q.m * q.n;
    if (q.build) {
      if ((st = launch_matrix_digits(PhaseAxis{}, q.axes + b0, items, q.m, q.M, e1.base, s))) return st;
      if ((st = launch_matrix_digits(PhaseAxis{}, q.axes + q.cols + b0, items, q.n, q.N, e2.base, s))) return st;
    }
    if (t.left)
      slice_cols_kernel<<<dim3(cdiv(q.n, SC_COLS), items), 32 * SC_WARPS, 0, s>>>(f, q.m, q.n, t.d1, t.exp1, S1,
                                                                                 t.lim1, t.err);
    else
      slice_rows_kernel<<<dim3(q.m, items), 128, 0, s>>>(f, q.m, q.n, t.d1, t.exp1, S1, t.lim1, t.err);
    LGB_CUDA(cudaGetLastError());
    const int own_items = own ? items : 1;
    if ((st = launch_gemm(t.d1, items, t.left ? e1 : e2, own_items, items, t.K1, t.deal1, t.lim1, BM, t.tile1,
                          t.P, t.stride, t.ld1, t.err, s)))
      return st;
    LGB_CUDA(launch_next(slice_product_kernel, dim3(t.rows1, items), 256, 0, s,
                         PartialSums{t.P, t.stride, t.ld1, t.rows1, t.vecs1, t.deal1, t.tile1, false}, t.exp1, t.d2,
                         t.exp2, S2, t.lim2));
    if ((st = launch_gemm(t.left ? e2 : t.d2, t.left ? own_items : items, t.left ? t.d2 : e1,
                          t.left ? items : own_items, items, t.K2, t.deal2, t.lim2, t.left ? BN : BM, t.tile2,
                          t.P, t.stride, t.ld2, t.err, s)))
      return st;
    FinishParams p{};
    p.q = PartialSums{t.P, t.stride, t.ld2, q.M, q.N, t.deal2, t.tile2, t.left};
    p.M = q.M;
    p.N = q.N;
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
    p.vec_exps = t.exp1;
    p.scratch = t.P;
    p.err = t.err;
    // four rows a block where that is a block per SM; below, one row (256^2: 64
    // blocks of four rows, the transform 34.9 us, 256 of one, 31.3; 512^2: 256
    // blocks of four, 57.7, 1024 of one, 60.6)
    const int blocks = cdiv(q.N, 256) * cdiv(q.M, FIN_ROWS) * items;
    if (blocks >= GPU_SMS)
      LGB_CUDA(launch_next(finish_kernel<FIN_ROWS>, dim3(cdiv(q.N, 256), cdiv(q.M, FIN_ROWS), items), 256, 0, s, p));
    else
      LGB_CUDA(launch_next(finish_kernel<1>, dim3(cdiv(q.N, 256), q.M, items), 256, 0, s, p));
    if (own && !q.build) {
      e1.base += (size_t)items * ND * e1.plane();
      e2.base += (size_t)items * ND * e2.plane();
    }
  }
  return LGB_OK;
}

// The armed stall: launches to go by first, and what the one after them holds back.
static std::mutex g_stall_mu;
static std::atomic<int> g_stall_launches{-1};       // -1: none (the launches' only look at it)
static SlicedStall g_stall;

SlicedStall take_sliced_stall() {
  SlicedStall none;
  if (g_stall_launches.load(std::memory_order_relaxed) < 0) return none;
  std::lock_guard<std::mutex> lock(g_stall_mu);
  if (g_stall_launches < 0 || g_stall_launches-- > 0) return none;
  return g_stall;
}

}  // namespace lgb

using namespace lgb;

extern "C" int lgb_test_stall_sliced(int launch, int stage, int release, double wait_ms) {
  LGB_REQUIRE(launch >= 0 && stage >= 0, LGB_EINVAL, "test_stall_sliced: launch and stage must be >= 0");
  LGB_REQUIRE(wait_ms > 0.0 && wait_ms <= 2000.0, LGB_EINVAL, "test_stall_sliced: wait_ms must lie in (0, 2000]");
  std::lock_guard<std::mutex> lock(g_stall_mu);
  g_stall.stage = stage;
  g_stall.release = release != 0;
  g_stall.wait_ns = (unsigned long long)(wait_ms * 1e6);
  g_stall_launches = launch;
  return LGB_OK;
}
