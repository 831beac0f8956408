// Pixel MTF of images whose size has no FFT here (pixelate.cu): |C img C^T|, C
// the circulant matrix of N taps c that fall off as 1/k^2, twice as
//     Y[r][a] = sum_q C[r][q] X[a][q],   X = img, then X = Y.
// The taps within w of the diagonal are summed in FP64, the others as digit
// products on the tensor cores (sliced.cuh), whose errors are relative to the
// largest far tap and the brightest pixel of a row.  Taking all of C so left
// pixels that are faint beside their row with errors of the nearest taps' size:
// 1.0e-14 of a pixel (median) behind a core 1e7 times as bright, 1e-11 behind
// 1e10, where the FP64 product has 3e-16 and 1e-15.  With w = N / 32 it is 3e-16
// and 1e-15 again (150^2 and 500^2 by 2 and 3, against extended precision), since
// a far tap is within 2^10 of the tap that couples a pixel to any other.
// Non-finite images, and a device-side wait that ran out, are evaluated in plain
// FP64 by the combining kernel.
#include "pixelate.cuh"
#include "sliced.cuh"

namespace lgb {
namespace {

// C[r][k] = c[(r - k) mod N] where r and k are more than w apart, else 0
struct FarTaps {
  const double* c;
  int N, w;
  __device__ __forceinline__ double at(int r, int k) const {
    const int d = r >= k ? r - k : r - k + N;
    return min(d, N - d) <= w ? 0.0 : c[d];
  }
};
struct DenseRows {
  const double* x;
  int N;
  __device__ __forceinline__ double at(int r, int k) const { return x[(size_t)r * N + k]; }
};

__device__ __forceinline__ double block_sum(double v, double* sm) {      // 256 threads; thread 0 has the sum
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < 8; ++w) v += sm[w];
  return v;
}

// Row r of a real N x N matrix -> digits and exponent, by one block.
template <typename Rows>
__device__ __forceinline__ int slice_real_row(const Rows& src, int r, const DigitRows& out, int* exps, int* flag) {
  const int N = src.N;
  __shared__ int se[8], sf[8];
  int e = 1, bad = 0;
  for (int k = threadIdx.x; k < N; k += 256) note_exponent(src.at(r, k), e, bad);
  e = __reduce_max_sync(0xffffffffu, e);
  bad = __reduce_or_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) { se[threadIdx.x >> 5] = e; sf[threadIdx.x >> 5] = bad; }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) { e = max(e, se[w]); bad |= sf[w]; }
  if (threadIdx.x == 0) {
    exps[r] = e - 1022;
    if (bad) atomicOr(flag, bad);
  }
  if (bad) return e;
  for (int k = 2 * threadIdx.x; k < out.kp; k += 512)
    store_digits(out, 0, r, k, k < N ? fixed_data(src.at(r, k), e) : 0,
                      k + 1 < N ? fixed_data(src.at(r, k + 1), e) : 0);
  return e;
}

// The rows of X, then (blocks from N on) those of the operator, whose first block
// also finds the unit of the sums: with L the sum of |C[0][q]| over the power of two
// above their largest, no sum exceeds L 2^16 of the digits' units, and S = 46 - lg L
// leaves it below 2^62.  (L is some 2 w, not N: six bits more than unit_shift.)
__global__ void __launch_bounds__(256) slice_real_kernel(DenseRows X, DigitRows dX, int* __restrict__ eX,
                                                         FarTaps op, DigitRows dR, int* __restrict__ eR,
                                                         int* __restrict__ flag, int* __restrict__ unit) {
  next_may_start();
  previous_done();
  const int r = blockIdx.x;
  if (r < X.N) {
    slice_real_row(X, r, dX, eX, flag);
    return;
  }
  const int e = slice_real_row(op, r - X.N, dR, eR, flag);
  if (r > X.N) return;
  __shared__ double sm[8];
  double sum = 0.0;
  for (int k = threadIdx.x; k < op.N; k += 256) sum += fabs(op.at(0, k));
  sum = block_sum(sum, sm);
  if (threadIdx.x == 0) {
    const int lg = sum > 0.0 ? ilogb(sum * (1.0 + 1e-9)) + 1 - (e - 1022) : 0;
    *unit = min(42, 46 - lg);
  }
}

constexpr int TILE = 32;                     // rows and columns of Y per combining block
constexpr int QC = 64;                       // entries of X's rows staged at once
constexpr int MAX_NEAR = 512;

struct Combine {
  PartialSums q;             // the far taps' products: rows r, cols a
  const int *ea, *eb;        // exponents of X's rows and of the operator's
  const int* unit;           // S
  const int* status;         // [0] expired wait, [1] non-finite input
  const double *X, *c;
  int N, w;
  double* Y;                 // [N][N], or null
  // of the last product: |Y|, its sum added to sums[0]; with d, every os-th
  // sample and their sum (sums[1])
  int os;
  double *d, *sums;
};

// Y = the FP64 sum over the near taps + the far taps' product.
//
// Bound by the FP64 pipe (16 clk a warp instruction): a lane is a column a, a warp
// four rows r with a window of 2 w + 4 entries, so that an entry of X and a tap from
// shared memory feed four FMAs.  1000^2, w = 32: 127 us, of which the 65 FMAs of
// each entry take 112 (all 1000 of them took 1730 in the FP64 GEMM).
template <bool LAST>
__global__ void __launch_bounds__(256) combine_kernel(const Combine p) {
  __shared__ double xs[QC][TILE + 1];
  __shared__ double taps[2 * MAX_NEAR + 2 * TILE];       // c[d] at d + w + TILE, 0 beyond w
  __shared__ double sm[8];
  next_may_start();
  previous_done();
  const int N = p.N, w = p.w;
  const int a0 = blockIdx.x * TILE, r0 = blockIdx.y * TILE;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = a0 + lane, r = r0 + 4 * warp;
  const bool plain = p.status[0] != 0 || p.status[1] != 0;
  for (int i = threadIdx.x; i < 2 * (w + TILE); i += 256) {
    const int d = i - w - TILE;
    taps[i] = d >= -w && d <= w ? p.c[d < 0 ? d + N : d] : 0.0;
  }
  double y[4] = {0.0, 0.0, 0.0, 0.0};
  const int first = plain ? 0 : r0 - w, last = plain ? N : r0 + TILE + w;
  for (int qb = first; qb < last; qb += QC) {
    __syncthreads();
    for (int i = threadIdx.x; i < TILE * QC; i += 256) {
      int q = qb + (i & (QC - 1));
      q = q < 0 ? q + N : q >= N ? q - N : q;
      const int row = a0 + i / QC;                          // (beyond the window: not used)
      xs[i & (QC - 1)][i / QC] = row < N && q < N ? p.X[(size_t)row * N + q] : 0.0;
    }
    __syncthreads();
    if (plain) {
      for (int t = 0; t < min(QC, N - qb); ++t) {
        const double x = xs[t][lane];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int d = r + i - (qb + t);
          if (r + i < N) y[i] = fma(p.c[d < 0 ? d + N : d], x, y[i]);
        }
      }
    } else {
      const int t0 = max(0, r - w - qb), t1 = min(QC, r + 4 + w - qb);
      const double* tap = taps + (r - qb + w + TILE);       // tap[-t + i]: row r + i, entry qb + t
      for (int t = t0; t < t1; ++t) {
        const double x = xs[t][lane];
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = fma(tap[i - t], x, y[i]);
      }
    }
  }
  if (!plain) {
    size_t at[4];
    int n[4];
    long long v[4];
    const int parts = r < N && a < N ? p.q.parts(0, r, a0) : 0;       // four rows, 32 columns: one tile
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      at[i] = (size_t)(r + i) * p.q.ld + a;
      n[i] = r + i < N ? parts : 0;
    }
    sum_parts<4>(p.q.P, p.q.part(), at, n, v);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (r + i < N && a < N) y[i] += scaled(v[i], p.ea[a] + p.eb[r + i] - 16 - *p.unit, 1.0);
  }
  double s = 0.0, sd = 0.0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = r + i;
    if (k >= N || a >= N) continue;
    if (LAST) {
      y[i] = fabs(y[i]);
      s += y[i];
      if (p.d && k % p.os == 0 && a % p.os == 0) {
        p.d[(size_t)(k / p.os) * (N / p.os) + a / p.os] = y[i];
        sd += y[i];
      }
    }
    if (!LAST || p.Y) p.Y[(size_t)k * N + a] = y[i];
  }
  if (LAST) {
    s = block_sum(s, sm);
    if (threadIdx.x == 0) atomicAdd(p.sums, s);
    if (p.d) {
      sd = block_sum(sd, sm);
      if (threadIdx.x == 0) atomicAdd(p.sums + 1, sd);
    }
  }
}
static_assert(BM % TILE == 0 && BN % TILE == 0, "a combining block lies in one tile of the GEMM");

// ------------------------------------------------------------------ host ---
DigitRows real_rows(uint16_t* base, int N) { return DigitRows{base, N, round_up(N, BK), 1}; }

struct Space {
  Deal deal;
  int ld;
  int *eX, *eR, *unit;
  uint16_t *dX, *dR;
  long long* P;
  double* Y;
  size_t bytes;
};

Space carve(int N, void* ws) {
  Space t{};
  t.deal = deal_of(N, N, cdiv(N, 2 * BK), 1);
  t.ld = round_up(N, BM);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    off = align_up(off, 256);
    char* q = ws ? static_cast<char*>(ws) + off : nullptr;
    off += bytes;
    return q;
  };
  const size_t digits = 2 * ND * real_rows(nullptr, N).plane();
  t.eX = reinterpret_cast<int*>(take(sizeof(int) * N));
  t.eR = reinterpret_cast<int*>(take(sizeof(int) * N));
  t.unit = reinterpret_cast<int*>(take(sizeof(int)));
  t.dX = reinterpret_cast<uint16_t*>(take(digits));
  t.dR = reinterpret_cast<uint16_t*>(take(digits));
  t.P = reinterpret_cast<long long*>(take(sizeof(long long) * (size_t)N * t.ld * max_parts(t.deal)));
  t.Y = reinterpret_cast<double*>(take(sizeof(double) * (size_t)N * N));
  t.bytes = off;
  return t;
}

}  // namespace

size_t pixel_sliced_workspace(int N) { return carve(N, nullptr).bytes; }

int launch_pixel_sliced(const double* img, int N, const double* c, void* ws, int* status, double* P, double* sums,
                        int os, double* d, cudaStream_t s) {
  const Space t = carve(N, ws);
  const DigitRows dX = real_rows(t.dX, N), dR = real_rows(t.dR, N);
  const int w = std::max(16, cdiv(N, 32));             // N <= 16384: at most MAX_NEAR
  Combine f{};
  f.q = PartialSums{t.P, 0, t.ld, N, N, t.deal, nullptr, false};
  f.ea = t.eX;
  f.eb = t.eR;
  f.unit = t.unit;
  f.status = status;
  f.c = c;
  f.N = N;
  f.w = w;
  f.os = os;
  const dim3 grid(cdiv(N, TILE), cdiv(N, TILE));
  for (int pass = 0; pass < 2; ++pass) {
    f.X = pass == 0 ? img : t.Y;
    LGB_CUDA(launch_next(slice_real_kernel, pass == 0 ? 2 * N : N, 256, 0, s, DenseRows{f.X, N}, dX, t.eX,
                         FarTaps{c, N, w}, dR, t.eR, status + 1, t.unit));
    const int st = launch_gemm(dX, 1, dR, 1, 1, N, t.deal, t.unit, 0, nullptr, t.P, 0, t.ld, status, s);
    if (st) return st;
    if (pass == 0) {
      f.Y = t.Y;
      LGB_CUDA(launch_next(combine_kernel<false>, grid, 256, 0, s, f));
    } else {
      f.Y = P;
      f.d = d;
      f.sums = sums;
      LGB_CUDA(launch_next(combine_kernel<true>, grid, 256, 0, s, f));
    }
  }
  return LGB_OK;
}

}  // namespace lgb
