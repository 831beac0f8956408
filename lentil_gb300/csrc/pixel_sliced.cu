// Pixel MTF and spline resampling of pixelate (pixelate.cu) as real matrix
// products out = L . X . R^T on the tensor cores, at FP64 accuracy (sliced.cuh):
//   - the MTF of images whose size has no FFT here: |C img C^T|, C circulant;
//   - the off-grid resampling G p G^T, G banded (64 taps a row).
// Each product is: digits of X's rows and of R's rows; GEMM (its output's
// contiguous index runs over X's rows, so the transposed product comes out
// row by row); digits of those rows; GEMM with L's digits; finish.
// The launches are chained (launch_next): 1000^2 by 3 takes 214 us, and took 246
// one by one.
// Non-finite images, and a device-side wait that ran out, are evaluated in
// plain FP64 by the finishing kernels.
#include "pixelate.cuh"
#include "sliced.cuh"

namespace lgb {
namespace {

// ------------------------------------------------------------ row sources ---
struct DenseRows {
  const double* x;
  int K;
  __device__ __forceinline__ double at(int r, int k) const { return x[(size_t)r * K + k]; }
};
struct CirculantRows {                       // C[r][k] = c[(r - k) mod N]
  const double* c;
  int K;
  __device__ __forceinline__ double at(int r, int k) const { return c[r >= k ? r - k : r - k + K]; }
};
struct BandedRows {                          // G[r][q0[r] + b] = Gt[b][r]
  const double* Gt;
  const int* q0;
  int K, S;
  __device__ __forceinline__ double at(int r, int k) const {
    const int b = k - q0[r];
    return b >= 0 && b < RS_BW ? Gt[(size_t)b * S + r] : 0.0;
  }
};

// Row r of a real matrix -> digits and exponent, by one block.
template <typename Rows>
__device__ __forceinline__ void slice_real_row(const Rows& src, int r, const DigitRows& out, int* exps, int* flag) {
  const int K = src.K;
  __shared__ int se[8], sf[8];
  int e = 1, bad = 0;
  for (int k = threadIdx.x; k < K; k += 256) note_exponent(src.at(r, k), e, bad);
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
  if (bad) return;
  for (int k = 2 * threadIdx.x; k < out.kp; k += 512)
    store_digits(out, 0, r, k, k < K ? fixed_data(src.at(r, k), e) : 0,
                      k + 1 < K ? fixed_data(src.at(r, k + 1), e) : 0);
}

// The rows of X, then those of the operator.
template <typename Rows>
__global__ void __launch_bounds__(256) slice_real_kernel(DenseRows X, int rows, DigitRows dX, int* __restrict__ eX,
                                                         Rows op, DigitRows dR, int* __restrict__ eR,
                                                         int* __restrict__ flag) {
  next_may_start();
  previous_done();
  const int r = blockIdx.x;
  if (r < rows) slice_real_row(X, r, dX, eX, flag);
  else slice_real_row(op, r - rows, dR, eR, flag);
}

// Row r of a product (entry a in units of 2^(ea[a] + eb[r] - 16 - S)) ->
// digits.  The first 2 KEEP entries of a thread stay in registers between the
// two passes.
__global__ void __launch_bounds__(256) slice_real_product_kernel(const PartialSums q,
                                                                 const int* ea,
                                                                 const int* eb, int S,
                                                                 DigitRows out, int* __restrict__ exps) {
  next_may_start();
  constexpr int KEEP = 4, NONE = -(1 << 28);
  const int r = blockIdx.x;
  const long long* P = q.P + (size_t)r * q.ld;
  __shared__ uint8_t parts[MAX_TILES_A];
  __shared__ int se[8];
  count_parts<1>(q, 0, r, parts);
  previous_done();
  long long kept[2 * KEEP], rest[2];
  int e = NONE;
  auto note = [&](int a, long long v) {
    if (v) e = max(e, ea[a] + bit_length(v));
  };
  {
    size_t at[2 * KEEP];
    int n[2 * KEEP];
#pragma unroll
    for (int i = 0; i < 2 * KEEP; ++i) {
      const int k = 2 * threadIdx.x + 512 * (i >> 1) + (i & 1);
      at[i] = k;
      n[i] = k < q.cols ? parts[k / BM] : 0;
    }
    sum_parts<2 * KEEP>(P, q.part(), at, n, kept);
#pragma unroll
    for (int i = 0; i < 2 * KEEP; ++i) note((int)at[i], kept[i]);
  }
  auto fetch = [&](int k) {
    const size_t at[2] = {(size_t)k, (size_t)k + 1};
    const int n[2] = {k < q.cols ? parts[k / BM] : 0, k + 1 < q.cols ? parts[(k + 1) / BM] : 0};
    sum_parts<2>(P, q.part(), at, n, rest);
  };
  for (int k = 512 * KEEP + 2 * threadIdx.x; k < q.cols; k += 512) {
    fetch(k);
    note(k, rest[0]);
    note(k + 1, rest[1]);
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) se[threadIdx.x >> 5] = e;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) e = max(e, se[w]);
  if (threadIdx.x == 0) exps[r] = e == NONE ? 0 : e + eb[r] - 16 - S;
  auto put = [&](int k, long long v0, long long v1) {
    store_digits(out, 0, r, k, k < q.cols ? shift_round(v0, ea[k] - e + XBITS) : 0,
                      k + 1 < q.cols ? shift_round(v1, ea[k + 1] - e + XBITS) : 0);
  };
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    const int k = 2 * threadIdx.x + 512 * i;
    if (k < out.kp) put(k, kept[2 * i], kept[2 * i + 1]);
  }
  for (int k = 512 * KEEP + 2 * threadIdx.x; k < out.kp; k += 512) {
    fetch(k);
    put(k, rest[0], rest[1]);
  }
}

constexpr int FIN_COLS = 4;                  // columns per thread of a finish pass

// Entries k of row r at l = l0 + 256 i of a product.
__device__ __forceinline__ void row_entries(const PartialSums& q, const uint8_t* parts, int r, int l0,
                                            long long (&v)[FIN_COLS]) {
  size_t at[FIN_COLS];
  int n[FIN_COLS];
#pragma unroll
  for (int i = 0; i < FIN_COLS; ++i) {
    const int l = l0 + 256 * i;
    at[i] = l;
    n[i] = l < q.cols ? parts[l / BM] : 0;
  }
  sum_parts<FIN_COLS>(q.P + (size_t)r * q.ld, q.part(), at, n, v);
}

__device__ __forceinline__ double block_sum(double v, double* sm) {      // 256 threads; thread 0 has the sum
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < 8; ++w) v += sm[w];
  return v;
}

struct FinishReal {
  PartialSums q;
  const int *ea, *eb;
  int S;
  const int* status;         // [0] expired wait, [1] non-finite input
  double* out;               // [rows][cols], or null
  double* sum;               // += sum of the results
};

// Row k of |C img C^T|: its entries, their sum, and, when d is set, the
// samples on the detector grid with their sum.
__global__ void __launch_bounds__(256) finish_pixel_kernel(const FinishReal p, const double* img,
                                                           const double* c,
                                                           double* __restrict__ scratch, int os,
                                                           double* __restrict__ d,
                                                           double* __restrict__ sum_d) {
  next_may_start();
  const int N = p.q.rows, k = blockIdx.x;
  __shared__ uint8_t parts[MAX_TILES_A];
  __shared__ double sm[8];
  count_parts<1>(p.q, 0, k, parts);
  previous_done();
  const bool plain = p.status[0] != 0 || p.status[1] != 0;
  double* T = scratch + (size_t)k * N;       // plain: row k of C img (P's memory)
  if (plain) {
    for (int j = threadIdx.x; j < N; j += 256) {
      double t = 0.0;
      for (int i = 0; i < N; ++i) t = fma(c[k >= i ? k - i : k - i + N], img[(size_t)i * N + j], t);
      T[j] = t;
    }
    __syncthreads();
  }
  double s = 0.0, sd = 0.0;
  const int Nd = N / os;
  for (int l0 = threadIdx.x; l0 < N; l0 += 256 * FIN_COLS) {
    long long z[FIN_COLS];
    if (!plain) row_entries(p.q, parts, k, l0, z);
#pragma unroll
    for (int i = 0; i < FIN_COLS; ++i) {
      const int l = l0 + 256 * i;
      if (l >= N) break;
      double v = 0.0;
      if (plain)
        for (int j = 0; j < N; ++j) v = fma(T[j], c[j >= l ? j - l : j - l + N], v);
      else
        v = scaled(z[i], p.ea[l] + p.eb[k] - 16 - p.S, 1.0);
      v = fabs(v);
      if (p.out) p.out[(size_t)k * N + l] = v;
      s += v;
      if (d && k % os == 0 && l % os == 0) {
        d[(size_t)(k / os) * Nd + l / os] = v;
        sd += v;
      }
    }
  }
  s = block_sum(s, sm);
  if (threadIdx.x == 0) atomicAdd(p.sum, s);
  if (d && k % os == 0) {
    sd = block_sum(sd, sm);
    if (threadIdx.x == 0) atomicAdd(sum_d, sd);
  }
}

// Row k of G p G^T and its sum.
__global__ void __launch_bounds__(256) finish_resample_kernel(const FinishReal p, const double* img,
                                                              const double* Gt,
                                                              const int* q0, int N) {
  next_may_start();
  const int S = p.q.rows, k = blockIdx.x;
  __shared__ uint8_t parts[MAX_TILES_A];
  __shared__ double sm[8];
  count_parts<1>(p.q, 0, k, parts);
  previous_done();
  const bool plain = p.status[0] != 0 || p.status[1] != 0;
  double s = 0.0;
  for (int l0 = threadIdx.x; l0 < S; l0 += 256 * FIN_COLS) {
    long long z[FIN_COLS];
    if (!plain) row_entries(p.q, parts, k, l0, z);
#pragma unroll
    for (int i = 0; i < FIN_COLS; ++i) {
      const int l = l0 + 256 * i;
      if (l >= S) break;
      double v = 0.0;
      if (plain) {
        const int nk = min(RS_BW, N - q0[k]), nl = min(RS_BW, N - q0[l]);
        for (int a = 0; a < nk; ++a) {
          double t = 0.0;
          for (int b = 0; b < nl; ++b)
            t = fma(Gt[(size_t)b * S + l], img[(size_t)(q0[k] + a) * N + q0[l] + b], t);
          v = fma(Gt[(size_t)a * S + k], t, v);
        }
      } else {
        v = scaled(z[i], p.ea[l] + p.eb[k] - 16 - p.S, 1.0);
      }
      p.out[(size_t)k * S + l] = v;
      s += v;
    }
  }
  s = block_sum(s, sm);
  if (threadIdx.x == 0) atomicAdd(p.sum, s);
}

// ------------------------------------------------------------------ host ---
DigitRows real_rows(uint16_t* base, int L, int K) { return DigitRows{base, L, round_up(K, BK), 1}; }

// Two products of one sandwich: X is p x q (rows of K = q), R has rows r of
// length q, L rows r of length p (both sides have the same operator here).
struct Sandwich {
  int p, q, r;
  Band band;                 // of the operator's rows
  Deal deal1, deal2;
  int ld1, ld2;
  size_t P_entries;
  Sandwich(int p_, int q_, int r_, int step) : p(p_), q(q_), r(r_) {
    const int total = cdiv(q, 2 * BK);
    band.step = step;
    band.total = total;
    band.count = step ? std::min(total, (96 * step + 68) / 64 + 2) : total;
    deal1 = deal_of(p, r, band.count, 1);                 // A: X's rows, B: operator rows
    deal2 = deal_of(r, r, band.count, 1);                 // A: rows of the first product
    ld1 = round_up(p, BM);
    ld2 = round_up(r, BM);
    P_entries = std::max((size_t)r * ld1 * max_parts(deal1), (size_t)r * ld2 * max_parts(deal2));
  }
};

size_t digit_entries(int L, int K) { return ND * real_rows(nullptr, L, K).plane(); }

struct Space {
  int *eX, *eR, *eT;
  uint16_t *dX, *dR, *dT;
  long long* P;
  size_t bytes;
};

Space carve(const Sandwich& w, void* ws) {
  Space t{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    off = align_up(off, 256);
    char* q = ws ? static_cast<char*>(ws) + off : nullptr;
    off += bytes;
    return q;
  };
  t.eX = reinterpret_cast<int*>(take(sizeof(int) * w.p));
  t.eR = reinterpret_cast<int*>(take(sizeof(int) * w.r));
  t.eT = reinterpret_cast<int*>(take(sizeof(int) * w.r));
  t.dX = reinterpret_cast<uint16_t*>(take(2 * digit_entries(w.p, w.q)));
  t.dR = reinterpret_cast<uint16_t*>(take(2 * digit_entries(w.r, w.q)));
  t.dT = reinterpret_cast<uint16_t*>(take(2 * digit_entries(w.r, w.p)));
  t.P = reinterpret_cast<long long*>(take(sizeof(long long) * w.P_entries));
  t.bytes = off;
  return t;
}

template <typename Rows>
int run_sandwich(const Sandwich& w, const Space& t, const double* X, const Rows& op, int* status, cudaStream_t s) {
  const int S = unit_shift(w.q, 1);
  const DigitRows dX = real_rows(t.dX, w.p, w.q), dR = real_rows(t.dR, w.r, w.q), dT = real_rows(t.dT, w.r, w.p);
  LGB_CUDA(launch_next(slice_real_kernel<Rows>, w.p + w.r, 256, 0, s, DenseRows{X, w.q}, w.p, dX, t.eX, op, dR, t.eR,
                       status + 1));
  int st = launch_gemm(dX, 1, dR, 1, 1, w.q, w.deal1, w.band, S, t.P, 0, w.ld1, status, s);
  if (st) return st;
  LGB_CUDA(launch_next(slice_real_product_kernel, w.r, 256, 0, s, PartialSums{t.P, 0, w.ld1, w.r, w.p, w.deal1}, t.eX,
                       t.eR, S, dT, t.eT));
  return launch_gemm(dT, 1, dR, 1, 1, w.q, w.deal2, w.band, S, t.P, 0, w.ld2, status, s);
}

}  // namespace

size_t pixel_sliced_workspace(int N) { return carve(Sandwich(N, N, N, 0), nullptr).bytes; }

int launch_pixel_sliced(const double* img, int N, const double* c, void* ws, int* status, double* P, double* sums,
                        int os, double* d, cudaStream_t s) {
  const Sandwich w(N, N, N, 0);
  const Space t = carve(w, ws);
  const int st = run_sandwich(w, t, img, CirculantRows{c, N}, status, s);
  if (st) return st;
  const FinishReal f{PartialSums{t.P, 0, w.ld2, N, N, w.deal2}, t.eT, t.eR, unit_shift(N, 1), status,
                     P, sums};
  LGB_CUDA(launch_next(finish_pixel_kernel, N, 256, 0, s, f, img, c, reinterpret_cast<double*>(t.P), os, d, sums + 1));
  return LGB_OK;
}

size_t resample_sliced_workspace(int N, int os, int S) { return carve(Sandwich(N, N, S, os), nullptr).bytes; }

int launch_resample_sliced(const double* P, int N, int os, int S, const double* Gt, const int* q0, void* ws,
                           int* status, double* raw, double* sum, cudaStream_t s) {
  const Sandwich w(N, N, S, os);
  const Space t = carve(w, ws);
  const int st = run_sandwich(w, t, P, BandedRows{Gt, q0, N, S}, status, s);
  if (st) return st;
  const FinishReal f{PartialSums{t.P, 0, w.ld2, S, S, w.deal2}, t.eT, t.eR, unit_shift(N, 1), status,
                     raw, sum};
  LGB_CUDA(launch_next(finish_resample_kernel, S, 256, 0, s, f, P, Gt, q0, N));
  return LGB_OK;
}

}  // namespace lgb
