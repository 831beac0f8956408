// K3: the plain FP64 (complex128) matrix triple product of lentil's dft2
// (lentil/fourier.py:95-101), as two tiled complex GEMMs on the FP64 pipe.
// This is the parity form (<= 1e-12 peak-normalised against numpy) and the
// baseline the split tensor-core form is measured against.
#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "kernels.cuh"

namespace lgb {

// 16 x 16 outputs per CTA of 64 threads.  The FP64 pipe (two FMAs a clock per
// SM) bounds every shape, and loads from shared memory cost little beside it,
// so the tile is small enough that even a 64 x 64 output spreads over all SMs
// (with K split): a 64^3 product took 134 us in 64 x 64 tiles, two CTAs of
// work, and takes 4 us here; at 512^3 the two tiles cost the same.
constexpr int ZBM = 16, ZBN = 16, ZBK = 8;

// blockIdx.x counts the tiles (fields of more than 16 x 65535 rows have more
// than y holds); blockIdx.z = b * splits + split: problem b, K range [split * kchunk,
// (split + 1) * kchunk); with splits > 1 each split writes its own partial
// product (C offset by split * sP) for zgemm_reduce_kernel to sum in order.
__global__ void __launch_bounds__(64) zgemm_kernel(int M, int N, int K,
                                                   const double2* __restrict__ A, int lda, long long sA,
                                                   const double2* __restrict__ B, int ldb, long long sB,
                                                   double2* __restrict__ C, int ldc, long long sC,
                                                   double alpha, int splits, int kchunk, long long sP) {
  __shared__ double2 As[ZBK][ZBM];
  __shared__ double2 Bs[ZBK][ZBN];
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3, tid = threadIdx.x;
  const int tiles_n = (N + ZBN - 1) / ZBN, tm = blockIdx.x / tiles_n;
  const int m0 = tm * ZBM, n0 = ((int)blockIdx.x - tm * tiles_n) * ZBN;
  const int b = blockIdx.z / splits, split = blockIdx.z - b * splits;
  A += (size_t)b * sA;
  B += (size_t)b * sB;
  C += (size_t)b * sC + (size_t)split * sP;
  const int kbeg = split * kchunk, kend = min(K, kbeg + kchunk);
  double cr[2][2] = {}, ci[2][2] = {};
  double2 ra[2], rb[2];                          // the next K block, loaded ahead
  const double2 zero = make_double2(0.0, 0.0);
  auto load = [&](int k0) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int e = tid + 64 * t;
      const int gr = m0 + (e >> 3), gk = k0 + (e & 7);          // A: 16 rows x 8 k
      ra[t] = (gr < M && gk < kend) ? A[(size_t)gr * lda + gk] : zero;
      const int hk = k0 + (e >> 4), gc = n0 + (e & 15);         // B: 8 k x 16 columns
      rb[t] = (hk < kend && gc < N) ? B[(size_t)hk * ldb + gc] : zero;
    }
  };
  load(kbeg);
  for (int k0 = kbeg; k0 < kend; k0 += ZBK) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int e = tid + 64 * t;
      As[e & 7][e >> 3] = ra[t];
      Bs[e >> 4][e & 15] = rb[t];
    }
    __syncthreads();
    if (k0 + ZBK < kend) load(k0 + ZBK);
#pragma unroll
    for (int k = 0; k < ZBK; ++k) {
      double2 a[2], bb[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) a[i] = As[k][ty + 8 * i];
#pragma unroll
      for (int j = 0; j < 2; ++j) bb[j] = Bs[k][tx + 8 * j];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          cr[i][j] = fma(a[i].x, bb[j].x, cr[i][j]);
          cr[i][j] = fma(-a[i].y, bb[j].y, cr[i][j]);
          ci[i][j] = fma(a[i].x, bb[j].y, ci[i][j]);
          ci[i][j] = fma(a[i].y, bb[j].x, ci[i][j]);
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = m0 + ty + 8 * i;
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = n0 + tx + 8 * j;
      if (c < N) C[(size_t)r * ldc + c] = make_double2(alpha * cr[i][j], alpha * ci[i][j]);
    }
  }
}

// C[b] = alpha * sum_s P[s][b] in split order (deterministic), P[s][b] M x N dense
__global__ void zgemm_reduce_kernel(const double2* __restrict__ P, int splits, long long sP,
                                    int M, int N, double2* __restrict__ C, int ldc, long long sC,
                                    double alpha) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y, b = blockIdx.z;
  if (c >= N) return;
  const double2* p = P + (size_t)b * M * N + (size_t)r * N + c;
  double re = 0.0, im = 0.0;
  for (int k = 0; k < splits; ++k) {
    const double2 v = p[(size_t)k * sP];
    re += v.x;
    im += v.y;
  }
  C[(size_t)b * sC + (size_t)r * ldc + c] = make_double2(alpha * re, alpha * im);
}

// The partials come from the device's default stream-ordered pool; by
// default the pool hands freed memory back at every synchronisation, so the
// next launch would map it again.  This process keeps up to 256 MiB cached
// (a property of the process's pool, gone when the process ends).
static void keep_pool_memory() {
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { (void)cudaGetLastError(); return; }
  std::lock_guard<std::mutex> lock(mu);
  if (done[dev]) return;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
    uint64_t keep = (uint64_t)256 << 20;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  }
  (void)cudaGetLastError();
  done[dev] = true;
}

// K splits of a launch (1: whole): see launch_zgemm.
static int zgemm_splits(int M, int N, int K, int batch) {
  const long long tiles = (long long)cdiv(N, ZBN) * cdiv(M, ZBM) * batch;
  const int sms = sm_count();
  if (tiles >= 2LL * sms || K <= ZBK) return 1;
  return (int)std::min<long long>({(2LL * sms + tiles - 1) / tiles, (long long)cdiv(K, ZBK), 16LL,
                                   65535LL / batch});
}

size_t zgemm_partial_bytes(int M, int N, int K, int batch) {
  const int splits = zgemm_splits(M, N, K, batch);
  return splits > 1 ? (size_t)splits * batch * M * N * sizeof(double2) : 0;
}

// A launch of fewer than two tiles per SM would leave FP64 pipes idle (a
// 64 x 64 output is 16 tiles), so such a launch splits K over up to 16 CTAs
// per tile, each writing a partial product to scratch (the caller's, or
// stream-ordered pool memory), and a second kernel sums the partials in split
// order.
int launch_zgemm(int M, int N, int K, const double2* A, int lda, long long sA, const double2* B,
                 int ldb, long long sB, double2* C, int ldc, long long sC, int batch, double alpha,
                 cudaStream_t s, const ZgemmScratch* scratch) {
  if (M <= 0 || N <= 0 || batch <= 0) return LGB_OK;
  LGB_REQUIRE(batch <= 65535, LGB_EINVAL, "zgemm: batch too large");
  int splits = zgemm_splits(M, N, K, batch);
  const long long sP = (long long)batch * M * N;          // one split's partials
  const size_t part_bytes = (size_t)sP * sizeof(double2);
  if (scratch) {                                          // as many splits as fit
    const size_t fit = scratch->ptr ? scratch->bytes / part_bytes : 0;
    if ((size_t)splits > fit) splits = (int)fit;
  } else if (splits > 1 && (size_t)splits * part_bytes > ((size_t)256 << 20)) {
    splits = 1;
  }
  if (splits <= 1) {
    dim3 grid(cdiv(N, ZBN) * cdiv(M, ZBM), 1, batch);
    zgemm_kernel<<<grid, 64, 0, s>>>(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, alpha, 1, K, 0);
    LGB_CUDA(cudaGetLastError());
    return LGB_OK;
  }
  const int kchunk = round_up(cdiv(K, splits), ZBK);
  splits = cdiv(K, kchunk);
  double2* P = nullptr;
  if (scratch) {
    P = static_cast<double2*>(scratch->ptr);
  } else {
    keep_pool_memory();
    LGB_CUDA(cudaMallocAsync(reinterpret_cast<void**>(&P), (size_t)splits * part_bytes, s));
  }
  dim3 grid(cdiv(N, ZBN) * cdiv(M, ZBM), 1, batch * splits);
  zgemm_kernel<<<grid, 64, 0, s>>>(M, N, K, A, lda, sA, B, ldb, sB, P, N, (long long)M * N, 1.0,
                                    splits, kchunk, sP);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) {
    dim3 rgrid(cdiv(N, 128), M, batch);
    zgemm_reduce_kernel<<<rgrid, 128, 0, s>>>(P, splits, sP, M, N, C, ldc, sC, alpha);
    e = cudaGetLastError();
  }
  if (!scratch) cudaFreeAsync(P, s);
  LGB_CUDA(e);
  return LGB_OK;
}

// out[b] += sum_l weights[b*L + l] * unit2[l] * |F[b*L + l]|^2 over the window (FP64);
// each output pixel is owned by one thread, so the wavelength sum is
// race-free and in a fixed order.
__global__ void intensity_accum_kernel(const double2* __restrict__ F, int M, int N, long long sF,
                                       int L, const double* __restrict__ weights,
                                       const double* __restrict__ unit2,
                                       double* __restrict__ out, int ld_out, long long s_out,
                                       int win_r0, int win_c0) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  const int u = blockIdx.y;
  const int b = blockIdx.z;
  if (v >= N || u >= M) return;
  double acc = 0.0;
  for (int l = 0; l < L; ++l) {
    const double2 z = F[((size_t)b * L + l) * sF + (size_t)u * N + v];
    const double w = (weights ? weights[(size_t)b * L + l] : 1.0) * unit2[l];
    acc = fma(w, z.x * z.x + z.y * z.y, acc);
  }
  out[(size_t)b * s_out + (size_t)(win_r0 + u) * ld_out + win_c0 + v] += acc;
}

int launch_intensity_accum_c128(const double2* F, int M, int N, long long sF, int batch_inner,
                                const double* weights, const double* unit2, double* out,
                                int ld_out, long long s_out, int win_r0, int win_c0, int n_outer,
                                cudaStream_t s) {
  if (M <= 0 || N <= 0) return LGB_OK;
  dim3 grid(cdiv(N, 128), M, n_outer);
  intensity_accum_kernel<<<grid, 128, 0, s>>>(F, M, N, sF, batch_inner, weights, unit2, out,
                                             ld_out, s_out, win_r0, win_c0);
  LGB_CUDA(cudaGetLastError());
  return LGB_OK;
}

}  // namespace lgb
