// Shared by pixelate.cu and pixel_sliced.cu.
#pragma once

#include "common.cuh"

namespace lgb {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// |C img C^T| for the circulant C of the taps c[N], 64 <= N <= 16384: P[N][N]
// (may be null), its sum added to sums[0]; with d, every os-th sample and their sum (sums[1])
// status: two words, zero: [0] an expired wait, [1] non-finite input
size_t pixel_sliced_workspace(int N);
int launch_pixel_sliced(const double* img, int N, const double* c, void* ws, int* status, double* P, double* sums,
                        int os, double* d, cudaStream_t s);

}  // namespace lgb
