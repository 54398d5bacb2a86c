// Scales of a product's inner index k: the exponents of the columns of its left
// operand, for the tensor-core updates whose operands are fixed point within a
// row or column (lu_oz.cu, lu_tc.cu).
//
// With A(:, k) 2^t_k and B(k, :) 2^-t_k, t_k the negative exponent of the largest
// entry of A(:, k), the operands are the same whatever powers of two scale the
// rows and columns of the matrix being factored: a factor of row k of U is a
// factor of 1 / l_ik in all of column k of L.
#pragma once

#include <cuda_runtime.h>

namespace bem2d_gpu {

constexpr int kColParts = 16;  // partial maxima per column at most

// exponent field (0: zero, subnormal or not finite)
__device__ __forceinline__ int col_expo(double x) {
  const int e = (__double2hiint(x) >> 20) & 2047;
  return e == 2047 ? 0 : e;
}
__device__ __forceinline__ int col_expo(float x) {
  const int e = (__float_as_int(x) >> 23) & 255;
  return e == 255 ? 0 : e;
}

// *out = largest exponent field of the rows of a column (M of them) in every np-th
// block of 256 from block p on; 256 threads.
template <typename T>
__device__ __forceinline__ void col_expo_part(const T* __restrict__ col, int M, int p, int np,
                                              int* __restrict__ out) {
  __shared__ int red[8];
  int e = 0;
#pragma unroll 4
  for (int r = p * 256 + threadIdx.x; r < M; r += np * 256) {
    const T v = col[r];
    e = max(e, max(col_expo(v.x), col_expo(v.y)));
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) e = max(e, red[w]);
    *out = e;
  }
}

// part[p K + k]: part p (blockIdx.y) of column k (blockIdx.x, K of them) of A (M rows)
template <typename T>
__global__ void __launch_bounds__(256)
col_expo_kernel(const T* __restrict__ A, long long lda, int M, int* __restrict__ part) {
  col_expo_part(A + (size_t)blockIdx.x * lda, M, blockIdx.y, gridDim.y,
                &part[blockIdx.y * gridDim.x + blockIdx.x]);
}

// Partial maxima per column of M rows.
inline int col_expo_parts(int M) {
  return M <= 1024 ? 1 : M >= 1024 * kColParts ? kColParts : (M + 1023) / 1024;
}

// Launches it; returns their number.
template <typename T>
int launch_col_expo(const T* A, long long lda, int M, int K, int* part, cudaStream_t s) {
  const int np = col_expo_parts(M);
  col_expo_kernel<T><<<dim3(K, np), 256, 0, s>>>(A, lda, M, part);
  return np;
}

// largest exponent field of column k
__device__ __forceinline__ int col_expo_max(const int* __restrict__ part, int np, int K, int k) {
  int e = 0;
#pragma unroll
  for (int p = 0; p < kColParts; ++p)  // all loads in flight at once
    if (p < np) e = max(e, __ldg(&part[p * K + k]));
  return e;
}

}  // namespace bem2d_gpu
