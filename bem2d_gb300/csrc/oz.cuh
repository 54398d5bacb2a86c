// Exact 8-bit digit splitting for products on the f16 tensor cores (lu_oz.cu,
// oz_gemm.cu): scale exponents, digits, the shared-memory layout and the MMA.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "tc.cuh"

namespace bem2d_gpu {
namespace oz {

// scale exponents: zero rows / columns, and rows / columns with a NaN or an
// infinity
constexpr int kZero = -100000, kNaN = 400000;

// K-major, no swizzle: core matrices of 8 rows x 16 bytes, 128 bytes along K,
// 256 bytes from one group of 8 rows to the next
__device__ __forceinline__ unsigned long long desc(unsigned addr) {
  return (unsigned long long)((addr & 0x3FFFF) >> 4) | ((unsigned long long)(128 >> 4) << 16) |
         ((unsigned long long)(256 >> 4) << 32) | (1ull << 46);
}
// byte offset of 8 consecutive k (k8 = 0, 1) of row r in a 16-deep block
__device__ __forceinline__ int off(int r, int k8) { return (r >> 3) * 256 + k8 * 128 + (r & 7) * 16; }

// D (128 x n, FP32) (+)= A (128 x 16) B^T (n x 16), f16
__device__ __forceinline__ void mma(unsigned d, unsigned a, unsigned b, unsigned n, unsigned acc) {
  // kind::f16: D f32 (bits 4-5 = 1), A and B f16 (0), K-major, N >> 3 at bit
  // 17, M >> 4 at bit 24
  const unsigned idesc = (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24);
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(desc(a)), "l"(desc(b)), "r"(idesc), "r"(acc));
}

// exponent field of a double (0: zero or subnormal, 2047: not finite), and the
// exponent that goes with the mantissa: subnormals have that of the smallest
// normal numbers
__device__ __forceinline__ int expo_field(double x) { return (__double2hiint(x) >> 20) & 2047; }
__device__ __forceinline__ int expo(double x) { return max(expo_field(x), 1); }
__device__ __forceinline__ bool is_zero(double2 v) {
  const int h = __double2hiint(v.x) | __double2hiint(v.y);
  return ((h & 0x7fffffff) | __double2loint(v.x) | __double2loint(v.y)) == 0;
}

__device__ __forceinline__ int scale_of(int emax) {
  return emax > 50000 ? kNaN : emax <= -5000 ? kZero : emax;
}

// x 2^p as a fixed-point integer F, |F| < 2^(8 S - 1): x 2^p = F 2^(erow -
// 1022 - (8 S - 1)), erow the largest exponent field plus p of the row, whose
// largest entry has |F| >= 2^(8 S - 2) if it is normal.  Rounded to nearest (S =
// 8: toward zero, below 2^-62 of the row's largest).
template <int S>
__device__ __forceinline__ long long fixed(double x, int p, int erow) {
  const long long b = __double_as_longlong(x);
  const int e = expo(x);
  const long long m = (b & 0xfffffffffffffll) | (expo_field(x) ? 0x10000000000000ll : 0ll);
  const int d = erow - (e + p) + 54 - 8 * S;  // shift to the right
  long long f;
  if (d <= 0)
    f = m << min(-d, 63);  // at most 10 for the entries of a scaled row
  else if (S == 8)
    f = d < 53 ? m >> d : 0;
  else
    f = d < 55 ? (m + (1ll << (d - 1))) >> d : 0;
  return b < 0 ? -f : f;
}

// The S balanced digits of 8 consecutive k of one real row, as f16.
template <int S>
struct Digits {
  unsigned w[S][4];
};
template <int S>
__device__ __forceinline__ void digits(const long long* f, Digits<S>* o) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    long long a = f[2 * q], b = f[2 * q + 1];
#pragma unroll
    for (int s = S - 1; s >= 0; --s) {
      const int da = s ? (int)(signed char)(a & 0xff) : (int)a;
      const int db = s ? (int)(signed char)(b & 0xff) : (int)b;
      a = (a - da) >> 8;
      b = (b - db) >> 8;
      // (1536 + d) - 1536 in f16: exact for |d| <= 512
      const unsigned w = 0x66006600u + (unsigned)da + ((unsigned)db << 16);
      const unsigned base = 0x66006600u;
      const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&w),
                                *reinterpret_cast<const __half2*>(&base));
      o->w[s][q] = *reinterpret_cast<const unsigned*>(&h);
    }
  }
}

}  // namespace oz
}  // namespace bem2d_gpu
