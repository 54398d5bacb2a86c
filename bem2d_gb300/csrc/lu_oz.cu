// Complex128 products on the 5th-generation tensor cores with FP64 accuracy:
// C = beta C + sign A B (column-major, any leading dimensions, K in slabs of
// 64), the trailing update of the complex128 LU.
//
// GB300's FP64 pipe issues 2 FMAs per clock and SM (1.06 TFLOP/s measured),
// its f16 tensor pipe 2 PFLOP/s.  The operands are therefore cut into 8-bit
// digits, products of digits are summed exactly, and FP64 is left only to add
// the sum to C (the error-free splitting of Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication by using fast routines
// of matrix multiplication and its applications", Numer. Algorithms 59, 2012, on tensor cores as
// in Mukunoki, Ozaki, Ogita and Imamura, ISC 2020).
//
// Digits.  Row i of A and column j of B are scaled by powers of two so that
// every entry is a 63-bit fixed-point integer F and a sign, and F = sum_s a_s
// 256^(7 - s), s = 0..7, with balanced digits |a_s| <= 128.  f16 holds each
// digit exactly.  A product of digits is at most 2^14 and one accumulator
// collects the pairs of one order s + t (at most 8) over K = 64: at most 2^23,
// exact in the FP32 accumulator.  Kept are the 36 pairs with s + t <= 7; what
// is dropped is below 2^-52 of (largest entry of the row) x (largest of the
// column) in the worst case and 2^-60 typically, where an FP64 sum of 64
// products rounds at about 2^-51 of its largest.  An entry's 53 bits survive
// whole while it is within 2^-10 of its row's largest.
//
// Rows and columns of very different size (graded meshes, unknowns in different
// units) must not meet in that bound:
//  - inner index k is scaled by the largest exponent of A(:, k) (colscale.cuh),
//    which makes the digits independent of powers of two on the rows and
//    columns of the matrix being factored.  (Scaled by the pivot's exponent, as
//    if A were read before the division by the pivot, columns of a system 2^60
//    apart left no correct digit in its solution.)
//  - an entry of the product whose 64 terms are all below 2^-kOzSpan of (row's
//    largest) x (column's largest) is summed in FP64 by the epilogue.  The pack
//    kernel marks rows and columns whose own entries span more than that; where
//    both are marked the terms' exponents are compared.  Disk, kite and random
//    systems have no such entries, squares and L-shapes graded over 8 levels 1
//    to 2 % of them in the updates behind a corner's panel.  Scales, marks and
//    comparisons together cost nothing that can be measured (disk N = 160 1.132
//    -> 1.127 ms, kite N = 2048 20.31 -> 20.33, N = 3001 21.1 -> 20.9, with one
//    pack kernel for both operands instead of two), the sums 9 % of the solve
//    on a graded square.
//
// Complex arithmetic as in lu_tc.cu: A' (rows 2i, 2i + 1 = re, im of row i)
// times [B_r B_i]; re C_i = D1[2i] - D2[2i+1], im C_i = D2[2i] + D1[2i+1].
//
// A tile is 64 complex rows by 16 complex columns: 32 accumulator columns for
// each of the 8 orders, 256 in all, two such sets in tensor memory.  Digit s
// of A against the digits 0 .. 7 - s of B, which lie one after another as
// rows of one operand, is one MMA of N = 32 (8 - s) whose result lands on the
// orders s .. 7: 8 MMAs per 16 of K, A read once for all of them.
//
// Persistent CTAs take contiguous runs of tiles (row block major) and keep
// the row block's A (128 KB) in shared memory:
//   warp 0     producer (bulk copies; A when the row block changes, B into a
//              ring of two 32 KB stages)
//   warp 1     MMA issuer
//   warps 2-9  epilogue: orders 0-3 and 4-7 of D1 and D2 become two 64-bit
//              integers each, partners exchange D2, two exact conversions, one
//              FMA to join them, one to add to C: 4 FP64 instructions per
//              real number, which bound the kernel (2,600 clocks of MMAs
//              against 4,100 of FP64 for a tile).
// Every wait is bounded as in lu_tc.cu.
//
// Measured against the FP64-pipe update it replaces: solve n = 3001 111.7 ->
// 49.7 ms; error of one K = 64 product of Gaussian matrices 8 times smaller
// (1.4e-13 against 1.2e-12, Frobenius; the same with entries spread over 2^10).
#include <cuda_runtime.h>

#include <algorithm>

#include "colscale.cuh"
#include "common.cuh"
#include "oz.cuh"

namespace bem2d_gpu {
namespace {

using namespace tc;
using namespace oz;

constexpr int kOzBM = 64;       // complex rows per tile (128 real rows = MMA M)
constexpr int kOzBN = 16;       // complex columns per tile
constexpr int kOzS = 8;         // digits
constexpr int kOzK = 64;        // K of a slab: 4 MMA steps of 16
constexpr int kOzStages = 2;
constexpr int kOzThreads = 320;  // producer, MMA, 8 epilogue warps
constexpr int kOzEpi = 256;
constexpr int kOzABlk = 128 * 16 * 2;              // one digit, one K-step of A'
constexpr int kOzBBlk = 2 * kOzBN * 16 * 2;        // the same of B
constexpr int kOzAStep = kOzS * kOzABlk;           // 32 KB per K-step
constexpr int kOzBStep = kOzS * kOzBBlk;           // 8 KB per K-step
constexpr int kOzKSteps = kOzK / 16;
constexpr int kOzABytes = kOzKSteps * kOzAStep;    // 128 KB
constexpr int kOzBBytes = kOzKSteps * kOzBStep;    // 32 KB
constexpr int kOzBarOff = kOzABytes + kOzStages * kOzBBytes;  // 192 KB
constexpr int kOzSmem = kOzBarOff + 256;
constexpr unsigned kOzAcc = 2 * kOzBN * kOzS;      // 256 TMEM columns
// exponents that a row's or column's entries, or an entry's terms, may span
constexpr int kOzSpan = 10;

// ---- packing -------------------------------------------------------------------
// A row's or column's scale exponent er and whether its entries span more than
// kOzSpan (a zero entry does), from the largest and smallest exponents.
__device__ __forceinline__ int oz_scale_word(int er, int emin) {
  const bool wide = er > kZero && er < kNaN && emin < er - kOzSpan;
  return 2 * er + (wide ? 1 : 0);
}

// Packs both operands; CTAs [0, mt) take a row block of A each, the others four
// column blocks of B.
//   A (M x K) -> per row block of 64: [K-step][digit][128 x 16]; ea[i]: the row's
//   scale word.  Eight threads per complex row, thread c takes k = 8 c .. 8 c + 7.
//   B (K x N) -> per block of 16 columns: [K-step][digit][32 x 16], rows 0..15 re
//   and 16..31 im of the columns; eb[j].  Eight threads per column.
// part, np: the columns' exponents (colscale.cuh), added to inner index k in A
// and subtracted in B.
// xa[i], xb[j]: the 64 exponents with their shifts as 16-bit integers (kOzNone:
// zero), for oz_apart.
constexpr int kOzPackThreads = 512;
constexpr int kOzNone = -16000;  // two of them still fit 16 bits
struct OzPack {
  unsigned char *A, *B;  // digits
  int *ea, *eb;          // scale words
  uint4 *xa, *xb;        // exponents, kOzK of them per row / column
  int* part;             // kOzK * kColParts partial maxima
};

__device__ __forceinline__ int oz_field(double2 v, int p) {
  const int e = max(expo(v.x), expo(v.y));
  return is_zero(v) ? kOzNone : e == 2047 ? kNaN : e + p;
}

__device__ __forceinline__ uint4 oz_pack_fields(const int (&x)[8]) {
  unsigned w[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int a = min(max(x[2 * q], kOzNone), -kOzNone), b = min(max(x[2 * q + 1], kOzNone), -kOzNone);
    w[q] = ((unsigned)a & 0xffffu) | ((unsigned)b << 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ void oz_pack_a(const double2* __restrict__ A, long long lda, int M,
                                          int K, int ksteps, const int* pk, int (*red)[kOzBM],
                                          int (*low)[kOzBM], const OzPack& o) {
  const int il = threadIdx.x & 63, c = threadIdx.x >> 6, i = blockIdx.x * kOzBM + il;
  double2 v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = 8 * c + q;
    v[q] = i < M && k < K ? A[(size_t)k * lda + i] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  int emax = -10000, emin = 100000, x[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    x[q] = oz_field(v[q], pk[8 * c + q]);
    emax = max(emax, x[q]);
    if (8 * c + q < K) emin = min(emin, x[q]);
  }
  if (i < M) o.xa[(size_t)i * 8 + c] = oz_pack_fields(x);
  red[c][il] = emax;
  low[c][il] = emin;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    emax = max(emax, red[q][il]);
    emin = min(emin, low[q][il]);
  }
  const int er = scale_of(emax);
  if (c == 0 && i < M) o.ea[i] = oz_scale_word(er, emin);
  if (c >= 2 * ksteps) return;
  const bool use = er > kZero && er < kNaN;
  unsigned char* blk = o.A + ((size_t)blockIdx.x * ksteps + (c >> 1)) * kOzAStep;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    long long f[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      f[q] = fixed<kOzS>(!use ? 0.0 : h ? v[q].y : v[q].x, pk[8 * c + q], er);
    Digits<kOzS> d;
    digits<kOzS>(f, &d);
#pragma unroll
    for (int s = 0; s < kOzS; ++s)
      *reinterpret_cast<uint4*>(blk + s * kOzABlk + off(2 * il + h, c & 1)) =
          make_uint4(d.w[s][0], d.w[s][1], d.w[s][2], d.w[s][3]);
  }
}

__device__ __forceinline__ void oz_pack_b(const double2* __restrict__ B, long long ldb, int K,
                                          int N, int ksteps, int nt, const int* pk,
                                          const OzPack& o) {
  const int c = threadIdx.x & 7, jl = threadIdx.x >> 3, j = nt * kOzBN + jl;
  double2 v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = 8 * c + q;
    v[q] = (j < N && k < K) ? B[(size_t)j * ldb + k] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  int emax = -10000, emin = 100000, x[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    x[q] = oz_field(v[q], -pk[8 * c + q]);
    emax = max(emax, x[q]);
    if (8 * c + q < K) emin = min(emin, x[q]);
  }
  if (j < N) o.xb[(size_t)j * 8 + c] = oz_pack_fields(x);
#pragma unroll
  for (int l = 4; l > 0; l >>= 1) {
    emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, l));
    emin = min(emin, __shfl_xor_sync(0xffffffffu, emin, l));
  }
  const int er = scale_of(emax);
  if (c == 0 && j < N) o.eb[j] = oz_scale_word(er, emin);
  // blocks of 16 columns lie one after another: block nt + jl / 16, column jl % 16
  if (c >= 2 * ksteps || j >= (N + kOzBN - 1) / kOzBN * kOzBN) return;
  const bool use = er > kZero && er < kNaN;
  unsigned char* blk =
      o.B + ((size_t)(nt + (jl >> 4)) * ksteps + (c >> 1)) * kOzBStep;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    long long f[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      f[q] = fixed<kOzS>(!use ? 0.0 : h ? v[q].y : v[q].x, -pk[8 * c + q], er);
    Digits<kOzS> d;
    digits<kOzS>(f, &d);
#pragma unroll
    for (int s = 0; s < kOzS; ++s)
      *reinterpret_cast<uint4*>(blk + s * kOzBBlk + off(h * kOzBN + (jl & 15), c & 1)) =
          make_uint4(d.w[s][0], d.w[s][1], d.w[s][2], d.w[s][3]);
  }
}

__global__ void __launch_bounds__(kOzPackThreads)
oz_pack_kernel(const double2* __restrict__ A, long long lda, const double2* __restrict__ B,
               long long ldb, int M, int N, int K, int ksteps, int mt,
               int np, OzPack o) {
  __shared__ int pk[kOzK], red[8][kOzBM], low[8][kOzBM];
  if (threadIdx.x < kOzK) {
    const int e = (int)threadIdx.x < K ? col_expo_max(o.part, np, K, threadIdx.x) : 0;
    pk[threadIdx.x] = e > 0 ? 1023 - e : 0;
  }
  if ((int)blockIdx.x < mt)  // (the barrier that pk needs stands behind their loads)
    oz_pack_a(A, lda, M, K, ksteps, pk, red, low, o);
  else
    oz_pack_b(B, ldb, K, N, ksteps, 4 * (blockIdx.x - mt), pk, o);
}

// ---- the product -----------------------------------------------------------------
#define OZ_LD8(dst, addr)                                                                   \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"      \
               : "=r"(dst[0]), "=r"(dst[1]), "=r"(dst[2]), "=r"(dst[3]), "=r"(dst[4]),      \
                 "=r"(dst[5]), "=r"(dst[6]), "=r"(dst[7])                                   \
               : "r"(addr))

// (double)v for |v| < 2^51, one FP64 instruction
__device__ __forceinline__ double oz_to_double(long long v) {
  return __longlong_as_double(v + 0x4338000000000000ll) - 6755399441055744.0;
}

// A whole warp, lanes 2 r and 2 r + 1 on the real and imaginary part of a row's
// eight entries (a: the row of A, k-th entry at a + k lda; er: its scale
// exponent; c: the lane's component of column u at c + u cstep).  Of the lane's
// columns in `cols` (eb[u], xb[8 u], k-th entry at b + u ldb + k) those whose sum
// has all of its terms more than kOzSpan exponents below the scale exponents of
// its row and column are finished here in FP64 and returned.
//   The largest of 64 sums of two exponents is 32 add-maximum instructions on
// pairs of 16-bit integers.  A sum takes the 32 lanes two terms each: 13 FP64
// instructions of the warp; such entries come a row or two at a time, and the
// lanes on their own would spend 128 on them (graded square N = 2064, combined
// operator: solve 11.9 ms without these sums, 15.4 by lanes, 13.0 by warps).
__device__ __noinline__ unsigned oz_apart(unsigned cols, int er, const int* __restrict__ eb,
                                          const uint4* __restrict__ xa,
                                          const uint4* __restrict__ xb,
                                          const double2* __restrict__ a, long long lda,
                                          const double2* __restrict__ b, long long ldb, int K,
                                          double* c, long long cstep, int beta, double sign) {
  const int lane = threadIdx.x & 31;
  unsigned done = 0u;
  if (cols) {
    uint4 x[kOzK / 8];
#pragma unroll
    for (int q = 0; q < kOzK / 8; ++q) x[q] = __ldg(xa + q);
    for (unsigned rest = cols; rest; rest &= rest - 1) {
      const int u = __ffs(rest) - 1;
      unsigned z = 0x80008000u;
#pragma unroll
      for (int q = 0; q < kOzK / 8; ++q) {
        const uint4 y = __ldg(xb + 8 * u + q);
        z = __viaddmax_s16x2(x[q].x, y.x, z);
        z = __viaddmax_s16x2(x[q].y, y.y, z);
        z = __viaddmax_s16x2(x[q].z, y.z, z);
        z = __viaddmax_s16x2(x[q].w, y.w, z);
      }
      const int top = max((int)(short)(z & 0xffffu), (int)(short)(z >> 16));
      if (top < er + (eb[u] >> 1) - kOzSpan) done |= 1u << u;
    }
  }
  __syncwarp();
  for (unsigned any = __reduce_or_sync(0xffffffffu, done); any; any &= any - 1) {
    const int u = __ffs(any) - 1;
    const double2* bu = b + (size_t)u * ldb;
    for (unsigned rows = __ballot_sync(0xffffffffu, (done >> u) & 1u) & 0x55555555u; rows;
         rows &= rows - 1) {
      const int l = __ffs(rows) - 1;
      const double2* al = a + ((l >> 1) - (lane >> 1));
      double sr = 0.0, si = 0.0;
#pragma unroll
      for (int k = lane; k < kOzK; k += 32) {
        if (k >= K) break;
        const double2 x = al[(size_t)k * lda], y = bu[k];
        sr = fma(x.x, y.x, fma(-x.y, y.y, sr));
        si = fma(x.x, y.y, fma(x.y, y.x, si));
      }
      // real parts to lanes 0-15, imaginary ones to lanes 16-31
      const bool up = lane & 16;
      double s = (up ? si : sr) + __shfl_xor_sync(0xffffffffu, up ? sr : si, 16);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const double re = __shfl_sync(0xffffffffu, s, 0), im = __shfl_sync(0xffffffffu, s, 16);
      if ((lane & ~1) == l)
        c[u * cstep] = fma(sign, lane & 1 ? im : re, beta ? c[u * cstep] : 0.0);
    }
  }
  return done;
}

// C[M x N] = beta C + sign A B, beta 0 or 1, sign +-1, from the packed operands
// (A, M x K, and B, K x N, themselves only for oz_apart).  grid: min(tiles,
// SMs).
__global__ void __launch_bounds__(kOzThreads, 1)
oz_zgemm_kernel(double2* __restrict__ C, long long ldc, OzPack o, const double2* __restrict__ A,
                long long lda, const double2* __restrict__ B, long long ldb, int M, int N, int K,
                int ksteps, int ntiles, int tiles, int beta, double sign, int* status) {
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned long long* full = reinterpret_cast<unsigned long long*>(sm + kOzBarOff);
  unsigned long long* empty = full + kOzStages;
  unsigned long long* afull = empty + kOzStages;
  unsigned long long* aempty = afull + 1;
  unsigned long long* acc_full = aempty + 1;
  unsigned long long* acc_empty = acc_full + 2;
  unsigned long long* fin = acc_empty + 2;
  unsigned* tslot = reinterpret_cast<unsigned*>(fin + 1);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tslot + 1);
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  const int t0 = (int)((long long)tiles * blockIdx.x / gridDim.x);
  const int t1 = (int)((long long)tiles * (blockIdx.x + 1) / gridDim.x);
  if (w == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
        smem_u32(tslot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (t == 32) {
    for (int s = 0; s < kOzStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(afull, 1);
    mbar_init(aempty, 1);
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], kOzEpi);
    }
    mbar_init(fin, 1);
    asm volatile("fence.mbarrier_init.release.cluster;");
    *s_abort = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const unsigned tmem = *tslot;
  bool ok = true;
  const unsigned abytes = (unsigned)ksteps * kOzAStep, bbytes = (unsigned)ksteps * kOzBStep;
  if (w == 0) {
    if (lane == 0) {  // ---- producer
      int it = 0, mt_prev = -1, na = 0;
      for (int tile = t0; tile < t1 && ok; ++tile, ++it) {
        const int mt = tile / ntiles, nt = tile - mt * ntiles;
        if (mt != mt_prev) {
          if (na > 0 && !mbar_wait(aempty, (unsigned)(na - 1) & 1u, s_abort)) {
            ok = false;
            break;
          }
          mbar_expect_tx(afull, abytes);
          for (int k = 0; k < ksteps; ++k)
            bulk_copy(sm + k * kOzAStep, o.A + (size_t)mt * abytes + (size_t)k * kOzAStep,
                      kOzAStep, afull);
          ++na;
          mt_prev = mt;
        }
        const int s = it % kOzStages;
        if (!mbar_wait(&empty[s], ((unsigned)(it / kOzStages) & 1u) ^ 1u, s_abort)) {
          ok = false;
          break;
        }
        mbar_expect_tx(&full[s], bbytes);
        bulk_copy(sm + kOzABytes + s * kOzBBytes, o.B + (size_t)nt * bbytes, bbytes, &full[s]);
      }
      if (!ok) {
        *s_abort = 1;
        // let the copies in flight land before the CTA's shared memory goes
        if (na > 0) mbar_wait(afull, (unsigned)(na - 1) & 1u, nullptr);
        for (int q = it - 1; q >= 0 && q >= it - kOzStages; --q)
          mbar_wait(&full[q % kOzStages], (unsigned)(q / kOzStages) & 1u, nullptr);
      }
    }
  } else if (w == 1) {
    if (lane == 0) {  // ---- MMA issuer
      int j = 0, mt_prev = -1, na = 0;
      for (int tile = t0; tile < t1 && ok; ++tile, ++j) {
        const int mt = tile / ntiles;
        if (mt != mt_prev) {
          if (!mbar_wait(afull, (unsigned)na & 1u, s_abort)) {
            ok = false;
            break;
          }
          ++na;
          mt_prev = mt;
        }
        const int a = j & 1, s = j % kOzStages;
        if (!mbar_wait(&acc_empty[a], ((unsigned)(j >> 1) & 1u) ^ 1u, s_abort) ||
            !mbar_wait(&full[s], (unsigned)(j / kOzStages) & 1u, s_abort)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const unsigned d = tmem + (unsigned)a * kOzAcc;
        const unsigned sa = smem_u32(sm), sb = smem_u32(sm + kOzABytes + s * kOzBBytes);
        for (int k = 0; k < ksteps; ++k) {
#pragma unroll
          for (int i = 0; i < kOzS; ++i) {
            mma(d + 2 * kOzBN * i, sa + k * kOzAStep + i * kOzABlk, sb + k * kOzBStep,
                2 * kOzBN * (kOzS - i), (k == 0 && i == 0) ? 0u : 1u);
          }
        }
        mma_commit(&empty[s]);
        mma_commit(&acc_full[a]);
        if (tile + 1 < t1 && (tile + 1) / ntiles != mt) mma_commit(aempty);
      }
      if (!ok) *s_abort = 1;
      // every MMA issued has completed before the tensor memory is released
      mma_commit(fin);
      if (!mbar_wait(fin, 0u, nullptr)) ok = false;
    }
  } else {  // ---- epilogue, warps 2-9
    // two warps per TMEM lane quarter (warp w may access lanes 32 (w % 4) ..),
    // one for each half of the tile's 16 columns
    const int q = w & 3, part = (w - 2) >> 2;
    const int tl = q * 32 + lane, cc = tl & 1;  // real row tl = 2 i + cc
    double* Cf = reinterpret_cast<double*>(C);
    int j = 0;
    for (int tile = t0; tile < t1; ++tile, ++j) {
      const int mt = tile / ntiles, nt = tile - mt * ntiles;
      const int i = mt * kOzBM + (tl >> 1), n0 = nt * kOzBN + part * 8;
      const int ew = i < M ? __ldg(&o.ea[i]) : 2 * kZero, er = ew >> 1;
      const int nlim = i < M ? min(8, N - n0) : 0;
      double* pc = Cf + 2 * ((size_t)n0 * ldc + i) + cc;
      const long long cstep = 2 * ldc;
      double cv[8];
      int ec[8];
      unsigned apart = 0u;  // marked columns, if the row is marked
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        cv[u] = u < nlim && beta ? pc[u * cstep] : 0.0;
        const int cw = n0 + u < N ? __ldg(&o.eb[n0 + u]) : 2 * kZero;
        ec[u] = cw >> 1;
        apart |= (unsigned)(ew & cw & 1) << u;
      }
      if (__any_sync(0xffffffffu, apart != 0u))
        apart = oz_apart(apart, er, o.eb + n0, o.xa + (size_t)i * 8, o.xb + (size_t)n0 * 8, A + i,
                         lda, B + (size_t)n0 * ldb, ldb, K, pc, cstep, beta, sign);
      const int a = j & 1;
      // (all lanes of a warp give up together: the rest of the loop needs them all)
      if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[a], (unsigned)(j >> 1) & 1u, s_abort))) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const unsigned lanes = tmem + (unsigned)a * kOzAcc + ((unsigned)(q * 32) << 16) +
                             (unsigned)(part * 8);
      double hi[8];
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        long long d1[8], d2[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) d1[u] = d2[u] = 0;
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          unsigned x1[8], x2[8];
          OZ_LD8(x1, lanes + (4 * half + o) * 2 * kOzBN);
          OZ_LD8(x2, lanes + (4 * half + o) * 2 * kOzBN + kOzBN);
          asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            d1[u] = (d1[u] << 8) + __float2int_rn(__uint_as_float(x1[u]));
            d2[u] = (d2[u] << 8) + __float2int_rn(__uint_as_float(x2[u]));
          }
        }
        if (half == 1) {  // the accumulator has been read
          asm volatile("tcgen05.fence::before_thread_sync;");
          mbar_arrive(&acc_empty[a]);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const long long p2 = __shfl_xor_sync(0xffffffffu, d2[u], 1);
          const double v = oz_to_double(d1[u] + (cc ? p2 : -p2));
          hi[u] = half == 0 ? v : fma(v, 2.3283064365386963e-10, hi[u]);  // 2^-32
        }
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (u >= nlim) break;
        // digit orders 0-3 weigh 256^11 = 2^88, the operands 2^(er - 1085)
        const int e = er + ec[u] - 2 * 1085 + 88;
        double v;
        if (e > -1000 && e < 960) {
          v = fma(sign * __hiloint2double((e + 1023) << 20, 0), hi[u], cv[u]);
        } else if (e > 50000) {
          v = __longlong_as_double(0x7ff8000000000000ll);
        } else {
          v = e < -3000 ? cv[u] : cv[u] + sign * ldexp(hi[u], e);
        }
        if (!((apart >> u) & 1u)) pc[u * cstep] = v;
      }
    }
    if (!ok) *s_abort = 1;
  }
  if (!ok) atomicExch(status, 1);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (w == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}
#undef OZ_LD8

size_t up256(size_t v) { return (v + 255) / 256 * 256; }

}  // namespace

// The pack buffer's parts for an M x N product; returns its bytes.
static size_t oz_parts(void* pack, int M, int N, OzPack* o) {
  const size_t mt = (size_t)(M + kOzBM - 1) / kOzBM, nt = (size_t)(N + kOzBN - 1) / kOzBN;
  char* p = static_cast<char*>(pack);
  size_t at = 0;
  auto take = [&](size_t bytes) {
    char* r = p ? p + at : nullptr;
    at += up256(bytes);
    return r;
  };
  o->A = reinterpret_cast<unsigned char*>(take(mt * kOzABytes));
  o->B = reinterpret_cast<unsigned char*>(take(nt * kOzBBytes));
  o->ea = reinterpret_cast<int*>(take(sizeof(int) * (size_t)M));
  o->eb = reinterpret_cast<int*>(take(sizeof(int) * (size_t)N));
  o->xa = reinterpret_cast<uint4*>(take(sizeof(uint4) * 8 * (size_t)M));
  o->xb = reinterpret_cast<uint4*>(take(sizeof(uint4) * 8 * (size_t)N));
  o->part = reinterpret_cast<int*>(take(sizeof(int) * kOzK * kColParts));
  return at;
}

size_t oz_pack_bytes(int M, int N) {
  OzPack o;
  return oz_parts(nullptr, M, N, &o);
}

int launch_oz_zgemm(double2* C, long long ldc, const double2* A, long long lda, const double2* B,
                    long long ldb, int M, int N, int K, int beta, double sign, void* pack,
                    size_t pack_bytes, int* status, cudaStream_t s, long long* launches) {
  if (!opt_in_smem<oz_zgemm_kernel>(kOzSmem)) return BEM2D_ERR_CUDA;
  if (M <= 0 || N <= 0 || K <= 0) return BEM2D_OK;
  OzPack o;
  if (!pack || oz_parts(pack, M, N, &o) > pack_bytes) return BEM2D_ERR_ARG;
  const int mt = (M + kOzBM - 1) / kOzBM, nt = (N + kOzBN - 1) / kOzBN;
  const int grid = std::min(mt * nt, device_sms());
  for (int k = 0; k < K; k += kOzK) {
    const int kk = std::min(kOzK, K - k), ksteps = (kk + 15) / 16;
    const double2* a = A + (size_t)k * lda;
    const double2* b = B + k;
    const int np = launch_col_expo(a, lda, M, kk, o.part, s);
    oz_pack_kernel<<<mt + (nt + 3) / 4, kOzPackThreads, 0, s>>>(a, lda, b, ldb, M, N, kk, ksteps,
                                                               mt, np, o);
    oz_zgemm_kernel<<<grid, kOzThreads, kOzSmem, s>>>(C, ldc, o, a, lda, b, ldb, M, N, kk, ksteps,
                                                      nt, mt * nt, k == 0 ? beta : 1, sign, status);
    *launches += 3;
  }
  return cudaPeekAtLastError() == cudaSuccess ? BEM2D_OK : BEM2D_ERR_CUDA;
}

}  // namespace bem2d_gpu
