// C = op(A) B for the numerical range's block Lanczos on the tensor cores:
// exact products of 8-bit digits (see lu_oz.cu for the splitting), A n x n
// packed once for all products of a scan, or, where its digits (8 S n^2 bytes for
// A and A^H) do not fit, a block of rows at a time in every product; B n x m
// packed per product.
//
// S digits (template): 8 where the products were FP64 (complex128 Lanczos), 7
// where they were float-float (error about 2^-51 of row maximum x column
// maximum against 2^-46), 4 where they were FP32 (2^-26 against about 2^-24
// for n = 2048).  Kept are the digit pairs of order s + t < S: 36, 28, 10 MMAs'
// worth.  Orders 0-3 and 4-(S-1) are joined to two 64-bit integers per real
// number, which run over the whole of K, so FP64 is met once per result.
//
// A tile is 64 complex rows by 32 complex columns: 64 S columns of tensor
// memory, one set for S = 7 or 8, two for S = 4.  After 128 of K (at most 8
// pairs x 128 x 2^14 = 2^24, exact in FP32) the epilogue drains the set; K
// steps of 16 (6 S KB: S digits of A and of B) arrive by bulk copies in a
// ring.  Digit s of A meets digits 0 .. S - 1 - s of B, which lie one after
// another as rows of one operand, in one or two MMAs (N <= 256).
//
// Roles as in lu_oz.cu, with 16 epilogue warps (four per lane quarter, 8
// columns each); every wait is bounded.  Bound by the tensor pipe and by L2 (42
// KB a step for 900 clocks of MMAs at S = 7).
// Measured, n = 2048, 360 angles, the mixed scan's products: float-float 96 ->
// 8.6 ms (7 digits), FP32 39 -> 15.6 ms (4 digits) with packing; error against
// long double, matrices with a dominant diagonal: 8 digits 1e-16 (FP64 pipe
// 8e-16), 7 digits 6e-15 (float-float 2e-14), 4 digits 9e-8 (FP32 4e-7).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "cplx.cuh"
#include "dense.cuh"
#include "oz.cuh"

namespace bem2d_gpu {
namespace {

using namespace tc;
using namespace oz;

constexpr int kGM = 64, kGN = 32;       // complex rows, columns per tile
constexpr int kGChunk = 8;              // K steps of 16 between drains
constexpr int kGThreads = 576, kGEpi = 512;
constexpr int kGA = 128 * 16 * 2;       // bytes of one digit of A, one K step
constexpr int kGB = 2 * kGN * 16 * 2;   // the same of B

template <int S>
struct Cfg {
  static constexpr int kStep = S * (kGA + kGB);
  static constexpr int kStages = std::min(8, 212 * 1024 / kStep);
  static constexpr int kSets = 512 / (2 * kGN * S);
  static constexpr int kBarOff = kStages * kStep;
  static constexpr int kSmem = kBarOff + 256;
};

__device__ __forceinline__ double2 widen(double2 v) { return v; }
__device__ __forceinline__ double2 widen(float2 v) { return make_double2(v.x, v.y); }

// Largest exponent field of each of `rows` rows of K entries, entry (r, k) at
// src[r ld + k] (TRANS: a warp per row, 8 rows per CTA) or src[k ld + r] (a
// lane per row, the 8 warps share K, 32 rows per CTA).
template <typename T, bool TRANS>
__global__ void __launch_bounds__(256)
row_expo_kernel(const T* __restrict__ src, long long ld, int rows, int K, int* __restrict__ ex) {
  __shared__ int red[8][33];
  const int a = threadIdx.x & 31, b = threadIdx.x >> 5;
  const int r = TRANS ? blockIdx.x * 8 + b : blockIdx.x * 32 + a;
  int e = -10000;
  if (r < rows) {
#pragma unroll 4
    for (int k = TRANS ? a : b; k < K; k += TRANS ? 32 : 8) {
      const double2 v = widen(src[TRANS ? (size_t)r * ld + k : (size_t)k * ld + r]);
      const int f = max(expo(v.x), expo(v.y));
      if (!is_zero(v)) e = max(e, f == 2047 ? kNaN : f);
    }
  }
  if (TRANS) {
    e = __reduce_max_sync(0xffffffffu, e);
    if (a == 0 && r < rows) ex[r] = scale_of(e);
  } else {
    red[b][a] = e;
    __syncthreads();
    if (b == 0 && r < rows) {
      for (int q = 1; q < 8; ++q) e = max(e, red[q][a]);
      ex[r] = scale_of(e);
    }
  }
}

// Digits of one K step (blockIdx.y) of R rows (blockIdx.x): [row block][K
// step][digit][2 R x 16].  BSIDE: rows 0 .. R - 1 re, R .. 2 R - 1 im (B);
// else re and im of a row one after the other (A).  CONJ: conjugated.
template <int S, typename T, bool TRANS, bool CONJ, bool BSIDE, int R>
__global__ void __launch_bounds__(2 * R)
pack_digits_kernel(const T* __restrict__ src, long long ld, int rows, int K,
                   const int* __restrict__ ex, unsigned char* __restrict__ dst) {
  const int il = threadIdx.x % R, c = threadIdx.x / R;
  const int r = blockIdx.x * R + il, k0 = blockIdx.y * 16 + 8 * c;
  const int er = r < rows ? ex[r] : kZero;
  const bool use = er > kZero && er < kNaN;
  double2 v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = k0 + q;
    v[q] = make_double2(0.0, 0.0);
    if (use && k < K) v[q] = widen(TRANS ? src[(size_t)r * ld + k] : src[(size_t)k * ld + r]);
    if (CONJ) v[q].y = -v[q].y;
  }
  constexpr int blk = 2 * R * 16 * 2;
  unsigned char* base = dst + ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * (S * blk);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    long long f[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) f[q] = fixed<S>(h ? v[q].y : v[q].x, 0, er);
    Digits<S> o;
    digits<S>(f, &o);
#pragma unroll
    for (int s = 0; s < S; ++s)
      *reinterpret_cast<uint4*>(base + s * blk + off(BSIDE ? h * R + il : 2 * il + h, c)) =
          make_uint4(o.w[s][0], o.w[s][1], o.w[s][2], o.w[s][3]);
  }
}

#define OZ_LD4(dst, addr)                                                        \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"      \
               : "=r"(dst[0]), "=r"(dst[1]), "=r"(dst[2]), "=r"(dst[3])          \
               : "r"(addr))

// One set of accumulators, 4 columns (re and im parts) of orders O0 .. O1 - 1,
// added to acc as integers.
template <int O0, int O1>
__device__ __forceinline__ void drain4(unsigned lanes, int cc, long long* acc) {
  long long d1[4] = {0, 0, 0, 0}, d2[4] = {0, 0, 0, 0};
#pragma unroll
  for (int o = O0; o < O1; ++o) {
    unsigned x1[4], x2[4];
    OZ_LD4(x1, lanes + o * 2 * kGN);
    OZ_LD4(x2, lanes + o * 2 * kGN + kGN);
    asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      d1[u] = (d1[u] << 8) + __float2int_rn(__uint_as_float(x1[u]));
      d2[u] = (d2[u] << 8) + __float2int_rn(__uint_as_float(x2[u]));
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    // re: D1 - D2 of the im row, im: D1 + D2 of the re row
    const long long p2 = __shfl_xor_sync(0xffffffffu, d2[u], 1);
    acc[u] += d1[u] + (cc ? p2 : -p2);
  }
}

// C (or the partial sums of K split z at C + z cz) = A B from packed digits.
// Unit u: row block u / (ntiles nz), column block, K split.
template <int S, typename T>
__global__ void __launch_bounds__(kGThreads, 1)
oz_gemm_kernel(T* __restrict__ C, long long ldc, long long cz,
               const unsigned char* __restrict__ Apk, const unsigned char* __restrict__ Bpk,
               const int* __restrict__ ea, const int* __restrict__ eb, int M, int N, int ksteps,
               int ntiles, int nz, int units, int* status) {
  typedef typename CTraits<T>::R R;
  typedef Cfg<S> F;
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned long long* full = reinterpret_cast<unsigned long long*>(sm + F::kBarOff);
  unsigned long long* empty = full + F::kStages;
  unsigned long long* acc_full = empty + F::kStages;
  unsigned long long* acc_empty = acc_full + F::kSets;
  unsigned long long* fin = acc_empty + F::kSets;
  unsigned* tslot = reinterpret_cast<unsigned*>(fin + 1);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tslot + 1);
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  const int chunks = (ksteps + kGChunk - 1) / kGChunk;
  if (w == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
        smem_u32(tslot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (t == 32) {
    for (int s = 0; s < F::kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < F::kSets; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], kGEpi);
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
  if (w == 0) {
    if (lane == 0) {  // ---- producer
      int it = 0;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const int z = u % nz, nt = (u / nz) % ntiles, mt = u / (nz * ntiles);
        const int k0 = (int)((long long)chunks * z / nz) * kGChunk;
        const int k1 = min(ksteps, (int)((long long)chunks * (z + 1) / nz) * kGChunk);
        for (int k = k0; k < k1; ++k, ++it) {
          const int s = it % F::kStages;
          if (!mbar_wait(&empty[s], ((unsigned)(it / F::kStages) & 1u) ^ 1u, s_abort)) {
            ok = false;
            break;
          }
          unsigned char* st = sm + s * F::kStep;
          mbar_expect_tx(&full[s], F::kStep);
          bulk_copy(st, Apk + ((size_t)mt * ksteps + k) * (S * kGA), S * kGA, &full[s]);
          bulk_copy(st + S * kGA, Bpk + ((size_t)nt * ksteps + k) * (S * kGB), S * kGB, &full[s]);
        }
      }
      if (!ok) {
        *s_abort = 1;
        // let the copies in flight land before the CTA's shared memory goes
        for (int q = it - 1; q >= 0 && q >= it - F::kStages; --q)
          mbar_wait(&full[q % F::kStages], (unsigned)(q / F::kStages) & 1u, nullptr);
      }
    }
  } else if (w == 1) {
    if (lane == 0) {  // ---- MMA issuer
      int it = 0, j = 0;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const int z = u % nz;
        const int c0 = (int)((long long)chunks * z / nz), c1 = (int)((long long)chunks * (z + 1) / nz);
        for (int c = c0; c < c1 && ok; ++c, ++j) {
          const int a = j % F::kSets;
          if (!mbar_wait(&acc_empty[a], ((unsigned)(j / F::kSets) & 1u) ^ 1u, s_abort)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const unsigned d = tmem + (unsigned)a * (2 * kGN * S);
          const int ke = min(ksteps, (c + 1) * kGChunk);
          for (int k = c * kGChunk; k < ke; ++k, ++it) {
            const int s = it % F::kStages;
            if (!mbar_wait(&full[s], (unsigned)(it / F::kStages) & 1u, s_abort)) {
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const unsigned sa = smem_u32(sm + s * F::kStep), sb = sa + S * kGA;
            const bool first = k == c * kGChunk;
#pragma unroll
            for (int i = 0; i < S; ++i) {
              // digits 0-3 of B, then the rest: N <= 256
              mma(d + 2 * kGN * i, sa + i * kGA, sb, 2 * kGN * min(4, S - i),
                  first && i == 0 ? 0u : 1u);
              if (S - i > 4)
                mma(d + 2 * kGN * (i + 4), sa + i * kGA, sb + 4 * kGB, 2 * kGN * (S - i - 4),
                    first && i == 0 ? 0u : 1u);
            }
            mma_commit(&empty[s]);
          }
          if (ok) mma_commit(&acc_full[a]);
        }
      }
      if (!ok) *s_abort = 1;
      // every MMA issued has completed before the tensor memory is released
      mma_commit(fin);
      if (!mbar_wait(fin, 0u, nullptr)) ok = false;
    }
  } else {  // ---- epilogue, warps 2-17
    const int q = w & 3, part = (w - 2) >> 2;
    const int tl = q * 32 + lane, cc = tl & 1;  // real row tl = 2 i + cc
    int j = 0;
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const int z = u % nz, nt = (u / nz) % ntiles, mt = u / (nz * ntiles);
      const int c0 = (int)((long long)chunks * z / nz), c1 = (int)((long long)chunks * (z + 1) / nz);
      long long hi[8], lo[8];
#pragma unroll
      for (int v = 0; v < 8; ++v) hi[v] = lo[v] = 0;
      for (int c = c0; c < c1; ++c, ++j) {
        const int a = j % F::kSets;
        if (!mbar_wait(&acc_full[a], (unsigned)(j / F::kSets) & 1u, s_abort)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const unsigned lanes = tmem + (unsigned)a * (2 * kGN * S) + ((unsigned)(q * 32) << 16) +
                               (unsigned)(part * 8);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          drain4<0, 4>(lanes + 4 * g, cc, hi + 4 * g);
          if (S > 4) drain4<4, S>(lanes + 4 * g, cc, lo + 4 * g);
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        mbar_arrive(&acc_empty[a]);
      }
      if (!ok) break;
      const int i = mt * kGM + (tl >> 1), n0 = nt * kGN + part * 8;
      const int er = i < M ? ea[i] : kZero;
      R* pc = reinterpret_cast<R*>(C + (size_t)z * cz) + 2 * ((size_t)n0 * ldc + i) + cc;
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        if (i >= M || n0 + v >= N) break;
        // order 3 weighs 256^(2 S - 5), order S - 1 256^(4 - S) of that
        const double x = S > 4 ? fma((double)lo[v], 1.0 / (double)(1ll << (8 * (S - 4))),
                                     (double)hi[v])
                               : (double)hi[v];
        const int e = er + eb[n0 + v] - 2 * (1022 + 8 * S - 1) + 8 * (2 * S - 5);
        double y;
        if (e > -900 && e < 900)
          y = __hiloint2double((e + 1023) << 20, 0) * x;
        else if (e > 50000)
          y = __longlong_as_double(0x7ff8000000000000ll);
        else
          y = e < -3000 ? 0.0 : ldexp(x, e);
        pc[2 * (size_t)v * ldc] = (R)y;
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
#undef OZ_LD4

template <typename T>
__global__ void oz_reduce_kernel(const T* __restrict__ P, long long cz, int nz, int n, int m,
                                 T* __restrict__ C, long long ldc) {
  const int j = blockIdx.y, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || j >= m) return;
  T s = P[(size_t)j * n + i];
  for (int z = 1; z < nz; ++z) {
    const T v = P[(size_t)z * cz + (size_t)j * n + i];
    s.x += v.x;
    s.y += v.y;
  }
  C[(size_t)j * ldc + i] = s;
}

size_t up256(size_t v) { return (v + 255) / 256 * 256; }

// rows of A (first at A), or columns (HERM), n entries each
template <int S, typename T, bool HERM>
void pack_a(const T* A, long long lda, int rows, int n, int ks, unsigned char* dst, int* ex,
            cudaStream_t s) {
  row_expo_kernel<T, HERM>
      <<<HERM ? (rows + 7) / 8 : (rows + 31) / 32, 256, 0, s>>>(A, lda, rows, n, ex);
  pack_digits_kernel<S, T, HERM, HERM, false, kGM>
      <<<dim3((rows + kGM - 1) / kGM, ks), 2 * kGM, 0, s>>>(A, lda, rows, n, ex, dst);
}

// K splits of a rows x m product: about two units per SM, at least two chunks each
int splits(int rows, int n, int m) {
  const long long tiles = (long long)((rows + kGM - 1) / kGM) * ((m + kGN - 1) / kGN);
  const int chunks = (n + 16 * kGChunk - 1) / (16 * kGChunk);
  return (int)std::max<long long>(1, std::min<long long>((2 * device_sms() + tiles - 1) / tiles, chunks / 2));
}

}  // namespace

size_t oz_gemm_a_bytes(int rows, int n, int S) {
  const size_t ks = (size_t)(n + 15) / 16, mt = (size_t)(rows + kGM - 1) / kGM;
  return up256(mt * ks * S * kGA) + up256(sizeof(int) * (size_t)rows);
}

// the packed B, and the partial sums of a K split
static size_t b_bytes(int n, int m, int S) {
  const size_t ks = (size_t)(n + 15) / 16, nt = (size_t)(m + kGN - 1) / kGN;
  return up256(nt * ks * S * kGB) + up256(sizeof(int) * (size_t)m);
}
size_t oz_gemm_work_bytes(int rows, int n, int m, int S, size_t elem) {
  const int z = splits(rows, n, m);
  return b_bytes(n, m, S) + (z > 1 ? elem * (size_t)z * rows * m : 0);
}

template <typename T>
void launch_oz_pack(bool herm, int S, const T* A, long long lda, int r0, int rows, int n, void* dst,
                    cudaStream_t s) {
  const int ks = (n + 15) / 16;
  unsigned char* d = static_cast<unsigned char*>(dst);
  const size_t mt = (size_t)(rows + kGM - 1) / kGM;
  A += herm ? (size_t)r0 * lda : (size_t)r0;
  int* ex = reinterpret_cast<int*>(d + up256(mt * ks * S * kGA));
  auto pack = [&](auto digits) {
    constexpr int D = decltype(digits)::value;
    if (herm)
      pack_a<D, T, true>(A, lda, rows, n, ks, d, ex, s);
    else
      pack_a<D, T, false>(A, lda, rows, n, ks, d, ex, s);
  };
  if constexpr (sizeof(T) == sizeof(float2))
    pack(std::integral_constant<int, 4>());
  else if (S == 7)
    pack(std::integral_constant<int, 7>());
  else
    pack(std::integral_constant<int, 8>());
}

template <int S, typename T>
static int gemm_t(const void* Apk, int rows, int n, int m, T* C, long long ldc, void* work,
                  int* status, cudaStream_t s) {
  if (!opt_in_smem<oz_gemm_kernel<S, T>>(Cfg<S>::kSmem)) return BEM2D_ERR_CUDA;
  const int ks = (n + 15) / 16, mt = (rows + kGM - 1) / kGM, nt = (m + kGN - 1) / kGN,
            nz = splits(rows, n, m);
  const unsigned char* ap = static_cast<const unsigned char*>(Apk);
  const int* ea = reinterpret_cast<const int*>(ap + up256((size_t)mt * ks * S * kGA));
  unsigned char* bp = static_cast<unsigned char*>(work);
  int* eb = reinterpret_cast<int*>(bp + up256((size_t)nt * ks * S * kGB));
  T* P = reinterpret_cast<T*>(bp + b_bytes(n, m, S));
  const int units = mt * nt * nz;
  oz_gemm_kernel<S, T><<<std::min(units, device_sms()), kGThreads, Cfg<S>::kSmem, s>>>(
      nz > 1 ? P : C, nz > 1 ? rows : ldc, (long long)rows * m, ap, bp, ea, eb, rows, m, ks, nt, nz,
      units, status);
  if (nz > 1)
    oz_reduce_kernel<T><<<dim3((rows + 255) / 256, m), 256, 0, s>>>(P, (long long)rows * m, nz, rows,
                                                                    m, C, ldc);
  return cudaPeekAtLastError() == cudaSuccess ? BEM2D_OK : BEM2D_ERR_CUDA;
}

template <int S, typename T>
static void pack_b(const T* B, long long ldb, int n, int m, void* work, cudaStream_t s) {
  const int ks = (n + 15) / 16, nt = (m + kGN - 1) / kGN;
  unsigned char* bp = static_cast<unsigned char*>(work);
  int* eb = reinterpret_cast<int*>(bp + up256((size_t)nt * ks * S * kGB));
  row_expo_kernel<T, true><<<(m + 7) / 8, 256, 0, s>>>(B, ldb, m, n, eb);
  pack_digits_kernel<S, T, true, false, true, kGN>
      <<<dim3(nt, ks), 2 * kGN, 0, s>>>(B, ldb, m, n, eb, bp);
}

template <typename T>
int launch_oz_gemm_pair(int S, const T* A, long long lda, int rows, void* Apk, int n, const T* B,
                        long long ldb, int m, T* C1, T* C2, long long ldc, void* work, int* status,
                        cudaStream_t s, long long* launches) {
  auto both = [&](auto digits) {
    constexpr int D = decltype(digits)::value;
    pack_b<D, T>(B, ldb, n, m, work, s);
    *launches += 2;
    for (int r0 = 0; r0 < n; r0 += rows) {
      const int r = std::min(rows, n - r0);
      for (int herm = 0; herm < 2; ++herm) {
        char* pk = static_cast<char*>(Apk) + (rows >= n ? herm * oz_gemm_a_bytes(n, n, D) : 0);
        if (rows < n) {
          launch_oz_pack<T>(herm != 0, D, A, lda, r0, r, n, pk, s);
          *launches += 2;
        }
        const int rc = gemm_t<D, T>(pk, r, n, m, (herm ? C2 : C1) + r0, ldc, work, status, s);
        if (rc) return rc;
        *launches += splits(r, n, m) > 1 ? 2 : 1;
      }
    }
    return (int)BEM2D_OK;
  };
  if constexpr (sizeof(T) == sizeof(float2))
    return both(std::integral_constant<int, 4>());
  else
    return S == 7 ? both(std::integral_constant<int, 7>()) : both(std::integral_constant<int, 8>());
}

#define BEM2D_OZ_INST(T)                                                                         \
  template void launch_oz_pack<T>(bool, int, const T*, long long, int, int, int, void*,          \
                                  cudaStream_t);                                                 \
  template int launch_oz_gemm_pair<T>(int, const T*, long long, int, void*, int, const T*,       \
                                      long long, int, T*, T*, long long, void*, int*,            \
                                      cudaStream_t, long long*);
BEM2D_OZ_INST(double2)
BEM2D_OZ_INST(float2)
#undef BEM2D_OZ_INST

}  // namespace bem2d_gpu
