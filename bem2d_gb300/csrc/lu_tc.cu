// Trailing update of the complex64 LU on the 5th-generation tensor cores:
// C -= A B (complex64, column-major, arbitrary leading dimensions), as
// tcgen05.mma kind::f16 with FP32 accumulators in tensor memory.
//
// Complex arithmetic as one real product.  The complex M x K operand A is
// read as a real (2M) x K matrix A' whose rows 2i and 2i + 1 hold re and im
// of row i (that is how complex column-major data lies in memory).  The
// complex K x N operand B becomes the real N' x K operand [B_r; B_i] with
// N' = 2N (the real parts of the tile's columns, then the imaginary parts),
// so one MMA of N = 256 gives D = A' [B_r B_i] with
//   D1 = A' B_r (columns 0..127),  D2 = A' B_i (columns 128..255),
//   re C_i = D1[2i] - D2[2i+1],   im C_i = D2[2i] + D1[2i+1].
// A tile is 64 complex rows (128 real rows = the MMA's M) by 128 complex
// columns: 256 tensor-memory columns per accumulator.
//
// Accuracy: row i of A and column j of B are scaled by powers of two so that
// their largest entry lies in [2^14, 2^15), and every scaled FP32 entry x is
// split into hi = x rounded to f16 and lo = x - hi rounded to f16 (11 bits
// each); a product is accumulated as hi*hi + hi*lo + lo*hi.  That keeps 22 bits
// of every entry within 2^-16 of its row's (column's) largest and an absolute
// error of 2^-40 of the largest below - no less than the 3xTF32 split it
// replaces (TF32 has the same 10 mantissa bits), at twice its rate: f16
// operands are half the bytes and an MMA covers 16 of K instead of 8.  With
// passes = 1 only hi*hi is issued: a third of the tensor work, products to
// about 2^-11 relative, for systems whose condition number the refinement
// tolerates at that precision.  Error against complex128 over (|A| |B|)_ij,
// rank-256 update of random 3000 x 3000: 7.8e-8 rms, 3.7e-7 at most (3xTF32:
// 1.5e-7, 7.1e-7); smaller too for rows, columns or entries over many decades.
// All updates of the L-shape's LU, N = 16384: 51.4 -> 30.1 ms, their packing
// (one kernel instead of two) 8.7 -> 3.9 ms; norm and condition number's, N =
// 8192: 19 -> 12.4 ms.
//   Inner index k is scaled first, by the largest exponent of A(:, k) and its
// inverse on B(k, :) (colscale.cuh), so that powers of two on the rows and
// columns of the matrix being factored do not meet in a column of U: without it
// one row 2^40 heavier than the others pushed the rest of its 64-row block of U
// below the split (refinement 3 -> 6 steps and 1e-8 in the solution; with 2^60
// no convergence at n = 1500).  The panels leave these exponents behind, the last
// step of an outer block forms those of its rank-256 update beside its own work:
// kite N = 2048 5.02 -> 5.06 ms, L-shape N = 16384 128.4 -> 129.1 ms.
//
// Operands are packed once per update (pack_kernel): scaled, split into hi/lo
// and laid out, per tile and per chunk of 32 along K, exactly as
// the MMA reads them from shared memory - the K-major, non-swizzled
// canonical layout (core matrices of 8 rows x 16 bytes, 128 bytes from one
// core matrix to the next along K, 512 bytes from one group of 8 rows to the
// next).  A chunk is then one contiguous block per operand: 16 KB of A'
// (hi, lo) and 32 KB of B (hi, lo).  The inverse scales (a byte each, the
// exponent field) are applied in the epilogue.
//
// The update kernel is persistent (one CTA per SM, tiles in a static
// round-robin) and warp-specialised:
//   warp 0      producer: two bulk copies (cp.async.bulk, completion counted
//               in bytes on the stage's `full` mbarrier) per chunk into a
//               ring of four 48 KB shared-memory stages;
//   warp 1      MMA issuer: six MMAs per chunk (two K-steps of 16, three products);
//               tcgen05.commit frees the stage (`empty`) once its MMAs have
//               read it, and marks the tile's accumulator complete (`acc_full`);
//   warps 2-17  epilogue: tcgen05.ld of the accumulator (warp w reads TMEM
//               lanes 32 (w % 4) ..., four warps per lane quarter, one per
//               quarter of the columns), rows 2i / 2i + 1 combined with one
//               shuffle; each thread loads its 32 C values before it waits
//               for the tile's accumulator (the loads overlap the tile's
//               MMAs; the next tile's C is prefetched into L2 meanwhile), C
//               is written with coalesced 128-byte accesses; then `acc_empty`.
// The two accumulators alternate between tiles (512 TMEM columns), so the
// epilogue of one tile overlaps the MMAs of the next.  Every wait is bounded
// (2 s of device time): on timeout the status flag is set, every role stops,
// the producer waits (bounded) for its copies in flight and the MMA thread
// for its MMAs, and the tensor memory is released before the kernel returns.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "colscale.cuh"
#include "common.cuh"
#include "cplx.cuh"
#include "tc.cuh"

namespace bem2d_gpu {
namespace {

using namespace tc;

constexpr int kTcBM = 64;    // complex rows per tile (128 real rows = MMA M)
constexpr int kTcBN = 128;   // complex columns per tile (MMA N = 256: re, im)
constexpr int kTcBK = 32;    // K per chunk (two MMAs of K = 16)
constexpr int kTcStages = 4;
constexpr int kTcThreads = 576;  // producer warp, MMA warp, 16 epilogue warps
constexpr int kTcEpiThreads = 512;
constexpr int kCoreBytes = 128;                   // 8 rows x 16 bytes
constexpr int kTcSBO = (kTcBK / 8) * kCoreBytes;  // 512
constexpr int kTcApart = 2 * kTcBM * kTcBK * 2;   // 8 KB: 128 real rows x 32
constexpr int kTcBpart = 2 * kTcBN * kTcBK * 2;   // 16 KB: 256 rows x 32
constexpr int kTcChunkA = 2 * kTcApart;           // hi, lo
constexpr int kTcChunkB = 2 * kTcBpart;           // hi, lo
constexpr int kTcStage = kTcChunkA + kTcChunkB;   // 48 KB
constexpr int kTcBarOff = kTcStages * kTcStage;   // 192 KB
constexpr int kTcSmem = kTcBarOff + 256;
constexpr unsigned kTcAcc = 2 * kTcBN;            // TMEM columns per accumulator

// tcgen05 shared-memory matrix descriptor: K-major, no swizzle
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr) {
  return (unsigned long long)((addr & 0x3FFFF) >> 4) |
         ((unsigned long long)(kCoreBytes >> 4) << 16) |
         ((unsigned long long)(kTcSBO >> 4) << 32) | (1ull << 46);
}
// byte offset of (row r, 8 consecutive k from 8 o) inside one packed chunk
__device__ __forceinline__ int kmajor_off(int r, int o) {
  return (r >> 3) * kTcSBO + o * kCoreBytes + (r & 7) * 16;
}

__device__ __forceinline__ void mma_f16(unsigned d, unsigned a, unsigned b, unsigned idesc,
                                        unsigned acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(smem_desc(a)), "l"(smem_desc(b)), "r"(idesc), "r"(acc));
}
#define TC_LD8(dst, addr)                                                                 \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"   \
               : "=r"(dst[0]), "=r"(dst[1]), "=r"(dst[2]), "=r"(dst[3]), "=r"(dst[4]),    \
                 "=r"(dst[5]), "=r"(dst[6]), "=r"(dst[7])                                 \
               : "r"(addr))

// ---- packing ---------------------------------------------------------------
// Exponent field of the power of two that brings a largest absolute value of m
// to [2^14, 2^15), within what a float holds on both sides (m = 0, infinite or
// below 2^-110 included), and of its inverse.
__device__ __forceinline__ int scale_exp(float m) {
  const int e = min(max((__float_as_int(m) >> 23) & 0xff, 17), 254);
  return 254 + 14 - e;
}
__device__ __forceinline__ float exp_float(int e) { return __int_as_float(e << 23); }

// 2^t of an inner index for A, 2^-t for B from the exponent of A's column (see
// colscale.cuh); t clamped to what the products of finite entries leave room for
__device__ __forceinline__ float inner_scale(int e, bool is_a) {
  const int t = e > 0 ? min(max(127 - e, -60), 100) : 0;
  return exp_float(127 + (is_a ? t : -t));
}

// 8 values times sc, split into f16 hi and lo, 16 bytes each
__device__ __forceinline__ void split8(const float (&v)[8], float sc, int passes,
                                       unsigned char* hi, unsigned char* lo) {
  unsigned h[4], l[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float x = v[2 * j] * sc, y = v[2 * j + 1] * sc;
    const __half2 p = __floats2half2_rn(x, y);
    const float2 f = __half22float2(p);
    const __half2 r = __floats2half2_rn(x - f.x, y - f.y);
    h[j] = *reinterpret_cast<const unsigned*>(&p);
    l[j] = *reinterpret_cast<const unsigned*>(&r);
  }
  *reinterpret_cast<uint4*>(hi) = make_uint4(h[0], h[1], h[2], h[3]);
  if (passes > 1) *reinterpret_cast<uint4*>(lo) = make_uint4(l[0], l[1], l[2], l[3]);
}

// Rows / columns r of an operand with their k octets, as the MMA reads them:
// A (M x K complex) -> Apk[mt][kc] = {hi, lo} chunks of kTcApart bytes each;
// B (K x N complex) -> Bpk[nt][kc] = {hi, lo} chunks of kTcBpart bytes, each
// with rows 0..127 = re and rows 128..255 = im of the tile's 128 columns;
// isa, isb: exponent fields of the inverse scales.
// part, np: the exponents of A's columns.
struct TcPack {
  unsigned char *A, *B, *isa, *isb;
  const int* part;
  int nkc, passes, np;
};
template <bool IS_A>
__device__ __forceinline__ void pack_octet(const TcPack& pk, int r, int o, const float (&re)[8],
                                           const float (&im)[8], float sc) {
  constexpr int T = IS_A ? kTcBM : kTcBN, part = IS_A ? kTcApart : kTcBpart;
  const int tl = r / T, il = r - tl * T;
  unsigned char* c = (IS_A ? pk.A : pk.B) + ((size_t)tl * pk.nkc + (o >> 2)) * (2 * part);
  unsigned char* cre = c + kmajor_off(IS_A ? 2 * il : il, o & 3);
  unsigned char* cim = c + kmajor_off(IS_A ? 2 * il + 1 : kTcBN + il, o & 3);
  split8(re, sc, pk.passes, cre, cre + part);
  split8(im, sc, pk.passes, cim, cim + part);
}
// 32 rows of A from row 32 blk (a warp 32 rows x 8 k at a time) or 8 columns of
// B from column 8 blk (a warp 8 columns x 32 k).  Each entry is read twice, for
// the largest and for the split (the second time from L1).  256 threads; fk:
// 32 nkc floats of shared memory for the inner indices' scales.
template <bool IS_A>
__device__ __forceinline__ void pack_block(const float2* __restrict__ P, long long ld, int lim,
                                           int K, int blk, const TcPack& pk, float (*red)[32],
                                           float* fk) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // row of A, or column of B; first octet of k and octet step of this thread
  const int r = IS_A ? blk * 32 + lane : blk * 8 + (lane & 7);
  const int o0 = IS_A ? w : 4 * w + (lane >> 3), os = IS_A ? 8 : 32;
  const bool ok = r < lim;
  const float2* src = IS_A ? P + r : P + (size_t)r * ld;
  const long long st = IS_A ? ld : 1;
  for (int k = threadIdx.x; k < pk.nkc * kTcBK; k += 256)
    fk[k] = inner_scale(k < K ? col_expo_max(pk.part, pk.np, K, k) : 0, IS_A);
  __syncthreads();
  float mx = 0.f;
  for (int o = o0; o < 4 * pk.nkc; o += os) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = 8 * o + j;
      const float2 v = ok && k < K ? src[k * st] : make_float2(0.f, 0.f);
      mx = fmaxf(mx, fmaxf(fabsf(v.x), fabsf(v.y)) * fk[k]);
    }
  }
  if (!IS_A) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
  }
  red[w][lane] = mx;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j) mx = fmaxf(mx, red[j][lane]);
  const int se = scale_exp(mx);
  const float sc = exp_float(se);
  if (w == 0 && (IS_A || lane < 8)) (IS_A ? pk.isa : pk.isb)[r] = (unsigned char)(254 - se);
  for (int o = o0; o < 4 * pk.nkc; o += os) {
    float re[8], im[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = 8 * o + j;
      const float2 v = ok && k < K ? src[k * st] : make_float2(0.f, 0.f);
      re[j] = v.x * fk[k];
      im[j] = v.y * fk[k];
    }
    pack_octet<IS_A>(pk, r, o, re, im, sc);
  }
}

// One launch for both operands: the first ab CTAs take A, the others B.
__global__ void __launch_bounds__(256)
pack_kernel(const float2* __restrict__ A, long long lda, const float2* __restrict__ B,
            long long ldb, int M, int N, int K, int ab, TcPack pk) {
  extern __shared__ float fk[];
  __shared__ float red[8][32];
  if ((int)blockIdx.x < ab)
    pack_block<true>(A, lda, M, K, blockIdx.x, pk, red, fk);
  else
    pack_block<false>(B, ldb, N, K, blockIdx.x - ab, pk, red, fk);
}

// ---- between a panel and its update ----------------------------------------
// Row swaps of the panel at k0 (ipiv, null: none) on the columns [cl, k0) and
// [rs, cr), U12 = L11^{-1} A12 on the latter and (packing) the operands of A22 -=
// L21 U12 for the M rows below the panel, in one launch.  CTAs:
//   [0, nright)  32 columns right of the panel each: swaps, U12, its pack;
//   then nleft   32 columns left of it: swaps;
//   then nexpo   a part of a column's exponents each, of the block that the
//                update after this launch takes (ex);
//   then         32 rows of L21 each: their pack.
// The swaps are applied as the permutation they amount to: 128 threads each
// follow one position (the panel's 64 rows; the other row of each swap) back
// through them, then every column is gathered and written once.  U12: warp w
// holds rows 8w .. 8w + 7 of its lane's column; block b of 8 rows is solved by
// warp b, then the warps below subtract L[w, b] x_b.
// Bound by latency (launch, loads, eight steps of the solve): 10.5 us per panel
// of the LU at N = 2048.  As three kernels - swaps by a thread per column in 64
// dependent steps, solve, packing - it took 21 us and two launches more.
constexpr int kStepCols = 32;
constexpr int kNBs = 64;  // panel width
constexpr size_t kStepSmem = sizeof(float2) * (kNBs * kNBs + kNBs * kStepCols);

__global__ void __launch_bounds__(256)
tc_step_kernel(float2* __restrict__ A, long long lda, int M, int k0, int nb, int cl, int rs,
               int cr, const int* __restrict__ ipiv, int nright, int nleft, int nexpo, bool packing,
               TcPack pk, TcExpo ex) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_ip[kNBs], s_src[kNBs], s_pos[kNBs], s_from[kNBs];
  __shared__ float red[8][32], fk[kNBs];
  __shared__ int s_le[4][kNBs];
  const int t = threadIdx.x, c = t & 31, w = t >> 5;
  const int b = blockIdx.x;
  if (b >= nright + nleft) {
    const int q = b - nright - nleft;
    if (q < nexpo)
      col_expo_part(ex.A + (size_t)(q % ex.K) * lda, ex.M, q / ex.K, ex.np, &ex.part[q]);
    else
      pack_block<true>(A + (size_t)k0 * lda + k0 + nb, lda, M, nb, q - nexpo, pk, red, fk);
    return;
  }
  const bool right = b < nright;
  const int cb = right ? rs + kStepCols * b : cl + kStepCols * (b - nright);
  const int nc = min(kStepCols, (right ? cr : k0) - cb);
  float2* L = reinterpret_cast<float2*>(smem);  // [kNBs][kNBs] column-major
  float2* X = L + kNBs * kNBs;                  // [kNBs][kStepCols]
  if (t < kNBs) {
    s_ip[t] = ipiv && t < nb ? ipiv[k0 + t] : k0 + t;
    s_src[t] = k0 + t;
    s_pos[t] = -1;
  }
  // inner index t & 63's exponent: a quarter of the parts each, used when packing
  int le = 0;
  if (right && packing) {
#pragma unroll
    for (int p = 0; p < kColParts / 4; ++p)
      if ((t >> 6) + 4 * p < pk.np) le = max(le, __ldg(&pk.part[((t >> 6) + 4 * p) * kNBs + (t & 63)]));
  }
  if (right) {  // nb = 64
#pragma unroll
    for (int v = 0; v < kNBs * kNBs / 256; ++v) {
      const int s = (v * 256 + t) >> 6, r = t & 63;
      L[s * kNBs + r] = A[(size_t)(k0 + s) * lda + k0 + r];
    }
  }
  __syncthreads();
  if (ipiv && t < 2 * kNBs) {  // the row that ends at position x
    const int x0 = t < kNBs ? k0 + t : s_ip[t - kNBs];
    int x = x0;
    for (int s = kNBs - 1; s >= 0; --s) {
      const int p = s_ip[s], q = k0 + s;
      x = x == q ? p : x == p ? q : x;
    }
    if (t < kNBs) {
      s_src[t] = x;
    } else {
      s_pos[t - kNBs] = x0 >= k0 + nb && x0 != x ? x0 : -1;
      s_from[t - kNBs] = x;
    }
  }
  __syncthreads();
  // gather: thread row t & 63, columns t >> 6, + 4, ..; the displaced rows wait
  // in registers until every column has been read
  const int r = t & 63, pos = s_pos[r], from = s_from[r], src = s_src[r];
  float2 top[kStepCols / 4], out[kStepCols / 4];
#pragma unroll
  for (int i = 0; i < kStepCols / 4; ++i) {
    const int cc = (t >> 6) + 4 * i;
    const float2* col = A + (size_t)(cb + cc) * lda;
    top[i] = cc < nc && r < nb ? col[src] : make_float2(0.f, 0.f);
    if (cc < nc && pos >= 0) out[i] = col[from];
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kStepCols / 4; ++i) {
    const int cc = (t >> 6) + 4 * i;
    float2* col = A + (size_t)(cb + cc) * lda;
    if (cc < nc && pos >= 0) col[pos] = out[i];
    if (right)
      X[r * kStepCols + cc] = top[i];
    else if (cc < nc && r < nb && src != k0 + r)
      col[k0 + r] = top[i];
  }
  if (!right) return;
  __syncthreads();
  float2 x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = X[(8 * w + i) * kStepCols + c];
  for (int q = 0; q < 8; ++q) {
    if (w == q) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = i + 1; j < 8; ++j) x[j] = cfms(x[j], L[(8 * q + i) * kNBs + 8 * q + j], x[i]);
#pragma unroll
      for (int i = 0; i < 8; ++i) X[(8 * q + i) * kStepCols + c] = x[i];
    }
    __syncthreads();
    if (w > q) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float2 xb = X[(8 * q + j) * kStepCols + c];
        const float4* l4 = reinterpret_cast<const float4*>(L + (8 * q + j) * kNBs + 8 * w);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 l = l4[i];
          x[2 * i] = cfms(x[2 * i], make_float2(l.x, l.y), xb);
          x[2 * i + 1] = cfms(x[2 * i + 1], make_float2(l.z, l.w), xb);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kStepCols / 4; ++i) {
    const int cc = (t >> 6) + 4 * i;
    if (cc < nc) A[(size_t)(cb + cc) * lda + k0 + r] = X[r * kStepCols + cc];
  }
  if (!packing) return;
  s_le[t >> 6][t & 63] = le;
  __syncthreads();
  if (t < kNBs)
    fk[t] = inner_scale(max(max(s_le[0][t], s_le[1][t]), max(s_le[2][t], s_le[3][t])), false);
  __syncthreads();
  // pack: thread (column c, octet w)
  float re[8], im[8], mx = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 v = X[(8 * w + j) * kStepCols + c];
    re[j] = v.x * fk[8 * w + j];
    im[j] = v.y * fk[8 * w + j];
    mx = fmaxf(mx, fmaxf(fabsf(re[j]), fabsf(im[j])));
  }
  red[w][c] = mx;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 8; ++j) mx = fmaxf(mx, red[j][c]);
  const int se = scale_exp(mx), col = kStepCols * b + c;
  if (w == 0) pk.isb[col] = (unsigned char)(254 - se);
  pack_octet<false>(pk, col, w, re, im, exp_float(se));
}

// ---- the update --------------------------------------------------------------
// grid: min(tiles, SMs) persistent CTAs, kTcThreads threads, kTcSmem bytes
// of shared memory (one CTA per SM).  Tile t: mt = t % mtiles, nt = t / mtiles.
__global__ void __launch_bounds__(kTcThreads, 1)
tc_cgemm_sub_kernel(float2* __restrict__ C, long long ldc, const unsigned char* __restrict__ Apk,
                    const unsigned char* __restrict__ Bpk, const unsigned char* __restrict__ isa,
                    const unsigned char* __restrict__ isb, int M, int N, int nkc, int mtiles,
                    int ntiles, int passes, int* status) {
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned long long* full = reinterpret_cast<unsigned long long*>(sm + kTcBarOff);
  unsigned long long* empty = full + kTcStages;
  unsigned long long* acc_full = empty + kTcStages;
  unsigned long long* acc_empty = acc_full + 2;
  unsigned long long* fin = acc_empty + 2;
  unsigned* tslot = reinterpret_cast<unsigned*>(fin + 1);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tslot + 1);
  const int t = threadIdx.x, w = t >> 5, lane = t & 31;
  const int ntl = mtiles * ntiles;
  if (w == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
        smem_u32(tslot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (t == 32) {
    for (int s = 0; s < kTcStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], kTcEpiThreads);
    }
    mbar_init(fin, 1);
    asm volatile("fence.mbarrier_init.release.cluster;");
    *s_abort = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const unsigned tmem = *tslot;
  // kind::f16: D f32 (bits 4-5 = 1), A and B f16 (0), both K-major, N >> 3 at
  // bit 17, M >> 4 at bit 24
  const unsigned idesc = (1u << 4) | ((kTcAcc >> 3) << 17) | ((128u >> 4) << 24);
  bool ok = true;
  if (w == 0) {
    if (lane == 0) {  // ---- producer
      int it = 0;
      for (int tile = blockIdx.x; tile < ntl && ok; tile += gridDim.x) {
        const int mt = tile % mtiles, nt = tile / mtiles;
        const unsigned char* asrc = Apk + (size_t)mt * nkc * kTcChunkA;
        const unsigned char* bsrc = Bpk + (size_t)nt * nkc * kTcChunkB;
        for (int c = 0; c < nkc; ++c, ++it) {
          const int s = it % kTcStages;
          const unsigned ph = (unsigned)(it / kTcStages) & 1u;
          if (!mbar_wait(&empty[s], ph ^ 1u, s_abort)) {
            ok = false;
            break;
          }
          unsigned char* st = sm + s * kTcStage;
          // one product: the hi halves only (the first half of each packed chunk)
          const unsigned abytes = passes > 1 ? kTcChunkA : kTcApart;
          const unsigned bbytes = passes > 1 ? kTcChunkB : kTcBpart;
          mbar_expect_tx(&full[s], abytes + bbytes);
          bulk_copy(st, asrc + (size_t)c * kTcChunkA, abytes, &full[s]);
          bulk_copy(st + kTcChunkA, bsrc + (size_t)c * kTcChunkB, bbytes, &full[s]);
        }
      }
      if (!ok) {
        *s_abort = 1;
        // let the copies in flight land before the CTA's shared memory goes
        for (int q = it - 1; q >= 0 && q >= it - kTcStages; --q)
          mbar_wait(&full[q % kTcStages], (unsigned)(q / kTcStages) & 1u, nullptr);
      }
    }
  } else if (w == 1) {
    if (lane == 0) {  // ---- MMA issuer
      int it = 0, j = 0;
      for (int tile = blockIdx.x; tile < ntl && ok; tile += gridDim.x, ++j) {
        const int a = j & 1;
        const unsigned aph = (unsigned)(j >> 1) & 1u;
        if (!mbar_wait(&acc_empty[a], aph ^ 1u, s_abort)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        const unsigned d = tmem + (unsigned)a * kTcAcc;
        for (int c = 0; c < nkc; ++c, ++it) {
          const int s = it % kTcStages;
          const unsigned ph = (unsigned)(it / kTcStages) & 1u;
          if (!mbar_wait(&full[s], ph, s_abort)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const unsigned base = smem_u32(sm + s * kTcStage);
          const unsigned ah = base, al = base + kTcApart;
          const unsigned bh = base + kTcChunkA, bl = bh + kTcBpart;
#pragma unroll
          for (int ks = 0; ks < kTcBK / 16; ++ks) {
            const unsigned o = 256u * ks;  // K = 16 f16 = two core matrices
            mma_f16(d, ah + o, bh + o, idesc, (c == 0 && ks == 0) ? 0u : 1u);
            if (passes > 1) {
              mma_f16(d, ah + o, bl + o, idesc, 1u);
              mma_f16(d, al + o, bh + o, idesc, 1u);
            }
          }
          mma_commit(&empty[s]);  // the stage may be refilled once these MMAs read it
        }
        if (!ok) break;
        mma_commit(&acc_full[a]);
      }
      if (!ok) *s_abort = 1;
      // every MMA issued has completed before the tensor memory is released
      mma_commit(fin);
      if (!mbar_wait(fin, 0u, nullptr)) ok = false;
    }
  } else {  // ---- epilogue, warps 2-17
    // four warps per TMEM lane quarter (warp w may access lanes 32 (w % 4)
    // ..), one for each quarter of the tile's 128 columns
    const int ew = w - 2, q = w & 3, part = ew >> 2;
    const int tl = q * 32 + lane;
    const int i = tl >> 1, cc = tl & 1;  // real row tl = 2i + cc
    float* Cf = reinterpret_cast<float*>(C);
    // the next tile's C columns into L2 while this tile's MMAs run: thread
    // et covers 128 of the 512 bytes of column et / 4 of the tile
    auto prefetch = [&](int tile) {
      if (tile >= ntl) return;
      const int et = ew * 32 + lane;
      const int i0 = (tile % mtiles) * kTcBM, n = (tile / mtiles) * kTcBN + (et >> 2);
      const int l = et & 3;
      if (n >= N || l * 16 >= M - i0) return;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(Cf + 2 * ((size_t)n * ldc + i0) + 32 * l));
    };
    prefetch(blockIdx.x);
    int j = 0;
    for (int tile = blockIdx.x; tile < ntl; tile += gridDim.x, ++j) {
      prefetch(tile + gridDim.x);
      const int mt = tile % mtiles, nt = tile / mtiles;
      const int i0 = mt * kTcBM, n0 = nt * kTcBN + part * (kTcBN / 4);
      const bool row_ok = i0 + i < M;
      float* crow = Cf + 2 * ((size_t)i0 + i) + cc;
      // this thread's 32 C values, loaded while the tile's MMAs still run
      const int nlim = row_ok ? min(kTcBN / 4, N - n0) : 0;
      const long long cstep = 2 * ldc;
      float cv[kTcBN / 4];
      {
        const float* pc = crow + (size_t)n0 * cstep;
        if (nlim == kTcBN / 4) {  // full tile: no per-column predicates
#pragma unroll
          for (int u = 0; u < kTcBN / 4; ++u, pc += cstep) cv[u] = *pc;
        } else {
#pragma unroll
          for (int u = 0; u < kTcBN / 4; ++u, pc += cstep) cv[u] = u < nlim ? *pc : 0.f;
        }
      }
      const float isr = exp_float(isa[i0 + i]);  // the row's inverse scale
      const int a = j & 1;
      const unsigned aph = (unsigned)(j >> 1) & 1u;
      if (!mbar_wait(&acc_full[a], aph, s_abort)) {
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const unsigned lanes = tmem + (unsigned)a * kTcAcc + ((unsigned)(q * 32) << 16) +
                             (unsigned)(part * (kTcBN / 4));
      float* pw = crow + (size_t)n0 * cstep;
#pragma unroll
      for (int h = 0; h < kTcBN / 4; h += 8) {
        unsigned d1[8], d2[8];
        TC_LD8(d1, lanes + h);
        TC_LD8(d2, lanes + kTcBN + h);
        // exponent fields of the 8 columns' inverse scales
        const uint2 iv = *reinterpret_cast<const uint2*>(isb + n0 + h);
        asm volatile("tcgen05.wait::ld.sync.aligned;");
        float o[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const float p2 = __shfl_xor_sync(0xffffffffu, __uint_as_float(d2[u]), 1);
          const float isc = exp_float(((u < 4 ? iv.x : iv.y) >> (8 * (u & 3))) & 0xff);
          o[u] = cv[h + u] - (__uint_as_float(d1[u]) + (cc ? p2 : -p2)) * isr * isc;
        }
        if (nlim == kTcBN / 4) {
#pragma unroll
          for (int u = 0; u < 8; ++u, pw += cstep) *pw = o[u];
        } else {
#pragma unroll
          for (int u = 0; u < 8; ++u, pw += cstep)
            if (h + u < nlim) *pw = o[u];
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      mbar_arrive(&acc_empty[a]);
    }
    if (!ok) *s_abort = 1;
  }
  if (!ok) atomicExch(status, 1);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (w == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

#undef TC_LD8

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

}  // namespace

// The pack buffer starts with the slots that panels leave L's exponents in, then
// those that an update forms of its own.
static size_t part_bytes(int K) { return align256(sizeof(int) * kColParts * (size_t)K); }

int* tc_update_part(void* pack) {
  return reinterpret_cast<int*>(static_cast<char*>(pack) + kPanelExpoBytes);
}

size_t tc_pack_bytes(int M, int N, int K) {
  const size_t nkc = (size_t)(K + kTcBK - 1) / kTcBK;
  const size_t mt = (size_t)(M + kTcBM - 1) / kTcBM, nt = (size_t)(N + kTcBN - 1) / kTcBN;
  return kPanelExpoBytes + part_bytes(K) + align256(mt * nkc * kTcChunkA) + align256(nt * nkc * kTcChunkB) +
         align256(mt * kTcBM) + align256(nt * kTcBN);
}

// The pack buffer's parts for an M x N x K update.
static TcPack pack_parts(void* pack, int M, int N, int K, int passes) {
  const int nkc = (K + kTcBK - 1) / kTcBK;
  const int mt = (M + kTcBM - 1) / kTcBM, nt = (N + kTcBN - 1) / kTcBN;
  TcPack pk;
  pk.part = nullptr;
  pk.np = 0;
  pk.A = static_cast<unsigned char*>(pack) + kPanelExpoBytes + part_bytes(K);
  pk.B = pk.A + align256((size_t)mt * nkc * kTcChunkA);
  pk.isa = pk.B + align256((size_t)nt * nkc * kTcChunkB);
  pk.isb = pk.isa + align256((size_t)mt * kTcBM);
  pk.nkc = nkc;
  pk.passes = passes;
  return pk;
}

// The update of packed operands.
static int update_packed(float2* C, long long ldc, int M, int N, const TcPack& pk, int* status,
                         cudaStream_t s, int max_ctas) {
  if (!opt_in_smem<tc_cgemm_sub_kernel>(kTcSmem)) return BEM2D_ERR_CUDA;
  const int mt = (M + kTcBM - 1) / kTcBM, nt = (N + kTcBN - 1) / kTcBN;
  const int grid = std::min(mt * nt, max_ctas > 0 ? max_ctas : device_sms());
  tc_cgemm_sub_kernel<<<grid, kTcThreads, kTcSmem, s>>>(C, ldc, pk.A, pk.B, pk.isa, pk.isb, M, N,
                                                        pk.nkc, mt, nt, pk.passes, status);
  return cudaPeekAtLastError() == cudaSuccess ? BEM2D_OK : BEM2D_ERR_CUDA;
}

int launch_tc_cgemm_sub(float2* C, long long ldc, const float2* A, long long lda,
                        const float2* B, long long ldb, int M, int N, int K, void* pack,
                        size_t pack_bytes, int* status, cudaStream_t s, int max_ctas,
                        int passes, const int* part, int np) {
  if (M <= 0 || N <= 0 || K <= 0) return BEM2D_OK;
  if (!pack || tc_pack_bytes(M, N, K) > pack_bytes) return BEM2D_ERR_ARG;
  if (passes != 1 && passes != 3) return BEM2D_ERR_ARG;
  TcPack pk = pack_parts(pack, M, N, K, passes);
  if (!part) {
    int* own = tc_update_part(pack);
    np = launch_col_expo(A, lda, M, K, own, s);
    part = own;
  }
  pk.part = part;
  pk.np = np;
  const int ab = (M + kTcBM - 1) / kTcBM * (kTcBM / 32), bb = (N + kTcBN - 1) / kTcBN * (kTcBN / 8);
  pack_kernel<<<ab + bb, 256, sizeof(float) * kTcBK * pk.nkc, s>>>(A, lda, B, ldb, M, N, K, ab, pk);
  return update_packed(C, ldc, M, N, pk, status, s, max_ctas);
}

int launch_tc_step(float2* A, long long lda, int M, int k0, int nb, int cl, int rs, int cr,
                   const int* ipiv, bool update, const int* part, int np, const TcExpo& ex,
                   void* pack, int* status, cudaStream_t s, int max_ctas, int passes) {
  if (!opt_in_smem<tc_step_kernel>((int)kStepSmem)) return BEM2D_ERR_CUDA;
  const int N = cr - rs;  // N > 0: nb = 64
  const int nright = (N + kStepCols - 1) / kStepCols, nleft = (k0 - cl + kStepCols - 1) / kStepCols;
  TcPack pk{};
  if (update) {
    pk = pack_parts(pack, M, N, nb, passes);
    pk.part = part;
    pk.np = np;
  }
  const int nexpo = ex.K * ex.np;
  const int grid = nright + nleft + nexpo + (update ? (M + 31) / 32 : 0);
  if (grid == 0) return BEM2D_OK;
  tc_step_kernel<<<grid, 256, kStepSmem, s>>>(A, lda, M, k0, nb, cl, rs, cr, ipiv, nright, nleft,
                                              nexpo, update, pk, ex);
  if (update)
    return update_packed(A + (size_t)rs * lda + k0 + nb, lda, M, N, pk, status, s, max_ctas);
  return cudaPeekAtLastError() == cudaSuccess ? BEM2D_OK : BEM2D_ERR_CUDA;
}

}  // namespace bem2d_gpu
