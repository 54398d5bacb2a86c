// Complex128 LU panels: 64 columns in blocks of 16, each factored by one
// thread-block cluster with the rows in registers.
//
// GB300's FP64 pipe takes 64 clocks of a scheduler for one warp instruction,
// so a panel column costs what its FP64 instructions cost on the critical
// path.  Per 16-column block:
//   panel16_kernel    up to 16 CTAs, one thread per row (two above 4096 rows),
//                     16 complex128 in registers; rank-1 updates stay inside
//                     the block (36 FP64 instructions a column on average
//                     instead of 128 for 64 columns); pivot search on the
//                     integer pipe (|re| + |im| as 64-bit keys, warp reduce
//                     instructions); candidates travel by asynchronous
//                     stores, no cluster barrier per column
//   panel_side_kernel row swaps on the panel's other columns and, right of the
//                     block, U = L11^{-1} A (a warp per column)
//   panel_update_kernel  A -= L U on the panel's columns right of the block,
//                     spread over the whole chip
// Measured: kite N = 2048, panels 24.7 -> 11.3 ms (4.4 us a column instead of
// 12) against one cluster kernel with 64 columns in shared memory.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "common.cuh"
#include "cplx.cuh"
#include "tc.cuh"

namespace cg = cooperative_groups;

namespace bem2d_gpu {
namespace {

constexpr int kZW = 16;            // block width
constexpr int kZMaxC = 16;         // CTAs of a cluster
constexpr int kZThreads = 256;

__device__ __forceinline__ int zexpo(double x) { return (__double2hiint(x) >> 20) & 2047; }

// 1/a: the reciprocal of |a|^2 by a third-order correction of the hardware's
// 2^-20 seed; a scaled by a power of two first unless |a|^2 is far from the
// ends of the range (subnormal or infinite a: the general routine).
__device__ __forceinline__ double2 zrcp(double2 a) {
  const int e = max(zexpo(a.x), zexpo(a.y));
  if (e == 0 || e == 2047) return crcp(a);
  double s = 1.0;
  if (e < 600 || e > 1400) {  // scaled parts below 2
    s = e < 2046 ? __hiloint2double((2046 - e) << 20, 0) : 1.1125369292536007e-308;
    a.x *= s;
    a.y *= s;
  }
  const double q = fma(a.x, a.x, a.y * a.y);
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(q));
  const double t = fma(-q, r, 1.0);
  r = fma(r, fma(t, t, t), r);
  a = make_double2(a.x * r, -a.y * r);
  return s == 1.0 ? a : make_double2(a.x * s, a.y * s);
}

struct ZKey {
  unsigned hi, lo, label;  // bits of |re| + |im| (0: none), row
};

// Largest key of the warp, ties to the smaller label; the same on every lane.
__device__ __forceinline__ ZKey zkey_max(ZKey k) {
  ZKey m;
  m.hi = __reduce_max_sync(0xffffffffu, k.hi);
  m.lo = __reduce_max_sync(0xffffffffu, k.hi == m.hi ? k.lo : 0u);
  m.label = __reduce_min_sync(
      0xffffffffu, (k.hi == m.hi && k.lo == m.lo && (m.hi | m.lo)) ? k.label : 0xffffffffu);
  return m;
}

// Columns kb .. kb + w of rows kb .. n.  Row exchanges by renaming: a row
// carries the matrix row it stands for; the pivot row takes kc, the row that
// held kc takes the pivot's, and rows are written to their names at the end.
template <int R>
__global__ void __launch_bounds__(kZThreads, 1)
panel16_kernel(double2* __restrict__ A, long long lda, int n, int kb, int w, int rpb,
               int* __restrict__ ipiv, int* info, int* status) {
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  // by column parity: the candidates' rows and keys, the warps' candidates,
  // the staged own row, the mbarrier that counts a column's bytes
  __shared__ __align__(16) double2 slot[2][kZMaxC][kZW];
  __shared__ __align__(16) uint4 key[2][kZMaxC];
  __shared__ ZKey wkey[2][kZThreads / 32];
  __shared__ __align__(16) double2 srow[2][kZW];
  __shared__ __align__(8) unsigned long long mb[2];
  __shared__ int s_ipiv[kZW], s_info, s_abort;
  const int T = (int)blockDim.x, tid = threadIdx.x, ln = tid & 31, lw = tid >> 5, nw = T >> 5;
  unsigned label[R];
  double2 a[R][kZW];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int lr = tid + r * T, gr = kb + rank * rpb + lr;
    label[r] = lr < rpb && gr < n ? (unsigned)gr : 0xffffffffu;
#pragma unroll
    for (int c = 0; c < kZW; ++c)
      a[r][c] = label[r] != 0xffffffffu && c < w ? A[(size_t)(kb + c) * lda + gr]
                                                 : make_double2(0.0, 0.0);
  }
  if (tid == 0) {
    s_info = 0;
    s_abort = 0;
    tc::mbar_init(&mb[0], 1);
    tc::mbar_init(&mb[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  cl.sync();  // every CTA of the cluster is running before any DSMEM access
#pragma unroll
  for (int c = 0; c < kZW; ++c) {
    if (c >= w) break;
    const unsigned kc = (unsigned)(kb + c);
    const int par = c & 1;
    // bytes of the C candidates: entries c .. 15 and a key each
    if (tid == 0) tc::mbar_expect_tx(&mb[par], (unsigned)C * 16u * (unsigned)(kZW - c + 1));
    // 1. the CTA's candidate
    ZKey k{0u, 0u, 0xffffffffu};
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (label[r] == 0xffffffffu || label[r] < kc) continue;
      const long long b = __double_as_longlong(cabs1(a[r][c]));
      if (b > 0x7ff0000000000000ll) continue;  // NaN
      const unsigned h = (unsigned)(b >> 32), l = (unsigned)b;
      if (h > k.hi || (h == k.hi && (l > k.lo || (l == k.lo && label[r] < k.label))))
        k = ZKey{h, l, label[r]};
    }
    k = zkey_max(k);
    if (ln == 0) wkey[par][lw] = k;
    __syncthreads();
    // every warp forms the CTA's candidate, whose thread stages its row; the
    // warps share the sends to the other CTAs, asynchronous stores that count
    // their bytes on the receiver's mbarrier.  A CTA sends its candidate of
    // column c + 1 after it has used the ones of column c, so two buffers do.
    k = zkey_max(ln < nw ? wkey[par][ln] : ZKey{0u, 0u, 0xffffffffu});
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (k.label != 0xffffffffu && label[r] == k.label) {
#pragma unroll
        for (int e = 0; e < kZW; ++e)
          if (e >= c) srow[par][e] = a[r][e];
      }
    }
    __syncthreads();
    {
      // lanes 0-15: entry ln to rank q, lanes 16-31 to rank q + 1
      const int e = ln & 15;
      const uint4 v = *reinterpret_cast<const uint4*>(&srow[par][e]);
      for (int q = 2 * lw + (ln >> 4); q < C; q += 2 * nw) {
        const unsigned bar = tc::map_rank(&mb[par], q);
        if (e >= c) tc::store_async(tc::map_rank(&slot[par][rank][e], q), v, bar);
        if (e == 0)
          tc::store_async(tc::map_rank(&key[par][rank], q), make_uint4(k.hi, k.lo, k.label, 0u),
                          bar);
      }
    }
    // 2. every candidate has arrived
    const bool live = tc::mbar_wait_cluster(&mb[par], (unsigned)(c >> 1) & 1u, &s_abort);
    // 3. the pivot, from the local slots (every warp)
    const uint4 kv = ln < C ? key[par][ln] : make_uint4(0u, 0u, 0xffffffffu, 0u);
    const ZKey mk{kv.x, kv.y, kv.z};
    k = zkey_max(mk);
    // after a wait that gave up nothing is used
    const bool zero = !__all_sync(0xffffffffu, live) || (k.hi | k.lo) == 0u || k.label < kc ||
                      k.label >= (unsigned)n;
    if (tid == 0) {
      s_ipiv[c] = zero ? (int)kc : (int)k.label;
      if (zero && s_info == 0) s_info = (int)kc + 1;
    }
    if (zero) continue;  // LAPACK: no swap and no elimination for a zero pivot
    const int win = __ffs(__ballot_sync(0xffffffffu, ln < C && mk.label == k.label)) - 1;
    const double2* p = slot[par][win];
    const double2 inv = zrcp(p[c]);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (label[r] == k.label)
        label[r] = kc;
      else if (label[r] == kc)
        label[r] = k.label;
      if (label[r] != 0xffffffffu && label[r] > kc) {
        const double2 l = cmul(a[r][c], inv);
        a[r][c] = l;
#pragma unroll
        for (int e = 0; e < kZW; ++e)
          if (e > c) a[r][e] = cfms(a[r][e], l, p[e]);
      }
    }
  }
  cl.sync();  // no CTA leaves while another may still write its shared memory
  if (tid == 0 && s_abort) atomicExch(status, 1);
  if (rank == 0) {
    if (tid < w) ipiv[kb + tid] = s_ipiv[tid];
    if (tid == 0 && s_info && *info == 0) *info = s_info;
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (label[r] != 0xffffffffu)
#pragma unroll
      for (int c = 0; c < kZW; ++c)
        if (c < w) A[(size_t)(kb + c) * lda + label[r]] = a[r][c];
}

// The interchanges ipiv[kb .. kb + w) on the panel columns [k0, kb) and
// [kb + w, kend), and U = L11^{-1} A on the latter; a warp per column.
__global__ void __launch_bounds__(128)
panel_side_kernel(double2* __restrict__ A, long long lda, const int* __restrict__ ipiv, int k0,
                  int kb, int w, int kend) {
  const int v = blockIdx.x * 4 + (threadIdx.x >> 5), ln = threadIdx.x & 31;
  const int left = kb - k0;
  if (v >= left + kend - kb - w) return;
  const int j = v < left ? k0 + v : kb + w + v - left;
  double2* col = A + (size_t)j * lda;
  const int p = ln < w ? ipiv[kb + ln] : 0;
  // lane l < 16: row kb + l, lane 16 + l: pivot row l; where its final value
  // comes from: the interchanges undone from the last to the first
  const int pp = __shfl_sync(0xffffffffu, p, ln & 15);
  const int row = (ln & 15) >= w ? -1 : ln < 16 ? kb + ln : pp;
  int src = row;
  for (int s = w - 1; s >= 0; --s) {
    const int ps = __shfl_sync(0xffffffffu, p, s);
    src = src == kb + s ? ps : src == ps ? kb + s : src;
  }
  double2 x = row >= 0 ? col[src] : make_double2(0.0, 0.0);
  __syncwarp();
  // a pivot row inside the block is stored by its own lane
  if (row >= 0 && ln >= 16 && row >= kb + w) col[row] = x;
  if (v >= left) {
    const double2* L = A + (size_t)kb * lda + kb + ln;
    double2 l[kZW];
#pragma unroll
    for (int s = 0; s < kZW; ++s)
      l[s] = s < w && ln < w && ln > s ? L[(size_t)s * lda] : make_double2(0.0, 0.0);
#pragma unroll
    for (int s = 0; s < kZW - 1; ++s) {
      const double2 xs = make_double2(__shfl_sync(0xffffffffu, x.x, s),
                                      __shfl_sync(0xffffffffu, x.y, s));
      x = cfms(x, l[s], xs);
    }
  }
  if (ln < w) col[kb + ln] = x;
}

// A[r, j] -= sum_k L[r, kb + k] U[kb + k, j], rows r0 .. n, columns j0 .. j1;
// a thread takes one row and 4 columns, a CTA 32 rows and 16 columns.
__global__ void __launch_bounds__(128)
panel_update_kernel(double2* __restrict__ A, long long lda, int n, int kb, int j0, int j1) {
  const int r = kb + kZW + blockIdx.x * 32 + (threadIdx.x & 31);
  const int j = j0 + blockIdx.y * 16 + (threadIdx.x >> 5) * 4;
  if (r >= n || j >= j1) return;
  const int nc = min(4, j1 - j);
  double2 acc[4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
    acc[u] = u < nc ? A[(size_t)(j + u) * lda + r] : make_double2(0.0, 0.0);
  const double2* L = A + (size_t)kb * lda + r;
  const double2* U = A + (size_t)j * lda + kb;
#pragma unroll 4
  for (int k = 0; k < kZW; ++k) {
    const double2 l = L[(size_t)k * lda];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (u < nc) acc[u] = cfms(acc[u], l, U[(size_t)u * lda + k]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (u < nc) A[(size_t)(j + u) * lda + r] = acc[u];
}

}  // namespace

// Factors columns [k0, k0 + nb) of rows k0 .. n (nb <= 64), interchanges
// applied to these columns only.  Returns 1 when the panel is too tall for
// the register kernel (more than 8192 rows) or clusters of its size are not
// available, having changed nothing.
int launch_zpanel(double2* A, long long lda, int n, int k0, int nb, const LuWork& w,
                  cudaStream_t s, long long* launches) {
  static std::atomic<int> max_cluster{kZMaxC};
  static std::once_flag attr;
  std::call_once(attr, [] {
    if (cudaFuncSetAttribute(panel16_kernel<1>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                             1) != cudaSuccess ||
        cudaFuncSetAttribute(panel16_kernel<2>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                             1) != cudaSuccess) {
      cudaGetLastError();
      max_cluster = 8;
    }
  });
  const int kend = k0 + nb;
  for (int kb = k0; kb < kend; kb += kZW) {
    const int bw = std::min(kZW, kend - kb), H = n - kb;
    // rows of a CTA: the fewest that 16 CTAs hold, in whole warps
    for (;;) {
      const int cmax = max_cluster;
      const int rpb = std::max(32, ((H + cmax - 1) / cmax + 31) / 32 * 32);
      const int R = rpb <= kZThreads ? 1 : 2;
      if (rpb > 2 * kZThreads) return kb == k0 ? 1 : BEM2D_ERR_CUDA;
      const int C = (H + rpb - 1) / rpb, threads = (rpb / R + 31) / 32 * 32;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(C);
      cfg.blockDim = dim3(threads);
      cfg.stream = s;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = C;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      const cudaError_t e =
          R == 1 ? cudaLaunchKernelEx(&cfg, panel16_kernel<1>, A, lda, n, kb, bw, rpb, w.ipiv, w.info, w.status)
                 : cudaLaunchKernelEx(&cfg, panel16_kernel<2>, A, lda, n, kb, bw, rpb, w.ipiv, w.info, w.status);
      if (e == cudaSuccess) break;
      cudaGetLastError();
      if (cmax <= 8) return kb == k0 ? 1 : BEM2D_ERR_CUDA;
      max_cluster = 8;
    }
    const int others = nb - bw;
    if (others > 0)
      panel_side_kernel<<<(others + 3) / 4, 128, 0, s>>>(A, lda, w.ipiv, k0, kb, bw, kend);
    const int j0 = kb + bw;
    if (j0 < kend && j0 < n)
      panel_update_kernel<<<dim3((n - j0 + 31) / 32, (kend - j0 + 15) / 16), 128, 0, s>>>(
          A, lda, n, kb, j0, kend);
    *launches += 1 + (others > 0) + (j0 < kend);
  }
  return cudaPeekAtLastError() == cudaSuccess ? BEM2D_OK : BEM2D_ERR_CUDA;
}

}  // namespace bem2d_gpu
