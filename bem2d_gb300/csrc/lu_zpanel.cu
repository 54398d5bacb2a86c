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
// Measured: kite N = 2048, panels 24.7 -> 9.3 ms (panel16_kernel 7.4 of them, 3.6
// us a column; one cluster kernel with 64 columns in shared memory: 12).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

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

// The factor r of a / p = a conj(p) r, r = 1 / |p|^2 by a third-order correction
// of the hardware's 2^-20 seed.  p is scaled by the power of two *s first where
// |p|^2 would leave the range (then a / p = a s conj(p) r).  Forming a conj(p)
// beside r keeps the chain of dependent FP64 instructions at seven.
// False for subnormal and non-finite p: use zdiv_general.
__device__ __forceinline__ bool zrcp(double2* p, double* s, double* r) {
  const int e = max(zexpo(p->x), zexpo(p->y));
  *s = 1.0;
  if (e == 0 || e == 2047) return false;
  if (e < 600 || e > 1400) {  // scaled parts below 2
    *s = e < 2046 ? __hiloint2double((2046 - e) << 20, 0) : 1.1125369292536007e-308;
    p->x *= *s;
    p->y *= *s;
  }
  const double q = fma(p->x, p->x, p->y * p->y);
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(q));
  const double t = fma(-q, y, 1.0);
  *r = fma(y, fma(t, t, t), y);
  return true;
}
__device__ __noinline__ double2 zdiv_general(double2 a, double2 p) { return cmul(a, crcp(p)); }

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
// R rows per thread, or TPR threads (neighbouring lanes) per row, thread t
// holding columns t, t + TPR, ...: a CTA of 32 or 64 rows then spreads its
// updates over all four schedulers.
template <int R, int TPR>
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
  constexpr int kL = kZW / TPR;  // columns per thread
  const int T = (int)blockDim.x, tid = threadIdx.x, ln = tid & 31, lw = tid >> 5, nw = T >> 5;
  const int t = tid % TPR;
  unsigned label[R];
  double2 a[R][kL];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int lr = tid / TPR + r * T, gr = kb + rank * rpb + lr;
    label[r] = lr < rpb && gr < n ? (unsigned)gr : 0xffffffffu;
#pragma unroll
    for (int i = 0; i < kL; ++i) {
      const int c = i * TPR + t;
      a[r][i] = label[r] != 0xffffffffu && c < w ? A[(size_t)(kb + c) * lda + gr]
                                                 : make_double2(0.0, 0.0);
    }
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
      if (label[r] == 0xffffffffu || label[r] < kc || t != c % TPR) continue;
      const unsigned long long b =
          (unsigned long long)__double_as_longlong(cabs1(a[r][c / TPR]));
      if (b > 0x7ff0000000000000ull) continue;  // NaN, whose sign bit may be set
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
        for (int i = 0; i < kL; ++i)
          if (i >= c / TPR) srow[par][i * TPR + t] = a[r][i];
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
    double2 ps = p[c];
    double sc, rc;
    const bool fast = zrcp(&ps, &sc, &rc);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (label[r] == k.label)
        label[r] = kc;
      else if (label[r] == kc)
        label[r] = k.label;
      // the row's column-c value, from the thread that holds it
      double2 v = a[r][c / TPR];
      if (TPR > 1) {
        v.x = __shfl_sync(0xffffffffu, v.x, (ln & ~(TPR - 1)) | (c % TPR));
        v.y = __shfl_sync(0xffffffffu, v.y, (ln & ~(TPR - 1)) | (c % TPR));
      }
      if (label[r] != 0xffffffffu && label[r] > kc) {
        double2 l;
        if (fast) {
          if (sc != 1.0) v = make_double2(v.x * sc, v.y * sc);
          l = make_double2(fma(v.x, ps.x, v.y * ps.y) * rc, fma(v.y, ps.x, -v.x * ps.y) * rc);
        } else {
          l = zdiv_general(v, p[c]);
        }
        if (TPR == 1) {
          a[r][c] = l;
        } else if (t >= c % TPR) {  // the slot of column c: l, or an update right of c
          const int i = c / TPR;
          a[r][i] = t == c % TPR ? l : cfms(a[r][i], l, p[i * TPR + t]);
        }
#pragma unroll
        for (int i = 0; i < kL; ++i)
          if (i > c / TPR) a[r][i] = cfms(a[r][i], l, p[i * TPR + t]);
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
      for (int i = 0; i < kL; ++i)
        if (i * TPR + t < w) A[(size_t)(kb + i * TPR + t) * lda + label[r]] = a[r][i];
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
  static PerDevice<int> largest(kZMaxC);
  static PerDeviceOnce attr;
  const int dev = current_device();
  std::atomic<int>& max_cluster = largest[dev];
  attr(dev, [&] {
    bool ok = true;
    for (auto k : {panel16_kernel<1, 1>, panel16_kernel<1, 2>, panel16_kernel<1, 4>,
                   panel16_kernel<2, 1>})
      ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                     cudaSuccess;
    if (!ok) {
      cudaGetLastError();
      max_cluster = 8;
    }
  });
  const int kend = k0 + nb;
  // this panel's own limit: another thread's refused launch must not make a block
  // too tall whose predecessors are already factored
  int cmax = max_cluster;
  for (int kb = k0; kb < kend; kb += kZW) {
    const int bw = std::min(kZW, kend - kb), H = n - kb;
    // rows of a CTA: the fewest that 16 CTAs hold, in whole warps
    for (;;) {
      const int rpb = std::max(32, ((H + cmax - 1) / cmax + 31) / 32 * 32);
      if (rpb > 2 * kZThreads) return kb == k0 ? 1 : BEM2D_ERR_CUDA;
      const int C = (H + rpb - 1) / rpb;
      const int threads = rpb <= 32    ? 4 * rpb
                          : rpb <= 64  ? 2 * rpb
                          : rpb <= kZThreads ? rpb
                                             : (rpb / 2 + 31) / 32 * 32;
      auto kern = rpb <= 32          ? panel16_kernel<1, 4>
                  : rpb <= 64        ? panel16_kernel<1, 2>
                  : rpb <= kZThreads ? panel16_kernel<1, 1>
                                     : panel16_kernel<2, 1>;
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
          cudaLaunchKernelEx(&cfg, kern, A, lda, n, kb, bw, rpb, w.ipiv, w.info, w.status);
      if (e == cudaSuccess) break;
      cudaGetLastError();
      if (cmax <= 8) return kb == k0 ? 1 : BEM2D_ERR_CUDA;
      cmax = max_cluster = 8;
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
