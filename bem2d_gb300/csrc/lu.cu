// Blocked right-looking LU with partial pivoting and the triangular solves,
// for complex128 (double2) and complex64 (float2).  Replaces LAPACK zgetrf +
// zgetrs as called by SolveSystem (lib/bem2d_mathroutines.cpp:323-351).
//
// Per panel of NB = 64 columns:
//   panel_cluster_kernel  one thread-block cluster (up to 16 CTAs) holds the
//                  panel rows in distributed shared memory; per column each CTA
//                  writes its pivot candidate (value, row, panel row) to its own
//                  shared memory, one cluster barrier, then every CTA reads the
//                  candidates over DSMEM, agrees on the pivot, swaps and
//                  updates.  Used while the panel fits in the cluster's smem.
//   panel_kernel   the same exchange through global-memory slots with
//                  sequence flags (bounded waits) across a cooperative grid,
//                  for taller panels.
//   laswp_kernel   the panel's row swaps on all other columns (LAPACK order)
//   trsm_kernel    U12 = L11^{-1} A12 (complex64 below kOuterMinN: both, and the
//                  update, in launch_tc_step)
//   gemm_kernel    A22 -= L21 U12  (register-tiled, 64 x 64 CTA tiles)
// After the factorisation: perm (the row permutation of the pivots) and the
// inverses of the 64 x 64 diagonal blocks of L and U, so that a solve is a
// chain of small matrix-vector products (trisolve64_kernel,
// trisolve_cluster_kernel, trisolve_wave_kernel).
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

#include <algorithm>
#include <atomic>
#include <climits>

#include "colscale.cuh"
#include "common.cuh"
#include "cplx.cuh"
#include "tc.cuh"

namespace bem2d_gpu {

constexpr int kNB = 64;              // panel width
constexpr int kPanelThreads = 256;
constexpr unsigned kSpinLimit = 1u << 25;  // polls of >= 32 ns: > 1 s

// (value, row) arg-max with ties to the smaller row, as LAPACK's izamax
// (first maximal |re| + |im|).
template <typename R>
__device__ __forceinline__ void argmax_merge(R& v, int& i, R v2, int i2) {
  if (v2 > v || (v2 == v && i2 < i)) {
    v = v2;
    i = i2;
  }
}

template <typename R>
__device__ void block_argmax(R& v, int& i) {
  __shared__ R sv[kPanelThreads / 32];
  __shared__ int si[kPanelThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const R v2 = __shfl_xor_sync(0xffffffffu, v, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, i, o);
    argmax_merge(v, i, v2, i2);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) {
    sv[w] = v;
    si[w] = i;
  }
  __syncthreads();
  v = sv[0];
  i = si[0];
  for (int k = 1; k < (int)(blockDim.x >> 5); ++k) argmax_merge(v, i, sv[k], si[k]);
}

// Panel exchange slots in global memory, two per block (column parity):
// {seq, row index, |pivot| value, the block's candidate panel row}, plus a
// slot for the current row kc from its owner.  A slot is valid for column kc
// when its seq equals kc + 1; the slots are zeroed before each factorisation.
constexpr int kMaxPanelBlocks = 1024;
constexpr int kSlotHead = 16;  // int seq, int idx, 8-byte value

template <typename T>
struct PanelSlots {
  char* base;
  __device__ __forceinline__ char* slot(int par, int b) const {
    return base + ((size_t)par * (kMaxPanelBlocks + 1) + b) * (kSlotHead + sizeof(T) * kNB);
  }
  __device__ __forceinline__ char* krow(int par) const { return slot(par, kMaxPanelBlocks); }
};


static size_t slots_bytes(size_t elem) {
  return (size_t)2 * (kMaxPanelBlocks + 1) * (kSlotHead + elem * kNB);
}

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Wait (bounded: `limit` polls) until *seq == want (acquire); returns false
// on timeout.  Spins without sleeping first: the expected wait is one L2
// round trip.
__device__ __forceinline__ bool wait_seq(const int* seq, int want, int* status,
                                         unsigned limit = kSpinLimit) {
  unsigned it = 0;
  while (ld_acquire(seq) != want) {
    if (++it > limit || (it > 1024 && *(volatile int*)status != 0)) {
      atomicExch(status, 1);
      return false;
    }
    if (it > 256) __nanosleep(32);
  }
  return true;
}

// Publish `epoch` at *flag after every thread of the block has written its
// data: bar.sync orders the block's writes before thread 0's release store.
__device__ __forceinline__ void block_publish(int* flag, int epoch) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    st_release(flag, epoch);
  }
}

template <typename T>
__global__ void __launch_bounds__(kPanelThreads)
panel_kernel(T* __restrict__ A, long long lda, int n, int k0, int nb, int rpb,
             int* __restrict__ ipiv, int* info, int* status, PanelSlots<T> sl, int nwait,
             unsigned spin) {
  typedef typename CTraits<T>::R R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* P = reinterpret_cast<T*>(smem_raw);  // [rpb][kNB] block's panel rows
  T* prow = P + (size_t)rpb * kNB;        // [kNB] pivot row
  T* lcol = prow + kNB;                   // [rpb] multipliers
  __shared__ int s_p, s_bw, s_ok;
  __shared__ R s_pv;

  const int b = blockIdx.x;
  const int r0 = k0 + b * rpb;
  const int r1 = min(r0 + rpb, n);
  const int nr = max(r1 - r0, 0);
  for (int v = threadIdx.x; v < nr * nb; v += blockDim.x) {
    const int c = v / nr, lr = v - c * nr;
    P[lr * kNB + c] = A[(size_t)(k0 + c) * lda + r0 + lr];
  }
  if (threadIdx.x == 0) s_ok = 1;
  __syncthreads();

  for (int c = 0; c < nb; ++c) {
    const int kc = k0 + c, par = kc & 1, epoch = kc + 1;
    // (a) local pivot candidate among rows >= kc
    R best = -1;
    int bidx = INT_MAX;
    for (int lr = threadIdx.x; lr < nr; lr += blockDim.x) {
      const int gr = r0 + lr;
      if (gr < kc) continue;
      argmax_merge(best, bidx, cabs1(P[lr * kNB + c]), gr);
    }
    block_argmax(best, bidx);
    // (b) publish the candidate (and row kc from its owner), then the seq
    char* my = sl.slot(par, b);
    T* myrow = reinterpret_cast<T*>(my + kSlotHead);
    if (bidx != INT_MAX)
      for (int j = threadIdx.x; j < nb; j += blockDim.x) myrow[j] = P[(bidx - r0) * kNB + j];
    const bool own_k = kc >= r0 && kc < r1;
    char* kr = sl.krow(par);
    if (own_k)
      for (int j = threadIdx.x; j < nb; j += blockDim.x)
        reinterpret_cast<T*>(kr + kSlotHead)[j] = P[(kc - r0) * kNB + j];
    if (threadIdx.x == 0) {
      reinterpret_cast<int*>(my)[1] = bidx;
      *reinterpret_cast<R*>(my + 8) = best;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      st_release(reinterpret_cast<int*>(my), epoch);
      if (own_k) st_release(reinterpret_cast<int*>(kr), epoch);
    }
    // (c) wait for every block's candidate (nwait = the grid size; a larger
    // value waits for slots nobody posts: the timeout check), agree on the
    // pivot
    R v = -1;
    int i = INT_MAX;
    if ((int)threadIdx.x < nwait) {
      const char* q = sl.slot(par, threadIdx.x);
      if (!wait_seq(reinterpret_cast<const int*>(q), epoch, status, spin)) {
        s_ok = 0;
      } else {
        i = __ldcg(reinterpret_cast<const int*>(q) + 1);
        v = __ldcg(reinterpret_cast<const R*>(q + 8));
      }
    }
    block_argmax(v, i);  // contains __syncthreads: s_ok visible after it
    if (!s_ok) return;
    if (threadIdx.x == 0) {
      // no finite candidate (all NaN): treat as a zero pivot at row kc
      if (i == INT_MAX || i < kc || i >= n) {
        i = kc;
        v = 0;
      }
      s_p = i;
      s_bw = (i - k0) / rpb;  // the owner block of row i published it
      s_pv = v;
    }
    __syncthreads();
    const int p = s_p, bw = s_bw;
    const bool zero = !(s_pv > 0);
    const T* wrow = reinterpret_cast<const T*>(sl.slot(par, bw) + kSlotHead);
    for (int j = threadIdx.x; j < nb; j += blockDim.x) prow[j] = __ldcg(&wrow[j]);
    if (b == 0 && threadIdx.x == 0) {
      ipiv[kc] = p;
      if (zero && *info == 0) *info = kc + 1;
    }
    if (!zero && p != kc && p >= r0 && p < r1) {
      if (threadIdx.x == 0 && !wait_seq(reinterpret_cast<const int*>(kr), epoch, status, spin))
        s_ok = 0;
      __syncthreads();
      if (!s_ok) return;
      for (int j = threadIdx.x; j < nb; j += blockDim.x)
        P[(p - r0) * kNB + j] = __ldcg(reinterpret_cast<const T*>(kr + kSlotHead) + j);
    }
    __syncthreads();
    if (!zero && p != kc && own_k)
      for (int j = threadIdx.x; j < nb; j += blockDim.x) P[(kc - r0) * kNB + j] = prow[j];
    __syncthreads();
    // (d) multipliers and rank-1 update of the block's rows below kc
    if (!zero) {
      const T inv = crcp(prow[c]);
      for (int lr = threadIdx.x; lr < nr; lr += blockDim.x) {
        if (r0 + lr > kc) {
          const T l = cmul(P[lr * kNB + c], inv);
          P[lr * kNB + c] = l;
          lcol[lr] = l;
        }
      }
      __syncthreads();
      const int w = nb - c - 1;
      if (w > 0) {
        for (int u = threadIdx.x; u < nr * w; u += blockDim.x) {
          const int lr = u / w, cc = c + 1 + (u - lr * w);
          if (r0 + lr > kc) P[lr * kNB + cc] = cfms(P[lr * kNB + cc], lcol[lr], prow[cc]);
        }
      }
    }
    __syncthreads();
  }
  for (int v2 = threadIdx.x; v2 < nr * nb; v2 += blockDim.x) {
    const int c = v2 / nr, lr = v2 - c * nr;
    A[(size_t)(k0 + c) * lda + r0 + lr] = P[lr * kNB + c];
  }
}

// Row swaps ipiv[k0 .. k0 + np) (LAPACK order) on columns [c0, c1).
template <typename T>
__global__ void laswp_cols_kernel(T* __restrict__ A, long long lda, const int* __restrict__ ipiv,
                                  int k0, int np, int c0, int c1) {
  const int j = c0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= c1) return;
  T* col = A + (size_t)j * lda;
  for (int s = 0; s < np; ++s) {
    const int p = ipiv[k0 + s];
    if (p != k0 + s) {
      const T t = col[k0 + s];
      col[k0 + s] = col[p];
      col[p] = t;
    }
  }
}
template <typename T>
static void laswp_cols(T* A, long long lda, const int* ipiv, int k0, int np, int c0, int c1,
                       cudaStream_t s, long long* launches) {
  if (c1 <= c0 || np <= 0) return;
  laswp_cols_kernel<T><<<(c1 - c0 + 127) / 128, 128, 0, s>>>(A, lda, ipiv, k0, np, c0, c1);
  ++*launches;
}

// Row swaps of panel [k0, k0+nb) on every column outside it.
template <typename T>
__global__ void laswp_kernel(T* __restrict__ A, long long lda, int n,
                             const int* __restrict__ ipiv, int k0, int nb) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n - nb) return;
  const int j = v < k0 ? v : v + nb;
  T* col = A + (size_t)j * lda;
  for (int s = 0; s < nb; ++s) {
    const int p = ipiv[k0 + s];
    if (p != k0 + s) {
      const T t = col[k0 + s];
      col[k0 + s] = col[p];
      col[p] = t;
    }
  }
}

// X = L11^{-1} X for X = A[k0:k0+nb, c0:c0+32), L11 unit lower.
template <typename T>
__global__ void __launch_bounds__(256)
trsm_kernel(T* __restrict__ A, long long lda, int k0, int nb, int c0, int ncols) {
  // U12 = L11^{-1} A12 for 32 columns per CTA, by blocks of 8 rows: warp w
  // holds rows 8w..8w+7 of its lane's column in registers; block b is
  // solved by warp b alone (8 steps in registers), then one __syncthreads
  // and every warp below subtracts L[w-block, b-block] x_b: 8 barriers
  // instead of one per row.
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* L = reinterpret_cast<T*>(smem_raw);  // [kNB][kNB] column-major
  T* X = L + kNB * kNB;                   // [kNB][32]: X[r*32 + c]
  const T zero = CTraits<T>::make(0, 0);
  const int cb = c0 + blockIdx.x * 32;
  const int nc = min(32, c0 + ncols - cb);
  for (int v = threadIdx.x; v < kNB * kNB; v += blockDim.x) {
    const int s = v >> 6, r = v & 63;
    L[s * kNB + r] = (s < nb && r < nb) ? A[(size_t)(k0 + s) * lda + k0 + r] : zero;
  }
  for (int v = threadIdx.x; v < kNB * 32; v += blockDim.x) {
    const int c = v >> 6, r = v & 63;
    X[r * 32 + c] = (c < nc && r < nb) ? A[(size_t)(cb + c) * lda + k0 + r] : zero;
  }
  __syncthreads();
  const int c = threadIdx.x & 31, w = threadIdx.x >> 5;
  T x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = X[(8 * w + i) * 32 + c];
  const int nbk = (nb + 7) >> 3;
  for (int b = 0; b < nbk; ++b) {
    if (w == b) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = i + 1; j < 8; ++j) x[j] = cfms(x[j], L[(8 * b + i) * kNB + 8 * b + j], x[i]);
#pragma unroll
      for (int i = 0; i < 8; ++i) X[(8 * b + i) * 32 + c] = x[i];
    }
    __syncthreads();
    if (w > b) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const T xb = X[(8 * b + j) * 32 + c];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = cfms(x[i], L[(8 * b + j) * kNB + 8 * w + i], xb);
      }
    }
  }
  __syncthreads();
  for (int v = threadIdx.x; v < nb * nc; v += blockDim.x) {
    const int cc = v / nb, r = v - cc * nb;
    A[(size_t)(cb + cc) * lda + k0 + r] = X[r * 32 + cc];
  }
}

// C[M x N] -= A[M x K] B[K x N], K <= kNB, column-major operands.
constexpr int kGB = 64;
constexpr int kTensorMinN = 256;  // update size from which complex64 uses tcgen05
constexpr int kOuterNB = 256;     // outer block width of the complex64 LU
constexpr int kOuterMinN = 8192;  // smaller matrices: the extra launches cost more
template <typename T>
__global__ void __launch_bounds__(256)
gemm_sub_kernel(const T* __restrict__ Am, long long lda, const T* __restrict__ Bm,
                long long ldb, T* __restrict__ C, long long ldc, int M, int N, int K) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* As = reinterpret_cast<T*>(smem_raw);  // [K][kGB]
  T* Bs = As + kNB * kGB;                  // [K][kGB]
  const int m0 = blockIdx.x * kGB, n0 = blockIdx.y * kGB;
  for (int v = threadIdx.x; v < K * kGB; v += blockDim.x) {
    const int k = v / kGB, i = v - k * kGB;
    As[k * kGB + i] = (m0 + i < M) ? Am[(size_t)k * lda + m0 + i] : CTraits<T>::make(0, 0);
  }
  for (int v = threadIdx.x; v < K * kGB; v += blockDim.x) {
    const int j = v / K, k = v - j * K;
    Bs[k * kGB + j] = (n0 + j < N) ? Bm[(size_t)(n0 + j) * ldb + k] : CTraits<T>::make(0, 0);
  }
  __syncthreads();
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  T acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[a][c] = CTraits<T>::make(0, 0);
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    T av[4], bv[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) av[a] = As[k * kGB + tx + 16 * a];
#pragma unroll
    for (int c = 0; c < 4; ++c) bv[c] = Bs[k * kGB + ty + 16 * c];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][c] = cfma(av[a], bv[c], acc[a][c]);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int j = n0 + ty + 16 * c;
    if (j >= N) continue;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i = m0 + tx + 16 * a;
      if (i < M) {
        T* p = C + (size_t)j * ldc + i;
        T v = *p;
        v.x -= acc[a][c].x;
        v.y -= acc[a][c].y;
        *p = v;
      }
    }
  }
}

template <typename T>
static int panel_blocks(int H) {
  const int nsm = device_sms();
  // at least 64 rows per block: fewer blocks make the per-column barrier
  // and the pivot agreement cheaper; one block per SM at most
  return std::max(1, std::min(nsm, (H + 63) / 64));
}

// ---- cluster panel ---------------------------------------------------------
// The panel's H rows are split over the C CTAs of one cluster (rpb rows
// each, at most kPanelRPT per thread) and held column-major in shared
// memory; thread t owns rows t, t + 256, ... and is the only thread that
// touches them, so the per-column update needs no intra-CTA barrier.
// Candidates are pushed, not pulled: per column
//   1. each thread: arg-max |re|+|im| over its rows >= kc, warp shuffles, one
//      __syncthreads, warp 0 merges the warps and writes the CTA's candidate
//      (value, row index, the whole row) into slot [parity][rank] of EVERY
//      CTA's shared memory (DSMEM stores); warp 1 of the owner of row kc
//      writes row kc into every CTA's krow[parity];
//   2. one cluster barrier (release/acquire): all C candidates and row kc
//      are now local to every CTA;
//   3. every warp picks the pivot from the C local slots (ties to the smaller
//      row, as izamax); the thread owning the pivot row takes row kc, the
//      thread owning row kc takes the pivot row (the row swap), and every
//      thread scales its rows below kc and applies the rank-1 update with the
//      pivot row read from the local slot.
// One __syncthreads and one cluster barrier per column, no DSMEM load on the
// critical path.  Slots are double-buffered by column parity: a CTA can only
// write the slots of column c + 1 after every CTA has left column c - 1.
constexpr int kPanelRPT = 4;        // panel rows per thread at most
constexpr int kMaxClusterPanel = 16;

template <typename T>
struct PanelSmem {
  // offsets in units of T, after the [kNB][ldp] panel
  static __host__ __device__ size_t slots(int ldp) { return (size_t)kNB * ldp; }
  static __host__ __device__ size_t krow(int ldp) {
    return slots(ldp) + (size_t)2 * kMaxClusterPanel * kNB;
  }
  static __host__ __device__ size_t total(int ldp) { return krow(ldp) + 2 * kNB; }
};

template <typename T>
__global__ void __launch_bounds__(kPanelThreads)
panel_cluster_kernel(T* __restrict__ A, long long lda, int n, int k0, int nb, int rpb,
                     int* __restrict__ ipiv, int* info) {
  typedef typename CTraits<T>::R R;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int ldp = rpb | 1;  // odd column stride
  T* P = reinterpret_cast<T*>(smem_raw);          // [kNB][ldp] panel rows, column-major
  T* slot = P + PanelSmem<T>::slots(ldp);         // [2][kMaxClusterPanel][kNB] candidate rows
  T* krow = P + PanelSmem<T>::krow(ldp);          // [2][kNB] row kc
  __shared__ R sval[2][kMaxClusterPanel];
  __shared__ int sidx[2][kMaxClusterPanel];
  __shared__ R wv[kPanelThreads / 32];
  __shared__ int wi[kPanelThreads / 32];
  __shared__ int s_ipiv[kNB];  // pivots, written to global memory at the end
  __shared__ int s_info;
  const int r0 = k0 + rank * rpb;
  const int r1 = min(r0 + rpb, n);
  const int nr = max(r1 - r0, 0);
  const int lw = threadIdx.x >> 5, ln = threadIdx.x & 31;
  const int nw = (int)(blockDim.x >> 5);
  for (int c = 0; c < nb; ++c)
    for (int lr = threadIdx.x; lr < nr; lr += blockDim.x)
      P[c * ldp + lr] = A[(size_t)(k0 + c) * lda + r0 + lr];
  if (threadIdx.x == 0) s_info = 0;
  __syncthreads();
  cl.sync();  // every CTA of the cluster is running before any DSMEM access
  for (int c = 0; c < nb; ++c) {
    const int kc = k0 + c, par = c & 1;
    // 1. local candidate, pushed to every CTA
    T vc[kPanelRPT];
    R best = -1;
    int bidx = INT_MAX;
#pragma unroll
    for (int i = 0; i < kPanelRPT; ++i) {
      const int lr = threadIdx.x + i * kPanelThreads;
      if (lr < nr) {
        vc[i] = P[c * ldp + lr];
        if (r0 + lr >= kc) argmax_merge(best, bidx, cabs1(vc[i]), r0 + lr);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const R v2 = __shfl_xor_sync(0xffffffffu, best, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, bidx, o);
      argmax_merge(best, bidx, v2, i2);
    }
    if (ln == 0) {
      wv[lw] = best;
      wi[lw] = bidx;
    }
    __syncthreads();
    if (lw == 0) {
      R v = ln < nw ? wv[ln] : R(-1);
      int i = ln < nw ? wi[ln] : INT_MAX;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const R v2 = __shfl_xor_sync(0xffffffffu, v, o);
        const int i2 = __shfl_xor_sync(0xffffffffu, i, o);
        argmax_merge(v, i, v2, i2);
      }
      if (ln < C) {
        *cl.map_shared_rank(&sval[par][rank], ln) = v;
        *cl.map_shared_rank(&sidx[par][rank], ln) = i;
      }
      if (i != INT_MAX) {
        const int lr = i - r0;
        const T a0 = P[ln * ldp + lr], a1 = P[(ln + 32) * ldp + lr];
        T* dst = slot + ((size_t)par * kMaxClusterPanel + rank) * kNB;
        for (int q = 0; q < C; ++q) {
          T* d = cl.map_shared_rank(dst, q);
          d[ln] = a0;
          d[ln + 32] = a1;
        }
      }
    } else if (lw == 1 && kc >= r0 && kc < r1) {
      const int lr = kc - r0;
      const T a0 = P[ln * ldp + lr], a1 = P[(ln + 32) * ldp + lr];
      T* dst = krow + (size_t)par * kNB;
      for (int q = 0; q < C; ++q) {
        T* d = cl.map_shared_rank(dst, q);
        d[ln] = a0;
        d[ln + 32] = a1;
      }
    }
    // 2. every candidate and row kc local to every CTA
    cl.sync();
    // 3. pivot (every warp, from local slots), swap, scale, update
    R v = -1;
    int p = INT_MAX, from = 0;
    if (ln < C) {
      v = sval[par][ln];
      p = sidx[par][ln];
      from = ln;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const R v2 = __shfl_xor_sync(0xffffffffu, v, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, p, o);
      const int f2 = __shfl_xor_sync(0xffffffffu, from, o);
      if (v2 > v || (v2 == v && i2 < p)) {
        v = v2;
        p = i2;
        from = f2;
      }
    }
    const bool zero = !(v > 0) || p == INT_MAX || p < kc || p >= n;
    if (threadIdx.x == 0) {
      s_ipiv[c] = zero ? kc : p;
      if (zero && s_info == 0) s_info = kc + 1;
    }
    if (zero) continue;  // LAPACK: no swap and no elimination for a zero pivot
    const T* prow = slot + ((size_t)par * kMaxClusterPanel + from) * kNB;
    const T* kr = krow + (size_t)par * kNB;
    const T inv = crcp(prow[c]);
#pragma unroll
    for (int i = 0; i < kPanelRPT; ++i) {
      const int lr = threadIdx.x + i * kPanelThreads;
      if (lr >= nr) break;
      const int gr = r0 + lr;
      if (gr < kc) continue;
      if (gr == kc) {
        if (p != kc)  // row kc becomes the pivot row
          for (int cc = 0; cc < nb; ++cc) P[cc * ldp + lr] = prow[cc];
        continue;
      }
      T a = vc[i];
      if (gr == p) {  // the pivot row takes row kc
        for (int cc = 0; cc < nb; ++cc) P[cc * ldp + lr] = kr[cc];
        a = kr[c];
      }
      const T l = cmul(a, inv);
      P[c * ldp + lr] = l;
      for (int cc0 = c + 1; cc0 < nb; cc0 += 8) {
        T pv[8], pr[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (cc0 + u < nb) {
            pv[u] = P[(cc0 + u) * ldp + lr];
            pr[u] = prow[cc0 + u];
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (cc0 + u < nb) P[(cc0 + u) * ldp + lr] = cfms(pv[u], l, pr[u]);
      }
    }
  }
  cl.sync();  // no CTA leaves while another may still write its shared memory
  if (rank == 0) {
    for (int c = threadIdx.x; c < nb; c += blockDim.x) ipiv[k0 + c] = s_ipiv[c];
    if (threadIdx.x == 0 && s_info && *info == 0) *info = s_info;
  }
  for (int c = 0; c < nb; ++c)
    for (int lr = threadIdx.x; lr < nr; lr += blockDim.x)
      A[(size_t)(k0 + c) * lda + r0 + lr] = P[c * ldp + lr];
}

// ---- row-resident complex64 panel -------------------------------------------
// Complex64 panels of up to 16 x 416 rows.  Thread t of CTA r owns rows t and
// t + blockDim of its CTA's slice, stored row-major in shared memory (stride
// 66 complex, 16-byte aligned rows) and is the only thread that ever changes
// them.  Row exchanges are done by renaming: each row carries the index
// (label) of the matrix row it currently represents; the pivot search runs
// over (|re|+|im|, label) with ties to the smaller label (izamax order), and
// at column c the pivot row takes label kc while the row labelled kc takes
// the pivot's label - the permutation LAPACK applies with physical swaps, so
// ipiv is the same.  At the end every row is written to the matrix row
// named by its label.
// A candidate is one 64-bit key: the bits of |re|+|im| (non-negative floats
// order like their bit patterns) above (2^23 - 1 - label) and the local row,
// so the arg-max is a plain maximum (one 64-bit shuffle per step).
// Per column: warp maxima and one __syncthreads form the CTA key; warp 0
// stages the candidate row (columns c..63) at a fixed place; one cluster
// barrier; the warps read every CTA's key and staged row (one DSMEM round
// trip) into local shared memory; a second __syncthreads; every warp picks
// the pivot from the local keys, and each thread scales its rows and
// applies the rank-1 update (16-byte shared-memory accesses, eight column
// pairs per batch).  The update streams the CTA's rows through shared
// memory, so the slices are kept short (64 rows per CTA while 16 CTAs
// suffice) and the CTA has one thread per row.
constexpr int kRowsMaxThreads = 256;
constexpr int kRowsRPT = 2;     // rows per thread
constexpr int kRowsLd = 66;     // complex64 per smem row (528 bytes)
constexpr int kRowsMaxRpb = 416;
constexpr int kRowsMinRpb = 64;
constexpr int kLabelBits = 23;  // labels (matrix rows) below 2^23

__host__ __device__ constexpr size_t panel_rows_smem(int rpb) {
  return sizeof(float2) * ((size_t)rpb * kRowsLd + (size_t)(2 + kMaxClusterPanel) * kNB);
}

__device__ __forceinline__ unsigned long long pivot_key(float a, int label, int lr) {
  return ((unsigned long long)__float_as_uint(a) << 32) |
         ((unsigned long long)((1u << kLabelBits) - 1u - (unsigned)label) << 9) | (unsigned)lr;
}

__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long k) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long k2 = __shfl_xor_sync(0xffffffffu, k, o);
    k = k2 > k ? k2 : k;
  }
  return k;
}

__global__ void __launch_bounds__(kRowsMaxThreads, 1)
panel_rows_kernel(float2* __restrict__ A, long long lda, int n, int k0, int nb, int rpb,
                  int* __restrict__ ipiv, int* info) {
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int T = (int)blockDim.x, nw = T >> 5;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* P = reinterpret_cast<float2*>(smem_raw);   // [rpb][kRowsLd]
  float2* cand = P + (size_t)rpb * kRowsLd;           // [2][kNB] this CTA's candidate row
  float2* stage = cand + 2 * kNB;                     // [kMaxClusterPanel][kNB] all candidates
  __shared__ unsigned long long ckey[2];
  __shared__ unsigned long long skey[kMaxClusterPanel];
  __shared__ unsigned long long wkey[kRowsMaxThreads / 32];
  __shared__ int s_ipiv[kNB];  // pivots, written to global memory at the end
  __shared__ int s_info;
  const int lw = threadIdx.x >> 5, ln = threadIdx.x & 31;
  const int r0 = k0 + rank * rpb;
  const int nr = max(min(rpb, n - r0), 0);
  int label[kRowsRPT];
#pragma unroll
  for (int i = 0; i < kRowsRPT; ++i) {
    const int lr = threadIdx.x + i * T;
    label[i] = lr < nr ? r0 + lr : INT_MAX;
  }
  // load: 16 columns of a row in flight per thread
  for (int lr = threadIdx.x; lr < nr; lr += T) {
    const float2* src = A + (size_t)k0 * lda + r0 + lr;
    for (int c0 = 0; c0 < kNB; c0 += 16) {
      float2 v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u)
        v[u] = c0 + u < nb ? src[(size_t)(c0 + u) * lda] : make_float2(0.f, 0.f);
#pragma unroll
      for (int u = 0; u < 16; ++u) P[lr * kRowsLd + c0 + u] = v[u];
    }
  }
  if (threadIdx.x == 0) s_info = 0;
  __syncthreads();
  cl.sync();  // every CTA of the cluster is running before any DSMEM access
  for (int c = 0; c < nb; ++c) {
    const int kc = k0 + c, par = c & 1;
    // 1. CTA candidate key
    unsigned long long key = 0;
    float2 vc[kRowsRPT];
#pragma unroll
    for (int i = 0; i < kRowsRPT; ++i) {
      const int lr = threadIdx.x + i * T;
      vc[i] = make_float2(0.f, 0.f);
      if (label[i] != INT_MAX) {
        vc[i] = P[lr * kRowsLd + c];
        const float a = cabs1(vc[i]);
        if (label[i] >= kc && a >= 0.f) {  // NaN never wins, as in izamax
          const unsigned long long k2 = pivot_key(a, label[i], lr);
          key = k2 > key ? k2 : key;
        }
      }
    }
    key = warp_max_key(key);
    if (ln == 0) wkey[lw] = key;
    __syncthreads();
    // 2. warp 0: the CTA key and its row, staged at a fixed place
    if (lw == 0) {
      key = warp_max_key(ln < nw ? wkey[ln] : 0ull);
      if (key) {
        const float2* src = P + (size_t)(key & 511ull) * kRowsLd;
        if (c + ln < kNB) cand[par * kNB + c + ln] = src[c + ln];
        if (c + 32 + ln < kNB) cand[par * kNB + c + 32 + ln] = src[c + 32 + ln];
      }
      if (ln == 0) ckey[par] = key;
    }
    cl.sync();
    // 3. every CTA's key and staged row into local shared memory
    for (int q = lw; q < C; q += nw) {
      const float2* src = cl.map_shared_rank(cand, q) + par * kNB;
      const unsigned long long kq = *cl.map_shared_rank(&ckey[par], q);
      if (c + ln < kNB) stage[q * kNB + c + ln] = src[c + ln];
      if (c + 32 + ln < kNB) stage[q * kNB + c + 32 + ln] = src[c + 32 + ln];
      if (ln == 0) skey[q] = kq;
    }
    __syncthreads();
    // 4. the pivot (every warp, from local keys)
    const unsigned long long mine = ln < C ? skey[ln] : 0ull;
    const unsigned long long best = warp_max_key(mine);
    const float v = __uint_as_float((unsigned)(best >> 32));
    const int p = (int)((1u << kLabelBits) - 1u - (unsigned)((best >> 9) & ((1u << kLabelBits) - 1u)));
    const bool zero = best == 0ull || !(v > 0.f) || p < kc || p >= n;
    if (threadIdx.x == 0) {
      // no global store inside the loop: the release of the next cluster
      // barrier would wait for it
      s_ipiv[c] = zero ? kc : p;
      if (zero && s_info == 0) s_info = kc + 1;
    }
    if (zero) continue;  // LAPACK neither swaps nor eliminates
    const int q = __ffsll((long long)__ballot_sync(0xffffffffu, mine == best)) - 1;
    const float2* prow = stage + q * kNB;
    const float4* pr4 = reinterpret_cast<const float4*>(prow);
    const float2 inv = crcp(prow[c]);
    const int j0 = c >> 1;
#pragma unroll
    for (int i = 0; i < kRowsRPT; ++i) {
      if (label[i] == p)
        label[i] = kc;
      else if (label[i] == kc)
        label[i] = p;
      if (label[i] <= kc || label[i] == INT_MAX) continue;
      const int lr = threadIdx.x + i * T;
      float4* row = reinterpret_cast<float4*>(P + (size_t)lr * kRowsLd);
      const float2 l = cmul(vc[i], inv);
      {  // the pair holding column c
        const float4 w = row[j0];
        float2 a = make_float2(w.x, w.y), b = make_float2(w.z, w.w);
        if (c & 1) {
          b = l;
        } else {
          a = l;
          b = cfms(b, l, prow[c + 1]);
        }
        row[j0] = make_float4(a.x, a.y, b.x, b.y);
      }
      for (int jb = j0 + 1; jb < kNB / 2; jb += 8) {
        float4 w[8], pq[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (jb + u < kNB / 2) {
            w[u] = row[jb + u];
            pq[u] = pr4[jb + u];
          }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          if (jb + u < kNB / 2) {
            const float2 a = cfms(make_float2(w[u].x, w[u].y), l, make_float2(pq[u].x, pq[u].y));
            const float2 b = cfms(make_float2(w[u].z, w[u].w), l, make_float2(pq[u].z, pq[u].w));
            row[jb + u] = make_float4(a.x, a.y, b.x, b.y);
          }
        }
      }
    }
  }
  cl.sync();  // no CTA leaves while another may still read its shared memory
  if (rank == 0) {
    for (int c = threadIdx.x; c < nb; c += T) ipiv[k0 + c] = s_ipiv[c];
    if (threadIdx.x == 0 && s_info && *info == 0) *info = s_info;
  }
#pragma unroll
  for (int i = 0; i < kRowsRPT; ++i) {
    if (label[i] == INT_MAX) continue;
    const int lr = threadIdx.x + i * T;
    for (int cc = 0; cc < nb; ++cc) A[(size_t)(k0 + cc) * lda + label[i]] = P[lr * kRowsLd + cc];
  }
}

// ---- register-window complex64 panel ----------------------------------------
// Complex64 panels of up to 16 x 256 rows, one thread per row, the row in
// registers.  Columns are processed in sub-blocks of 8: the rank-1 updates of a
// column touch its sub-block only (w, shifted by one per column so that the
// current column is always w[0]), and the columns right of it (R) take the 8
// pivots at once.  Finished columns go to shared memory (Fin).  Rows are
// exchanged by renaming, as in the shared-memory panels (same ipiv).
// Candidates are compared by (bits of |re|+|im|) + 1 (0 = no candidate;
// non-negative floats order like their bits); the lowest label wins a tie.
// Per column: every warp's candidate stages its key, reciprocal and row; after
// one __syncthreads every warp finds the CTA's candidate and sends its share of
// it to the other CTAs with asynchronous stores that count their bytes on the
// receiver's mbarrier; every warp waits there (bounded), picks the pivot and
// updates w.  No cluster barrier: a CTA sends its candidate of column c + 1
// after it has used the ones of column c, so with two buffers (column parity)
// whoever holds all candidates of c + 1 may overwrite those of c.
// Per sub-block: the CTAs that own its pivot rows send them (multipliers and
// right part) to every CTA with bulk copies, one per run of consecutive
// pivots; every CTA solves L11 U = right part for itself and applies U to its
// rows.  Every entry still takes its updates in the order of the columns.
// Bound by the latency of a column's chain: about 330 instructions at two
// clocks each and a one-way exchange of 600.  64 columns of 2048 rows take 66
// us; with rank-1 updates and exchanges of all 64 columns 70 us, with cluster
// barriers instead of asynchronous stores 109 us; in sub-blocks of 16 as long
// for one panel, 2 % longer for many at once.
// lexp (null: none): every CTA leaves the largest exponents of its part of L21's
// columns there (colscale.cuh), read from Fin across its rows: 0.85 us (with a
// warp reduce instruction per column 2.9 us, by a kernel of its own 5 us).
constexpr int kWinMaxRows = 256;
constexpr int kSub = 8;          // columns of a sub-block
constexpr int kSubP = kSub / 2;   // 16-byte words of a candidate

__host__ __device__ constexpr int win_threads(int rpb) {
  return rpb <= 64 ? 64 : (rpb + 31) / 32 * 32;
}
__host__ __device__ constexpr size_t panel_win_smem(int rpb) {
  return sizeof(float2) * (size_t)win_threads(rpb) * kNB +
         sizeof(float4) * (2 * (kWinMaxRows / 32) * (kSubP + 1) + 2 * kMaxClusterPanel * kSubP +
                           2 * kSub * (kNB / 2 + 1));
}

// 1/a = conj(a) / |a|^2 with the components scaled by a power of two near
// 1/max(|re|,|im|): |a|^2 in [1, 8), its reciprocal by Newton's iteration from
// the hardware's approximation.
__device__ __forceinline__ float2 crcp_fast(float2 a) {
  const int e = (__float_as_int(fmaxf(fabsf(a.x), fabsf(a.y))) >> 23) & 0xff;
  const float sc = __int_as_float((254 - min(max(e, 1), 253)) << 23);
  const float ar = a.x * sc, ai = a.y * sc;
  const float d = fmaf(ar, ar, ai * ai);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(r, fmaf(-d, r, 1.f), r) * sc;
  return make_float2(ar * r, -ai * r);
}

__global__ void __launch_bounds__(kWinMaxRows, 1)
panel_win_kernel(float2* __restrict__ A, long long lda, int n, int k0, int nb, int rpb,
                 int* __restrict__ ipiv, int* info, int* status, int* __restrict__ lexp) {
  constexpr int kR = kNB - kSub;
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int T = (int)blockDim.x, nw = T >> 5, lr = (int)threadIdx.x;
  const int lw = lr >> 5, ln = lr & 31;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* Fin = reinterpret_cast<float2*>(smem_raw);     // [kNB][T] finished columns
  float4* cand2 = reinterpret_cast<float4*>(Fin + (size_t)kNB * T);  // [2][warps][key, row]
  float4* stage2 = cand2 + 2 * (kWinMaxRows / 32) * (kSubP + 1);     // [2][kMaxClusterPanel][kSubP]
  float4* prow = stage2 + 2 * kMaxClusterPanel * kSubP;  // [kSub][<= kNB/2 + 1] own pivot rows
  float4* pin = prow + kSub * (kNB / 2 + 1);             // [kSub][<= kNB/2 + 1] all pivot rows
  // by column parity: candidates' keys {value, label, 1/pivot}, the warps'
  // maxima, and the mbarrier that counts the bytes of a column's candidates;
  // mb[2]: the bytes of a sub-block's pivot rows
  __shared__ __align__(16) uint4 skey[2][kMaxClusterPanel];
  __shared__ unsigned wk[2][kWinMaxRows / 32];
  __shared__ float4 s_zero[kSubP];
  __shared__ __align__(8) unsigned long long mb[3];
  __shared__ int s_abort;
  __shared__ unsigned s_own[kNB / kSub];  // pivots of the sub-block held by this CTA
  __shared__ int s_ipiv[kNB];
  __shared__ int s_info;
  __shared__ unsigned char s_exp[kWinMaxRows / 32][kNB];
  const int r0 = k0 + rank * rpb;
  const bool active = lr < max(min(rpb, n - r0), 0);
  unsigned label = active ? (unsigned)(r0 + lr) : 0xffffffffu;
  float2 w[kSub], R[kR];
#pragma unroll
  for (int i = 0; i < kNB; ++i) {
    const float2 a = active && i < nb ? A[(size_t)(k0 + i) * lda + label] : make_float2(0.f, 0.f);
    if (i < kSub)
      w[i < kSub ? i : 0] = a;
    else
      R[i < kSub ? 0 : i - kSub] = a;
  }
  if (lr < kNB / kSub) s_own[lr] = 0u;
  if (lr < kSubP) s_zero[lr] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (lr == 0) {
    s_info = 0;
    s_abort = 0;
    for (int i = 0; i < 3; ++i) tc::mbar_init(&mb[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  __syncthreads();
  cl.sync();  // every CTA of the cluster is running before any DSMEM access
  // a warp sends word pr of the row to CTAs q0, q0 + kTgt nw (two at most: T >= 64)
  constexpr int kTgt = 32 / kSubP;
  const int pr = ln & (kSubP - 1), q0 = kTgt * lw + ln / kSubP, q1 = q0 + kTgt * nw;
  const int qa = min(q0, C - 1), qb = min(q1, C - 1);
  const unsigned ra = tc::map_rank(&stage2[rank * kSubP + pr], qa),
                 ka = tc::map_rank(&skey[0][rank], qa), ba = tc::map_rank(&mb[0], qa),
                 rb = tc::map_rank(&stage2[rank * kSubP + pr], qb),
                 kb = tc::map_rank(&skey[0][rank], qb), bb = tc::map_rank(&mb[0], qb);
  for (int sb = 0; kSub * sb < nb; ++sb) {
    unsigned zmask = 0u;  // columns of the sub-block without a pivot
    const int cend = min(kSub, nb - kSub * sb);
    // the row's key for the current column, and the warp's largest
    auto key_of = [&](unsigned kc) {
      const float a = cabs1(w[0]);
      return (active && label >= kc && a >= 0.f) ? __float_as_uint(a) + 1u : 0u;
    };
    unsigned vb = key_of((unsigned)(k0 + kSub * sb));
    unsigned m = __reduce_max_sync(0xffffffffu, vb);
#pragma unroll 1
    for (int cs = 0; cs < cend; ++cs) {
      const int c = kSub * sb + cs, par = c & 1;
      const unsigned kc = (unsigned)(k0 + c);
      // 1. the warp's candidate (the lowest label where several rows share the
      //    largest key) stages its key and row; without one lane 0 a key of 0
      float4* slots = cand2 + par * (kWinMaxRows / 32) * (kSubP + 1);
      {
        unsigned at = __ballot_sync(0xffffffffu, vb == m);
        if (m && (at & (at - 1))) {
          const unsigned lo = __reduce_min_sync(0xffffffffu, vb == m ? label : 0xffffffffu);
          at = __ballot_sync(0xffffffffu, vb == m && label == lo);
        }
        const float2 rcp = crcp_fast(w[0]);
        if (ln == (m ? __ffs(at) - 1 : 0)) {
          wk[par][lw] = m;
          float4* d = slots + lw * (kSubP + 1);
          *reinterpret_cast<uint4*>(d) =
              make_uint4(m, label, __float_as_uint(rcp.x), __float_as_uint(rcp.y));
#pragma unroll
          for (int i = 0; i < kSubP; ++i)
            d[1 + i] = make_float4(w[2 * i].x, w[2 * i].y, w[2 * i + 1].x, w[2 * i + 1].y);
        }
      }
      __syncthreads();
      // 2. every warp finds the CTA's candidate and sends its share of it
      {
        const unsigned x = ln < nw ? wk[par][ln] : 0u;
        const unsigned xm = __reduce_max_sync(0xffffffffu, x);
        unsigned at = __ballot_sync(0xffffffffu, ln < nw && x == xm);
        if (xm && (at & (at - 1))) {
          const unsigned xl = ((at >> ln) & 1u)
                                  ? reinterpret_cast<const uint4*>(slots + ln * (kSubP + 1))->y
                                  : 0xffffffffu;
          const unsigned lo = __reduce_min_sync(0xffffffffu, xl);
          at = __ballot_sync(0xffffffffu, xl == lo);
        }
        const uint4* d = reinterpret_cast<const uint4*>(slots + (__ffs(at) - 1) * (kSubP + 1));
        const uint4 key = d[0], v = d[1 + pr];
        const unsigned ro = par * kMaxClusterPanel * kSubP * 16u, ko = par * kMaxClusterPanel * 16u,
                       bo = par * 8u;
        if (q0 < C) {
          tc::store_async(ra + ro, v, ba + bo);
          if (pr == 0) tc::store_async(ka + ko, key, ba + bo);
        }
        if (q1 < C) {
          tc::store_async(rb + ro, v, bb + bo);
          if (pr == 0) tc::store_async(kb + ko, key, bb + bo);
        }
      }
      // bytes of the C candidates: the row's part and a key each
      if (lr == 0) tc::mbar_expect_tx(&mb[par], (unsigned)C * 16u * (kSubP + 1));
      // 3. every candidate has arrived
      const bool live = tc::mbar_wait_cluster(&mb[par], (unsigned)(c >> 1) & 1u, &s_abort);
      // 4. the pivot, from the local keys (every warp)
      const unsigned kv = ln < C && live ? skey[par][ln].x : 0u;
      const unsigned bm = __reduce_max_sync(0xffffffffu, kv);
      unsigned at = __ballot_sync(0xffffffffu, ln < C && kv == bm);
      if (bm && (at & (at - 1))) {
        const unsigned kl = ((at >> ln) & 1u) ? skey[par][ln].y : 0xffffffffu;
        const unsigned lo = __reduce_min_sync(0xffffffffu, kl);
        at = __ballot_sync(0xffffffffu, kl == lo);
      }
      const int q = __ffs(at) - 1;
      const uint4 pk = skey[par][q];
      const unsigned p = pk.y;
      // bm == 1: |pivot| = 0; after a wait that gave up nothing is used
      const bool zero = bm <= 1u || p < kc || p >= (unsigned)n;
      if (!zero) label = label == p ? kc : label == kc ? p : label;
      // 5. the update: l = 0 for the rows that are done; the next column's key
      //    as soon as it is there
      const float4* u4 = zero ? s_zero : stage2 + (par * kMaxClusterPanel + q) * kSubP;
      const bool upd = !zero && active && label > kc;
      float2 l = cmul(w[0], make_float2(__uint_as_float(pk.z), __uint_as_float(pk.w)));
      Fin[(size_t)c * T + lr] = upd ? l : w[0];
      l.x = upd ? l.x : 0.f;
      l.y = upd ? l.y : 0.f;
      const float4 u0 = u4[0];
      w[0] = cfms(w[1], l, make_float2(u0.z, u0.w));
      vb = key_of(kc + 1);
      m = __reduce_max_sync(0xffffffffu, vb);
#pragma unroll
      for (int i = 1; i < kSubP; ++i) {
        const float4 u = u4[i];
        w[2 * i - 1] = cfms(w[2 * i], l, make_float2(u.x, u.y));
        w[2 * i] = cfms(w[2 * i + 1], l, make_float2(u.z, u.w));
      }
      zmask |= zero ? 1u << cs : 0u;
      if (lr == 0) {
        s_ipiv[c] = zero ? (int)kc : (int)p;
        if (zero && s_info == 0) s_info = (int)kc + 1;
      }
    }
    const int cr = kSub * (sb + 1);  // first column right of the sub-block
    if (cr >= nb) break;
    // 5. pivot rows to every CTA: the sub-block's columns and those right of it
    const int np = (kNB - kSub * sb) / 2 + 1;                // 16-byte words of a row (odd)
    const int ng = kNB / kSub - 1 - sb;                      // groups of 16 columns right
    const unsigned pj = label - (unsigned)(k0 + kSub * sb);  // pivot of the sub-block if < 16
    if (lr == 0) tc::mbar_expect_tx(&mb[2], (unsigned)(kSub * np * 16));
    if (active && pj < (unsigned)kSub) {
      float4* d = prow + pj * np;
#pragma unroll
      for (int i = 0; i < kSubP; ++i) {
        const float2 x = Fin[(size_t)(kSub * sb + 2 * i) * T + lr],
                     y = Fin[(size_t)(kSub * sb + 2 * i + 1) * T + lr];
        d[i] = make_float4(x.x, x.y, y.x, y.y);
      }
#pragma unroll
      for (int i = 0; i < kR / 2; ++i)
        if (i < ng * kSubP)
          d[kSubP + i] = make_float4(R[2 * i].x, R[2 * i].y, R[2 * i + 1].x, R[2 * i + 1].y);
      atomicOr(&s_own[sb], 1u << pj);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (lw == 0 && ln < C && !*reinterpret_cast<volatile int*>(&s_abort)) {
      unsigned own = s_own[sb];
      while (own) {
        const int j0 = __ffs(own) - 1, len = __ffs(~(own >> j0)) - 1;
        tc::copy_to_rank(tc::map_rank(pin + j0 * np, ln), prow + j0 * np,
                         (unsigned)(len * np * 16), tc::map_rank(&mb[2], ln));
        own &= ~(((1u << len) - 1u) << j0);
      }
    }
    const bool live =
        __all_sync(0xffffffffu, tc::mbar_wait_cluster(&mb[2], (unsigned)sb & 1u, &s_abort));
    // 6. U = L11^{-1} (right part): a thread per column
    if (live && lr < kNB - cr) {
      float2* pf = reinterpret_cast<float2*>(pin) + kSub + lr;
      float2 u[kSub];
#pragma unroll
      for (int i = 0; i < kSub; ++i) u[i] = pf[i * 2 * np];
      const float2* L = reinterpret_cast<const float2*>(pin);
#pragma unroll
      for (int q = 0; q < kSub - 1; ++q)
        if (!((zmask >> q) & 1u)) {
#pragma unroll
          for (int i = q + 1; i < kSub; ++i) u[i] = cfms(u[i], L[i * 2 * np + q], u[q]);
        }
#pragma unroll
      for (int i = 1; i < kSub; ++i) pf[i * 2 * np] = u[i];
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the next copies land here
    }
    __syncthreads();
    // 7. the rows below take U, the pivot rows become U
    if (live && active && label >= (unsigned)(k0 + kSub * sb)) {
      const bool piv = pj < (unsigned)kSub;
      const int q0 = piv ? (int)pj : 0, q1 = piv ? q0 + 1 : kSub;
#pragma unroll 1
      for (int q = q0; q < q1; ++q) {
        if (!piv && ((zmask >> q) & 1u)) continue;
        const float2 l = Fin[(size_t)(kSub * sb + q) * T + lr];
        const float4* u4 = pin + q * np + kSubP;
#pragma unroll
        for (int g = 0; g < kR / kSub; ++g) {
          if (g >= ng) break;
#pragma unroll
          for (int i = 0; i < kSubP; ++i) {
            const float4 u = u4[g * kSubP + i];
            float2& x = R[g * kSub + 2 * i];
            float2& y = R[g * kSub + 2 * i + 1];
            x = piv ? make_float2(u.x, u.y) : cfms(x, l, make_float2(u.x, u.y));
            y = piv ? make_float2(u.z, u.w) : cfms(y, l, make_float2(u.z, u.w));
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kSub; ++i) w[i] = R[i];
#pragma unroll
    for (int i = 0; i < kR - kSub; ++i) R[i] = R[i + kSub];
  }
  cl.sync();  // no CTA leaves while another may still write its shared memory
  if (lr == 0 && s_abort) atomicExch(status, 1);
  if (rank == 0) {
    for (int c = lr; c < nb; c += T) ipiv[k0 + c] = s_ipiv[c];
    if (lr == 0 && s_info && *info == 0) *info = s_info;
  }
  if (active)
    for (int c = 0; c < nb; ++c) A[(size_t)(k0 + c) * lda + label] = Fin[(size_t)c * T + lr];
  if (!lexp) return;
  __syncwarp();
  // this CTA's largest exponent in every column of L21 (nb = 64): lane l reads
  // columns l and l + 32 of its warp's rows, starting at row l (other banks)
  const unsigned below = __ballot_sync(0xffffffffu, active && label >= (unsigned)(k0 + kNB));
  const unsigned mine = __funnelshift_r(below, below, ln);
  float m0 = 0.f, m1 = 0.f;
  const float2* f = Fin + (size_t)ln * T + 32 * lw;
#pragma unroll 16
  for (int i = 0; i < 32; ++i) {
    const float2 a = f[(ln + i) & 31], b = f[32 * T + ((ln + i) & 31)];
    const bool in = (mine >> i) & 1u;
    m0 = in ? fmaxf(m0, fmaxf(fabsf(a.x), fabsf(a.y))) : m0;
    m1 = in ? fmaxf(m1, fmaxf(fabsf(b.x), fabsf(b.y))) : m1;
  }
  s_exp[lw][ln] = (unsigned char)col_expo(m0);
  s_exp[lw][ln + 32] = (unsigned char)col_expo(m1);
  __syncthreads();
  if (lr < kNB) {
    int e = 0;
    for (int k = 0; k < nw; ++k) e = max(e, (int)s_exp[k][lr]);
    lexp[rank * kNB + lr] = e;
  }
}

template <typename K, typename... Args>
static cudaError_t launch_cluster(K kern, int C, int threads, size_t smem, cudaStream_t s,
                                  Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// ---- tournament pivoting for tall complex64 panels --------------------------
// A complex64 panel taller than the register-window cluster holds (16 x 256
// rows) is factored with tournament pivoting (TSLU: Grigori, Demmel and
// Xiang, "CALU: a communication optimal LU factorization algorithm", SIAM J.
// Matrix Anal. Appl. 32, 2011):
//   1. select: G blocks of R rows, one CTA each, run partial pivoting on
//      their own rows in shared memory (no exchange between CTAs) and name
//      the nb rows they pivoted on;
//   2. the G nb candidate rows, with their original values, are gathered and
//      factored with partial pivoting by the register-window cluster kernel:
//      its nb pivot rows are the panel's, its top nb rows are L11 \ U11;
//   3. every other row a of the panel becomes L21 = a U11^{-1} (substitution
//      across the columns, a thread per row), and the panel is written back
//      in pivot order; the pivot sequence is returned as LAPACK row
//      interchanges (ipiv), so the rest of the factorisation is unchanged.
// One exchange between CTAs per panel instead of one per column.  The pivots
// can differ from partial pivoting's (its growth is as small in practice);
// the complex64 factor is the preconditioner of the FP64 refinement, whose
// backward-error test decides the result.
constexpr int kTsluMaxRows = 384;  // rows of one select CTA (one row per thread)
constexpr int kTsluMinRows = 256;
constexpr int kTsluMaxCand = kMaxClusterPanel * kWinMaxRows;  // 4096
constexpr int kTsluFinalCand = 1024;  // capacity of the second candidates' buffer
// candidates left for the final factorisation (a cluster of four CTAs);
// measured on the graded L-shape (N = 16384): LU 127 ms against 140 ms when
// the rounds go on to 256 candidates and one CTA
constexpr int kTsluLastCand = 1024;
constexpr int kTsluMaxH = 64 * kTsluMaxRows;                  // tallest panel (24576)

// Scratch of the tournament, behind the panel exchange slots in
// LuWork::scratch.
struct TsluScratch {
  float2* Cb;    // [kTsluMaxCand][kNB] candidates of rounds 1, 3, ... (original values)
  float2* Cb2;   // [kTsluFinalCand][kNB] candidates of rounds 2, 4, ...
  float2* P;     // [H][kNB] the factored panel
  int* sel;      // [kTsluMaxCand] a round's picks (rows of its input)
  int* mapX;     // [kTsluMaxCand] rows of A of a round's candidates
  int* mapY;     // [kTsluMaxCand] (alternating with mapX)
  int* ipc;      // [kNB] the final candidates' interchanges
  int* infc;     // [1] their first zero pivot
  int* moved;    // [2 kNB + 1] count, then (position, row) pairs beyond the pivots
};
static size_t slots_region() {
  return ((size_t)2 * (kMaxPanelBlocks + 1) * (kSlotHead + sizeof(double2) * kNB) + 511) / 256 *
         256;
}
static size_t tslu_bytes(int n) {
  if (n <= kTsluMaxCand) return 0;
  return sizeof(float2) * (size_t)(kTsluMaxCand + kTsluFinalCand + n) * kNB +
         sizeof(int) * ((size_t)3 * kTsluMaxCand + 4 * kNB + 64) + 2048;
}
static TsluScratch tslu_scratch(void* base, int n) {
  auto al = [](char* q) { return reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(q) + 255) / 256 * 256); };
  char* p = al(static_cast<char*>(base));
  TsluScratch t;
  t.Cb = reinterpret_cast<float2*>(p);
  p = al(p + sizeof(float2) * (size_t)kTsluMaxCand * kNB);
  t.Cb2 = reinterpret_cast<float2*>(p);
  p = al(p + sizeof(float2) * (size_t)kTsluFinalCand * kNB);
  t.P = reinterpret_cast<float2*>(p);
  p = al(p + sizeof(float2) * (size_t)n * kNB);
  t.sel = reinterpret_cast<int*>(p);
  t.mapX = t.sel + kTsluMaxCand;
  t.mapY = t.mapX + kTsluMaxCand;
  t.ipc = t.mapY + kTsluMaxCand;
  t.infc = t.ipc + kNB;
  t.moved = t.infc + 32;
  return t;
}

size_t lu_scratch_bytes(int n) { return slots_region() + tslu_bytes(n); }

// One tournament round: grid G, R threads (one row each, R a multiple of
// 32, at most kTsluMaxRows).  Block b runs partial pivoting on rows r0 ..
// r0 + R - 1 (r0 = k0 + b R) of columns k0 .. k0 + nb - 1 and writes the
// rows it pivoted on (absolute indices) to cand[b nb + c], -1 for steps not
// taken.  Columns in sub-blocks of 8 as in the register-window panel: per
// column the warps' candidates stage their key and row, one barrier, every
// warp picks the block's best and updates the sub-block's columns; after a
// sub-block the columns right of it take its pivots at once.  64 columns of 256
// rows take 42 us; with rank-1 updates of all 64 columns 67 us.
__global__ void __launch_bounds__(kTsluMaxRows, 1)
tslu_select_kernel(const float2* __restrict__ A, long long lda, int n, int k0, int nb, int R,
                   int* __restrict__ cand) {
  constexpr int kW = kTsluMaxRows / 32, kR = kNB - kSub;
  __shared__ __align__(16) float4 slots[2][kW][kSubP + 1];  // by column parity: key, row
  __shared__ unsigned wk[2][kW];
  __shared__ float2 Ls[kSub][kTsluMaxRows];                 // the sub-block's multipliers
  __shared__ __align__(16) float4 pin[kSub][kNB / 2 + 1];   // its pivot rows
  const int t = threadIdx.x, ln = t & 31, lw = t >> 5, nw = (int)blockDim.x >> 5;
  const int r0 = k0 + blockIdx.x * R;
  const int nr = max(0, min(R, n - r0));
  bool active = t < nr;
  float2 w[kSub], Rt[kR];
#pragma unroll
  for (int i = 0; i < kNB; ++i) {
    const float2 a =
        active && i < nb ? A[(size_t)(k0 + i) * lda + r0 + t] : make_float2(0.f, 0.f);
    if (i < kSub)
      w[i < kSub ? i : 0] = a;
    else
      Rt[i < kSub ? 0 : i - kSub] = a;
  }
  int* out = cand + (size_t)blockIdx.x * nb;
  const int npiv = min(nb, nr);  // a row is left at each of these steps
  // bits of |re| + |im| plus one (non-negative floats order like their bits; 0
  // = not a candidate, NaN counts as zero); among equals the smallest row,
  // which is the lowest lane of the lowest warp (LAPACK's izamax)
  auto key_of = [&]() {
    float v = cabs1(w[0]);
    if (!(v >= 0.f)) v = 0.f;
    return active ? __float_as_uint(v) + 1u : 0u;
  };
  for (int sb = 0; kSub * sb < npiv; ++sb) {
    unsigned zmask = 0u;
    int pj = -1;  // step of the sub-block that picked this row
    const int cend = min(kSub, npiv - kSub * sb);
    unsigned vb = key_of();
    unsigned m = __reduce_max_sync(0xffffffffu, vb);
#pragma unroll 1
    for (int cs = 0; cs < cend; ++cs) {
      const int par = cs & 1;
      const unsigned at = __ballot_sync(0xffffffffu, vb == m);
      const float2 rcp = crcp_fast(w[0]);
      if (ln == __ffs(at) - 1) {  // the warp's candidate stages its key and row
        wk[par][lw] = m;
        float4* d = slots[par][lw];
        d[0] = make_float4(__uint_as_float(m), __int_as_float(t), rcp.x, rcp.y);
#pragma unroll
        for (int i = 0; i < kSubP; ++i)
          d[1 + i] = make_float4(w[2 * i].x, w[2 * i].y, w[2 * i + 1].x, w[2 * i + 1].y);
      }
      __syncthreads();
      const unsigned x = ln < nw ? wk[par][ln] : 0u;
      const unsigned bm = __reduce_max_sync(0xffffffffu, x);
      const unsigned aw = __ballot_sync(0xffffffffu, ln < nw && x == bm);
      const float4* u4 = slots[par][__ffs(aw) - 1];
      const float4 key = u4[0];
      if (t == __float_as_int(key.y)) {
        out[kSub * sb + cs] = r0 + t;
        active = false;  // the pivot row is not updated from here on
        pj = cs;
      }
      const bool upd = active && bm > 1u;  // bm == 1: a zero column
      float2 l = cmul(w[0], make_float2(key.z, key.w));
      l.x = upd ? l.x : 0.f;
      l.y = upd ? l.y : 0.f;
      Ls[cs][t] = l;
      const float4 u0 = u4[1];
      w[0] = cfms(w[1], l, make_float2(u0.z, u0.w));
      vb = key_of();
      m = __reduce_max_sync(0xffffffffu, vb);
#pragma unroll
      for (int i = 1; i < kSubP; ++i) {
        const float4 u = u4[1 + i];
        w[2 * i - 1] = cfms(w[2 * i], l, make_float2(u.x, u.y));
        w[2 * i] = cfms(w[2 * i + 1], l, make_float2(u.z, u.w));
      }
      zmask |= bm > 1u ? 0u : 1u << cs;
    }
    if (kSub * (sb + 1) >= npiv) break;
    // the pivot rows' multipliers and right parts, U = L11^{-1} (right parts),
    // then the rows left take U
    const int np = (kNB - kSub * (sb + 1)) / 2;  // 16-byte words right of the sub-block
    if (pj >= 0) {
      float4* d = pin[pj];
#pragma unroll
      for (int i = 0; i < kSubP; ++i) {
        const float2 x = Ls[2 * i][t], y = Ls[2 * i + 1][t];
        d[i] = make_float4(x.x, x.y, y.x, y.y);
      }
#pragma unroll
      for (int i = 0; i < kR / 2; ++i)
        if (i < np)
          d[kSubP + i] = make_float4(Rt[2 * i].x, Rt[2 * i].y, Rt[2 * i + 1].x, Rt[2 * i + 1].y);
    }
    __syncthreads();
    for (int c = t; c < 2 * np; c += blockDim.x) {
      float2 u[kSub];
#pragma unroll
      for (int i = 0; i < kSub; ++i) u[i] = reinterpret_cast<const float2*>(pin[i])[kSub + c];
#pragma unroll
      for (int q = 0; q < kSub - 1; ++q)
#pragma unroll
        for (int i = q + 1; i < kSub; ++i)
          u[i] = cfms(u[i], reinterpret_cast<const float2*>(pin[i])[q], u[q]);
#pragma unroll
      for (int i = 1; i < kSub; ++i) reinterpret_cast<float2*>(pin[i])[kSub + c] = u[i];
    }
    __syncthreads();
    if (active) {
#pragma unroll 1
      for (int q = 0; q < kSub; ++q) {
        if ((zmask >> q) & 1u) continue;
        const float2 l = Ls[q][t];
        const float4* u4 = pin[q] + kSubP;
#pragma unroll
        for (int g = 0; g < kR / kSub; ++g) {
          if (g * kSubP >= np) break;
#pragma unroll
          for (int i = 0; i < kSubP; ++i) {
            const float4 u = u4[g * kSubP + i];
            float2& x = Rt[g * kSub + 2 * i];
            float2& y = Rt[g * kSub + 2 * i + 1];
            x = cfms(x, l, make_float2(u.x, u.y));
            y = cfms(y, l, make_float2(u.z, u.w));
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kSub; ++i) w[i] = Rt[i];
#pragma unroll
    for (int i = 0; i < kR - kSub; ++i) Rt[i] = Rt[i + kSub];
  }
  for (int j = npiv + t; j < nb; j += blockDim.x) out[j] = -1;  // steps not taken
}

// Cb (Gc x nb, column-major, ld Gc) = rows src[j] of S (column-major, ld
// lds; zero rows for -1); optionally map[j] = idx[src[j]].
// grid (ceil(Gc / 256), nb), 256 threads.
__global__ void tslu_gather_kernel(const float2* __restrict__ S, long long lds, int k0, int nb,
                                   const int* __restrict__ src, int Gc, float2* __restrict__ Cb,
                                   const int* __restrict__ idx, int* __restrict__ map) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
  if (j >= Gc || c >= nb) return;
  const int r = src[j];
  Cb[(size_t)c * Gc + j] = r >= 0 ? S[(size_t)(k0 + c) * lds + r] : make_float2(0.f, 0.f);
  if (map && c == 0) map[j] = (r >= 0 && idx) ? idx[r] : r;
}

// The panel's interchanges from the final candidates' factorisation (ipc,
// infc): ipiv[k0 + c] (LAPACK), and the rows that end beyond the pivots at
// positions other than their own: moved[0] = count, then (position, row)
// pairs.  Positions relative to k0 live in shared memory (2 H ints).  One
// CTA of 1024 threads.  lexp (null: none): set to zero, for tslu_rows_kernel.
__global__ void __launch_bounds__(1024)
tslu_perm_kernel(int n, int k0, int nb, const int* __restrict__ candF, int Gc,
                 const int* __restrict__ ipc, const int* __restrict__ infc, int* __restrict__ ipiv,
                 int* info, int* __restrict__ moved, int* __restrict__ lexp) {
  extern __shared__ int sh[];
  const int H = n - k0;
  static_assert(kColParts * kNB == 1024, "");
  if (lexp) lexp[threadIdx.x] = 0;
  int* pos = sh;       // [H] position of row k0 + i
  int* at = sh + H;    // [H] row at position k0 + i
  __shared__ int cw[kTsluMaxCand];
  __shared__ int sp[kNB], ic[kNB], m;  // the panel's pivots, the candidates' pivots, moved rows
  if (threadIdx.x < nb) ic[threadIdx.x] = ipc[threadIdx.x];
  if (threadIdx.x == 0) m = 0;
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    pos[i] = i;
    at[i] = i;
  }
  Gc = min(Gc, kTsluMaxCand);  // the caller passes at most kTsluMaxCand
  for (int j = threadIdx.x; j < Gc; j += blockDim.x) cw[j] = candF[j];
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int c = 0; c < nb; ++c) {  // the candidates' interchanges: cw[c] = pivot row c
      const int q = ic[c];
      if (q != c && q >= 0 && q < Gc) {
        const int tmp = cw[c];
        cw[c] = cw[q];
        cw[q] = tmp;
      }
    }
    for (int c = 0; c < nb; ++c) {
      const int r = cw[c] - k0;
      if (r < 0 || r >= H) {  // a zero column: no interchange (info is set)
        sp[c] = c;
        continue;
      }
      const int p = pos[r], rt = at[c];
      sp[c] = p;
      at[p] = rt;
      pos[rt] = p;
      at[c] = r;
      pos[r] = c;
    }
    if (*infc && *info == 0) *info = k0 + *infc;
  }
  __syncthreads();
  // a thread per step: its pivot, and the row that an interchange left at the
  // pivot's position (listed once, by the first step that names it)
  if (threadIdx.x < nb) {
    const int c = threadIdx.x, p = sp[c];
    ipiv[k0 + c] = k0 + p;
    bool first = p >= nb && at[p] != p;
    for (int u = 0; u < c; ++u) first &= sp[u] != p;
    if (first) {
      const int j = atomicAdd(&m, 1);
      moved[1 + 2 * j] = k0 + p;
      moved[2 + 2 * j] = k0 + at[p];
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) moved[0] = m;
}

// P (H x nb, column-major, ld H = n - k0): the factored panel in its final
// row order.  Positions k0 .. k0 + nb - 1: rows 0 .. nb - 1 of the
// candidates' factor (L11 \ U11, Cf: ld Gc); position i beyond: the row r
// there (i itself unless listed in `moved`), x U11 = A(r, :) solved for x =
// L21(i).  A thread per position, the row in registers; columns in sub-blocks of
// 8 as in the panels: the sub-block's triangle, then the columns right of it.
// FP32 issue bounds it (2016 complex multiply-subtracts per row); 16384 x 64 take
// 22 us, as a warp per row with lanes on columns (a shuffle per column, strided
// loads) 41 us.  lexp (null: none): the largest exponents of L21's columns, CTA b
// adds its rows' to part b % kColParts.
constexpr int kRowsCta = 128, kULd = kNB + 2;
__global__ void __launch_bounds__(kRowsCta)
tslu_rows_kernel(const float2* __restrict__ A, long long lda, int n, int k0, int nb,
                 const float2* __restrict__ Cf, int Gc, const int* __restrict__ moved,
                 float2* __restrict__ P, int* __restrict__ lexp) {
  constexpr int kR = kNB - kSub;
  __shared__ __align__(16) float2 U[kNB][kULd];  // row c of U11
  __shared__ float2 dv[kNB];
  __shared__ float2 Xs[kSub][kRowsCta];
  __shared__ int src[kRowsCta];
  const int t = threadIdx.x, H = n - k0, i = blockIdx.x * kRowsCta + t;
  src[t] = k0 + min(i, H - 1);  // beyond H: the last row once more, not stored
  for (int e = t; e < kNB * kNB; e += kRowsCta) {
    const int c = e / kNB, r = e - c * kNB;  // coalesced: consecutive rows of column c
    U[r][c] = c < nb && r < nb ? Cf[(size_t)c * Gc + r] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  for (int c = t; c < kNB; c += kRowsCta) {
    const float2 d = U[c][c];
    dv[c] = (d.x != 0.f || d.y != 0.f) ? crcp(d) : make_float2(0.f, 0.f);
  }
  for (int u = t; u < moved[0]; u += kRowsCta) {  // the rows moved to positions of this CTA
    const int q = moved[1 + 2 * u] - k0 - blockIdx.x * kRowsCta;
    if (q >= 0 && q < kRowsCta) src[q] = moved[2 + 2 * u];
  }
  __syncthreads();
  if (i < nb) {
    for (int c = 0; c < nb; ++c) P[(size_t)c * H + i] = Cf[(size_t)c * Gc + i];
    return;
  }
  int* my = lexp ? lexp + (blockIdx.x % kColParts) * kNB : nullptr;
  const float2* row = A + (size_t)k0 * lda + src[t];
  float2 w[kSub], R[kR];
#pragma unroll
  for (int c = 0; c < kNB; ++c) {
    const float2 a = c < nb ? row[(size_t)c * lda] : make_float2(0.f, 0.f);
    if (c < kSub)
      w[c < kSub ? c : 0] = a;
    else
      R[c < kSub ? 0 : c - kSub] = a;
  }
#pragma unroll 1
  for (int c0 = 0; c0 < nb; c0 += kSub) {
#pragma unroll
    for (int q = 0; q < kSub; ++q) {
      const float2 x = cmul(w[q], dv[c0 + q]);
      w[q] = x;
      Xs[q][t] = x;
#pragma unroll
      for (int j = q + 1; j < kSub; ++j) w[j] = cfms(w[j], x, U[c0 + q][c0 + j]);
    }
#pragma unroll
    for (int q = 0; q < kSub; ++q)
      if (c0 + q < nb && i < H) P[(size_t)(c0 + q) * H + i] = w[q];
    if (my) {  // (nb = 64: whole warps) four lanes per column, 8 of the warp's rows each
      __syncwarp();
      const int l = t & 31, q = l >> 2, r0 = t - l + 8 * (l & 3);
      float m = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) {  // starting at row q: other banks
        const float2 v = Xs[q][r0 + ((r + q) & 7)];
        m = fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y)));
      }
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
      if ((l & 3) == 0) atomicMax(&my[c0 + q], col_expo(m));
      __syncwarp();
    }
    const int ng = (kNB - c0) / kSub - 1;  // groups of 8 columns right
#pragma unroll 1
    for (int q = 0; q < kSub; ++q) {
      const float2 x = Xs[q][t];
      const float4* u4 = reinterpret_cast<const float4*>(&U[c0 + q][c0 + kSub]);
#pragma unroll
      for (int g = 0; g < kR / kSub; ++g) {
        if (g >= ng) break;
#pragma unroll
        for (int j = 0; j < kSubP; ++j) {
          const float4 u = u4[g * kSubP + j];
          R[g * kSub + 2 * j] = cfms(R[g * kSub + 2 * j], x, make_float2(u.x, u.y));
          R[g * kSub + 2 * j + 1] = cfms(R[g * kSub + 2 * j + 1], x, make_float2(u.z, u.w));
        }
      }
    }
#pragma unroll
    for (int j = 0; j < kSub; ++j) w[j] = R[j];
#pragma unroll
    for (int j = 0; j < kR - kSub; ++j) R[j] = R[j + kSub];
  }
}

// Tournament-pivoted panel of columns k0 .. k0 + nb - 1 (rows k0 .. n - 1).
// false: not applicable (taller than the tournament holds, scratch too
// small, or the cluster launch refused); A and ipiv are then untouched.
// lexp (null: none): kColParts partial maxima of the exponents of L21's columns.
static bool tslu_panel(float2* A, long long lda, int n, int k0, int nb, const LuWork& w, int cmax,
                       int* lexp, cudaStream_t s, long long* launches) {
  const int H = n - k0;
  if (H > kTsluMaxH || tslu_bytes(n) == 0 ||
      w.scratch_bytes < slots_region() + tslu_bytes(n))
    return false;
  const int gmax = kTsluMaxCand / nb;
  const int R0 = std::max(kTsluMinRows, ((H + gmax - 1) / gmax + 31) / 32 * 32);
  if (R0 > kTsluMaxRows) return false;
  const TsluScratch ts = tslu_scratch(static_cast<char*>(w.scratch) + slots_region(), n);
  // rounds: blocks of the current candidates (the panel's rows first), one
  // CTA each, until at most kTsluLastCand are left; a launch the GPU refuses
  // leaves the panel to the other kernels (A is only read until the end)
  const float2* src = A;
  long long lds = lda;
  int koff = k0, rows = H, round = 0, R = R0;
  int* mapPrev = nullptr;
  int* mapNext = ts.mapX;
  float2* Cf = ts.Cb;
  int Gf = 0;
  cudaGetLastError();
  for (;;) {
    const int G = (rows + R - 1) / R;
    Gf = G * nb;
    Cf = (round & 1) ? ts.Cb2 : ts.Cb;
    if (Gf > ((round & 1) ? kTsluFinalCand : kTsluMaxCand)) return false;
    tslu_select_kernel<<<G, R, 0, s>>>(src, lds, koff + rows, koff, nb, R, ts.sel);
    if (cudaGetLastError() != cudaSuccess) return false;
    tslu_gather_kernel<<<dim3((Gf + 255) / 256, nb), 256, 0, s>>>(src, lds, koff, nb, ts.sel, Gf,
                                                                  Cf, mapPrev, mapNext);
    *launches += 2;
    if (Gf <= kTsluLastCand || G == 1) break;
    src = Cf;
    lds = Gf;
    koff = 0;
    rows = Gf;
    R = kTsluMinRows;
    mapPrev = mapNext;
    mapNext = (mapNext == ts.mapX) ? ts.mapY : ts.mapX;
    ++round;
  }
  const int* candF = mapNext;
  const int ld = Gf;
  if (Gf > kTsluMaxCand || sizeof(int) * (2 * (size_t)H + kTsluMaxCand) > 220 * 1024)
    return false;  // the permutation kernel's shared memory
  // the final candidates: partial pivoting in one cluster (one CTA for up to
  // 256 rows)
  int C = std::max(1, (Gf + kWinMaxRows - 1) / kWinMaxRows);
  if (C > cmax) return false;
  const int rpb = (Gf + C - 1) / C;
  const int threads = win_threads(rpb);
  cudaMemsetAsync(ts.infc, 0, sizeof(int), s);
  if (launch_cluster(panel_win_kernel, C, threads, panel_win_smem(rpb), s, Cf, (long long)ld, Gf,
                     0, nb, rpb, ts.ipc, ts.infc, w.status, (int*)nullptr) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  tslu_perm_kernel<<<1, 1024, sizeof(int) * 2 * (size_t)H, s>>>(n, k0, nb, candF, Gf, ts.ipc,
                                                                ts.infc, w.ipiv, w.info, ts.moved,
                                                                 lexp);
  tslu_rows_kernel<<<(H + kRowsCta - 1) / kRowsCta, kRowsCta, 0, s>>>(A, lda, n, k0, nb, Cf, ld,
                                                                      ts.moved, ts.P, lexp);
  cudaMemcpy2DAsync(A + (size_t)k0 * lda + k0, sizeof(float2) * lda, ts.P, sizeof(float2) * H,
                    sizeof(float2) * H, nb, cudaMemcpyDeviceToDevice, s);
  *launches += 2;  // + the cluster launch the caller counts
  return true;
}

constexpr int kMaxCluster = 16;
constexpr size_t kClusterSmem = 220 * 1024;

template <typename T>
static size_t panel_cluster_smem(int rpb) {
  return sizeof(T) * PanelSmem<T>::total(rpb | 1);
}

// Row permutation of the pivots: perm[i] = the original row that ends at i.
// A thread per i follows its position back through the swaps; swap s moves the
// positions s and ipiv[s] >= s only, so it starts at s = i.  2048 rows: 76 us as
// n swaps in a row by one thread, 24 us.
constexpr int kPermThreads = 64, kPermTile = 1024;
__global__ void __launch_bounds__(kPermThreads)
perm_kernel(int n, const int* __restrict__ ipiv, int* __restrict__ perm) {
  __shared__ __align__(16) int ip[kPermTile];
  const int i = blockIdx.x * kPermThreads + threadIdx.x;
  const int last = min(n, (int)(blockIdx.x + 1) * kPermThreads) - 1;
  int x = i;
  for (int t0 = last / kPermTile * kPermTile; t0 >= 0; t0 -= kPermTile) {
    __syncthreads();
    for (int v = threadIdx.x; v < kPermTile; v += kPermThreads)
      ip[v] = t0 + v <= last ? ipiv[t0 + v] : t0 + v;
    __syncthreads();
    for (int v = min(kPermTile, last - t0 + 4) / 4 * 4 - 4; v >= 0; v -= 4) {
      const int4 p = *reinterpret_cast<const int4*>(ip + v);
      const int s = t0 + v;
      x = x == s + 3 ? p.w : x == p.w ? s + 3 : x;
      x = x == s + 2 ? p.z : x == p.z ? s + 2 : x;
      x = x == s + 1 ? p.y : x == p.y ? s + 1 : x;
      x = x == s ? p.x : x == p.x ? s : x;
    }
  }
  if (i < n) perm[i] = x;
}

// X = L^{-1} X for a unit lower 64 x 64 L in shared memory (column-major, zero
// on and above the diagonal) and 8 columns, one CTA of 16 warps: lane (g, c),
// c = lane % 8, of warp w holds row 4 w + g of column c in x.  Block b of 4
// rows is solved inside warp b (3 shuffle steps), its rows go to X, and after
// one barrier every warp below subtracts 4 products.  Bound by the FP64
// pipe: a warp instruction takes 64 clocks of a scheduler, so the 8-column
// tiles are there to spread the 2,112 instructions of a tile over all SMs.
constexpr int kTriThreads = 512;
template <typename T>
__device__ __forceinline__ T tri64_solve(const T* L, T* X, T x) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = lane & 7, r = 4 * w + (lane >> 3);
  for (int b = 0; b < 16; ++b) {
    if (w == b) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        T xi;
        xi.x = __shfl_sync(0xffffffffu, x.x, 8 * i + c);
        xi.y = __shfl_sync(0xffffffffu, x.y, 8 * i + c);
        x = cfms(x, L[(4 * b + i) * kNB + r], xi);  // zero for rows above
      }
      X[r * 8 + c] = x;
    }
    __syncthreads();
    if (w > b) {
#pragma unroll
      for (int i = 0; i < 4; ++i) x = cfms(x, L[(4 * b + i) * kNB + r], X[(4 * b + i) * 8 + c]);
    }
  }
  return x;
}

template <typename T>
constexpr size_t tri64_smem() {
  return sizeof(T) * (kNB * kNB + kNB * 8 + kNB);
}

// Complex128 U12 = L11^{-1} A12, 8 columns per CTA (kite N =
// 2048, all panels: 3.4 ms with 32 columns per CTA on at most 64 SMs, 1.1 ms).
__global__ void __launch_bounds__(kTriThreads)
trsm8_kernel(double2* __restrict__ A, long long lda, int k0, int nb, int c0, int ncols) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* L = reinterpret_cast<double2*>(smem_raw);
  double2* X = L + kNB * kNB;
  for (int v = threadIdx.x; v < kNB * kNB; v += kTriThreads) {
    const int s = v >> 6, r = v & 63;
    L[v] = s < r && r < nb ? A[(size_t)(k0 + s) * lda + k0 + r] : make_double2(0.0, 0.0);
  }
  const int lane = threadIdx.x & 31, r = 4 * (threadIdx.x >> 5) + (lane >> 3);
  const int j = blockIdx.x * 8 + (lane & 7);
  const bool in = j < ncols && r < nb;
  double2* p = A + (size_t)(c0 + j) * lda + k0 + r;
  double2 x = in ? *p : make_double2(0.0, 0.0);
  __syncthreads();
  x = tri64_solve(L, X, x);
  if (in) *p = x;
}

// Inverses of the diagonal blocks: dinv[(2 k) * 64 * 64 ...] = L_kk^{-1}
// (unit lower), dinv[(2 k + 1) * 64 * 64 ...] = U_kk^{-1}; column-major 64 x 64.
// blockIdx.y: 8 columns of L^{-1} (0-7) or U^{-1} (8-15) by the same solve on
// columns of the identity; U read backwards (row and column order reversed,
// rows divided by their pivots) is unit lower too.  (kite N = 2048, complex128:
// 420 us with one thread per column, 92 us.)
template <typename T>
__global__ void __launch_bounds__(kTriThreads)
dinv_kernel(const T* __restrict__ LU, long long lda, int n, T* __restrict__ dinv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* L = reinterpret_cast<T*>(smem_raw);
  T* X = L + kNB * kNB;
  T* iv = X + kNB * 8;
  const int k0 = blockIdx.x * kNB, nb = min(kNB, n - k0);
  const bool up = blockIdx.y >= 8;
  const T zero = CTraits<T>::make(0, 0);
  const T* D = LU + (size_t)k0 * lda + k0;
  if (threadIdx.x < kNB) {
    const int d = nb - 1 - (int)threadIdx.x;
    iv[threadIdx.x] = up && d >= 0 ? crcp(D[(size_t)d * lda + d]) : CTraits<T>::make(1, 0);
  }
  __syncthreads();
  for (int v = threadIdx.x; v < kNB * kNB; v += kTriThreads) {
    const int s = v >> 6, r = v & 63;
    T l = zero;
    if (s < r && r < nb)
      l = up ? cmul(D[(size_t)(nb - 1 - s) * lda + nb - 1 - r], iv[r]) : D[(size_t)s * lda + r];
    L[v] = l;
  }
  const int lane = threadIdx.x & 31, r = 4 * (threadIdx.x >> 5) + (lane >> 3);
  const int j = (blockIdx.y & 7) * 8 + (lane & 7);
  T x = zero;
  if (j < nb && r == (up ? nb - 1 - j : j)) x = iv[r];
  __syncthreads();
  x = tri64_solve(L, X, x);
  T* out = dinv + (size_t)(2 * blockIdx.x + (up ? 1 : 0)) * kNB * kNB + (size_t)j * kNB;
  if (r < nb)
    out[up ? nb - 1 - r : r] = x;
  else
    out[r] = zero;
}

size_t lu_pack_bytes(int n, size_t elem) {
  return elem == sizeof(double2) ? oz_pack_bytes(n, n)
                                 : tc_pack_bytes(n, n, n >= kOuterMinN ? kOuterNB : kNB);
}

// SMs left to the panels while a look-ahead update runs beside them: one for each
// CTA of the tournament's first round (L-shape N = 16384: 141.4 ms with 40, 138.7
// with 64, 139.5 with 80; N = 8192 the same with all three)
constexpr int kLookaheadFreeSMs = 64;
#ifndef BEM2D_LOOKAHEAD_MIN_N
#define BEM2D_LOOKAHEAD_MIN_N 8192
#endif
bool lu_lookahead(int n) { return n >= BEM2D_LOOKAHEAD_MIN_N; }
int lu_lookahead_ctas() {
  return std::max(1, device_sms() - kLookaheadFreeSMs);
}

size_t lu_aux_bytes(int n, size_t elem) {
  const size_t nk = (n + kNB - 1) / kNB;
  return sizeof(int) * (size_t)n + 2 * nk * kNB * kNB * elem + 256;
}

// Updates large enough for the tensor cores on their own account: at least
// kTensorMinN rows and columns, or tall and narrow ones (the columns inside an
// outer block), or short wide ones (the rows of an outer block right of it).
static bool tensor_sized(int M, int N) {
  return (M >= kTensorMinN && N >= kTensorMinN) || (M >= 4 * kTensorMinN && N >= kNB) ||
         (N >= 4 * kTensorMinN && M >= kNB);
}

// C -= Am Bm (M x N, inner dimension K; all three column-major with leading
// dimension ld inside the matrix being factored).  complex64 updates of at
// least kTensorMinN rows and columns run on the tensor cores, the rest on the
// CUDA cores in slices of K = 64.
// part, np: as for launch_tc_cgemm_sub.
template <typename T>
static int update_sub(T* C, const T* Am, const T* Bm, long long ld, int M, int N, int K,
                      const LuWork& w, cudaStream_t s, long long* launches,
                      const int* part = nullptr, int np = 0) {
  if (M <= 0 || N <= 0 || K <= 0) return BEM2D_OK;
  if constexpr (sizeof(T) == sizeof(double2)) {
    if (w.pack && oz_pack_bytes(M, N) <= w.pack_bytes)
      return launch_oz_zgemm(C, ld, Am, ld, Bm, ld, M, N, K, 1, -1.0, w.pack, w.pack_bytes,
                             w.status, s, launches);
  }
  if constexpr (sizeof(T) == sizeof(float2)) {
    if (tensor_sized(M, N)) {
      ++*launches;
      if (w.pack && tc_pack_bytes(M, N, K) <= w.pack_bytes) {
        *launches += part ? 1 : 2;  // + the packing kernel and the one for its scales
        return launch_tc_cgemm_sub(reinterpret_cast<float2*>(C), ld,
                                   reinterpret_cast<const float2*>(Am), ld,
                                   reinterpret_cast<const float2*>(Bm), ld, M, N, K, w.pack,
                                   w.pack_bytes, w.status, s, w.tc_ctas, w.tc_passes, part, np)
                   ? BEM2D_ERR_CUDA
                   : BEM2D_OK;
      }
      --*launches;
    }
  }
  dim3 g((M + kGB - 1) / kGB, (N + kGB - 1) / kGB);
  for (int k = 0; k < K; k += kNB) {
    gemm_sub_kernel<T><<<g, 256, sizeof(T) * 2 * kNB * kGB, s>>>(
        Am + (size_t)k * ld, ld, Bm + k, ld, C, ld, M, N, std::min(kNB, K - k));
    ++*launches;
  }
  return BEM2D_OK;
}

template <typename T>
static void trsm_rows(T* A, long long lda, int k0, int nb, int c0, int nc, cudaStream_t s,
                      long long* launches) {
  if (nc <= 0) return;
  ++*launches;
  if constexpr (sizeof(T) == sizeof(double2)) {
    trsm8_kernel<<<(nc + 7) / 8, kTriThreads, tri64_smem<T>(), s>>>(A, lda, k0, nb, c0, nc);
  } else {
    trsm_kernel<T><<<(nc + 31) / 32, 256, sizeof(T) * (kNB * kNB + kNB * 32), s>>>(A, lda, k0, nb,
                                                                                  c0, nc);
  }
}

template <typename T>
int lu_factor(T* A, long long lda, int n, const LuWork& w, cudaStream_t s,
              long long* launches) {
  PanelSlots<T> sl;
  sl.base = static_cast<char*>(w.scratch);
  cudaMemsetAsync(w.info, 0, sizeof(int), s);
  cudaMemsetAsync(w.status, 0, sizeof(int), s);
  cudaMemsetAsync(sl.base, 0, slots_bytes(sizeof(T)), s);
  // one-time function attributes; thread-safe (workers of a sweep factor
  // concurrently from several host threads)
  static PerDevice<bool> c16(true);
  static PerDeviceOnce attr;
  const int dev = current_device();
  std::atomic<bool>& cluster16 = c16[dev];
  attr(dev, [&] {
    cudaFuncSetAttribute(panel_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(panel_cluster_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kClusterSmem);
    cudaFuncSetAttribute(panel_win_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaFuncSetAttribute(panel_win_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)panel_win_smem(kWinMaxRows));
    cudaFuncSetAttribute(panel_rows_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaFuncSetAttribute(panel_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)panel_rows_smem(kRowsMaxRpb));
    if (cudaFuncSetAttribute(panel_cluster_kernel<T>,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      cluster16 = false;
    }
    if constexpr (sizeof(T) == sizeof(float2))
      cudaFuncSetAttribute(trsm_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(sizeof(T) * (kNB * kNB + kNB * 32)));
    cudaFuncSetAttribute(gemm_sub_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(sizeof(T) * 2 * kNB * kGB));
    cudaFuncSetAttribute(dinv_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)tri64_smem<T>());
    cudaFuncSetAttribute(trsm8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)tri64_smem<double2>());
    cudaFuncSetAttribute(tslu_perm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(sizeof(int) * 2 * kTsluMaxH));
  });
  // complex64 matrices are factored in outer blocks of kOuterNB columns:
  // inside a block each 64-column panel updates only the block's columns;
  // the columns right of the block receive one rank-kOuterNB update (K =
  // kOuterNB on the tensor cores), which reads and writes the trailing
  // matrix once per block instead of once per panel.
  const int outer = (sizeof(T) == sizeof(float2) && n >= kOuterMinN) ? kOuterNB : kNB;
  // look-ahead (complex64, from BEM2D_LOOKAHEAD_MIN_N on; a block is an
  // outer block, or a single panel below kOuterMinN): block b's update of the columns
  // beyond block b + 1 runs on w.aux while block b + 1's panels run here;
  // until that update is done, block b + 1 applies its row swaps to its own
  // columns only (the update reads block b's L21 and writes the columns
  // beyond), then to the rest
  const bool la = sizeof(T) == sizeof(float2) && lu_lookahead(n) && w.aux && w.ev_u12 &&
                  w.ev_far && w.pack2 && w.pack2_bytes >= lu_pack_bytes(n, sizeof(T));
  LuWork w2 = w;  // the far updates' work: second packing buffer, fewer CTAs
  if (la) {
    w2.pack = w.pack2;
    w2.pack_bytes = w.pack2_bytes;
    w2.tc_ctas = w.aux_ctas;
  }
  bool far_pending = false;
  static_assert(kOuterNB <= 4 * kNB && kPanelExpoBytes == sizeof(int) * 4 * kColParts * kNB, "");
  for (int K0 = 0; K0 < n; K0 += outer) {
  const int bend = std::min(n, K0 + outer);
  int lparts[4] = {0, 0, 0, 0};  // parts of L's exponents of the block's panels in w.pack
  for (int k0 = K0; k0 < bend; k0 += kNB) {
    const int nb = std::min(kNB, n - k0);
    const int H = n - k0;
    // cluster panel.  complex64: about one row per thread (256 rows per
    // CTA; the update is cheap on the FP32 pipe, fewer CTAs make the
    // per-column barrier cheaper).  complex128: 64 rows per CTA, as many CTAs
    // as allowed, since the rank-1 updates are bound by the FP64 pipe.  More
    // CTAs when the rows do not fit in shared memory; at most 16 (8
    // portable) CTAs and kPanelRPT rows per thread.
    const int rows_target = sizeof(T) == sizeof(float2) ? kPanelThreads : 64;
    bool done = false;
    // where the panel leaves the exponents of L21's columns
    const int slot = (k0 - K0) / kNB;
    int* lexp = nullptr;
    if (sizeof(T) == sizeof(float2) && nb == kNB && H > nb && w.pack &&
        w.pack_bytes >= tc_pack_bytes(H - nb, 1, nb))
      lexp = static_cast<int*>(w.pack) + slot * kColParts * kNB;
    if constexpr (sizeof(T) == sizeof(double2)) {
      const int rc = launch_zpanel(A, lda, n, k0, nb, w, s, launches);
      if (rc < 0) return rc;
      done = rc == 0;
      if (done) --*launches;  // counted below
    }
    if (sizeof(T) == sizeof(float2)) {  // register-window panel
      const int min_rpb = std::min(kWinMaxRows, w.min_rows > 0 ? w.min_rows : kRowsMinRpb);
      for (int cmax : {cluster16 ? kMaxClusterPanel : 8, 8}) {
        int C = std::max(1, std::min(cmax, (H + min_rpb - 1) / min_rpb));
        while ((H + C - 1) / C > kWinMaxRows) ++C;
        if (C > cmax) continue;
        const int rpb = (H + C - 1) / C;
        const int threads = win_threads(rpb);
        cudaError_t e = launch_cluster(panel_win_kernel, C, threads, panel_win_smem(rpb), s,
                                       reinterpret_cast<float2*>(A), lda, n, k0, nb, rpb,
                                       w.ipiv, w.info, w.status, lexp);
        if (e == cudaSuccess) {
          done = true;
          lparts[slot] = lexp ? C : 0;
          break;
        }
        cudaGetLastError();
        if (cmax > 8) cluster16 = false;
      }
    }
    if (!done && sizeof(T) == sizeof(float2)) {  // taller: shared-memory rows panel
      for (int cmax : {cluster16 ? kMaxClusterPanel : 8, 8}) {
        int C = std::max(1, std::min(cmax, (H + kRowsMinRpb - 1) / kRowsMinRpb));
        while ((H + C - 1) / C > kRowsMaxRpb) ++C;
        if (C > cmax) continue;
        const int rpb = (H + C - 1) / C;
        const int threads = rpb <= kRowsMaxThreads ? (rpb + 31) / 32 * 32 : kRowsMaxThreads;
        cudaError_t e = launch_cluster(panel_rows_kernel, C, threads, panel_rows_smem(rpb), s,
                                       reinterpret_cast<float2*>(A), lda, n, k0, nb, rpb,
                                       w.ipiv, w.info);
        if (e == cudaSuccess) {
          done = true;
          break;
        }
        cudaGetLastError();
        if (cmax > 8) cluster16 = false;
      }
    }
    if (!done && sizeof(T) == sizeof(float2)) {
      // taller still: tournament pivoting (measured against the shared-memory
      // rows panel above: ~200 us per 64 columns for it up to 16 x 416 rows,
      // about as much for the tournament there; beyond, the grid panel: ~370 us)
      done = tslu_panel(reinterpret_cast<float2*>(A), lda, n, k0, nb, w,
                        cluster16 ? kMaxClusterPanel : 8, lexp, s, launches);
      if (done && lexp) lparts[slot] = kColParts;
    }
    for (int cmax : {cluster16 ? kMaxClusterPanel : 8, 8}) {
      if (done) break;
      int C = std::max(1, std::min(cmax, (H + rows_target - 1) / rows_target));
      while (C < cmax && panel_cluster_smem<T>((H + C - 1) / C) > kClusterSmem) ++C;
      const int rpb = (H + C - 1) / C;
      const size_t smem = panel_cluster_smem<T>(rpb);
      if (smem > kClusterSmem || rpb > kPanelRPT * kPanelThreads) continue;
      cudaError_t e = launch_cluster(panel_cluster_kernel<T>, C, kPanelThreads, smem, s, A, lda,
                                     n, k0, nb, rpb, w.ipiv, w.info);
      if (e == cudaSuccess) {
        done = true;
        break;
      }
      cudaGetLastError();
      if (cmax > 8) cluster16 = false;
    }
    if (!done) {
      int nblk = panel_blocks<T>(H);
      int rpb = (H + nblk - 1) / nblk;
      nblk = (H + rpb - 1) / rpb;
      const size_t smem = sizeof(T) * ((size_t)rpb * kNB + kNB + rpb);
      if (smem > 200 * 1024) return BEM2D_ERR_ARG;
      unsigned spin = kSpinLimit;
      void* args[] = {(void*)&A,      (void*)&lda,    (void*)&n,      (void*)&k0,
                      (void*)&nb,     (void*)&rpb,    (void*)&w.ipiv, (void*)&w.info,
                      (void*)&w.status, (void*)&sl,   (void*)&nblk,   (void*)&spin};
      cudaError_t e = cudaLaunchCooperativeKernel((void*)panel_kernel<T>, dim3(nblk),
                                                  dim3(kPanelThreads), args, smem, s);
      if (e != cudaSuccess) return BEM2D_ERR_CUDA;
    }
    ++*launches;
    if (sizeof(T) == sizeof(float2) && (la || outer == kNB)) {
      // swaps, U12 and the update of the block's own columns with la (the rest
      // after the far update), of all others without (a panel is its own
      // block)
      const int cl = la ? K0 : 0, cr = la ? bend : n, c1 = k0 + nb, M = n - c1, N = cr - c1;
      const bool tc = N > 0 && w.pack && tc_pack_bytes(M, N, nb) <= w.pack_bytes;
      if (lexp && !lparts[slot]) {  // panels that leave none
        lparts[slot] = launch_col_expo(A + (size_t)k0 * lda + c1, lda, M, nb, lexp, s);
        ++*launches;
      }
      // (one product per term only where the work is worth it: small updates cost
      // no less with one than with three)
      const int passes = tensor_sized(M, N) ? w.tc_passes : 3;
      if (N > 0 || k0 > cl) {
        if (launch_tc_step(reinterpret_cast<float2*>(A), lda, M, k0, nb, cl, c1, cr, w.ipiv, tc,
                           lexp, lparts[slot], TcExpo(), w.pack, w.status, s, w.tc_ctas,
                           passes))
          return BEM2D_ERR_CUDA;
        *launches += tc ? 2 : 1;
      }
      if (!tc) {
        const int rc = update_sub(A + (size_t)c1 * lda + c1, A + (size_t)k0 * lda + c1,
                                  A + (size_t)c1 * lda + k0, lda, M, N, nb, w, s, launches);
        if (rc) return rc;
      }
      continue;
    } else if (n > nb) {
      laswp_kernel<T><<<(n - nb + 127) / 128, 128, 0, s>>>(A, lda, n, w.ipiv, k0, nb);
      ++*launches;
    }
    // columns of the block right of this panel
    const int c0 = k0 + nb, ncb = bend - c0;
    if (ncb > 0) {
      trsm_rows(A, lda, k0, nb, c0, ncb, s, launches);
      int rc = update_sub(A + (size_t)c0 * lda + c0, A + (size_t)k0 * lda + c0,
                          A + (size_t)c0 * lda + k0, lda, n - c0, ncb, nb, w, s, launches);
      if (rc) return rc;
    }
  }
  if (la) {  // the block's swaps on the columns outside it
    if (far_pending && cudaStreamWaitEvent(s, w.ev_far, 0) != cudaSuccess) return BEM2D_ERR_CUDA;
    far_pending = false;
    laswp_cols(A, lda, w.ipiv, K0, bend - K0, 0, K0, s, launches);
    laswp_cols(A, lda, w.ipiv, K0, bend - K0, bend, n, s, launches);
  }
  // columns right of the block: U12 = L11^{-1} A12 block row by block row,
  // then A22 -= L21 U12 with K = the block width
  const int nc = n - bend;
  const bool stepped = sizeof(T) == sizeof(float2) && outer == kNB && !la;
  TcExpo ex;  // the exponents of the block's L21, by the last step's launch
  if (nc > 0 && !stepped) {
    for (int j0 = K0; j0 < bend; j0 += kNB) {
      const int r1 = j0 + kNB, slot = (j0 - K0) / kNB;
      if (la && lparts[slot] && tc_pack_bytes(bend - r1, nc, kNB) <= w.pack_bytes) {
        if (r1 >= bend && tc_pack_bytes(nc, 1, bend - K0) <= w.pack_bytes) {
          ex.A = reinterpret_cast<const float2*>(A) + (size_t)K0 * lda + bend;
          ex.M = nc;
          ex.K = bend - K0;
          ex.np = std::min(4, col_expo_parts(nc));  // CTAs of the step's size: few
          ex.part = tc_update_part(w.pack);
        }
        if (launch_tc_step(reinterpret_cast<float2*>(A), lda, bend - r1, j0, kNB, j0, bend, n,
                           nullptr, r1 < bend,
                           static_cast<const int*>(w.pack) + slot * kColParts * kNB, lparts[slot],
                           ex, w.pack, w.status, s, w.tc_ctas,
                           tensor_sized(bend - r1, nc) ? w.tc_passes : 3))
          return BEM2D_ERR_CUDA;
        *launches += r1 < bend ? 2 : 1;
        continue;
      }
      trsm_rows(A, lda, j0, kNB, bend, nc, s, launches);
      if (r1 < bend) {
        int rc = update_sub(A + (size_t)bend * lda + r1, A + (size_t)j0 * lda + r1,
                            A + (size_t)bend * lda + j0, lda, bend - r1, nc, kNB, w, s, launches);
        if (rc) return rc;
      }
    }
    if (la) {
      // the next block's columns here; the columns beyond it on w.aux
      const int next = std::min(n, bend + outer);
      int rc = update_sub(A + (size_t)bend * lda + bend, A + (size_t)K0 * lda + bend,
                          A + (size_t)bend * lda + K0, lda, nc, next - bend, bend - K0, w, s,
                          launches, ex.part, ex.np);
      if (rc) return rc;
      if (next < n) {
        if (cudaEventRecord(w.ev_u12, s) != cudaSuccess ||
            cudaStreamWaitEvent(w.aux, w.ev_u12, 0) != cudaSuccess)
          return BEM2D_ERR_CUDA;
        rc = update_sub(A + (size_t)next * lda + bend, A + (size_t)K0 * lda + bend,
                        A + (size_t)next * lda + K0, lda, nc, n - next, bend - K0, w2, w.aux,
                        launches, ex.part, ex.np);  // (rewritten after ev_far only)
        if (rc) return rc;
        if (cudaEventRecord(w.ev_far, w.aux) != cudaSuccess) return BEM2D_ERR_CUDA;
        far_pending = true;
      }
    } else {
      int rc = update_sub(A + (size_t)bend * lda + bend, A + (size_t)K0 * lda + bend,
                          A + (size_t)bend * lda + K0, lda, nc, nc, bend - K0, w, s, launches);
      if (rc) return rc;
    }
  }
  }
  if (far_pending && cudaStreamWaitEvent(s, w.ev_far, 0) != cudaSuccess) return BEM2D_ERR_CUDA;
  // solve aids: permutation and diagonal-block inverses
  const int nk = (n + kNB - 1) / kNB;
  perm_kernel<<<(n + kPermThreads - 1) / kPermThreads, kPermThreads, 0, s>>>(n, w.ipiv, w.perm);
  dinv_kernel<T><<<dim3(nk, 16), kTriThreads, tri64_smem<T>(), s>>>(A, lda, n,
                                                                   reinterpret_cast<T*>(w.dinv));
  *launches += 2;
  return BEM2D_OK;
}

// ---- triangular solves ----------------------------------------------------
// The solves are templated on the arithmetic type T and the factor's
// storage type TS (TS = complex64, T = complex128: the complex64 factor
// applied exactly in FP64, a fixed operator, as GMRES-IR needs).
template <typename T, typename TS>
__device__ __forceinline__ T cvt(TS v) {
  return CTraits<T>::make(v.x, v.y);
}
// x = U^{-1} L^{-1} P b in one cluster launch, arithmetic in complex128.  CTA r owns rows
// [r rpb, (r+1) rpb) of b in shared memory (rpb a multiple of 64).  Step k of
// the forward sweep: the owner of block k forms y_k = L_kk^{-1} b_k from the
// stored inverse; one cluster barrier; every CTA reads y_k over DSMEM and
// updates its rows below the block.  The backward sweep is the mirror with
// U_kk^{-1}.  One cluster barrier per block step.  bin and xout may be the
// same vector (every read of bin precedes the first write of xout), so
// neither is declared __restrict__.
template <typename T, typename TS = T>
__global__ void __launch_bounds__(256)
trisolve_cluster_kernel(const TS* __restrict__ LU, long long lda, int n,
                        const int* __restrict__ perm, const TS* __restrict__ dinv,
                        const T* bin, T* xout, int rpb) {
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* bc = reinterpret_cast<T*>(smem_raw);  // [rpb] this CTA's rows of b
  T* ys = bc + rpb;                         // [kNB] the current block solution
  T* ps = ys + kNB;                         // [4][max(rpb, kNB)] partial sums
  const int r0 = rank * rpb, r1 = min(n, r0 + rpb), nr = max(r1 - r0, 0);
  for (int i = threadIdx.x; i < nr; i += blockDim.x) bc[i] = bin[perm[r0 + i]];
  const int nk = (n + kNB - 1) / kNB;
  cl.sync();
  for (int step = 0; step < 2 * nk; ++step) {
    const bool fwd = step < nk;
    const int kb = fwd ? step : 2 * nk - 1 - step;
    const int k0 = kb * kNB, nb = min(kNB, n - k0);
    const int owner = k0 / rpb;
    if (rank == owner) {
      // y = D_k^{-1} b_k: four column groups of 16 per row, partial sums in ps
      const TS* Di = dinv + (size_t)(2 * kb + (fwd ? 0 : 1)) * kNB * kNB;
      const T* bk = bc + (k0 - r0);
      const int r = threadIdx.x & 63, g = threadIdx.x >> 6;
      T acc = CTraits<T>::make(0, 0);
      if (r < nb) {
        T l[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) l[u] = cvt<T>(Di[(g * 16 + u) * kNB + r]);
#pragma unroll
        for (int u = 0; u < 16; ++u)
          if (g * 16 + u < nb) acc = cfma(l[u], bk[g * 16 + u], acc);
      }
      ps[g * kNB + r] = acc;
      __syncthreads();
      if ((int)threadIdx.x < nb) {
        const int t = threadIdx.x;
        T v = ps[t];
        v.x += ps[kNB + t].x + ps[2 * kNB + t].x + ps[3 * kNB + t].x;
        v.y += ps[kNB + t].y + ps[2 * kNB + t].y + ps[3 * kNB + t].y;
        bc[k0 - r0 + t] = v;
      }
    }
    cl.sync();
    const T* yk = cl.map_shared_rank(bc, owner) + (k0 - owner * rpb);
    if ((int)threadIdx.x < nb) ys[threadIdx.x] = yk[threadIdx.x];
    __syncthreads();
    // rows below (forward) / above (backward) the block: work items
    // (row, group of 16 columns), 16 independent loads in flight per item
    const int lo = fwd ? max(r0, k0 + nb) : r0;
    const int hi = fwd ? r1 : min(r1, k0);
    const int nrows = max(hi - lo, 0);
    for (int it = threadIdx.x; it < 4 * nrows; it += blockDim.x) {
      const int g = it / nrows, r = lo + (it - g * nrows);
      const TS* col = LU + (size_t)(k0 + g * 16) * lda + r;
      T l[16];
#pragma unroll
      for (int u = 0; u < 16; ++u)
        l[u] = (g * 16 + u < nb) ? cvt<T>(col[(size_t)u * lda]) : CTraits<T>::make(0, 0);
      T acc = CTraits<T>::make(0, 0);
#pragma unroll
      for (int u = 0; u < 16; ++u) acc = cfma(l[u], ys[(g * 16 + u) & (kNB - 1)], acc);
      ps[g * rpb + (r - r0)] = acc;
    }
    __syncthreads();
    for (int r = lo + threadIdx.x; r < hi; r += blockDim.x) {
      const int i = r - r0;
      T v = bc[i];
      v.x -= ps[i].x + ps[rpb + i].x + ps[2 * rpb + i].x + ps[3 * rpb + i].x;
      v.y -= ps[i].y + ps[rpb + i].y + ps[2 * rpb + i].y + ps[3 * rpb + i].y;
      bc[i] = v;
    }
    __syncthreads();
  }
  cl.sync();
  for (int i = threadIdx.x; i < nr; i += blockDim.x) xout[r0 + i] = bc[i];
}

// ---- complex64 triangular solves in one cluster --------------------------------
// x = U^{-1} L^{-1} P b.  Block b of 64 rows belongs to CTA b % C.  Whoever
// holds y_k subtracts L[m, k] y_k from its blocks m > k; the owner of block k +
// 1 takes that block first, forms y_{k+1} = L_{k+1,k+1}^{-1} b_{k+1} from the
// stored inverse and sends it to the CTAs with a block after it before it turns
// to its other blocks.  Going back the same with U, to every CTA.  A step of the
// chain is then one 512-byte message (asynchronous stores counted on the
// receiver's mbarrier; every block has its own slot and mbarrier) and two
// products of 64 x 64, whose matrices are loaded a step ahead.  x_k takes the
// slot and the next phase of y_k: whoever was sent y_k has a block m > k, x_k
// depends on y_m, and that left only after all of y_k had arrived and been
// read.  A CTA without a later block is not sent y_k (nothing would order that
// message before x_k); x_k is the first phase of its mbarrier.  Thread (row r,
// quarter g) = lane 4 (r % 8) + g of warp r / 8 takes the columns 8 u + 2 g, + 1.
// Bound by that chain: 2048 rows take 100 us; with contiguous rows per CTA and a
// cluster barrier in every step 270 us.  The FP64 solve keeps that scheme: there
// a 64 x 64 product costs 4 us of one SM's FP64 pipe, not the exchange.
constexpr int kSolveThreads = 256;

__host__ __device__ constexpr size_t solve64_smem(int nk, int C) {
  // y slots, own blocks' right-hand sides, mbarriers
  return sizeof(float2) * ((size_t)nk + (nk + C - 1) / C) * kNB + sizeof(long long) * nk;
}

__global__ void __launch_bounds__(kSolveThreads, 1)
trisolve64_kernel(const float2* __restrict__ LU, long long lda, int n,
                  const int* __restrict__ perm, const float2* __restrict__ dinv,
                  const float2* bin, float2* xout, int* status) {
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int nk = (n + kNB - 1) / kNB, own = (nk + C - 1) / C;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* ys = reinterpret_cast<float2*>(smem_raw);  // [nk][64] solution blocks
  float2* bl = ys + (size_t)nk * kNB;                // [own][64] own blocks, i = b / C
  unsigned long long* mb = reinterpret_cast<unsigned long long*>(bl + (size_t)own * kNB);  // [nk]
  __shared__ int s_abort;
  const int t = threadIdx.x, ln = t & 31, lw = t >> 5;
  const int r = 8 * lw + (ln >> 2), g = ln & 3;
  constexpr unsigned kBytes = kNB * sizeof(float2);
  for (int i = t; i < own * kNB; i += kSolveThreads) {
    const int row = ((i >> 6) * C + rank) * kNB + (i & 63);
    bl[i] = row < n ? bin[perm[row]] : make_float2(0.f, 0.f);
  }
  if (t == 0) {
    s_abort = 0;
    for (int k = 0; k < nk; ++k) tc::mbar_init(&mb[k], 1);
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  __syncthreads();
  if (t == 0)
    for (int k = 0; k < nk; ++k)
      if (k % C != rank) tc::mbar_expect_tx(&mb[k], kBytes);
  cl.sync();  // every mbarrier is set, every read of bin done (xout may be bin)
  // the CTAs this thread sends its row's value to: lane quarters g take ranks
  // rank + 1 + g, + 4, ..; the next block's owner (either direction) is among
  // the first
  unsigned ya[4], ma[4];
  bool to[4];
  int lastq[4];
  auto last_own = [&](int q) { return nk - 1 - (nk - 1 - q) % C; };  // last block of CTA q
  const int last = last_own(rank);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int d = (i & 1) ? C - 1 - (g + 4 * (i >> 1)) : 1 + g + 4 * (i >> 1);
    // forward distances 1..8 (i = 0, 2), backward ones C-1..C-8 (i = 1, 3), each rank once
    to[i] = d >= 1 && d < C && ((i & 1) ? d > 8 : d <= 8);
    const int q = (rank + (to[i] ? d : 0)) % C;
    lastq[i] = last_own(q);
    ya[i] = tc::map_rank(ys + r, q);
    ma[i] = tc::map_rank(mb, q);
  }
  auto load = [&](float2 (&m)[16], const float2* base, long long ld, int rows, int cols) {
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int c = 8 * (u >> 1) + 2 * g + (u & 1);
      m[u] = r < rows && c < cols ? base[(size_t)c * ld + r] : make_float2(0.f, 0.f);
    }
  };
  // sum over a row's 64 columns of m times v, in all four lanes of the row
  auto dot = [&](const float2 (&m)[16], const float2* v) {
    float2 a = make_float2(0.f, 0.f), b = make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float4 x = *reinterpret_cast<const float4*>(v + 8 * u + 2 * g);
      a = cfma(m[2 * u], make_float2(x.x, x.y), a);
      b = cfma(m[2 * u + 1], make_float2(x.z, x.w), b);
    }
    a.x += b.x;
    a.y += b.y;
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
      a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
    }
    return a;
  };
  bool ok = true;
  for (int dir = 0; dir < 2; ++dir) {
    // step s of the direction is block k(s); L or U block (m, k); D_k^{-1}
    const int st = dir ? -1 : 1, kfirst = dir ? nk - 1 : 0;
    auto lblock = [&](float2 (&m)[16], int mr, int k) {
      load(m, LU + (size_t)k * kNB * lda + (size_t)mr * kNB, lda, min(kNB, n - mr * kNB),
           min(kNB, n - k * kNB));
    };
    auto dblock = [&](float2 (&m)[16], int k) {
      const int nb = min(kNB, n - k * kNB);
      load(m, dinv + (size_t)(2 * k + dir) * kNB * kNB, kNB, nb, nb);
    };
    // solves block k (held here) and sends the result
    auto solve = [&](const float2 (&d)[16], int k) {
      const float2 y = dot(d, bl + (size_t)(k / C) * kNB);
      const unsigned yo = (unsigned)k * kBytes, mo = (unsigned)k * 8u;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (to[i] && (dir || k < lastq[i])) tc::store_async8(ya[i] + yo, y, ma[i] + mo);
      if (g == 0) {
        ys[(size_t)k * kNB + r] = y;
        if (dir && k * kNB + r < n) xout[(size_t)k * kNB + r] = y;
      }
    };
    // the first own block after k, in the order of this direction
    auto next_own = [&](int k) {
      int m = k + st;
      const int dlt = dir ? ((m - rank) % C + C) % C : ((rank - m) % C + C) % C;
      return m + st * dlt;
    };
    auto inside = [&](int m) { return m >= 0 && m < nk; };
    float2 d[16], p[16], o[16];
    int mn = kfirst % C == rank ? kfirst : next_own(kfirst);  // whose D is in d
    if (inside(mn)) dblock(d, mn);
    if (dir) {  // the own blocks' right-hand side is y
      __syncthreads();
      for (int i = t; i < own * kNB; i += kSolveThreads) {
        const int b = (i >> 6) * C + rank;
        if (b < nk) bl[i] = ys[(size_t)b * kNB + (i & 63)];
      }
      __syncthreads();
    }
    if (kfirst % C == rank) {
      solve(d, kfirst);
      mn = next_own(kfirst);
      if (inside(mn)) dblock(d, mn);
    }
    if (inside(mn)) lblock(p, mn, kfirst);
    if (inside(mn + st * C)) lblock(o, mn + st * C, kfirst);
    const int steps = dir ? nk - 1 : last;  // forward up to the last own block
    for (int s = 0; s < steps; ++s) {
      const int k = kfirst + st * s;
      if (k % C == rank) {
        __syncthreads();  // this CTA's y_k
      } else {
        ok = tc::mbar_wait_cluster(&mb[k], dir && k < last ? 1u : 0u, &s_abort) && ok;
        if (!dir && t == 0) tc::mbar_expect_tx(&mb[k], kBytes);  // x_k, on the way back
      }
      const float2* yk = ys + (size_t)k * kNB;
      const int m0 = next_own(k);
      if (!inside(m0)) continue;
      // the first own block (p holds its factor block), then its solution if it is next
      {
        const float2 v = dot(p, yk);
        if (g == 0) {
          float2& x = bl[(size_t)(m0 / C) * kNB + r];
          x.x -= v.x;
          x.y -= v.y;
        }
      }
      if (m0 == k + st) {
        __syncthreads();
        solve(d, m0);
        mn = next_own(m0);
        if (inside(mn)) dblock(d, mn);
      }
      const bool more = s + 1 < steps;
      if (more && inside(mn)) lblock(p, mn, k + st);
      // the others, the second own block from o
      auto sub = [&](const float2 (&l)[16], int m) {
        const float2 v = dot(l, yk);
        if (g == 0) {
          float2& x = bl[(size_t)(m / C) * kNB + r];
          x.x -= v.x;
          x.y -= v.y;
        }
      };
      int m = m0 + st * C;
      if (inside(m)) sub(o, m);
      if (more && inside(mn + st * C)) lblock(o, mn + st * C, k + st);
      for (m += st * C; inside(m); m += st * C) {
        float2 l[16];
        lblock(l, m, k);
        sub(l, m);
      }
    }
  }
  // x_0 has no readers, but must arrive before this CTA's shared memory goes
  if (rank != 0) ok = tc::mbar_wait_cluster(&mb[0], last > 0 ? 1u : 0u, &s_abort) && ok;
  if (!ok) atomicExch(status, 1);
  cl.sync();  // no CTA leaves while another may still write its shared memory
}

// ---- wavefront triangular solves (large n) -----------------------------------
// One cooperative launch per triangle.  The 64-row blocks are dealt to the G
// CTAs round-robin (block b to CTA b % G); each CTA keeps its blocks' entries
// of the right-hand side in shared memory.  Step k (ascending going forward,
// descending going back): the owner of block k, which has already applied
// every earlier step to that block, forms y_k = D_k^{-1} x_k from the stored
// inverse of the diagonal block, writes y_k to the output and to a slot in
// global memory and posts the slot's flag (release); every other CTA that
// still has blocks beyond k waits for the flag (acquire, bounded), reads y_k
// and subtracts L[rows, k] y_k (U[rows, k] y_k going back) from those blocks.
// There is no grid-wide barrier: a CTA waits only for the block it needs
// next, and it loads the factor entries of that step and, if it owns the
// next block, that block's inverse before it waits, so the chain of owners
// costs about one L2 round trip and two 64 x 64 products per step.  The
// factor streams through every SM at once.
constexpr int kWaveThreads = 256;
constexpr int kWaveMinN = 8192;  // below: the single-cluster solve (fewer launches)

template <typename T, bool FWD, typename TS = T>
__global__ void __launch_bounds__(kWaveThreads)
trisolve_wave_kernel(const TS* __restrict__ LU, long long lda, int n, const TS* __restrict__ dinv,
                     const int* __restrict__ perm, const T* bin, T* xout, T* ybuf, int* flags,
                     int* status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const T zero = CTraits<T>::make(0, 0);
  const int G = gridDim.x, g = blockIdx.x;
  const int nk = (n + kNB - 1) / kNB;
  const int nown = (nk - g + G - 1) / G;  // this CTA's blocks: g, g + G, ...
  T* xs = reinterpret_cast<T*>(smem_raw);  // [nown][kNB]
  T* ys = xs + (size_t)nown * kNB;          // [kNB] y of the current step
  T* ps = ys + kNB;                         // [4][kNB] partial sums
  __shared__ int s_ok;
  const int r = threadIdx.x & (kNB - 1), q = threadIdx.x >> 6;  // row, 16-column group
  for (int v = threadIdx.x; v < nown * kNB; v += blockDim.x) {
    const int row = (g + (v / kNB) * G) * kNB + (v % kNB);
    xs[v] = row < n ? (FWD ? bin[perm[row]] : bin[row]) : zero;
  }
  if (threadIdx.x == 0) s_ok = 1;
  __syncthreads();
  if (nown == 0) return;
  const int first = g, last = g + (nown - 1) * G;  // owned block range
  // entries of the diagonal-block inverse of block k for thread (r, q)
  auto load_dinv = [&](int kb, T* d) {
    const TS* Di = dinv + (size_t)(2 * kb + (FWD ? 0 : 1)) * kNB * kNB;
#pragma unroll
    for (int u = 0; u < 16; ++u) d[u] = cvt<T>(Di[(q * 16 + u) * kNB + r]);
  };
  // factor entries of block row `blk` in the columns of block kb
  auto load_l = [&](int blk, int kb, T* l) {
    const int row = blk * kNB + r, c0 = kb * kNB + q * 16;
    const TS* col = LU + (size_t)c0 * lda + row;
#pragma unroll
    for (int u = 0; u < 16; ++u)
      l[u] = (row < n && c0 + u < n) ? cvt<T>(col[(size_t)u * lda]) : zero;
  };
  // first owned block strictly beyond kb in the sweep direction, or -1
  auto next_owned = [&](int kb) -> int {
    if (FWD) {
      if (kb >= last) return -1;
      const int b = kb < first ? first : first + ((kb - first) / G + 1) * G;
      return b <= last ? b : -1;
    }
    if (kb <= first) return -1;
    const int b = kb > last ? last : first + ((kb - first - 1) / G) * G;
    return b >= first ? b : -1;
  };
  T dpre[16], lpre[16];
  int kb = FWD ? 0 : nk - 1;
  if (kb % G == g) load_dinv(kb, dpre);
  for (int s = 0; s < nk; ++s, kb += FWD ? 1 : -1) {
    if (FWD ? kb > last : kb < first) break;  // nothing of this CTA left to update
    const int jb = next_owned(kb);
    if (jb >= 0) load_l(jb, kb, lpre);
    const int kn = FWD ? kb + 1 : kb - 1;  // the next step's block
    if (kb % G == g) {
      // owner: y = D_k^{-1} x_k, published through ybuf / flags[kb]
      const T* xk = xs + (size_t)((kb - first) / G) * kNB;
      T acc = zero;
#pragma unroll
      for (int u = 0; u < 16; ++u) acc = cfma(dpre[u], xk[q * 16 + u], acc);
      ps[q * kNB + r] = acc;
      __syncthreads();
      if ((int)threadIdx.x < kNB) {
        const int t = threadIdx.x;
        T v = ps[t];
        v.x += ps[kNB + t].x + ps[2 * kNB + t].x + ps[3 * kNB + t].x;
        v.y += ps[kNB + t].y + ps[2 * kNB + t].y + ps[3 * kNB + t].y;
        ys[t] = v;
        if (kb * kNB + t < n) {
          xout[kb * kNB + t] = v;
          ybuf[kb * kNB + t] = v;
        }
      }
      block_publish(&flags[kb], 1);
      if (kn >= 0 && kn < nk && kn % G == g) load_dinv(kn, dpre);
    } else {
      if (kn >= 0 && kn < nk && kn % G == g) load_dinv(kn, dpre);  // before the wait
      if (threadIdx.x == 0 && !wait_seq(&flags[kb], 1, status)) s_ok = 0;
      __syncthreads();
      if (!s_ok) return;
      if ((int)threadIdx.x < kNB)
        ys[threadIdx.x] = kb * kNB + (int)threadIdx.x < n ? __ldcg(&ybuf[kb * kNB + threadIdx.x])
                                                          : zero;
    }
    __syncthreads();
    // update the owned blocks beyond kb: the first with the prefetched
    // entries, the others loading theirs
    for (int blk = jb; blk >= 0 && blk >= first && blk <= last; blk += FWD ? G : -G) {
      T l[16];
      if (blk == jb) {
#pragma unroll
        for (int u = 0; u < 16; ++u) l[u] = lpre[u];
      } else {
        load_l(blk, kb, l);
      }
      T acc = zero;
#pragma unroll
      for (int u = 0; u < 16; ++u) acc = cfma(l[u], ys[q * 16 + u], acc);
      ps[q * kNB + r] = acc;
      __syncthreads();
      if ((int)threadIdx.x < kNB) {
        const int t = threadIdx.x;
        T* xv = xs + (size_t)((blk - first) / G) * kNB + t;
        T v = *xv;
        v.x -= ps[t].x + ps[kNB + t].x + ps[2 * kNB + t].x + ps[3 * kNB + t].x;
        v.y -= ps[t].y + ps[kNB + t].y + ps[2 * kNB + t].y + ps[3 * kNB + t].y;
        *xv = v;
      }
      __syncthreads();
    }
  }
}

template <typename T, typename TS = T>
static int lu_solve_wave(const TS* LU, long long lda, int n, const LuWork& w, const T* b, T* x,
                         cudaStream_t s, long long* launches) {
  const int nk = (n + kNB - 1) / kNB;
  // scratch: forward result v [n], y slots [nk * kNB], flags [2 * nk]
  const size_t need = sizeof(T) * ((size_t)n + (size_t)nk * kNB) + sizeof(int) * 2 * nk;
  if (w.scratch_bytes < need) return BEM2D_ERR_ARG;
  T* v = static_cast<T*>(w.scratch);
  T* ybuf = v + n;
  int* flags = reinterpret_cast<int*>(ybuf + (size_t)nk * kNB);
  const int G = std::min(nk, device_sms());
  const size_t smem = sizeof(T) * ((size_t)((nk + G - 1) / G) * kNB + 5 * kNB);
  if (smem > 48 * 1024) return BEM2D_ERR_ARG;
  cudaMemsetAsync(flags, 0, sizeof(int) * 2 * nk, s);
  const TS* dinv = reinterpret_cast<const TS*>(w.dinv);
  const int* perm = w.perm;
  int* fl = flags;
  int* status = w.status;
  T* vo = v;
  void* af[] = {(void*)&LU, (void*)&lda, (void*)&n, (void*)&dinv, (void*)&perm, (void*)&b,
                (void*)&vo, (void*)&ybuf, (void*)&fl, (void*)&status};
  if (cudaLaunchCooperativeKernel((void*)trisolve_wave_kernel<T, true, TS>, dim3(G),
                                  dim3(kWaveThreads), af, smem, s) != cudaSuccess)
    return BEM2D_ERR_CUDA;
  const T* vin = v;
  int* fb = flags + nk;
  void* ab[] = {(void*)&LU, (void*)&lda, (void*)&n, (void*)&dinv, (void*)&perm, (void*)&vin,
                (void*)&x, (void*)&ybuf, (void*)&fb, (void*)&status};
  if (cudaLaunchCooperativeKernel((void*)trisolve_wave_kernel<T, false, TS>, dim3(G),
                                  dim3(kWaveThreads), ab, smem, s) != cudaSuccess)
    return BEM2D_ERR_CUDA;
  *launches += 2;
  return BEM2D_OK;
}

template <typename T>
static int lu_solve_cluster(const T* LU, long long lda, int n, const LuWork& w, const T* b, T* x,
                            cudaStream_t s, long long* launches) {
  static PerDevice<int> largest(kMaxCluster);
  static PerDeviceOnce attr;
  const int dev = current_device();
  std::atomic<int>& cmax = largest[dev];
  attr(dev, [&] {
    cudaFuncSetAttribute(trisolve_cluster_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kClusterSmem);
    if (cudaFuncSetAttribute(trisolve_cluster_kernel<T>,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      cmax = 8;
    }
  });
  for (;;) {
    const int nk = (n + kNB - 1) / kNB;
    const int C = std::max(1, std::min(cmax.load(), nk));
    const int rpb = ((nk + C - 1) / C) * kNB;
    const size_t smem = sizeof(T) * ((size_t)rpb + kNB + 4 * (size_t)std::max(rpb, kNB));
    if (smem > kClusterSmem) return BEM2D_ERR_ARG;
    cudaError_t e = launch_cluster(trisolve_cluster_kernel<T>, C, 256, smem, s, LU, lda, n,
                                   (const int*)w.perm, (const T*)w.dinv, b, x, rpb);
    if (e == cudaSuccess) break;
    cudaGetLastError();
    if (cmax == 8) return BEM2D_ERR_CUDA;
    cmax = 8;
  }
  ++*launches;
  return BEM2D_OK;
}

static int lu_solve64(const float2* LU, long long lda, int n, const LuWork& w, const float2* b,
                      float2* x, cudaStream_t s, long long* launches) {
  static PerDevice<int> largest(kMaxCluster);
  static PerDeviceOnce attr;
  const int dev = current_device();
  std::atomic<int>& cmax = largest[dev];
  attr(dev, [&] {
    cudaFuncSetAttribute(trisolve64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kClusterSmem);
    if (cudaFuncSetAttribute(trisolve64_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed,
                             1) != cudaSuccess) {
      cudaGetLastError();
      cmax = 8;
    }
  });
  const int nk = (n + kNB - 1) / kNB;
  for (;;) {
    const int C = std::max(1, std::min(cmax.load(), nk));
    const cudaError_t e =
        launch_cluster(trisolve64_kernel, C, kSolveThreads, solve64_smem(nk, C), s, LU, lda, n,
                       (const int*)w.perm, (const float2*)w.dinv, b, x, w.status);
    if (e == cudaSuccess) break;
    cudaGetLastError();
    if (cmax == 8) return BEM2D_ERR_CUDA;
    cmax = 8;
  }
  ++*launches;
  return BEM2D_OK;
}

template <typename T>
int lu_solve(const T* LU, long long lda, int n, const LuWork& w, const T* b, T* x,
             cudaStream_t s, long long* launches) {
  if (n >= kWaveMinN) return lu_solve_wave(LU, lda, n, w, b, x, s, launches);
  if constexpr (sizeof(T) == sizeof(float2))
    return lu_solve64(LU, lda, n, w, b, x, s, launches);
  else
    return lu_solve_cluster(LU, lda, n, w, b, x, s, launches);
}

// x = A^{-1} b with a complex64 factor, the arithmetic in complex128.
int lu_solve_mixed(const float2* LU, long long lda, int n, const LuWork& w, const double2* b,
                   double2* x, cudaStream_t s, long long* launches) {
  if (n >= kWaveMinN) return lu_solve_wave<double2, float2>(LU, lda, n, w, b, x, s, launches);
  static PerDevice<int> largest(kMaxCluster);
  static PerDeviceOnce attr;
  const int dev = current_device();
  std::atomic<int>& cmax = largest[dev];
  attr(dev, [&] {
    cudaFuncSetAttribute(trisolve_cluster_kernel<double2, float2>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterSmem);
    if (cudaFuncSetAttribute(trisolve_cluster_kernel<double2, float2>,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      cmax = 8;
    }
  });
  for (;;) {
    const int nk = (n + kNB - 1) / kNB;
    const int C = std::max(1, std::min(cmax.load(), nk));
    const int rpb = ((nk + C - 1) / C) * kNB;
    const size_t smem = sizeof(double2) * ((size_t)rpb + kNB + 4 * (size_t)std::max(rpb, kNB));
    if (smem > kClusterSmem) return BEM2D_ERR_ARG;
    cudaError_t e = launch_cluster(trisolve_cluster_kernel<double2, float2>, C, 256, smem, s, LU,
                                   lda, n, (const int*)w.perm, (const float2*)w.dinv, b, x, rpb);
    if (e == cudaSuccess) break;
    cudaGetLastError();
    if (cmax == 8) return BEM2D_ERR_CUDA;
    cmax = 8;
  }
  ++*launches;
  return BEM2D_OK;
}

// x = A^{-H} b = P^T L^{-H} U^{-H} b in one cluster launch.  Forward sweep
// with U^H (lower), backward with L^H (upper, unit diagonal).  Per step
// every CTA forms the partial sums sum_r conj(M[r, k0+c]) x_r over its own,
// already final rows; one cluster barrier; the owner of block k adds the
// partials over DSMEM and applies the conjugate transpose of the stored
// diagonal-block inverse.  Partial buffers alternate by step parity.
template <typename T>
__global__ void __launch_bounds__(256)
trisolve_h_cluster_kernel(const T* __restrict__ LU, long long lda, int n,
                          const int* __restrict__ perm, const T* __restrict__ dinv,
                          const T* __restrict__ bin, T* __restrict__ xout, int rpb) {
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), C = (int)cl.num_blocks();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* bc = reinterpret_cast<T*>(smem_raw);  // [rpb]
  T* part = bc + rpb;                       // [2][kNB]
  T* v = part + 2 * kNB;                    // [kNB]
  const int r0 = rank * rpb, r1 = min(n, r0 + rpb), nr = max(r1 - r0, 0);
  for (int i = threadIdx.x; i < nr; i += blockDim.x) bc[i] = bin[r0 + i];
  const int nk = (n + kNB - 1) / kNB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  cl.sync();
  for (int step = 0; step < 2 * nk; ++step) {
    const bool fwd = step < nk;
    const int kb = fwd ? step : 2 * nk - 1 - step;
    const int k0 = kb * kNB, nb = min(kNB, n - k0), par = step & 1;
    const int lo = fwd ? r0 : max(r0, k0 + nb);
    const int hi = fwd ? min(r1, k0) : r1;
    for (int c = warp * 8; c < warp * 8 + 8; ++c) {
      double sr = 0, si = 0;
      if (c < nb) {
        const T* col = LU + (size_t)(k0 + c) * lda;
        for (int r = lo + lane; r < hi; r += 32) {
          const T a = col[r], b = bc[r - r0];
          sr += (double)a.x * b.x + (double)a.y * b.y;
          si += (double)a.x * b.y - (double)a.y * b.x;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sr += __shfl_xor_sync(0xffffffffu, sr, o);
        si += __shfl_xor_sync(0xffffffffu, si, o);
      }
      if (lane == 0) part[par * kNB + c] = CTraits<T>::make(sr, si);
    }
    cl.sync();
    const int owner = k0 / rpb;
    if (rank == owner) {
      const int t = threadIdx.x;
      if (t < nb) {
        T acc = bc[k0 - r0 + t];
        for (int q = 0; q < C; ++q) {
          const T pq = cl.map_shared_rank(part, q)[par * kNB + t];
          acc.x -= pq.x;
          acc.y -= pq.y;
        }
        v[t] = acc;
      }
      __syncthreads();
      // x_k = D^{-H} v with D^{-1} = (U or L)_kk^{-1} stored column-major
      const T* Di = dinv + (size_t)(2 * kb + (fwd ? 1 : 0)) * kNB * kNB;
      if (t < nb) {
        T acc = CTraits<T>::make(0, 0);
        for (int m = 0; m < nb; ++m) {
          const T d = Di[t * kNB + m];  // D^{-1}[m, t]
          // conj(d) * v[m]
          acc.x += d.x * v[m].x + d.y * v[m].y;
          acc.y += d.x * v[m].y - d.y * v[m].x;
        }
        bc[k0 - r0 + t] = acc;
      }
      __syncthreads();
    }
  }
  cl.sync();
  for (int i = threadIdx.x; i < nr; i += blockDim.x) xout[perm[r0 + i]] = bc[i];
}

template <typename T>
int lu_solve_h(const T* LU, long long lda, int n, const LuWork& w, const T* b, T* x,
               cudaStream_t s, long long* launches) {
  static PerDevice<int> largest(kMaxCluster);
  static PerDeviceOnce attr;
  const int dev = current_device();
  std::atomic<int>& cmax = largest[dev];
  attr(dev, [&] {
    cudaFuncSetAttribute(trisolve_h_cluster_kernel<T>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClusterSmem);
    if (cudaFuncSetAttribute(trisolve_h_cluster_kernel<T>,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      cmax = 8;
    }
  });
  if (b == x) return BEM2D_ERR_ARG;  // the scatter at the end needs distinct buffers
  for (;;) {
    const int nk = (n + kNB - 1) / kNB;
    const int C = std::max(1, std::min(cmax.load(), nk));
    const int rpb = ((nk + C - 1) / C) * kNB;
    const size_t smem = sizeof(T) * ((size_t)rpb + 3 * kNB);
    if (smem > kClusterSmem) return BEM2D_ERR_ARG;
    cudaError_t e = launch_cluster(trisolve_h_cluster_kernel<T>, C, 256, smem, s, LU, lda, n,
                                   (const int*)w.perm, (const T*)w.dinv, b, x, rpb);
    if (e == cudaSuccess) break;
    cudaGetLastError();
    if (cmax == 8) return BEM2D_ERR_CUDA;
    cmax = 8;
  }
  ++*launches;
  return BEM2D_OK;
}

template int lu_solve_h<double2>(const double2*, long long, int, const LuWork&, const double2*,
                                 double2*, cudaStream_t, long long*);
template int lu_solve_h<float2>(const float2*, long long, int, const LuWork&, const float2*,
                                float2*, cudaStream_t, long long*);

// Timeout check of the grid panel's bounded waits: one panel of the
// complex64 matrix A (n x 64, n >= 256, lda) on two cooperative blocks whose
// waits expect three candidates, so each waits for a slot that is never
// posted; every wait gives up after `polls` polls, sets *w.status and the
// kernel returns.  The caller reads *w.status after synchronising.
int lu_panel_timeout_probe(float2* A, long long lda, int n, const LuWork& w, unsigned polls,
                           cudaStream_t s) {
  if (n < 256 || lda < n || polls < 1) return BEM2D_ERR_ARG;
  PanelSlots<float2> sl;
  sl.base = static_cast<char*>(w.scratch);
  cudaMemsetAsync(w.info, 0, sizeof(int), s);
  cudaMemsetAsync(w.status, 0, sizeof(int), s);
  cudaMemsetAsync(sl.base, 0, slots_bytes(sizeof(float2)), s);
  static PerDeviceOnce attr;
  attr(current_device(), [] {
    cudaFuncSetAttribute(panel_kernel<float2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         200 * 1024);
  });
  int nblk = 2, k0 = 0, nb = kNB;
  int rpb = (n + nblk - 1) / nblk;
  const size_t smem = sizeof(float2) * ((size_t)rpb * kNB + kNB + rpb);
  if (smem > 200 * 1024) return BEM2D_ERR_ARG;
  int nwait = nblk + 1;
  unsigned spin = polls;
  void* args[] = {(void*)&A,      (void*)&lda,    (void*)&n,      (void*)&k0,
                  (void*)&nb,     (void*)&rpb,    (void*)&w.ipiv, (void*)&w.info,
                  (void*)&w.status, (void*)&sl,   (void*)&nwait,  (void*)&spin};
  return cudaLaunchCooperativeKernel((void*)panel_kernel<float2>, dim3(nblk),
                                     dim3(kPanelThreads), args, smem, s) == cudaSuccess
             ? BEM2D_OK
             : BEM2D_ERR_CUDA;
}

template int lu_factor<double2>(double2*, long long, int, const LuWork&, cudaStream_t, long long*);
template int lu_factor<float2>(float2*, long long, int, const LuWork&, cudaStream_t, long long*);
template int lu_solve<double2>(const double2*, long long, int, const LuWork&, const double2*,
                               double2*, cudaStream_t, long long*);
template int lu_solve<float2>(const float2*, long long, int, const LuWork&, const float2*, float2*,
                              cudaStream_t, long long*);

// ---- refinement helpers -----------------------------------------------------
// r = b - A x in FP64: column chunks give partial sums per row; the kernel that
// adds them also forms the partial sums of |r|^2 and |x|^2.  FP64 pipe: 4 n^2
// FMAs.  Chunks of 64 columns below 4096 rows, so that every SM has several
// blocks (n = 2048: 39 us, with chunks of 256 72 us; 28 us is the pipe's time);
// above, longer chunks fill the GPU too and write fewer partial sums.
constexpr int kResChunk = 256;
static int res_chunk(int n) { return n < 4096 ? kResChunk / 4 : n < 8192 ? kResChunk / 2 : kResChunk; }
__global__ void __launch_bounds__(128)
residual_partial_kernel(const double2* __restrict__ A, long long lda, int n, int chunk,
                        const double2* __restrict__ x, double2* part) {
  __shared__ double2 xs[kResChunk];
  const int c0 = blockIdx.y * chunk;
  const int nc = min(chunk, n - c0);
  for (int v = threadIdx.x; v < nc; v += blockDim.x) xs[v] = x[c0 + v];
  __syncthreads();
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  double2 acc = make_double2(0, 0);
  const double2* col = A + (size_t)c0 * lda + r;
#pragma unroll 8
  for (int c = 0; c < nc; ++c) acc = cfma(col[(size_t)c * lda], xs[c], acc);
  part[(size_t)blockIdx.y * n + r] = acc;
}

// With nchunk > 0: r = b - the partial sums.  red[2 block], + 1: the block's sums
// of |r|^2 and |x|^2.
__global__ void __launch_bounds__(256)
residual_final_kernel(int n, int nchunk, const double2* __restrict__ part,
                      const double2* __restrict__ b, double2* r, const double2* __restrict__ x,
                      double* __restrict__ red) {
  double s[2] = {0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double2 acc;
    if (nchunk > 0) {
      acc = b[i];
#pragma unroll 8
      for (int c = 0; c < nchunk; ++c) {
        const double2 p = part[(size_t)c * n + i];
        acc.x -= p.x;
        acc.y -= p.y;
      }
      r[i] = acc;
    } else {
      acc = r[i];
    }
    const double2 v = x[i];
    s[0] = fma(acc.x, acc.x, fma(acc.y, acc.y, s[0]));
    s[1] = fma(v.x, v.x, fma(v.y, v.y, s[1]));
  }
  __shared__ double w[2][8];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
    if ((threadIdx.x & 31) == 0) w[j][threadIdx.x >> 5] = s[j];
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double a = 0.0;
    for (int k = 0; k < 8; ++k) a += w[threadIdx.x][k];
    red[2 * blockIdx.x + threadIdx.x] = a;
  }
}

// out[j] = sum of red[2 i + j], i < nb: a warp for each j
__global__ void __launch_bounds__(64)
sum2_kernel(int nb, const double* __restrict__ red, double* out) {
  const int j = threadIdx.x >> 5;
  double s = 0.0;
  for (int i = threadIdx.x & 31; i < nb; i += 32) s += red[2 * i + j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) out[j] = s;
}

constexpr int kSumsqBlocks = 304;
static void final_norms(int n, int nchunk, const double2* part, const double2* b, double2* r,
                        const double2* x, double* red, double* out, cudaStream_t s) {
  const int nb = std::min((n + 255) / 256, kSumsqBlocks / 2);
  residual_final_kernel<<<nb, 256, 0, s>>>(n, nchunk, part, b, r, x, red);
  sum2_kernel<<<1, 64, 0, s>>>(nb, red, out);
}

void launch_residual(const double2* A, long long lda, int n, const double2* x,
                     const double2* b, double2* r, double2* part, double* red, double* out,
                     cudaStream_t s) {
  const int chunk = res_chunk(n), nchunk = (n + chunk - 1) / chunk;
  dim3 g((n + 127) / 128, nchunk);
  residual_partial_kernel<<<g, 128, 0, s>>>(A, lda, n, chunk, x, part);
  final_norms(n, nchunk, part, b, r, x, red, out, s);
}

void launch_norms(int n, double2* r, const double2* x, double* red, double* out, cudaStream_t s) {
  final_norms(n, 0, nullptr, nullptr, r, x, red, out, s);
}

size_t residual_part_bytes(int n) {
  const int chunk = res_chunk(n);
  return sizeof(double2) * (size_t)n * ((n + chunk - 1) / chunk);
}

__global__ void to_c64_kernel(const double2* __restrict__ src, long long lds,
                              float2* __restrict__ dst, long long ldd, int rows, int cols) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= (long long)rows * cols) return;
  const int j = (int)(v / rows), i = (int)(v - (long long)j * rows);
  const double2 a = src[(size_t)j * lds + i];
  dst[(size_t)j * ldd + i] = make_float2((float)a.x, (float)a.y);
}

void launch_to_c64(const double2* src, long long lds, float2* dst, long long ldd,
                   int rows, int cols, cudaStream_t s) {
  const long long tot = (long long)rows * cols;
  to_c64_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(src, lds, dst, ldd, rows, cols);
}

// dst = (complex64)(src * scale)
__global__ void scale_to_c64_kernel(int n, const double2* __restrict__ src, double scale,
                                    float2* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = make_float2((float)(src[i].x * scale), (float)(src[i].y * scale));
}
// x += scale * d
__global__ void axpy_c64_kernel(int n, double scale, const float2* __restrict__ d,
                                double2* __restrict__ x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) {
    x[i].x = fma(scale, (double)d[i].x, x[i].x);
    x[i].y = fma(scale, (double)d[i].y, x[i].y);
  }
}

// ---- explicit inverse of a complex64 factor ---------------------------------
// W = U^{-1} L^{-1} from the factor P A = L U of lu_factor<float2>, so that
// A^{-1} x = W (P x) and A^{-H} x = P^T (W^H x).  Blocked substitution on
// the identity, 64 rows at a time inside outer blocks of 256 rows (64 when
// the packing buffer only holds rank-64 operands):
//   forward  Y_k = L_kk^{-1} Y_k, then the outer block's rows below k, and
//            after the outer block the rows below it (Y stays lower
//            triangular: only the columns left of the block are touched);
//   backward W_k = U_kk^{-1} W_k, then the outer block's rows above k, and
//            after the outer block the rows above it.
// The diagonal-block inverses are lu_factor's (w.dinv); the updates run on
// the tensor cores (the trailing-update kernel).  About 2.7 N^3
// complex flops; an inverse pays for itself once an iteration needs more
// than a few dozen solves with the factor (a product with W streams N^2
// entries; the substitution is a chain of 2 N / 64 dependent steps).

// Xb (rows r0 .. r0 + bs - 1 of X, column-major, ld ldx) = D Xb, D a 64 x 64
// column-major block (zero beyond bs).  grid ceil(ncols / 16), 256 threads.
__global__ void __launch_bounds__(256)
block_apply_kernel(const float2* __restrict__ D, float2* __restrict__ X, long long ldx, int bs,
                   int ncols) {
  __shared__ float2 Ds[kNB * kNB];  // Ds[k * 64 + r] = D(r, k)
  __shared__ float2 T[kNB * 17];    // T[k * 17 + c] = X(r0 + k, c0 + c)
  const int c0 = blockIdx.x * 16;
  for (int e = threadIdx.x; e < kNB * kNB; e += blockDim.x) Ds[e] = D[e];
  for (int e = threadIdx.x; e < kNB * 16; e += blockDim.x) {
    const int c = e / kNB, k = e - c * kNB;  // coalesced along k (rows)
    T[k * 17 + c] = (k < bs && c0 + c < ncols) ? X[(size_t)(c0 + c) * ldx + k]
                                                : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const int c = threadIdx.x & 15, rb = threadIdx.x >> 4;  // rows rb + 16 q
  float2 acc[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) acc[q] = make_float2(0.f, 0.f);
  for (int k = 0; k < bs; ++k) {
    const float2 t = T[k * 17 + c];
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] = cfma(Ds[k * kNB + rb + 16 * q], t, acc[q]);
  }
  if (c0 + c >= ncols) return;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = rb + 16 * q;
    if (r < bs) X[(size_t)(c0 + c) * ldx + r] = acc[q];
  }
}

__global__ void identity_c64_kernel(int n, float2* __restrict__ X, long long ldx) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) X[(size_t)i * ldx + i] = make_float2(1.f, 0.f);
}

// The exponents of every column k of LU (colscale.cuh), for all updates of the
// inverse in one launch: ex[k] of the rows below k's 64-column block, ex[n + k]
// of those below its outer block of ob columns, ex[2 n + k] and ex[3 n + k] of
// those above them.
__global__ void __launch_bounds__(256)
inverse_expo_kernel(const float2* __restrict__ LU, long long lda, int n, int ob,
                    int* __restrict__ ex) {
  __shared__ int red[4][8];
  const int k = blockIdx.x, b0 = k / kNB * kNB, b1 = b0 + kNB, q0 = k / ob * ob, q1 = q0 + ob;
  int e[4] = {0, 0, 0, 0};
#pragma unroll 4
  for (int r = threadIdx.x; r < n; r += 256) {
    const float2 v = LU[(size_t)k * lda + r];
    const int x = max(col_expo(v.x), col_expo(v.y));
    if (r >= b1) e[0] = max(e[0], x);
    if (r >= q1) e[1] = max(e[1], x);
    if (r < b0) e[2] = max(e[2], x);
    if (r < q0) e[3] = max(e[3], x);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    e[i] = __reduce_max_sync(0xffffffffu, e[i]);
    if ((threadIdx.x & 31) == 0) red[i][threadIdx.x >> 5] = e[i];
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    int m = 0;
    for (int w = 0; w < 8; ++w) m = max(m, red[threadIdx.x][w]);
    ex[(size_t)threadIdx.x * n + k] = m;
  }
}

int lu_inverse_c64(const float2* LU, long long lda, int n, const LuWork& w, float2* W,
                   long long ldw, cudaStream_t s, long long* launches) {
  if (n <= 0) return BEM2D_OK;
  if (!w.pack || !w.dinv) return BEM2D_ERR_ARG;
  if (tc_pack_bytes(n, n, kNB) > w.pack_bytes) return BEM2D_ERR_ARG;
  // outer blocks of kOuterNB rows where the packing buffer holds rank-256
  // operands (one pass over the rest of W per outer block, not per 64 rows)
  const int ob = tc_pack_bytes(n, n, kOuterNB) <= w.pack_bytes ? kOuterNB : kNB;
  // the panels' scratch is free by now
  int* ex = w.scratch_bytes >= sizeof(int) * 4 * (size_t)n ? static_cast<int*>(w.scratch) : nullptr;
  if (ex) {
    inverse_expo_kernel<<<n, 256, 0, s>>>(LU, lda, n, ob, ex);
    ++*launches;
  }
  // set 0 .. 3 of the exponents, of the columns from k on
  auto upd = [&](float2* C, const float2* Am, const float2* Bm, int M, int N, int K, int set,
                 int k) -> int {
    if (M <= 0 || N <= 0 || K <= 0) return BEM2D_OK;
    if (launch_tc_cgemm_sub(C, ldw, Am, lda, Bm, ldw, M, N, K, w.pack, w.pack_bytes, w.status, s,
                            0, 3, ex ? ex + (size_t)set * n + k : nullptr, 1))
      return BEM2D_ERR_CUDA;
    *launches += ex ? 2 : 3;
    return BEM2D_OK;
  };
  if (cudaMemset2DAsync(W, sizeof(float2) * ldw, 0, sizeof(float2) * n, n, s) != cudaSuccess)
    return BEM2D_ERR_CUDA;
  identity_c64_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, W, ldw);
  ++*launches;
  const float2* dinv = static_cast<const float2*>(w.dinv);
  int rc = 0;
  for (int R0 = 0; R0 < n; R0 += ob) {  // forward: Y = L^{-1} (lower triangular)
    const int R1 = std::min(n, R0 + ob);
    for (int k0 = R0; k0 < R1; k0 += kNB) {
      const int kb = k0 / kNB, bs = std::min(kNB, n - k0), nc = k0 + bs;
      block_apply_kernel<<<(nc + 15) / 16, 256, 0, s>>>(dinv + (size_t)(2 * kb) * kNB * kNB,
                                                        W + k0, ldw, bs, nc);
      ++*launches;
      // the rest of this outer block's rows
      if ((rc = upd(W + nc, LU + (size_t)k0 * lda + nc, W + k0, R1 - nc, nc, bs, 0, k0))) return rc;
    }
    // the rows below the outer block, columns 0 .. R1 - 1 (Y is zero beyond)
    if ((rc = upd(W + R1, LU + (size_t)R0 * lda + R1, W + R0, n - R1, R1, R1 - R0, 1, R0)))
      return rc;
  }
  const int nob = (n + ob - 1) / ob;
  for (int q = nob - 1; q >= 0; --q) {  // backward: W = U^{-1} Y
    const int R0 = q * ob, R1 = std::min(n, R0 + ob);
    for (int k0 = ((R1 - 1) / kNB) * kNB; k0 >= R0; k0 -= kNB) {
      const int kb = k0 / kNB, bs = std::min(kNB, n - k0);
      block_apply_kernel<<<(n + 15) / 16, 256, 0, s>>>(dinv + (size_t)(2 * kb + 1) * kNB * kNB,
                                                       W + k0, ldw, bs, n);
      ++*launches;
      if ((rc = upd(W + R0, LU + (size_t)k0 * lda + R0, W + k0, k0 - R0, n, bs, 2, k0))) return rc;
    }
    if ((rc = upd(W, LU + (size_t)R0 * lda, W + R0, R0, n, R1 - R0, 3, R0))) return rc;
  }
  return cudaPeekAtLastError() == cudaSuccess ? BEM2D_OK : BEM2D_ERR_CUDA;
}

// dst[i] = (complex64) (scale src[perm[i]]): P x of an FP64 vector.
__global__ void gather_to_c64_kernel(int n, const double2* __restrict__ src,
                                     const int* __restrict__ perm, double scale,
                                     float2* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2 v = src[perm[i]];
  dst[i] = make_float2((float)(v.x * scale), (float)(v.y * scale));
}
// dst[perm[i]] = src[i]: P^T y (complex64).
__global__ void scatter_c64_kernel(int n, const float2* __restrict__ src,
                                   const int* __restrict__ perm, float2* __restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[perm[i]] = src[i];
}
void launch_gather_to_c64(int n, const double2* src, const int* perm, double scale, float2* dst,
                          cudaStream_t s) {
  gather_to_c64_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, src, perm, scale, dst);
}
void launch_scatter_c64(int n, const float2* src, const int* perm, float2* dst, cudaStream_t s) {
  scatter_c64_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, src, perm, dst);
}

void launch_scale_to_c64(int n, const double2* src, double scale, float2* dst, cudaStream_t s) {
  scale_to_c64_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, src, scale, dst);
}
void launch_axpy_c64(int n, double scale, const float2* d, double2* x, cudaStream_t s) {
  axpy_c64_kernel<<<(n + 255) / 256, 256, 0, s>>>(n, scale, d, x);
}

// Sum of |a_ij|^2 over a rows x cols column-major block: per-block partial
// sums, then one block adds them (deterministic order).
__global__ void __launch_bounds__(256)
sumsq_partial_kernel(const double2* __restrict__ A, long long ld, long long rows, int cols,
                     double* part) {
  __shared__ double red[8];
  // blocks of 1024 consecutive rows of a column
  const long long per = (rows + 1023) / 1024, tot = per * cols;
  double acc = 0.0;
  for (long long v = blockIdx.x; v < tot; v += gridDim.x) {
    const long long j = cols == 1 ? 0 : v / per, i0 = (v - j * per) * 1024;
    const double2* col = A + j * ld;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long i = i0 + u * 256 + threadIdx.x;
      const double2 a = i < rows ? col[i] : make_double2(0.0, 0.0);
      acc = fma(a.x, a.x, fma(a.y, a.y, acc));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int k = 0; k < 8; ++k) s += red[k];
    part[blockIdx.x] = s;
  }
}

__global__ void sum_kernel(int n, const double* __restrict__ part, double* out) {
  __shared__ double red[256];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += part[i];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

void launch_sumsq(const double2* A, long long ld, int rows, int cols, double* part,
                  double* out, cudaStream_t s) {
  // a contiguous matrix is one column
  const bool one = ld == rows;
  const long long r = one ? (long long)rows * cols : rows;
  sumsq_partial_kernel<<<kSumsqBlocks, 256, 0, s>>>(A, ld, r, one ? 1 : cols, part);
  sum_kernel<<<1, 256, 0, s>>>(kSumsqBlocks, part, out);
}
size_t sumsq_part_bytes() { return sizeof(double) * kSumsqBlocks; }

// *flag |= 1 if any entry of the rows x cols column-major block is NaN or
// infinite: one coalesced pass (rows fastest), one atomic per warp that saw
// a non-finite value.
__global__ void nonfinite_kernel(const double2* __restrict__ A, long long ld, int rows, int cols,
                                 int* flag) {
  bool bad = false;
  for (int j = blockIdx.y; j < cols; j += gridDim.y)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) {
      const double2 a = A[(size_t)j * ld + i];
      bad |= !(isfinite(a.x) && isfinite(a.y));
    }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

void launch_nonfinite_scan(const double2* A, long long ld, int rows, int cols, int* flag,
                           cudaStream_t s) {
  const int bx = std::min(8, (rows + 255) / 256);
  const int by = std::min(cols, 1024);
  nonfinite_kernel<<<dim3(bx, by), 256, 0, s>>>(A, ld, rows, cols, flag);
}

}  // namespace bem2d_gpu
