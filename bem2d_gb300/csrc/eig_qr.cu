// Eigenvalues of a complex upper Hessenberg matrix by pipelined shifted QR in
// one thread-block cluster (Eigenvalues without eigenvectors,
// lib/bem2d_mathroutines.cpp:437-466).
//
// Single-shift implicit QR (Golub & Van Loan, sec. 7.5), up to 16 sweeps at a
// time: sweep b chases its bulge 3 rows behind sweep b - 1 (Braman, Byers and
// Mathias, "The multishift QR algorithm. Part I", SIAM J. Matrix Anal. Appl.
// 23, 2002, with one-element bulges).  Rotations of different sweeps act on
// disjoint row pairs and disjoint column pairs, and a left rotation of one
// commutes with a right rotation of another, so a step applies all row
// rotations, then all column rotations: what sequential sweeps with the same
// shifts compute.  The shifts are the eigenvalues of the trailing block.
//
// One sweep at a time is bound by the latency of its chain: forming one
// rotation, two updates and three barriers took 4.7 us (n = 255: 300 ms).
// Here a step costs about as much for up to 16 rotations, which lanes of one
// warp form together, and the updates run on 16 SMs: a warp's
// FP64 instruction takes 64 clocks of a scheduler, and one SM alone would need
// 34 ms for the 12 instructions per element pair.  n = 255: 50 ms, 6,300 steps
// in 30 rounds.
//
// The matrix stays in L2 (loads and stores bypass L1: CTAs read each other's
// elements after a cluster barrier).  CTA 0 deflates, solves blocks of at most
// 16 rows outright and picks shifts with one warp in shared memory while the
// others wait at the barrier.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <float.h>

#include "common.cuh"
#include "cplx.cuh"

namespace cg = cooperative_groups;

namespace bem2d_gpu {
namespace {

constexpr int kQrSweeps = 16;   // sweeps at a time, and the small block's order
constexpr int kQrGap = 3;       // rows between bulges
constexpr int kQrCta = 128;
constexpr int kQrMaxIt = 30;    // sweeps per eigenvalue at most

__device__ __forceinline__ double2 conj2(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double abs1(double2 a) { return fabs(a.x) + fabs(a.y); }

__device__ __forceinline__ double shfl1(double v) { return __shfl_xor_sync(0xffffffffu, v, 1); }

// 1/sqrt(v) to FP64 accuracy for v in the normal range: a third-order
// correction of the hardware's 2^-20 seed.
__device__ __forceinline__ double rsqrt3(double v) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
  const double e = fma(-v * y, y, 1.0);
  return fma(y, e * fma(0.375, e, 0.5), y);
}

// Rotation with  c x + s y = r, -conj(s) x + c y = 0  (c real), formed by a
// pair of lanes: the even one brings v = x, the odd one v = y, both get c and
// s.  What the two halves have in common then costs one FP64 instruction, 17
// in all.  Components are scaled by a power of two first, so squares neither
// overflow nor vanish.  All 32 lanes take part.
__device__ __forceinline__ void rotation(double2 v, double* c, double2* s) {
  const bool odd = threadIdx.x & 1;
  int e = max(__double2hiint(v.x) & 0x7ff00000, __double2hiint(v.y) & 0x7ff00000);
  e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
  // 2^(1022 - exponent): scaled components below 1 (2 at the top of the range)
  const double f = __hiloint2double(max(0x7fd00000 - e, 0x00100000), 0);
  v = make_double2(v.x * f, v.y * f);
  const double n = fma(v.x, v.x, v.y * v.y), o = shfl1(n), r = n + o;
  const double X = odd ? o : n;
  const double q = rsqrt3(odd ? r : n);  // 1 / r, 1 / |x|
  const double qo = shfl1(q);
  const double2 vo = make_double2(shfl1(v.x), shfl1(v.y));
  const double2 x = odd ? vo : v, y = odd ? v : vo;
  if (!(r > 0.0)) {  // both zero
    *c = 1.0;
    *s = make_double2(0.0, 0.0);
  } else if (X == 0.0) {
    const double iy = odd ? q : qo;
    *c = 0.0;
    *s = make_double2(y.x * iy, -y.y * iy);  // conj(y) / |y|
  } else {
    // c = |x| / r, s = (x / |x|) conj(y) / r
    const double g = q * qo;
    *c = X * g;
    const double tx = x.x * g, ty = x.y * g;
    // re = tx y.x + ty y.y (even lane), im = ty y.x - tx y.y (odd lane)
    const double m = fma(odd ? ty : tx, y.x, (odd ? -tx : ty) * y.y);
    s->x = m;
    s->y = m;
  }
  // one exchange for both components, outside the branch (lanes of a pair agree)
  const double mo = shfl1(odd ? s->y : s->x), own = odd ? s->y : s->x;
  const bool general = r > 0.0 && X != 0.0;
  if (general) *s = odd ? make_double2(mo, own) : make_double2(own, mo);
}

// c h + t g.  Rows: (h1, h2) <- (c h1 + s h2, c h2 - conj(s) h1); columns the
// same with conj(s) and s.
__device__ __forceinline__ double2 rot(double c, double2 t, double2 h, double2 g) {
  return cfma(t, g, make_double2(c * h.x, c * h.y));
}

// Principal square root.
__device__ __forceinline__ double2 sqrt2c(double2 w) {
  const double m = hypot(w.x, w.y);
  if (m == 0.0) return make_double2(0.0, 0.0);
  if (w.x >= 0) {
    const double s = sqrt(0.5 * (m + w.x));
    return make_double2(s, w.y / (2 * s));
  }
  const double t = sqrt(0.5 * (m - w.x));
  return make_double2(fabs(w.y) / (2 * t), w.y >= 0 ? t : -t);
}

// Power of two that scales the largest component of a, b, c, d to [1/2, 2).
__device__ __forceinline__ double scale4(double2 a, double2 b, double2 c, double2 d) {
  auto ex = [](double2 v) {
    return max(__double2hiint(v.x) & 0x7ff00000, __double2hiint(v.y) & 0x7ff00000);
  };
  const int e = max(max(ex(a), ex(b)), max(ex(c), ex(d)));
  return __hiloint2double(max(0x7fd00000 - e, 0x00100000), 0);
}

// Eigenvalues of [a b; c d].
__device__ void eig22(double2 a, double2 b, double2 c, double2 d, double2* l1, double2* l2) {
  const double f = scale4(a, b, c, d), g = 1.0 / f;
  const double2 t = make_double2(0.5 * f * (a.x - d.x), 0.5 * f * (a.y - d.y));
  const double2 q = sqrt2c(cfma(t, t, cmul(make_double2(b.x * f, b.y * f),
                                           make_double2(c.x * f, c.y * f))));
  const double2 h = make_double2(0.5 * (a.x + d.x), 0.5 * (a.y + d.y));
  *l1 = make_double2(fma(q.x, g, h.x), fma(q.y, g, h.y));
  *l2 = make_double2(fma(-q.x, g, h.x), fma(-q.y, g, h.y));
}

// Eigenvalue of [a b; c d] nearer d, as a shift: d - bc / (t +- sqrt(t^2 + bc)),
// t = (a - d)/2, the larger denominator, roots and reciprocal to the hardware's
// 2^-20 (the correction to d shrinks with bc, and its error with it).
__device__ __forceinline__ double2 wilkinson(double2 a, double2 b, double2 c, double2 d) {
  const double f = scale4(a, b, c, d);
  const double2 t = make_double2(0.5 * f * (a.x - d.x), 0.5 * f * (a.y - d.y));
  b = make_double2(b.x * f, b.y * f);
  const double2 cs = make_double2(c.x * f, c.y * f);
  const double2 bc = cmul(b, cs), w = cfma(t, t, bc);
  auto root = [](double v) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(fmax(v, DBL_MIN)));
    return y;
  };
  const double n = fma(w.x, w.x, w.y * w.y), m = n * root(n);
  const double h = 0.5 * (m + fabs(w.x)), ih = root(h);
  const double p = h * ih, r = 0.5 * w.y * ih;  // |Re|, Im of the root (or swapped)
  const double2 q = w.x >= 0 ? make_double2(p, r) : make_double2(fabs(r), copysign(p, w.y));
  const double2 p1 = make_double2(t.x + q.x, t.y + q.y), p2 = make_double2(t.x - q.x, t.y - q.y);
  const double2 den = abs1(p1) >= abs1(p2) ? p1 : p2;
  const double dn = fma(den.x, den.x, den.y * den.y);
  if (!(dn > DBL_MIN)) return d;  // bc = 0 with a = d, or not finite
  double id;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(id) : "d"(dn));
  const double2 z = cmul(bc, make_double2(den.x * id, -den.y * id));
  const double g = 1.0 / f;
  return make_double2(d.x - z.x * g, d.y - z.y * g);
}

// Negligible subdiagonal between diagonal entries a and d.
__device__ __forceinline__ bool negligible(double2 sub, double2 a, double2 d) {
  const double v = abs1(sub);
  return v <= DBL_EPSILON * (abs1(a) + abs1(d)) || v < DBL_MIN;
}

typedef double2 SmallMat[kQrSweeps][kQrSweeps + 1];

// Eigenvalues of the Hessenberg S (m x m, m <= 16) into w by single-shift QR;
// one warp, S in shared memory.  Returns false when the iteration limit is
// reached (w then holds the diagonal).
__device__ bool small_eigs(SmallMat& S, int m, double2* w) {
  const int ln = threadIdx.x & 31, j = ln & 15, half = ln >> 4;
  int hi = m - 1, its = 0;
  for (int total = 0; hi >= 0;) {
    // smallest active block ending at hi
    const bool neg = j >= 1 && j <= hi && negligible(S[j][j - 1], S[j - 1][j - 1], S[j][j]);
    const unsigned bits = __ballot_sync(0xffffffffu, neg && half == 0);
    const int lo = bits ? 31 - __clz(bits) : 0;
    if (lo == hi) {
      if (ln == 0) w[hi] = S[hi][hi];
      --hi;
      its = 0;
      continue;
    }
    if (lo == hi - 1) {
      if (ln == 0) {
        double2 l1, l2;
        eig22(S[lo][lo], S[lo][hi], S[hi][lo], S[hi][hi], &l1, &l2);
        w[lo] = l1;
        w[hi] = l2;
      }
      hi -= 2;
      its = 0;
      continue;
    }
    if (++total > 30 * kQrSweeps) {
      for (int i = ln; i <= hi; i += 32) w[i] = S[i][i];
      __syncwarp();
      return false;
    }
    ++its;
    double2 mu = S[hi][hi];
    if (its % 10 == 0)
      mu.x += 0.75 * fabs(S[hi][hi - 1].x);
    else
      mu = wilkinson(S[hi - 1][hi - 1], S[hi - 1][hi], S[hi][hi - 1], mu);
    for (int k = lo; k < hi; ++k) {
      double2 v = S[k + (ln & 1)][max(k - 1, lo)];
      if (k == lo && (ln & 1) == 0) v = make_double2(v.x - mu.x, v.y - mu.y);
      double c;
      double2 s;
      rotation(v, &c, &s);
      // lane (j, half): column j of row k + half; then row j of column k + half
      const int jl = max(lo, k - 1);
      const double2 t = half ? make_double2(-s.x, s.y) : s;  // -conj(s), s
      if (j >= jl && j <= hi) v = rot(c, t, S[k + half][j], S[k + 1 - half][j]);
      if (half && j < k) v = make_double2(0.0, 0.0);
      __syncwarp();
      if (j >= jl && j <= hi) S[k + half][j] = v;
      __syncwarp();
      const int il = min(k + 2, hi);
      const double2 u = half ? make_double2(-s.x, -s.y) : conj2(s);  // -s, conj(s)
      if (j >= lo && j <= il) v = rot(c, u, S[j][k + half], S[j][k + 1 - half]);
      __syncwarp();
      if (j >= lo && j <= il) S[j][k + half] = v;
      __syncwarp();
    }
  }
  __syncwarp();
  return true;
}

struct QrControl {
  int mode, lo, hi, ns;  // mode 0: done, 1: sweep rows lo .. hi with ns shifts
  double2 mu[kQrSweeps];
};

__global__ void __launch_bounds__(kQrCta)
hess_eigenvalues_kernel(double2* __restrict__ H, long long ld, int n, double2* __restrict__ w,
                        int* __restrict__ status, QrControl* ctl) {
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int tid = threadIdx.x, ln = tid & 31, lw = tid >> 5;
  __shared__ SmallMat S;
  __shared__ double2 s_w[kQrSweeps];
  __shared__ int s_defl;
  __shared__ double s_c[kQrSweeps];
  __shared__ double2 s_s[kQrSweeps], s_mu[kQrSweeps];
  auto at = [&](int i, int j) { return __ldcg(&H[(size_t)j * ld + i]); };
  // CTA 0's state
  int hi0 = n - 1, total = 0, stuck = 0;
  for (;;) {
    if (rank == 0) {
      // deflate until a block of more than kQrSweeps rows is active
      for (;;) {
        if (hi0 < 0) {
          if (tid == 0) ctl->mode = 0;
          break;
        }
        if (tid == 0) s_defl = 0;
        __syncthreads();
        for (int k = hi0 - tid; k >= 1; k -= kQrCta)
          if (negligible(at(k, k - 1), at(k - 1, k - 1), at(k, k))) {
            atomicMax(&s_defl, k);
            break;  // smaller k of this thread cannot beat it
          }
        __syncthreads();
        const int lo = s_defl, m = hi0 - lo + 1;
        const int ns = min(kQrSweeps, m < 48 ? 8 : kQrSweeps);
        const int base = m <= kQrSweeps ? lo : hi0 - ns + 1, mm = m <= kQrSweeps ? m : ns;
        for (int v = tid; v < mm * mm; v += kQrCta) S[v % mm][v / mm] = at(base + v % mm, base + v / mm);
        __syncthreads();
        if (lw == 0) {
          // entries below the subdiagonal are zero in memory (bulges are
          // cleared, reflectors are not stored there)
          const bool good = small_eigs(S, mm, s_w);
          if (ln == 0) s_defl = good ? 1 : 0;
        }
        __syncthreads();
        const bool good = s_defl != 0;
        if (m <= kQrSweeps) {
          if (tid < m) w[lo + tid] = s_w[tid];
          if (!good && tid == 0) status[0] = hi0 + 1;
          hi0 = lo - 1;
          stuck = 0;
          __syncthreads();
          if (!good) {
            if (tid == 0) ctl->mode = 0;
            break;
          }
          continue;
        }
        total += ns;
        if (total > kQrMaxIt * max(10, n)) {
          if (tid == 0) {
            status[0] = hi0 + 1;
            ctl->mode = 0;
          }
          break;
        }
        if (tid == 0) {
          ctl->mode = 1;
          ctl->lo = lo;
          ctl->hi = hi0;
          ctl->ns = ns;
        }
        if (tid < ns) {
          double2 mu = s_w[tid];
          // every sixth time without a deflation at the end: exceptional shifts
          if (stuck % 6 == 5) {
            mu = at(hi0 - tid, hi0 - tid);
            mu.x += 0.75 * abs1(at(hi0 - tid, hi0 - tid - 1));
          }
          ctl->mu[tid] = mu;
        }
        ++stuck;
        break;
      }
    }
    cl.sync();
    const int mode = __ldcg(&ctl->mode);
    if (mode == 0) break;
    const int lo = __ldcg(&ctl->lo), hi = __ldcg(&ctl->hi), ns = __ldcg(&ctl->ns);
    if (tid < ns) s_mu[tid] = __ldcg(&ctl->mu[tid]);
    __syncthreads();
    const int gw = rank * (kQrCta / 32) + lw, nwarps = C * (kQrCta / 32);
    const int b = gw % ns, per = nwarps / ns;        // this warp's sweep, warps per sweep
    const int part = gw / ns;                        // parts beyond `per` idle
    const int steps = hi - lo + kQrGap * (ns - 1);
    for (int t = 0; t < steps; ++t) {
      // all rotations of the step, two lanes each, in every CTA
      if (lw == 0) {
        const int q = ln >> 1, k = lo + t - kQrGap * q;
        const bool live = q < ns && k >= lo && k < hi;
        double2 v = make_double2(0.0, 0.0);
        if (live) v = at(k + (ln & 1), max(k - 1, lo));
        if (live && k == lo && (ln & 1) == 0) v = make_double2(v.x - s_mu[q].x, v.y - s_mu[q].y);
        double c;
        double2 s;
        rotation(v, &c, &s);
        if (live && (ln & 1) == 0) {
          s_c[q] = c;
          s_s[q] = s;
        }
      }
      // The row phase leaves column k - 1 alone (the column phase writes it),
      // so only a starting sweep's elements could change while another CTA
      // still reads them.
      if (t % kQrGap == 0 && t / kQrGap < ns)
        cl.sync();
      else
        __syncthreads();
      const int k = lo + t - kQrGap * b;
      const bool on = part < per && k >= lo && k < hi;
      double c = 1.0;
      double2 s = make_double2(0.0, 0.0);
      if (on) {
        c = s_c[b];
        s = s_s[b];
        for (int j = k + part * 32 + ln; j <= hi; j += per * 32) {
          double2* p = H + (size_t)j * ld + k;
          const double2 h1 = __ldcg(p), h2 = __ldcg(p + 1);
          __stcg(p, rot(c, s, h1, h2));
          __stcg(p + 1, rot(c, make_double2(-s.x, s.y), h2, h1));
        }
      }
      cl.sync();
      if (on) {
        const int il = min(k + 2, hi);
        for (int i = lo + part * 32 + ln; i <= il; i += per * 32) {
          double2* p = H + (size_t)k * ld + i;
          const double2 h1 = __ldcg(p), h2 = __ldcg(p + ld);
          __stcg(p, rot(c, conj2(s), h1, h2));
          __stcg(p + ld, rot(c, make_double2(-s.x, -s.y), h2, h1));
        }
        if (k > lo && part == 0 && ln == 0) {
          double2* p = H + (size_t)(k - 1) * ld + k;
          __stcg(p, rot(c, s, __ldcg(p), __ldcg(p + 1)));
          __stcg(p + 1, make_double2(0.0, 0.0));
        }
      }
      cl.sync();
    }
  }
}

}  // namespace

size_t hess_eigenvalues_work_bytes() { return sizeof(QrControl); }

int launch_hess_eigenvalues(double2* H, int n, double2* w, int* status, void* work,
                            cudaStream_t s) {
  static PerDevice<bool> non_portable(false);
  static PerDeviceOnce attr;
  const int dev = current_device();
  attr(dev, [&] {
    non_portable[dev] =
        cudaFuncSetAttribute(hess_eigenvalues_kernel,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  });
  const bool big = non_portable[dev];
  cudaMemsetAsync(status, 0, sizeof(int), s);
  for (int C : {big ? 16 : 8, 8}) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(kQrCta);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, hess_eigenvalues_kernel, H, (long long)n, n, w, status,
                           static_cast<QrControl*>(work)) == cudaSuccess)
      return BEM2D_OK;
    cudaGetLastError();
  }
  return BEM2D_ERR_CUDA;
}

}  // namespace bem2d_gpu
