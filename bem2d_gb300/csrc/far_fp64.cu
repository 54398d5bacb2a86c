// FP64 far field and potentials (sm_103a): node pairs evaluated with the
// table form of H0 and H1 (hankel_tab.cuh), real and complex wavenumbers.
//
//  hankel_tab_kernel  fills the table of one ray arg z
//  far_fp64_kernel    tensor Gauss rule (Integrate<kernel, Gauss2D>,
//                     lib/bem2d_quadrature.h:37-65, for the pairs selected at
//                     :283-287), both orientations of a pair in one pass
//  potential_kernel   EvalKernel (lib/bem2d_quadrature.h:184-228)
#include <algorithm>
#include <cmath>
#include <mutex>

#include "common.cuh"
#include "hankel_tab.cuh"

namespace bem2d_gpu {

// ---- table -------------------------------------------------------------------
// One half-warp per interval: lane l evaluates Chebyshev point l, the
// discrete Chebyshev sums a_j = (2/16) sum_l f_l cos(j theta_l), j <= 6, are
// formed by all lanes, and lane 0 converts sum a_j T_j(2w) to powers of w.
__global__ void __launch_bounds__(128)
hankel_tab_kernel(double ur, double ui, double2* __restrict__ tcd, float* __restrict__ tct,
                  double2* __restrict__ tsc) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id < kHtTrig) {
    double s, c;
    sincospi((double)id / (kHtTrig / 2), &s, &c);
    tsc[id] = make_double2(c, s);
  }
  const int bin = min(id / kHtNodes, kHtBins - 1), l = id % kHtNodes;
  const int oct = bin / kHtPerOct, j0 = bin % kHtPerOct;
  const double scale = ldexp(1.0, kHtOct0 + oct - 6);  // interval length
  const double lo = (double)(kHtPerOct + j0) * scale;
  double sv, v;  // Chebyshev point
  sincospi((l + 0.5) / kHtNodes, &sv, &v);
  const double x = fma(0.5 * (v + 1.0), scale, lo);
  cd g0, g1;
  hankel_scaled(x, ur, ui, &g0, &g1);
  const double f[4] = {g0.re, g0.im, g1.re, g1.im};
#pragma unroll 1
  for (int fn = 0; fn < 4; ++fn) {
    double a[7];
#pragma unroll
    for (int j = 0; j < 7; ++j) {
      double t = f[fn] * cospi(j * (l + 0.5) / kHtNodes);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      a[j] = t * (2.0 / kHtNodes);
    }
    if (l != 0 || id / kHtNodes >= kHtBins) continue;
    // powers of v, then of w = v / 2
    const double c0 = 0.5 * a[0] - a[2] + a[4] - a[6], c1 = a[1] - 3 * a[3] + 5 * a[5],
                 c2 = 2 * a[2] - 8 * a[4] + 18 * a[6], c3 = 4 * a[3] - 20 * a[5],
                 c4 = 8 * a[4] - 48 * a[6], c5 = 16 * a[5], c6 = 32 * a[6];
    double2* c = tcd + (size_t)bin * 8 + 2 * fn;
    c[0] = make_double2(c0, 2 * c1);
    c[1] = make_double2(4 * c2, 8 * c3);
    float* t = tct + (size_t)bin * 12 + fn;
    t[0] = (float)(16 * c4);
    t[4] = (float)(32 * c5);
    t[8] = (float)(64 * c6);
  }
}

void launch_hankel_tab(void* tab, double k, double ki, cudaStream_t s) {
  const HankelTab t = hankel_tab_at(tab);
  const double ka = ki == 0.0 ? std::abs(k) : std::hypot(k, ki);
  hankel_tab_kernel<<<(kHtBins * kHtNodes + 127) / 128, 128, 0, s>>>(
      ki == 0.0 ? 1.0 : k / ka, ki == 0.0 ? 0.0 : ki / ka, const_cast<double2*>(t.cd),
      reinterpret_cast<float*>(const_cast<float4*>(t.ct)), const_cast<double2*>(t.sc));
}

// The table of real wavenumbers (one per device, the same for all of them).
static const void* hankel_tab_real() {
  constexpr int kMaxDev = 64;
  static std::mutex mu;
  static void* tab[kMaxDev] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= kMaxDev) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (!tab[dev]) {
    void* d = nullptr;
    cudaStream_t s = nullptr;
    if (cudaMalloc(&d, kHtBytes) != cudaSuccess) return nullptr;
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) {
      cudaFree(d);
      return nullptr;
    }
    launch_hankel_tab(d, 1.0, 0.0, s);
    const cudaError_t e = cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
    if (e != cudaSuccess) {
      cudaFree(d);
      return nullptr;
    }
    tab[dev] = d;
  }
  return tab[dev];
}

size_t hankel_tab_bytes() { return kHtBytes; }

// ---- far field ---------------------------------------------------------------
// Bound by the FP64 pipe (90 % of its rate by ncu at kite N = 2048).  Per node
// pair 70 FP64 instructions serve entry (i, j) and entry (j, i) of every
// basis-function pair of the two elements: the distance, 1/d, H0 and H1 are
// shared, an orientation adds its normal factor n . (x - y), a basis function
// its weight.  Measured against one direct evaluation (hankel01_d, ~175
// instructions) per entry and node pair: kite N = 2048 31.2 -> 7.5 ms; 801
// elements of PolBasis(2), N = 2403, 32.3 -> 1.24 ms; disk N = 160 2.1 -> 0.15
// ms; complex wavenumber, N = 512, 113.6 -> 1.5 ms (hankel01_c sums up to 105
// complex square roots per evaluation).
//
// Unknowns are taken in groups: runs of up to NB consecutive unknowns of one
// element (the element-major order of Geometry::FlatMap).  A CTA takes 32
// groups as rows, one per lane, against `cols` groups as columns, and only
// the pairs with row < column.
//  NB = 1: warp w integrates the test nodes w, w + warps, ... of the batch's
//    columns, one after another; the warps' partial sums meet in shared
//    memory and warp w stores column w of the batch.  Splitting a pair over
//    warps keeps the chip busy at small orders (160 unknowns are 400
//    (32-row, column) tasks of 25 node pairs for 152 SMs).
//  NB > 1: a warp owns a column; 2 NB^2 sums per lane stay in registers.
constexpr int kFarWarps = 5;

struct FarGroups {
  const int2* grp;  // first unknown, count; null: group i = unknown i
  int n;
};

template <int KERNEL, int NB, bool CK>
__global__ void __launch_bounds__(32 * kFarWarps)
far_fp64_kernel(DevGeom g, NodeTable t, FarGroups fg, int ng, int cols, HankelTab tb,
                double kr, double ki, double ka, double eta, double alpha,
                double2* __restrict__ out, long long ld) {
  constexpr bool kH0 = KERNEL == BEM2D_KERNEL_SINGLE || KERNEL == BEM2D_KERNEL_COMBINED;
  constexpr bool kH1 = KERNEL != BEM2D_KERNEL_SINGLE;
  const int row0 = blockIdx.y * 32, col0 = blockIdx.x * cols;
  if (col0 + cols <= row0 + 1) return;  // no pair with row < column
  extern __shared__ double smem[];
  const int SZ = ng * 32;
  double* rs = smem;                       // [4 + NB][ng][32] x, y, nx, ny, weights
  double* cs = rs + (4 + NB) * SZ;         // [cols][ng][4 + NB]
  double* red = cs + (size_t)cols * ng * (4 + NB);  // NB = 1: [warps cols][warps][4][32]
  __shared__ long long lk[3][32];
  const int nw = blockDim.x >> 5;
  for (int v = threadIdx.x; v < SZ; v += blockDim.x) {
    const int q = v >> 5, l = v & 31;
    const int gi = min(row0 + l, fg.n - 1);
    const int2 u = fg.grp ? fg.grp[gi] : make_int2(gi, 1);
    const size_t o = (size_t)u.x * ng + q;
    rs[v] = t.x[o];
    rs[SZ + v] = t.y[o];
    rs[2 * SZ + v] = t.nx[o];
    rs[3 * SZ + v] = t.ny[o];
#pragma unroll
    for (int b = 0; b < NB; ++b) rs[(4 + b) * SZ + v] = b < u.y ? t.w[o + (size_t)b * ng] : 0.0;
  }
  for (int v = threadIdx.x; v < cols * ng; v += blockDim.x) {
    const int c = v / ng, q = v - c * ng;
    const int gi = min(col0 + c, fg.n - 1);
    const int2 u = fg.grp ? fg.grp[gi] : make_int2(gi, 1);
    const size_t o = (size_t)u.x * ng + q;
    double* p = cs + (size_t)v * (4 + NB);
    p[0] = t.x[o];
    p[1] = t.y[o];
    p[2] = t.nx[o];
    p[3] = t.ny[o];
#pragma unroll
    for (int b = 0; b < NB; ++b) p[4 + b] = b < u.y ? t.w[o + (size_t)b * ng] : 0.0;
  }
  if (threadIdx.x < 32) {
    const int gi = min(row0 + (int)threadIdx.x, fg.n - 1);
    const int e = g.unk_elem[fg.grp ? fg.grp[gi].x : gi];
    lk[0][threadIdx.x] = g.index[e];
    lk[1][threadIdx.x] = g.next[e];
    lk[2][threadIdx.x] = g.prev[e];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = row0 + lane;
  const long long ri = lk[0][lane], rn = lk[1][lane], rp = lk[2][lane];
  const int2 ur = fg.grp ? fg.grp[min(row, fg.n - 1)] : make_int2(row, 1);

  // The kernels as  F H1 (n . w) / d + E H0:  F = -i k/4, E = eta/4 (combined)
  // or i/4 (single layer)
  const double fr = CK ? 0.25 * ki : 0.0, fi = -0.25 * kr, eq = 0.25 * eta;

  // wanted orientations of (row, column c): rc = entry (row, col), cr = (col, row)
  auto wanted = [&](int c, bool* rc, bool* cr) {
    const int col = col0 + c;
    *rc = *cr = false;
    if (c >= cols || col >= fg.n || row >= col) return;
    const int e = g.unk_elem[fg.grp ? fg.grp[col].x : col];
    const long long ci = g.index[e];
    *rc = !(ri == ci || rn == ci || rp == ci);
    *cr = !(ci == ri || g.next[e] == ri || g.prev[e] == ri);
  };

  if constexpr (NB == 1) {
    for (int c0 = 0; c0 < cols; c0 += nw) {
      const int cend = min(c0 + nw, cols);
      for (int c = c0; c < cend; ++c) {
        bool rc, cr;
        wanted(c, &rc, &cr);
        double a1r = 0, a1i = 0, a2r = 0, a2i = 0;
        if (rc || cr) {
          for (int q1 = warp; q1 < ng; q1 += nw) {
            const int o1 = q1 * 32 + lane;
            const double x1 = rs[o1], y1 = rs[SZ + o1], n1x = rs[2 * SZ + o1],
                         n1y = rs[3 * SZ + o1], w1 = rs[4 * SZ + o1];
            const double* cp = cs + (size_t)c * ng * 5;
            double t1r = 0, t1i = 0, t2r = 0, t2i = 0, s0r = 0, s0i = 0;
#pragma unroll 1
            for (int q2 = 0; q2 < ng; ++q2, cp += 5) {
              const double wx = x1 - cp[0], wy = y1 - cp[1], w2 = cp[4];
              double rd, h0r, h0i, h1r, h1i;
              hankel_tab_eval<kH0, kH1, CK>(tb, wx, wy, kr, ki, ka, &rd, &h0r, &h0i, &h1r, &h1i);
              if (kH0) {
                s0r = fma(w2, h0r, s0r);
                s0i = fma(w2, h0i, s0i);
              }
              if (kH1) {
                const double gw = w2 * rd, gr = gw * h1r, gi = gw * h1i;
                const double n1w = fma(n1x, wx, n1y * wy), n2w = fma(cp[2], wx, cp[3] * wy);
                // -n2w, n1w (double layer); n1w, -n2w (its adjoint)
                const double m1 = KERNEL == BEM2D_KERNEL_DOUBLE ? -n2w : n1w;
                const double m2 = KERNEL == BEM2D_KERNEL_DOUBLE ? n1w : -n2w;
                t1r = fma(m1, gr, t1r);
                t1i = fma(m1, gi, t1i);
                t2r = fma(m2, gr, t2r);
                t2i = fma(m2, gi, t2i);
              }
            }
            if (KERNEL == BEM2D_KERNEL_SINGLE) {
              a1r = fma(w1, s0r, a1r);
              a1i = fma(w1, s0i, a1i);
            } else {
              const double er = kH0 ? eq * s0r : 0.0, ei = kH0 ? eq * s0i : 0.0;
              double zr = fma(-fi, t1i, er), zi = fma(fi, t1r, ei);
              if (CK) {
                zr = fma(fr, t1r, zr);
                zi = fma(fr, t1i, zi);
              }
              a1r = fma(w1, zr, a1r);
              a1i = fma(w1, zi, a1i);
              zr = fma(-fi, t2i, er);
              zi = fma(fi, t2r, ei);
              if (CK) {
                zr = fma(fr, t2r, zr);
                zi = fma(fr, t2i, zi);
              }
              a2r = fma(w1, zr, a2r);
              a2i = fma(w1, zi, a2i);
            }
          }
        }
        double* rd_ = red + ((size_t)(c - c0) * nw + warp) * 128 + lane;
        rd_[0] = a1r;
        rd_[32] = a1i;
        rd_[64] = a2r;
        rd_[96] = a2i;
      }
      __syncthreads();
      {
        const int c = c0 + warp, col = col0 + c;
        bool rc = false, cr = false;
        if (c < cend) wanted(c, &rc, &cr);
        if (rc || cr) {
          double a1r = 0, a1i = 0, a2r = 0, a2i = 0;
          for (int k = 0; k < nw; ++k) {
            const double* p = red + ((size_t)warp * nw + k) * 128 + lane;
            a1r += p[0];
            a1i += p[32];
            a2r += p[64];
            a2i += p[96];
          }
          if (KERNEL == BEM2D_KERNEL_SINGLE) {  // (i/4) H0, both orientations
            const double zr = -0.25 * a1i, zi = 0.25 * a1r;
            a1r = a2r = zr;
            a1i = a2i = zi;
          }
          const int uc = fg.grp ? fg.grp[col].x : col;
          if (rc) out[(size_t)uc * ld + ur.x] = make_double2(alpha * a1r, alpha * a1i);
          if (cr) out[(size_t)ur.x * ld + uc] = make_double2(alpha * a2r, alpha * a2i);
        }
      }
      __syncthreads();
    }
  } else {
    for (int c = warp; c < cols; c += nw) {
      bool rc, cr;
      wanted(c, &rc, &cr);
      if (!rc && !cr) continue;
      // acc[a][b]: row basis a, column basis b
      double2 A1[NB][NB], A2[NB][NB];
#pragma unroll
      for (int a = 0; a < NB; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b) A1[a][b] = A2[a][b] = make_double2(0.0, 0.0);
#pragma unroll 1
      for (int q1 = 0; q1 < ng; ++q1) {
        const int o1 = q1 * 32 + lane;
        const double x1 = rs[o1], y1 = rs[SZ + o1], n1x = rs[2 * SZ + o1], n1y = rs[3 * SZ + o1];
        double2 p1[NB], p2[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) p1[b] = p2[b] = make_double2(0.0, 0.0);
        const double* cp = cs + (size_t)c * ng * (4 + NB);
#pragma unroll 1
        for (int q2 = 0; q2 < ng; ++q2, cp += 4 + NB) {
          const double wx = x1 - cp[0], wy = y1 - cp[1];
          double rd, h0r, h0i, h1r, h1i;
          hankel_tab_eval<kH0, kH1, CK>(tb, wx, wy, kr, ki, ka, &rd, &h0r, &h0i, &h1r, &h1i);
          double k1r, k1i, k2r, k2i;
          if (KERNEL == BEM2D_KERNEL_SINGLE) {
            k1r = k2r = h0r;  // times i/4 at the end
            k1i = k2i = h0i;
          } else {
            const double n1w = fma(n1x, wx, n1y * wy), n2w = fma(cp[2], wx, cp[3] * wy);
            const double m1 = rd * (KERNEL == BEM2D_KERNEL_DOUBLE ? -n2w : n1w);
            const double m2 = rd * (KERNEL == BEM2D_KERNEL_DOUBLE ? n1w : -n2w);
            // F H1
            double zr = -fi * h1i, zi = fi * h1r;
            if (CK) {
              zr = fma(fr, h1r, zr);
              zi = fma(fr, h1i, zi);
            }
            if (kH0) {
              const double er = eq * h0r, ei = eq * h0i;
              k1r = fma(m1, zr, er);
              k1i = fma(m1, zi, ei);
              k2r = fma(m2, zr, er);
              k2i = fma(m2, zi, ei);
            } else {
              k1r = m1 * zr;
              k1i = m1 * zi;
              k2r = m2 * zr;
              k2i = m2 * zi;
            }
          }
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            const double w2 = cp[4 + b];
            p1[b].x = fma(w2, k1r, p1[b].x);
            p1[b].y = fma(w2, k1i, p1[b].y);
            if (KERNEL != BEM2D_KERNEL_SINGLE) {
              p2[b].x = fma(w2, k2r, p2[b].x);
              p2[b].y = fma(w2, k2i, p2[b].y);
            }
          }
        }
#pragma unroll
        for (int a = 0; a < NB; ++a) {
          const double w1 = rs[(4 + a) * SZ + o1];
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            A1[a][b].x = fma(w1, p1[b].x, A1[a][b].x);
            A1[a][b].y = fma(w1, p1[b].y, A1[a][b].y);
            if (KERNEL != BEM2D_KERNEL_SINGLE) {
              A2[a][b].x = fma(w1, p2[b].x, A2[a][b].x);
              A2[a][b].y = fma(w1, p2[b].y, A2[a][b].y);
            }
          }
        }
      }
      const int2 uc = fg.grp ? fg.grp[col0 + c] : make_int2(col0 + c, 1);
#pragma unroll
      for (int a = 0; a < NB; ++a)
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          if (a >= ur.y || b >= uc.y) continue;
          double2 v1 = A1[a][b], v2 = A2[a][b];
          if (KERNEL == BEM2D_KERNEL_SINGLE) v1 = v2 = make_double2(-0.25 * v1.y, 0.25 * v1.x);
          if (rc)
            out[(size_t)(uc.x + b) * ld + ur.x + a] = make_double2(alpha * v1.x, alpha * v1.y);
          if (cr)
            out[(size_t)(ur.x + a) * ld + uc.x + b] = make_double2(alpha * v2.x, alpha * v2.y);
        }
    }
  }
}

template <int KERNEL, int NB, bool CK>
static void launch_far_nb(const DevGeom& g, const NodeTable& t, const FarGroups& fg, int ng,
                          double k, double ki, double eta, double alpha, const HankelTab& tb,
                          double2* out, long long ld, cudaStream_t s) {
  const double ka = CK ? std::hypot(k, ki) : k;
  const int nw = NB == 1 ? std::min(ng, kFarWarps) : kFarWarps;
  const int rows = (fg.n + 31) / 32;
  // columns per CTA: up to 40, fewer while the triangle of CTAs would not
  // give every SM a few (their cost is the staging of 32 + cols groups)
  int cols = 8 * kFarWarps;
  while (cols > kFarWarps && (long long)rows * ((fg.n + cols - 1) / cols) / 2 < 8LL * device_sms())
    cols /= 2;
  const size_t per_col = sizeof(double) * ng * (4 + NB);
  const size_t fixed = sizeof(double) * ((size_t)(4 + NB) * ng * 32 +
                                         (NB == 1 ? (size_t)nw * nw * 128 : 0));
  while (cols > 1 && fixed + per_col * cols > 200 * 1024) cols /= 2;
  const size_t smem = fixed + per_col * cols;
  const dim3 grid((fg.n + cols - 1) / cols, rows);
  auto fn = far_fp64_kernel<KERNEL, NB, CK>;
  // one value for all rules: calls of several threads must not undo each other
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)std::max<size_t>(smem, 208 * 1024));
  fn<<<grid, 32 * nw, smem, s>>>(g, t, fg, ng, cols, tb, k, ki, ka, eta, alpha, out, ld);
}

template <int KERNEL, bool CK>
static void launch_far_k(const DevGeom& g, const NodeTable& t, const int2* grp, int ngrp, int nb,
                         int ng, double k, double ki, double eta, double alpha,
                         const HankelTab& tb, double2* out, long long ld, cudaStream_t s) {
  if (nb <= 1)
    launch_far_nb<KERNEL, 1, CK>(g, t, FarGroups{nullptr, g.n_unk}, ng, k, ki, eta, alpha, tb,
                                 out, ld, s);
  else if (nb == 2)
    launch_far_nb<KERNEL, 2, CK>(g, t, FarGroups{grp, ngrp}, ng, k, ki, eta, alpha, tb, out, ld,
                                 s);
  else
    launch_far_nb<KERNEL, 3, CK>(g, t, FarGroups{grp, ngrp}, ng, k, ki, eta, alpha, tb, out, ld,
                                 s);
}

template <bool CK>
static void launch_far_any(const DevGeom& g, const NodeTable& t, const int2* grp, int ngrp,
                           int nb, int ng, int kernel, double k, double ki, double eta,
                           double alpha, const HankelTab& tb, double2* out, long long ld,
                           cudaStream_t s) {
  switch (kernel) {
    case BEM2D_KERNEL_SINGLE:
      launch_far_k<BEM2D_KERNEL_SINGLE, CK>(g, t, grp, ngrp, nb, ng, k, ki, eta, alpha, tb, out,
                                            ld, s);
      break;
    case BEM2D_KERNEL_DOUBLE:
      launch_far_k<BEM2D_KERNEL_DOUBLE, CK>(g, t, grp, ngrp, nb, ng, k, ki, eta, alpha, tb, out,
                                            ld, s);
      break;
    case BEM2D_KERNEL_CONJDOUBLE:
      launch_far_k<BEM2D_KERNEL_CONJDOUBLE, CK>(g, t, grp, ngrp, nb, ng, k, ki, eta, alpha, tb,
                                                out, ld, s);
      break;
    default:
      launch_far_k<BEM2D_KERNEL_COMBINED, CK>(g, t, grp, ngrp, nb, ng, k, ki, eta, alpha, tb, out,
                                              ld, s);
  }
}

int launch_far_fp64(const DevGeom& g, const NodeTable& t, const int2* grp, int ngrp, int nb,
                    int ng, int kernel, double k, double ki, double eta, double alpha,
                    double2* out, long long ld, void* ck_tab, cudaStream_t s) {
  if (ki != 0.0) {
    launch_hankel_tab(ck_tab, k, ki, s);
    launch_far_any<true>(g, t, grp, ngrp, nb, ng, kernel, k, ki, eta, alpha,
                         hankel_tab_at(ck_tab), out, ld, s);
    return BEM2D_OK;
  }
  const void* tab = hankel_tab_real();
  if (!tab) return BEM2D_ERR_NOMEM;
  launch_far_any<false>(g, t, grp, ngrp, nb, ng, kernel, k, 0.0, eta, alpha,
                        hankel_tab_at(const_cast<void*>(tab)), out, ld, s);
  return BEM2D_OK;
}

// ---- potentials ----------------------------------------------------------------
// out[p] = sum_u c_u sum_q K(x_p, y_uq) W_uq, both normals the source node's.
// One thread per point; blockIdx.y takes a slice of the nodes, staged through
// shared memory with c_u W_uq formed once per CTA; the slices' partial sums
// are added in order by potential_sum_kernel.  Slices make the work even:
// 40,000 points alone are 313 CTAs, which 152 SMs finish in three rounds of
// which the last is nearly empty.  FP64 pipe: about 45 instructions per
// (point, node) for the single layer; 40,000 points, 1,024 elements, 57.9 ->
// 16.5 ms against one slice and direct evaluation.
constexpr int kPotThreads = 128;
constexpr int kPotCtas = 24;  // per SM

template <int KERNEL, bool CK>
__global__ void __launch_bounds__(kPotThreads)
potential_kernel(int total, int slice, NodeTable t, int ng, HankelTab tb, double kr, double ki,
                 double ka, double eta, const double2* __restrict__ coef, int npts,
                 const double* __restrict__ pts, double2* __restrict__ part) {
  constexpr bool kH0 = KERNEL == BEM2D_KERNEL_SINGLE || KERNEL == BEM2D_KERNEL_COMBINED;
  constexpr bool kH1 = KERNEL != BEM2D_KERNEL_SINGLE;
  __shared__ double sx[kPotThreads], sy[kPotThreads], snx[kPotThreads], sny[kPotThreads];
  __shared__ double2 sc[kPotThreads];  // c_u W_uq
  const int p = blockIdx.x * kPotThreads + threadIdx.x;
  const double px = p < npts ? pts[2 * p] : 0.0, py = p < npts ? pts[2 * p + 1] : 0.0;
  const double fr = CK ? 0.25 * ki : 0.0, fi = -0.25 * kr, eq = 0.25 * eta;
  double ar = 0.0, ai = 0.0, br = 0.0, bi = 0.0;  // H0 sum, H1 sum
  const int v0 = blockIdx.y * slice, v1 = min(v0 + slice, total);
  for (int base = v0; base < v1; base += kPotThreads) {
    const int v = base + threadIdx.x;
    __syncthreads();
    if (v < v1) {
      sx[threadIdx.x] = t.x[v];
      sy[threadIdx.x] = t.y[v];
      snx[threadIdx.x] = t.nx[v];
      sny[threadIdx.x] = t.ny[v];
      const double2 c = coef[v / ng];
      const double w = t.w[v];
      sc[threadIdx.x] = make_double2(c.x * w, c.y * w);
    }
    __syncthreads();
    const int cnt = min(kPotThreads, v1 - base);
    if (p < npts) {
#pragma unroll 1
      for (int i = 0; i < cnt; ++i) {
        const double wx = px - sx[i], wy = py - sy[i];
        double rd, h0r, h0i, h1r, h1i;
        hankel_tab_eval<kH0, kH1, CK>(tb, wx, wy, kr, ki, ka, &rd, &h0r, &h0i, &h1r, &h1i);
        const double2 c = sc[i];
        if (kH0) {
          ar = fma(c.x, h0r, fma(-c.y, h0i, ar));
          ai = fma(c.x, h0i, fma(c.y, h0r, ai));
        }
        if (kH1) {
          const double nw = fma(snx[i], wx, sny[i] * wy);
          const double m = rd * (KERNEL == BEM2D_KERNEL_DOUBLE ? -nw : nw);
          const double cx = c.x * m, cy = c.y * m;
          br = fma(cx, h1r, fma(-cy, h1i, br));
          bi = fma(cx, h1i, fma(cy, h1r, bi));
        }
      }
    }
  }
  if (p >= npts) return;
  double2 r;
  if (KERNEL == BEM2D_KERNEL_SINGLE) {
    r = make_double2(-0.25 * ai, 0.25 * ar);
  } else {
    r = make_double2(fr * br - fi * bi, fma(fi, br, fr * bi));
    if (kH0) {
      r.x = fma(eq, ar, r.x);
      r.y = fma(eq, ai, r.y);
    }
  }
  part[(size_t)blockIdx.y * npts + p] = r;
}

__global__ void potential_sum_kernel(int npts, int slices, const double2* __restrict__ part,
                                     double2* __restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npts) return;
  double2 r = part[p];
  for (int s = 1; s < slices; ++s) {
    const double2 v = part[(size_t)s * npts + p];
    r.x += v.x;
    r.y += v.y;
  }
  out[p] = r;
}

// Slices of the nodes (whole staging chunks): about 24 CTAs per SM, one slice
// (no partial sums) once the points alone give that many.
static int potential_slices(int npts, int nodes) {
  const int blocks = (npts + kPotThreads - 1) / kPotThreads;
  const int chunks = (nodes + kPotThreads - 1) / kPotThreads;
  return std::max(1, std::min(chunks, (kPotCtas * device_sms() + blocks - 1) / blocks));
}

size_t potential_part_bytes(int npts, int nodes) {
  const int s = potential_slices(npts, nodes);
  return s > 1 ? sizeof(double2) * (size_t)s * npts : 0;
}

template <int KERNEL>
static void launch_potential_k(const NodeTable& t, int total, int slice, int slices, int ng,
                               double k, double ki, double eta, const HankelTab& tb,
                               const double2* coef, int npts, const double* pts, double2* part,
                               cudaStream_t s) {
  const dim3 grid((npts + kPotThreads - 1) / kPotThreads, slices);
  if (ki != 0.0)
    potential_kernel<KERNEL, true><<<grid, kPotThreads, 0, s>>>(
        total, slice, t, ng, tb, k, ki, std::hypot(k, ki), eta, coef, npts, pts, part);
  else
    potential_kernel<KERNEL, false><<<grid, kPotThreads, 0, s>>>(total, slice, t, ng, tb, k, 0.0,
                                                                 k, eta, coef, npts, pts, part);
}

int launch_potential(const DevGeom& g, const NodeTable& t, int ng, int kernel, double k,
                     double ki, double eta, const double2* coef, int npts, const double* pts,
                     double2* out, double2* part, void* ck_tab, cudaStream_t s) {
  const void* tab = ck_tab;
  if (ki != 0.0)
    launch_hankel_tab(ck_tab, k, ki, s);
  else if (!(tab = hankel_tab_real()))
    return BEM2D_ERR_NOMEM;
  const HankelTab tb = hankel_tab_at(const_cast<void*>(tab));
  const int total = g.n_unk * ng, chunks = (total + kPotThreads - 1) / kPotThreads;
  const int per = (chunks + potential_slices(npts, total) - 1) / potential_slices(npts, total);
  const int slice = per * kPotThreads, slices = (chunks + per - 1) / per;
  if (slices == 1) part = out;
  switch (kernel) {
    case BEM2D_KERNEL_SINGLE:
      launch_potential_k<BEM2D_KERNEL_SINGLE>(t, total, slice, slices, ng, k, ki, eta, tb, coef,
                                              npts, pts, part, s);
      break;
    case BEM2D_KERNEL_DOUBLE:
      launch_potential_k<BEM2D_KERNEL_DOUBLE>(t, total, slice, slices, ng, k, ki, eta, tb, coef,
                                              npts, pts, part, s);
      break;
    case BEM2D_KERNEL_CONJDOUBLE:
      launch_potential_k<BEM2D_KERNEL_CONJDOUBLE>(t, total, slice, slices, ng, k, ki, eta, tb,
                                                  coef, npts, pts, part, s);
      break;
    default:
      launch_potential_k<BEM2D_KERNEL_COMBINED>(t, total, slice, slices, ng, k, ki, eta, tb, coef,
                                                npts, pts, part, s);
  }
  if (slices > 1)
    potential_sum_kernel<<<(npts + 127) / 128, 128, 0, s>>>(npts, slices, part, out);
  return BEM2D_OK;
}

}  // namespace bem2d_gpu
