// The near-field kernel and its launch, for the translation units that
// instantiate it: real wavenumbers (assembly.cu) and complex ones (near_ck.cu).
// Two, because a program loads a translation unit's kernels with its first launch.
#pragma once

#include <algorithm>

#include "common.cuh"
#include "ff.cuh"
#include "kernel_ff.cuh"

namespace bem2d_gpu {

// ---------------------------------------------------------------------------
// Near field: one warp per (test, trial) pair of adjacent or identical
// elements.  Lanes stride over the rule's points; a shuffle tree reduces.
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// mass-matrix entry of a same-index pair (EvalIdent's inner loop)
__device__ __forceinline__ double mass_entry(const DevGeom& g, const DevRules& r,
                                             int ui, int uj) {
  const int ej = g.unk_elem[uj];
  double m = 0.0;
  for (int q = 0; q < r.ng; ++q) {
    const double tq = r.gx[q];
    const ElemPt p = elem_eval(g.kind[ej], g.param + 8 * (size_t)ej, tq);
    m += elem_jac(p) * basis_eval(g.unk_kind[ui], g.unk_param[ui], tq) *
         basis_eval(g.unk_kind[uj], g.unk_param[uj], tq) * r.gw[q];
  }
  return m;
}

// Element geometry at the distinct coordinates of a rule, per warp in shared
// memory (structure of arrays): Map, Normal and |J| phi, phi the basis
// functions of the pair's unknowns on that element (basis b at f + b cap).
struct GeoTab {
  double* x;
  double* y;
  double* nx;
  double* ny;
  double* f;
  int cap;
};

// Geometry of element e and the basis functions of its unknowns u .. u + nu - 1.
template <int NB>
__device__ __forceinline__ void geo_fill(const DevGeom& g, int e, int u, int nu,
                                         const double* vals, int n, bool mirror, const GeoTab& tb,
                                         int off, int lane) {
  const double* prm = g.param + 8 * (size_t)e;
  for (int v = lane; v < n; v += 32) {
    const double s = mirror ? 1 - vals[v] : vals[v];
    const ElemPt p = elem_eval(g.kind[e], prm, s);
    double nx, ny;
    elem_normal(p, &nx, &ny);
    tb.x[off + v] = p.mx;
    tb.y[off + v] = p.my;
    tb.nx[off + v] = nx;
    tb.ny[off + v] = ny;
    const double jac = elem_jac(p);
#pragma unroll
    for (int b = 0; b < NB; ++b)
      if (NB == 1 || b < nu)
        tb.f[b * tb.cap + off + v] = jac * basis_eval(g.unk_kind[u + b], g.unk_param[u + b], s);
  }
}

// K(x, y) (re1, im1) and, if PAIR, K(y, x) (re2, im2) at a test point x
// (normal n1) and a trial point y (normal n2).  FP64: kernel_d; MIXED: the
// distance and the normal factors from the FP64 difference w = x - y, the
// Bessel functions and the kernel in float-float.  CK (FP64 only): complex
// wavenumber k + i ki.
template <int KERNEL, bool MIXED, bool PAIR, bool CK>
__device__ __forceinline__ void near_point(double k, double ki, double kq, double eq,
                                           const KConstFF& kc,
                                           const float* tab, double ax, double ay, double n1x,
                                           double n1y, double bx, double by, double n2x,
                                           double n2y, double* re1, double* im1, double* re2,
                                           double* im2) {
  if (CK) {
    if (PAIR)
      kernel_c_pair<KERNEL>(k, ki, eq, ax, ay, bx, by, n1x, n1y, n2x, n2y, re1, im1, re2, im2);
    else
      kernel_c<KERNEL>(k, ki, eq, ax, ay, bx, by, n1x, n1y, n2x, n2y, re1, im1);
    return;
  }
  if (!MIXED) {
    if (PAIR)
      kernel_d_pair<KERNEL>(k, kq, eq, ax, ay, bx, by, n1x, n1y, n2x, n2y, re1, im1, re2, im2);
    else
      kernel_d<KERNEL>(k, kq, eq, ax, ay, bx, by, n1x, n1y, n2x, n2y, re1, im1);
    return;
  }
  const double wx = ax - bx, wy = ay - by;
  const ff dx = ff_from_double(wx), dy = ff_from_double(wy);
  const ff d2 = ff_add_fast(ff_sqr(dx), ff_sqr(dy));
  const ff id = ff_rsqrt(d2);  // 1/d
  const BesselFF b = bessel01_ff(ff_mul(ff_mul(d2, id), kc.k), ff_mul(id, kc.invk), tab);
  ff cd1 = ff_make(0.0f, 0.0f), cd2 = ff_make(0.0f, 0.0f);
  if (KERNEL != BEM2D_KERNEL_SINGLE) {
    const double n1w = fma(n1x, wx, n1y * wy);  // n_x . (x - y)
    const double n2w = fma(n2x, wx, n2y * wy);  // n_y . (x - y)
    cd1 = ff_mul(ff_from_double(KERNEL == BEM2D_KERNEL_DOUBLE ? -n2w : n1w), id);
    if (PAIR) cd2 = ff_mul(ff_from_double(KERNEL == BEM2D_KERNEL_DOUBLE ? n1w : -n2w), id);
  }
  const ffc K1 = kernel_from_bessel<KERNEL>(b, cd1, kc);
  *re1 = ff_to_double(K1.re);
  *im1 = ff_to_double(K1.im);
  if (PAIR) {
    if (KERNEL == BEM2D_KERNEL_SINGLE) {
      *re2 = *re1;
      *im2 = *im1;
    } else {
      const ffc K2 = kernel_from_bessel<KERNEL>(b, cd2, kc);
      *re2 = ff_to_double(K2.re);
      *im2 = ff_to_double(K2.im);
    }
  }
}

// Sums over a rule's points of K f_i f_j w for the NB x NB basis functions of a
// pair: f_i at stride sa from fa, f_j w in gb.
template <int NB>
struct NearSums {
  double re[NB][NB], im[NB][NB];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) re[i][j] = im[i][j] = 0.0;
  }
  __device__ __forceinline__ void add(double r, double m, const double (&fa)[NB],
                                      const double (&gb)[NB]) {
    if constexpr (NB == 1) {
      const double f = fa[0] * gb[0];
      re[0][0] = fma(r, f, re[0][0]);
      im[0][0] = fma(m, f, im[0][0]);
    } else {
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const double rj = r * gb[j], mj = m * gb[j];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          re[i][j] = fma(rj, fa[i], re[i][j]);
          im[i][j] = fma(mj, fa[i], im[i][j]);
        }
      }
    }
  }
  __device__ __forceinline__ void reduce() {
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        re[i][j] = warp_sum(re[i][j]);
        im[i][j] = warp_sum(im[i][j]);
      }
  }
};

// One pair of groups: runs of up to NB consecutive unknowns of one element (NB
// = 1: of unknowns).  Every point's kernel value, the work that counts, serves
// all NB x NB entries: 801 elements of PolBasis(2), N = 2403, double layer,
// 1.46 ms with a warp per entry, 0.27 so.
template <int KERNEL, bool MIXED, bool CK, int NB>
__global__ void __launch_bounds__(256)
near_kernel(DevGeom g, DevRules r, const NearPair* __restrict__ pairs, int npairs, double k,
            double ki, double eta, double alpha, double beta, KConstFF kc, const float* gtab, int cap_s,
            int cap_t, double2* __restrict__ out, long long ld, float2* __restrict__ out32,
            long long ld32) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float* tab = reinterpret_cast<float*>(smem_raw);  // e^{ix} table (MIXED)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cap = cap_s + cap_t;
  double* base = reinterpret_cast<double*>(smem_raw + 1024) + (size_t)warp * (4 + NB) * cap;
  const GeoTab S{base, base + cap, base + 2 * cap, base + 3 * cap, base + 4 * cap, cap};
  if (MIXED) {
    for (int v = threadIdx.x; v < 256; v += blockDim.x) tab[v] = gtab[v];
    __syncthreads();
  }
  const int wid = blockIdx.x * (blockDim.x >> 5) + warp;
  if (wid >= npairs) return;
  const NearPair pr = pairs[wid];
  const int e1 = g.unk_elem[pr.i], e2 = g.unk_elem[pr.j];
  const double kq = 0.25 * k, eq = 0.25 * eta;
  NearSums<NB> acc, acc2;  // acc2: the second orientation of RULE_G3_PAIR
  acc.clear();
  double u1, u2;  // unused second orientation
  if (pr.rule == RULE_SELF) {
    // IntegrateIdent: Duffy split, points (x, (1-y)x) and (1-x, 1-x+yx),
    // both weighted by x * w.  Test-side geometry from the table (x values,
    // then 1 - x); trial-side evaluated per point.
    geo_fill<NB>(g, e1, pr.i, pr.ni, r.u1, r.nu1, false, S, 0, lane);
    geo_fill<NB>(g, e1, pr.i, pr.ni, r.u1, r.nu1, true, S, r.nu1, lane);
    __syncwarp();
    const double* p2 = g.param + 8 * (size_t)e2;
    for (int p = lane; p < r.n1; p += 32) {
      const double x = r.r1[3 * p], y = r.r1[3 * p + 1], w = r.r1[3 * p + 2];
      const int si = r.k1[p] & 0xffff;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int a = si + h * r.nu1;
        const double t = h == 0 ? (1 - y) * x : 1 - x + y * x;
        const ElemPt b = elem_eval(g.kind[e2], p2, t);
        double n2x, n2y, re, im;
        elem_normal(b, &n2x, &n2y);
        near_point<KERNEL, MIXED, false, CK>(k, ki, kq, eq, kc, tab, S.x[a], S.y[a], S.nx[a],
                                             S.ny[a], b.mx, b.my, n2x, n2y, &re, &im, &u1,
                                             &u2);
        const double jw = elem_jac(b) * (x * w);
        double fa[NB], gb[NB];
#pragma unroll
        for (int v = 0; v < NB; ++v) {
          fa[v] = NB == 1 || v < pr.ni ? S.f[v * cap + a] : 0.0;
          gb[v] = NB == 1 || v < pr.nj
                      ? jw * basis_eval(g.unk_kind[pr.j + v], g.unk_param[pr.j + v], t)
                      : 0.0;
        }
        acc.add(re, im, fa, gb);
      }
    }
  } else {
    // AdaptedGauss2 / AdaptedGauss3: test geometry at the rule's x values,
    // trial geometry at its y values.  RULE_G3_PAIR: (i, j) with
    // AdaptedGauss3 at (x, y) and (j, i) with its mirror AdaptedGauss2 at
    // (y, x), the same point pairs, one evaluation each.
    const bool g2 = pr.rule == RULE_G2;
    const double* rule = g2 ? r.r2 : r.r3;
    const int* key = g2 ? r.k2 : r.k3;
    const int np = g2 ? r.n2 : r.n3;
    geo_fill<NB>(g, e1, pr.i, pr.ni, g2 ? r.u2 : r.u3, g2 ? r.nu2 : r.nu3, false, S, 0, lane);
    geo_fill<NB>(g, e2, pr.j, pr.nj, g2 ? r.v2 : r.v3, g2 ? r.nv2 : r.nv3, false, S, cap_s, lane);
    __syncwarp();
    auto weights = [&](int p, int* a, int* b, double (&fa)[NB], double (&gb)[NB]) {
      const int kk = key[p];
      *a = kk & 0xffff;
      *b = cap_s + (kk >> 16);
      const double w = rule[3 * p + 2];
#pragma unroll
      for (int v = 0; v < NB; ++v) {
        fa[v] = NB == 1 || v < pr.ni ? S.f[v * cap + *a] : 0.0;
        gb[v] = NB == 1 || v < pr.nj ? S.f[v * cap + *b] * w : 0.0;
      }
    };
    if (pr.rule == RULE_G3_PAIR) {
      acc2.clear();
      for (int p = lane; p < np; p += 32) {
        int a, b;
        double fa[NB], gb[NB], r1, i1, r2, i2;
        weights(p, &a, &b, fa, gb);
        near_point<KERNEL, MIXED, true, CK>(k, ki, kq, eq, kc, tab, S.x[a], S.y[a], S.nx[a],
                                            S.ny[a], S.x[b], S.y[b], S.nx[b], S.ny[b], &r1,
                                            &i1, &r2, &i2);
        acc.add(r1, i1, fa, gb);
        acc2.add(r2, i2, fa, gb);
      }
      acc2.reduce();
#pragma unroll
      for (int i = 0; i < NB; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j)
          if (lane == i * NB + j && (NB == 1 || (i < pr.ni && j < pr.nj))) {
            const double re = alpha * acc2.re[i][j], im = alpha * acc2.im[i][j];
            const size_t row = pr.j + j, col = pr.i + i;
            out[col * ld + row] = make_double2(re, im);
            if (MIXED) out32[col * ld32 + row] = make_float2((float)re, (float)im);
          }
    } else {
      for (int p = lane; p < np; p += 32) {
        int a, b;
        double fa[NB], gb[NB], re, im;
        weights(p, &a, &b, fa, gb);
        near_point<KERNEL, MIXED, false, CK>(k, ki, kq, eq, kc, tab, S.x[a], S.y[a], S.nx[a],
                                             S.ny[a], S.x[b], S.y[b], S.nx[b], S.ny[b], &re,
                                             &im, &u1, &u2);
        acc.add(re, im, fa, gb);
      }
    }
  }
  acc.reduce();
#pragma unroll
  for (int i = 0; i < NB; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (lane == i * NB + j && (NB == 1 || (i < pr.ni && j < pr.nj))) {
        const int row = pr.i + i, col = pr.j + j;
        double re = alpha * acc.re[i][j], im = alpha * acc.im[i][j];
        if (pr.same && beta != 0.0) re = fma(beta, mass_entry(g, r, row, col), re);
        out[(size_t)col * ld + row] = make_double2(re, im);
        if (MIXED) out32[(size_t)col * ld32 + row] = make_float2((float)re, (float)im);
      }
}

// Table capacities (entries per warp) of the near-field kernel for rules r.
static void near_caps(const DevRules& r, int* cap_s, int* cap_t) {
  *cap_s = std::max(2 * r.nu1, std::max(r.nu2, r.nu3));
  *cap_t = std::max(r.nv2, r.nv3);
}

static size_t near_table_bytes(const DevRules& r, int nb) {
  int cs, ct;
  near_caps(r, &cs, &ct);
  return sizeof(double) * (size_t)(nb > 1 ? 4 + kNearBasis : 5) * (cs + ct);
}

template <int KERNEL, bool MIXED, bool CK, int NB>
static void launch_near_k(const DevGeom& g, const DevRules& r, const NearPair* pairs, int npairs,
                          double k, double ki, double eta, double alpha, double beta,
                          const float* tab,
                          double2* out, long long ld, float2* out32, long long ld32,
                          cudaStream_t s) {
  int cs, ct;
  near_caps(r, &cs, &ct);
  const size_t per_warp = std::max<size_t>(near_table_bytes(r, NB), 8);  // L = 0: empty rules
  // warps per block: up to 8, within 96 KB of shared memory; fewer while the
  // blocks would not give every SM eight of them (self and neighbour pairs
  // differ in cost; kite N = 2048, FP64: 20.25 -> 19.9 ms of the whole solve).
  // Two are enough in the mixed path, where every block copies the e^{ix} table
  // (kite N = 2048: 414 us with 8 warps, 427 with 2).
  int wpb = (int)std::max<size_t>(1, std::min<size_t>(8, (96 * 1024 - 1024) / per_warp));
  while (wpb > 1 && (npairs + wpb - 1) / wpb < (MIXED ? 2 : 8) * device_sms()) wpb /= 2;
  const size_t smem = 1024 + per_warp * wpb;
  const int blocks = (npairs + wpb - 1) / wpb;
  auto fn = near_kernel<KERNEL, MIXED, CK, NB>;
  // (one value for all rules: calls of several threads must not undo each other)
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  fn<<<blocks, 32 * wpb, smem, s>>>(g, r, pairs, npairs, k, ki, eta, alpha, beta,
                                     make_kconst(k, eta), tab, cs, ct, out, ld, out32, ld32);
}

template <bool MIXED, bool CK, int NB>
static void launch_near_m(const DevGeom& g, const DevRules& r, const NearPair* pairs, int npairs,
                          int kernel, double k, double ki, double eta, double alpha, double beta,
                          const float* tab, double2* out, long long ld, float2* out32,
                          long long ld32, cudaStream_t s) {
  switch (kernel) {
    case BEM2D_KERNEL_SINGLE:
      launch_near_k<BEM2D_KERNEL_SINGLE, MIXED, CK, NB>(g, r, pairs, npairs, k, ki, eta, alpha,
                                                    beta, tab, out, ld, out32, ld32, s);
      break;
    case BEM2D_KERNEL_DOUBLE:
      launch_near_k<BEM2D_KERNEL_DOUBLE, MIXED, CK, NB>(g, r, pairs, npairs, k, ki, eta, alpha,
                                                    beta, tab, out, ld, out32, ld32, s);
      break;
    case BEM2D_KERNEL_CONJDOUBLE:
      launch_near_k<BEM2D_KERNEL_CONJDOUBLE, MIXED, CK, NB>(g, r, pairs, npairs, k, ki, eta, alpha,
                                                        beta, tab, out, ld, out32, ld32, s);
      break;
    default:
      launch_near_k<BEM2D_KERNEL_COMBINED, MIXED, CK, NB>(g, r, pairs, npairs, k, ki, eta, alpha,
                                                      beta, tab, out, ld, out32, ld32, s);
  }
}

}  // namespace bem2d_gpu
