// Mixed-precision far-field assembly (sm_103a): the bulk of the Galerkin
// matrix evaluated in float-float arithmetic on the FP32 pipe.
//
// 32 x 32 tiles, one lane per test unknown, node data staged in shared
// memory; H0 and H1 from the table of hankel_tab_ff.cuh.  Pair geometry: the centre
// difference of the two elements in FP64, node offsets from the centres in
// float-float, so |x - y| keeps ~48 bits relative to itself even for
// neighbouring elements.  Entries whose element pair admits k|x - y| <= 4
// anywhere (bounded with the element radii) are deferred to a second
// float-float pass (deferred_ff_kernel, one thread per element pair), which
// carries the small-argument Bessel branch; keeping them out of the tile
// loop keeps its warps on one branch.  Adjacent and identical pairs belong to
// the near-field kernel as in the FP64 path.  Each entry is stored twice:
// complex128 (refinement residual) and complex64 (the LU).
#include <algorithm>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "ff.cuh"
#include "hankel_tab_ff.cuh"
#include "kernel_ff.cuh"

namespace bem2d_gpu {

// amp P0, amp Q0, (amp/x) P1, (amp/x) Q1 (amp = sqrt(2/(pi x))) and
// e^{i(x - pi/4)} by the general evaluator: arguments outside the table's octaves.
__device__ __noinline__ void hankel_direct_ff(ff x, const float* etab, ff* p0, ff* q0, ff* p1,
                                              ff* q1, ffc* e) {
  const ff ix = ff_rcp(x);
  const ff amp = ff_mul(ff_make(0.7978845834732056f, -2.2670340271702116e-08f), ff_rsqrt(x));
  const ff ampx = ff_mul(amp, ix);
  pq_ff(x.hi, ix, p0, q0, p1, q1);
  *p0 = ff_mul(amp, *p0);
  *q0 = ff_mul(amp, *q0);
  *p1 = ff_mul(ampx, *p1);
  *q1 = ff_mul(ampx, *q1);
  *e = expi_ff(x, etab);
}

// E (P + i Q)
__device__ __forceinline__ ffc ffcu_mul_pq(const ffc& e, ff p, ff q) {
  ffc r;
  r.re = ffu_dot2(e.re, p, ff_neg(e.im), q);
  r.im = ffu_dot2(e.re, q, e.im, p);
  return r;
}

// acc += v without renormalising acc: acc.lo gathers the hi sums' rounding
// errors and the lo parts (ff_acc_norm restores |lo| <= ulp(hi)/2 after a
// few steps, so that the FP32 sum in lo stays ~2^-48 |acc| accurate)
__device__ __forceinline__ void ff_acc(ff& acc, ff v) {
  const ff s = two_sum(acc.hi, v.hi);
  acc.hi = s.hi;
  acc.lo += s.lo + v.lo;
}
__device__ __forceinline__ void ff_acc_norm(ff& acc) { acc = fast_two_sum(acc.hi, acc.lo); }

// One entry in FP64 from the FP64 node table (deferred entries).
template <int KERNEL>
__device__ __forceinline__ void entry_fp64(const NodeTable& t, int ng, int row, int col,
                                           double k, double kq, double eq, double* re,
                                           double* im) {
  double ar = 0.0, ai = 0.0;
  for (int q1 = 0; q1 < ng; ++q1) {
    const size_t a = (size_t)row * ng + q1;
    const double x1 = t.x[a], y1 = t.y[a], n1x = t.nx[a], n1y = t.ny[a], w1 = t.w[a];
    for (int q2 = 0; q2 < ng; ++q2) {
      const size_t b = (size_t)col * ng + q2;
      double vr, vi;
      kernel_d<KERNEL>(k, kq, eq, x1, y1, t.x[b], t.y[b], n1x, n1y, t.nx[b], t.ny[b], &vr, &vi);
      const double ww = w1 * t.w[b];
      ar = fma(vr, ww, ar);
      ai = fma(vi, ww, ai);
    }
  }
  *re = ar;
  *im = ai;
}

constexpr int kTileF = 32;
constexpr int kDeferRC = 1 << 30;  // deferred item: entry (row, col) wanted
constexpr int kDeferCR = 1 << 29;  // deferred item: entry (col, row) wanted
constexpr int kDeferIdx = kDeferCR - 1;
constexpr int kFarFFThreads = 256;
constexpr float kDeferX = 4.001f;
// table intervals in shared memory (27 KB: with rules of 64 nodes a CTA takes 214 KB)
constexpr int kFtCap = 192;

// Tiles are processed in symmetric pairs: CTA b owns tile (I, J), I <= J,
// and computes both (I, J) and (J, I).  The distance-dependent work at a node
// pair (the Hankel terms, most of the cost) is the same for entry (r, c) and
// entry (c, r); only the normal factor of the double-layer kernels differs.
// Entry (r, c) is stored directly (a warp writes 32 consecutive rows of a
// column); entry (c, r) goes to a shared-memory copy of tile (J, I) that is
// written out, column by column, at the end.  A pair that is near in either
// direction is left, in that direction, to the near-field kernel; the
// small-argument test depends on the distance only, so a deferred pair is
// deferred in both directions.  On a diagonal tile only r < c is computed.
__device__ __forceinline__ void tile_of(unsigned b, int* I, int* J) {
  int j = (int)((sqrt(8.0 * (double)b + 1.0) - 1.0) * 0.5);
  while ((long long)(j + 1) * (j + 2) / 2 <= (long long)b) ++j;
  while ((long long)j * (j + 1) / 2 > (long long)b) --j;
  *J = j;
  *I = (int)((long long)b - (long long)j * (j + 1) / 2);
}

// Bound by FP32 issue (76 % of the issue slots, 65 % of the FMA pipe): 704
// thread instructions per node pair with pq_ff (1/d, 1/sqrt(x), four
// polynomials of degree 9-12 and e^{ix} each), 472 with the table; 1.24 ->
// 0.85 ms at kite N = 2048, 69 -> 51 ms at L-shape N = 16384, with about half
// the error against FP64.  More warps (3 CTAs at 80 registers, 22 warps at 80,
// 20 at 96) measured no faster.  All coordinates are scaled by k first, so that x = |k (x - y)| is
// one square root and H1 comes as H1/x, the factor the normal product needs;
// k, eta and alpha enter once per entry.  The CTA's arguments lie between two
// bounds from its 1024 centre distances; when the table intervals between them
// fit (kFtCap of 144 bytes: stride 9 x 16 bytes, so that neighbouring
// intervals fall into different banks), they are copied to shared memory,
// otherwise they are read from the global table.
template <int KERNEL, int NG>
__global__ void __launch_bounds__(kFarFFThreads, 2)
far_ff_kernel(DevGeom g, NodeTable t, NodeTableFF tf, int ng_rt, KConstFF kc, double k,
              double eta, double alpha, double2* __restrict__ out, long long ld,
              float2* __restrict__ out32, long long ld32, DeferList dl,
              const float4* __restrict__ ftab, const float* __restrict__ etab) {
  constexpr bool kH0 = KERNEL == BEM2D_KERNEL_SINGLE || KERNEL == BEM2D_KERNEL_COMBINED;
  constexpr bool kH1 = KERNEL != BEM2D_KERNEL_SINGLE;
  const int ng = NG > 0 ? NG : ng_rt;
  const int SZ = ng * kTileF;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* tT = reinterpret_cast<double2*>(smem_raw);          // [32][33] tile (J, I)
  double2* cen = tT + kTileF * (kTileF + 1);                   // rows 32, cols 32
  float4* rxy = reinterpret_cast<float4*>(cen + 2 * kTileF);   // [ng][32] k (x, y) offsets
  float4* rnn = rxy + SZ;                                      // [ng][32] normals
  float4* cxy = rnn + SZ;
  float4* cnn = cxy + SZ;
  float4* bins = cnn + SZ;                                     // [kFtCap][9]
  float4* trig = bins + kFtCap * (kFtWords / 4);               // [512]
  float2* rw = reinterpret_cast<float2*>(trig + kFtTrig);      // [ng][32] weights
  float2* cw = rw + SZ;
  long long* links = reinterpret_cast<long long*>(cw + SZ);    // 6 x 32
  float* rad = reinterpret_cast<float*>(links + 6 * kTileF);   // rows 32, cols 32
  unsigned* vT = reinterpret_cast<unsigned*>(rad + 2 * kTileF);  // [32] masks
  float* red = reinterpret_cast<float*>(vT + kTileF);          // 2 x 8

  int I, J;
  tile_of(blockIdx.x, &I, &J);
  const int row0 = I * kTileF, col0 = J * kTileF;
  const bool diag = I == J;
  const int n = g.n_unk;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int v = threadIdx.x; v < kFtTrig; v += blockDim.x)
    trig[v] = ftab[kFtBins * (kFtWords / 4) + v];
  if (threadIdx.x < kTileF) vT[threadIdx.x] = 0u;
  for (int v = threadIdx.x; v < 2 * SZ; v += blockDim.x) {
    const bool isc = v >= SZ;
    const int o = isc ? v - SZ : v, q = o / kTileF, l = o - q * kTileF;
    const size_t i = (size_t)min((isc ? col0 : row0) + l, n - 1) * ng + q;
    const float2 ox = tf.ox[i], oy = tf.oy[i], nx = tf.nx[i], ny = tf.ny[i];
    const ff X = ff_mul(ff_make(ox.x, ox.y), kc.k), Y = ff_mul(ff_make(oy.x, oy.y), kc.k);
    (isc ? cxy : rxy)[o] = make_float4(X.hi, X.lo, Y.hi, Y.lo);
    (isc ? cnn : rnn)[o] = make_float4(nx.x, nx.y, ny.x, ny.y);
    (isc ? cw : rw)[o] = tf.w[i];
  }
  if (threadIdx.x < kTileF) {
    const int l = threadIdx.x;
    const int ur = min(row0 + l, n - 1), uc = min(col0 + l, n - 1);
    cen[l] = tf.c[ur];
    cen[kTileF + l] = tf.c[uc];
    rad[l] = tf.rad[ur];
    rad[kTileF + l] = tf.rad[uc];
    const int er = g.unk_elem[ur], ec = g.unk_elem[uc];
    links[l] = g.index[er];
    links[kTileF + l] = g.next[er];
    links[2 * kTileF + l] = g.prev[er];
    links[3 * kTileF + l] = g.index[ec];
    links[4 * kTileF + l] = g.next[ec];
    links[5 * kTileF + l] = g.prev[ec];
  }
  __syncthreads();

  const int row = row0 + lane;
  const float kf = (float)k;

  // the table intervals between the smallest and the largest argument
  float xlo = INFINITY, xhi = 0.0f;
  for (int cc = warp; cc < kTileF; cc += kFarFFThreads / 32) {
    const float dx = (float)(cen[lane].x - cen[kTileF + cc].x),
                dy = (float)(cen[lane].y - cen[kTileF + cc].y);
    const float dist = sqrtf(dx * dx + dy * dy), rr = rad[lane] + rad[kTileF + cc];
    xlo = fminf(xlo, kf * (dist * (1.0f - 1e-6f) - rr));
    xhi = fmaxf(xhi, kf * (dist * (1.0f + 1e-6f) + rr));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    xlo = fminf(xlo, __shfl_xor_sync(0xffffffffu, xlo, o));
    xhi = fmaxf(xhi, __shfl_xor_sync(0xffffffffu, xhi, o));
  }
  if (lane == 0) {
    red[warp] = xlo;
    red[kFarFFThreads / 32 + warp] = xhi;
  }
  __syncthreads();
#pragma unroll
  for (int v = 0; v < kFarFFThreads / 32; ++v) {
    xlo = fminf(xlo, red[v]);
    xhi = fmaxf(xhi, red[kFarFFThreads / 32 + v]);
  }
  // one interval to spare on each side; a pair outside them takes the general
  // evaluator
  int bin0 = max(ft_bin(fmaxf(xlo, 4.0f)) - 1, 0);
  int nbin = max(min(ft_bin(xhi) + 1, kFtBins - 1) - bin0 + 1, 0);
  const float4* fb = bins;
  if (nbin <= kFtCap) {
    for (int v = threadIdx.x; v < nbin * (kFtWords / 4); v += blockDim.x)
      bins[v] = ftab[bin0 * (kFtWords / 4) + v];
  } else {
    bin0 = 0;
    nbin = kFtBins;
    fb = ftab;
  }
  __syncthreads();

#pragma unroll 1
  for (int cc = warp; cc < kTileF; cc += kFarFFThreads / 32) {
    const int col = col0 + cc;
    const long long ri = links[lane], rn = links[kTileF + lane], rp = links[2 * kTileF + lane];
    const long long ci = links[3 * kTileF + cc], cn = links[4 * kTileF + cc],
                    cp = links[5 * kTileF + cc];
    // rc: entry (row, col); cr: entry (col, row)
    bool rc = row < n && col < n && !((ri == ci) || (rn == ci) || (rp == ci));
    bool cr = row < n && col < n && !((ci == ri) || (cn == ri) || (cp == ri));
    if (diag && lane >= cc) rc = cr = false;
    if (!rc && !cr) continue;
    const ff dxc = ff_from_double(cen[lane].x - cen[kTileF + cc].x),
             dyc = ff_from_double(cen[lane].y - cen[kTileF + cc].y);
    const float dist = sqrtf(dxc.hi * dxc.hi + dyc.hi * dyc.hi);
    if (kf * (dist * (1.0f - 1e-6f) - rad[lane] - rad[kTileF + cc]) <= kDeferX) {
      // small arguments somewhere on this pair: second pass (or here, in
      // FP64, if the list is full).  One list item per pair: (row, col) with the flags
      // kDeferRC / kDeferCR in the top bits of .x for the directions needed.
      const unsigned slot = atomicAdd(dl.count, 1u);
      if (slot < dl.capacity) {
        dl.ij[slot] = make_int2(row | (rc ? kDeferRC : 0) | (cr ? kDeferCR : 0), col);
      } else {
        for (int dir = 0; dir < 2; ++dir) {
          if (!(dir == 0 ? rc : cr)) continue;
          const int a = dir == 0 ? row : col, b = dir == 0 ? col : row;
          double re, im;
          entry_fp64<KERNEL>(t, ng, a, b, k, 0.25 * k, 0.25 * eta, &re, &im);
          out[(size_t)b * ld + a] = make_double2(alpha * re, alpha * im);
          out32[(size_t)b * ld32 + a] = make_float2((float)(alpha * re), (float)(alpha * im));
        }
      }
      continue;
    }
    const ff Dx = ff_mul(dxc, kc.k), Dy = ff_mul(dyc, kc.k);
    // With X = k (x - y), Z0 = w_x w_y amp E (P0 + i Q0) and
    // Z1 = w_x w_y (amp/x) E (P1 + i Q1):
    //   single layer  (i/4) sum Z0
    //   combined      (eta/4) sum Z0 - (k/4) sum (n . X) Z1 (double layers
    //                 without the Z0 term), n . X = n_y . (y - x) k for the
    //                 double layer at (x, y), n_x . (x - y) k otherwise
    // s0 = sum Z0, t1 = sum (n_x . X) Z1, t2 = sum (n_y . X) Z1 (x on the row
    // element) serve both entries of the pair.
    ffc s0, t1, t2;
    s0.re = s0.im = t1.re = t1.im = t2.re = t2.im = ff_make(0.0f, 0.0f);
#pragma unroll 1
    for (int q1 = 0; q1 < ng; ++q1) {
      const int o1 = q1 * kTileF + lane;
      const float4 a0 = rxy[o1], a1 = rnn[o1];
      const float2 a2 = rw[o1];
      // the row node's position relative to the column element's centre
      const ff Px = ff_add_fast(Dx, ff_make(a0.x, a0.y));
      const ff Py = ff_add_fast(Dy, ff_make(a0.z, a0.w));
#pragma unroll 1
      for (int q2 = 0; q2 < ng; ++q2) {
        const int o2 = q2 * kTileF + cc;
        const float4 b0 = cxy[o2], b1 = cnn[o2];
        const float2 b2 = cw[o2];
        const ff dx = ffu_add(Px, ff_make(-b0.x, -b0.y));
        const ff dy = ffu_add(Py, ff_make(-b0.z, -b0.w));
        const ff x = ff_sqrt(ffu_dot2(dx, dx, dy, dy));
        ff p0, q0, p1, q1v;
        ffc E;
        const int bin = ft_bin(x.hi) - bin0;
        if ((unsigned)bin < (unsigned)nbin) {
          ft_pq<kH0, kH1>(fb + bin * (kFtWords / 4), x, &p0, &q0, &p1, &q1v);
          E = ft_expi(x, trig);
        } else {
          hankel_direct_ff(x, etab, &p0, &q0, &p1, &q1v, &E);
        }
        const ff ww = ffu_mul(ff_make(a2.x, a2.y), ff_make(b2.x, b2.y));
        E.re = ffu_mul(E.re, ww);
        E.im = ffu_mul(E.im, ww);
        if (kH0) {
          const ffc Z0 = ffcu_mul_pq(E, p0, q0);
          ff_acc(s0.re, Z0.re);
          ff_acc(s0.im, Z0.im);
        }
        if (kH1) {
          const ffc Z1 = ffcu_mul_pq(E, p1, q1v);
          const ff n1 = ffu_dot2(ff_make(a1.x, a1.y), dx, ff_make(a1.z, a1.w), dy);
          const ff n2 = ffu_dot2(ff_make(b1.x, b1.y), dx, ff_make(b1.z, b1.w), dy);
          ff_acc(t1.re, ffu_mul(n1, Z1.re));
          ff_acc(t1.im, ffu_mul(n1, Z1.im));
          ff_acc(t2.re, ffu_mul(n2, Z1.re));
          ff_acc(t2.im, ffu_mul(n2, Z1.im));
        }
      }
      if (kH0) {
        ff_acc_norm(s0.re);
        ff_acc_norm(s0.im);
      }
      if (kH1) {
        ff_acc_norm(t1.re);
        ff_acc_norm(t1.im);
        ff_acc_norm(t2.re);
        ff_acc_norm(t2.im);
      }
    }
    ffc arc, acr;
    if (KERNEL == BEM2D_KERNEL_SINGLE) {
      arc.re = ff_scale2(ff_neg(s0.im), 0.25f);
      arc.im = ff_scale2(s0.re, 0.25f);
      acr = arc;
    } else {
      // -n . X of entry (row, col): n2 (double layer) or -n1; (col, row): the reverse
      const ff kq = kc.kq, mkq = ff_neg(kc.kq);
      const ffc& trc = KERNEL == BEM2D_KERNEL_DOUBLE ? t2 : t1;
      const ffc& tcr = KERNEL == BEM2D_KERNEL_DOUBLE ? t1 : t2;
      const ff frc = KERNEL == BEM2D_KERNEL_DOUBLE ? kq : mkq;
      const ff fcr = KERNEL == BEM2D_KERNEL_DOUBLE ? mkq : kq;
      arc.re = ff_mul(frc, trc.re);
      arc.im = ff_mul(frc, trc.im);
      acr.re = ff_mul(fcr, tcr.re);
      acr.im = ff_mul(fcr, tcr.im);
      if (KERNEL == BEM2D_KERNEL_COMBINED) {
        const ff er = ff_mul(kc.eq, s0.re), ei = ff_mul(kc.eq, s0.im);
        arc.re = ff_add(arc.re, er);
        arc.im = ff_add(arc.im, ei);
        acr.re = ff_add(acr.re, er);
        acr.im = ff_add(acr.im, ei);
      }
    }
    if (rc) {
      const double re = alpha * ff_to_double(arc.re), im = alpha * ff_to_double(arc.im);
      out[(size_t)col * ld + row] = make_double2(re, im);
      out32[(size_t)col * ld32 + row] = make_float2((float)re, (float)im);
    }
    if (cr) {
      tT[cc * (kTileF + 1) + lane] =
          make_double2(alpha * ff_to_double(acr.re), alpha * ff_to_double(acr.im));
      atomicOr(&vT[cc], 1u << lane);
    }
  }
  __syncthreads();
  // tile (J, I): entry (col0 + cc, row0 + l) = tT[cc][l]; a warp writes 32
  // consecutive rows (cc) of one column (row0 + l)
  for (int l = warp; l < kTileF; l += kFarFFThreads / 32) {
    const int cc = lane;
    if (!((vT[cc] >> l) & 1u)) continue;
    const double2 v = tT[cc * (kTileF + 1) + l];
    out[(size_t)(row0 + l) * ld + col0 + cc] = v;
    out32[(size_t)(row0 + l) * ld32 + col0 + cc] = make_float2((float)v.x, (float)v.y);
  }
}

template <int KERNEL>
__global__ void __launch_bounds__(128)
deferred_ff_kernel(NodeTableFF tf, int ng, KConstFF kc, double alpha, const int2* __restrict__ ij,
                   const unsigned* count, unsigned cap, double2* __restrict__ out, long long ld,
                   float2* __restrict__ out32, long long ld32, const float* gtab) {
  // one item = one element pair; both orientations share every distance
  // and Bessel evaluation.  Same pair geometry as far_ff_kernel: the centre
  // difference in FP64, node offsets in ff.
  __shared__ float tab[256];
  for (int v = threadIdx.x; v < 256; v += blockDim.x) tab[v] = gtab[v];
  __syncthreads();
  const unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= min(*count, cap)) return;
  const int2 e = ij[p];
  const int row = e.x & kDeferIdx, col = e.y;
  const bool want_rc = (e.x & kDeferRC) != 0, want_cr = (e.x & kDeferCR) != 0;
  const double2 cr0 = tf.c[row], cc0 = tf.c[col];
  const ff Dx = ff_from_double(cr0.x - cc0.x), Dy = ff_from_double(cr0.y - cc0.y);
  ffc arc, acr;
  arc.re = arc.im = acr.re = acr.im = ff_make(0.0f, 0.0f);
#pragma unroll 1
  for (int q1 = 0; q1 < ng; ++q1) {
    const size_t a = (size_t)row * ng + q1;
    const float2 a0 = tf.ox[a], a1 = tf.oy[a], a2 = tf.nx[a], a3 = tf.ny[a], a4 = tf.w[a];
    const ff ox1 = ff_make(a0.x, a0.y), oy1 = ff_make(a1.x, a1.y);
    const ff n1x = ff_make(a2.x, a2.y), n1y = ff_make(a3.x, a3.y), w1 = ff_make(a4.x, a4.y);
#pragma unroll 1
    for (int q2 = 0; q2 < ng; ++q2) {
      const size_t b = (size_t)col * ng + q2;
      const float2 b0 = tf.ox[b], b1 = tf.oy[b], b2 = tf.nx[b], b3 = tf.ny[b], b4 = tf.w[b];
      // w = x - y, x a node of the row element, y of the column element
      const ff dx = ff_add_fast(Dx, ff_add_fast(ox1, ff_make(-b0.x, -b0.y)));
      const ff dy = ff_add_fast(Dy, ff_add_fast(oy1, ff_make(-b1.x, -b1.y)));
      const ff d2 = ff_add_fast(ff_sqr(dx), ff_sqr(dy));
      const ff id = ff_rsqrt(d2);  // 1/d
      const ff x = ff_mul(ff_mul(d2, id), kc.k);
      const BesselFF bs = bessel01_ff(x, ff_mul(id, kc.invk), tab);
      const ff ww = ff_mul(w1, ff_make(b4.x, b4.y));
      ff cd_rc = ff_make(0.0f, 0.0f), cd_cr = ff_make(0.0f, 0.0f);
      if (KERNEL != BEM2D_KERNEL_SINGLE) {
        const ff n1w = ff_mul(ff_add_fast(ff_mul(n1x, dx), ff_mul(n1y, dy)), id);
        const ff n2w = ff_mul(ff_add_fast(ff_mul(ff_make(b2.x, b2.y), dx),
                                          ff_mul(ff_make(b3.x, b3.y), dy)), id);
        if (KERNEL == BEM2D_KERNEL_DOUBLE) {
          cd_rc = ff_neg(n2w);  // (row, col): n_y . (y - x) / d
          cd_cr = n1w;          // (col, row): n_x . (x - y) / d
        } else {
          cd_rc = n1w;
          cd_cr = ff_neg(n2w);
        }
      }
      const ffc K1 = kernel_from_bessel<KERNEL>(bs, cd_rc, kc);
      arc.re = ff_add_fast(arc.re, ff_mul(K1.re, ww));
      arc.im = ff_add_fast(arc.im, ff_mul(K1.im, ww));
      if (KERNEL == BEM2D_KERNEL_SINGLE) {
        acr = arc;
      } else {
        const ffc K2 = kernel_from_bessel<KERNEL>(bs, cd_cr, kc);
        acr.re = ff_add_fast(acr.re, ff_mul(K2.re, ww));
        acr.im = ff_add_fast(acr.im, ff_mul(K2.im, ww));
      }
    }
  }
  if (want_rc) {
    const double re = alpha * ff_to_double(arc.re), im = alpha * ff_to_double(arc.im);
    out[(size_t)col * ld + row] = make_double2(re, im);
    out32[(size_t)col * ld32 + row] = make_float2((float)re, (float)im);
  }
  if (want_cr) {
    const double re = alpha * ff_to_double(acr.re), im = alpha * ff_to_double(acr.im);
    out[(size_t)row * ld + col] = make_double2(re, im);
    out32[(size_t)row * ld32 + col] = make_float2((float)re, (float)im);
  }
}

// A table of `count` floats made by `build` on the host and kept on the current
// device.
template <typename B>
static const float* device_table(float* (&tab)[64], std::mutex& mu, size_t count, B build) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (!tab[dev]) {
    std::vector<float> h(count);
    build(h.data());
    float* d = nullptr;
    if (cudaMalloc(&d, sizeof(float) * count) != cudaSuccess) return nullptr;
    if (cudaMemcpy(d, h.data(), sizeof(float) * count, cudaMemcpyHostToDevice) != cudaSuccess) {
      cudaFree(d);
      return nullptr;
    }
    tab[dev] = d;
  }
  return tab[dev];
}

const float* expi_table_dev() {
  static std::mutex mu;
  static float* tab[64] = {};
  return device_table(tab, mu, 256, expi_table);
}

// The far field's table (see hankel_tab_ff.cuh).
static const float* ft_table_dev() {
  static std::mutex mu;
  static float* tab[64] = {};
  return device_table(tab, mu, kFtFloats, ft_build);
}

template <int KERNEL>
static int launch_far_ff_k(const DevGeom& g, const NodeTable& t, const NodeTableFF& tf, int ng,
                            double k, double eta, double alpha, double2* out, long long ld,
                            float2* out32, long long ld32, DeferList dl, cudaStream_t s) {
  const KConstFF kc = make_kconst(k, eta);
  const size_t smem = sizeof(double2) * (kTileF * (kTileF + 1) + 2 * kTileF) +
                      (4 * sizeof(float4) + 2 * sizeof(float2)) * (size_t)ng * kTileF +
                      sizeof(float) * kFtWords * kFtCap + sizeof(float4) * kFtTrig +
                      sizeof(long long) * 6 * kTileF + sizeof(float) * (3 * kTileF + 16);
  const unsigned nt = (unsigned)((g.n_unk + kTileF - 1) / kTileF);
  dim3 grid(nt * (nt + 1) / 2);  // tile pairs (I, J), I <= J
  const float* ftab = ft_table_dev();
  const float* etab = expi_table_dev();
  if (!ftab || !etab) return BEM2D_ERR_NOMEM;
  auto fn = ng == 5 ? far_ff_kernel<KERNEL, 5> : far_ff_kernel<KERNEL, 0>;
  // one value for all rules: calls of several threads must not undo each other
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  fn<<<grid, kFarFFThreads, smem, s>>>(g, t, tf, ng, kc, k, eta, alpha, out, ld, out32, ld32, dl,
                                       reinterpret_cast<const float4*>(ftab), etab);
  return BEM2D_OK;
}

int launch_far_ff(const DevGeom& g, const NodeTable& t, const NodeTableFF& tf, int ng,
                  int kernel, double k, double eta, double alpha, double2* out,
                  long long ld, float2* out32, long long ld32, DeferList dl,
                  cudaStream_t s) {
  switch (kernel) {
    case BEM2D_KERNEL_SINGLE:
      return launch_far_ff_k<BEM2D_KERNEL_SINGLE>(g, t, tf, ng, k, eta, alpha, out, ld, out32,
                                                  ld32, dl, s);
    case BEM2D_KERNEL_DOUBLE:
      return launch_far_ff_k<BEM2D_KERNEL_DOUBLE>(g, t, tf, ng, k, eta, alpha, out, ld, out32,
                                                  ld32, dl, s);
    case BEM2D_KERNEL_CONJDOUBLE:
      return launch_far_ff_k<BEM2D_KERNEL_CONJDOUBLE>(g, t, tf, ng, k, eta, alpha, out, ld, out32,
                                                      ld32, dl, s);
    default:
      return launch_far_ff_k<BEM2D_KERNEL_COMBINED>(g, t, tf, ng, k, eta, alpha, out, ld, out32,
                                                    ld32, dl, s);
  }
}

// Grid sized by the list capacity; threads beyond the device-side count exit.
int launch_deferred(const NodeTableFF& tf, int ng, int kernel, double k, double eta,
                    double alpha, const DeferList& dl, double2* out, long long ld,
                    float2* out32, long long ld32, cudaStream_t s) {
  if (dl.capacity == 0) return BEM2D_OK;
  const float* tab = expi_table_dev();
  if (!tab) return BEM2D_ERR_NOMEM;
  const KConstFF kc = make_kconst(k, eta);
  const unsigned blocks = (dl.capacity + 127) / 128;
  switch (kernel) {
    case BEM2D_KERNEL_SINGLE:
      deferred_ff_kernel<BEM2D_KERNEL_SINGLE><<<blocks, 128, 0, s>>>(tf, ng, kc, alpha, dl.ij, dl.count, dl.capacity, out, ld, out32, ld32, tab);
      break;
    case BEM2D_KERNEL_DOUBLE:
      deferred_ff_kernel<BEM2D_KERNEL_DOUBLE><<<blocks, 128, 0, s>>>(tf, ng, kc, alpha, dl.ij, dl.count, dl.capacity, out, ld, out32, ld32, tab);
      break;
    case BEM2D_KERNEL_CONJDOUBLE:
      deferred_ff_kernel<BEM2D_KERNEL_CONJDOUBLE><<<blocks, 128, 0, s>>>(tf, ng, kc, alpha, dl.ij, dl.count, dl.capacity, out, ld, out32, ld32, tab);
      break;
    default:
      deferred_ff_kernel<BEM2D_KERNEL_COMBINED><<<blocks, 128, 0, s>>>(tf, ng, kc, alpha, dl.ij, dl.count, dl.capacity, out, ld, out32, ld32, tab);
  }
  return BEM2D_OK;
}

}  // namespace bem2d_gpu
