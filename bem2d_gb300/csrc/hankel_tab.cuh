// H0(z) and H1(z) on the ray z = k d of one wavenumber from a table of short
// polynomials: the evaluator of the FP64 far field and of the potentials.
//
// Why a table: GB300's FP64 pipe issues 2 FMAs per clock and SM, 1/64 of the
// FP32 pipe, so an FP64 kernel evaluation costs what its FP64 instructions
// cost and everything else (table loads, integer and FP32 instructions) is
// nearly free.  hankel01_d spends about 170 FP64 instructions on a node pair
// (two square roots, two divisions, four polynomials of degree 12-16, sincos
// with its reduction); the table form below about 45.
//
// With x = |k| d, H_nu(z) = e^{iz} g_nu(x).  g is smooth (algebraic in x), so
// on each of 64 equal intervals of every octave of x a polynomial of degree 6
// in w = (x - centre) / (2 half-widths), |w| <= 1/2, carries g to 2^-55 |g|
// (the nearest singularity, x = 0, lies 64 widths away).  Terms w^4 .. w^6
// (below 2^-28 |g|) are summed in FP32.  The octaves cover
// 1/2 <= x < 4096; other arguments (and NaN) take the direct evaluators.
//   e^{iz}: Re z = n (2 pi / 256) + r, the 256 values e^{2 pi i n / 256} from
//   a table, e^{ir} - 1 from short Taylor polynomials (|r| <= pi/256); for a
//   complex wavenumber times exp(-Im z).
//
// A table entry is filled from 16 Chebyshev points of the direct evaluator
// (least squares: the discrete Chebyshev sums up to degree 6), so evaluation
// noise of the points is averaged, not interpolated.
#pragma once

#include "hankel_c.cuh"

namespace bem2d_gpu {

constexpr int kHtOct0 = -1;                    // first octave: x in [1/2, 1)
constexpr int kHtOctaves = 13;                 // up to x < 4096
constexpr int kHtPerOct = 64;
constexpr int kHtBins = kHtOctaves * kHtPerOct;
constexpr int kHtNodes = 16;                   // points per interval
constexpr int kHtTrig = 256;
constexpr int kHtBase = (1023 + kHtOct0) * kHtPerOct;  // bin 0's exponent | mantissa bits

// Device table: per interval and function (Re g0, Im g0, Re g1, Im g1) the
// coefficients c0..c3 in FP64, c4..c6 in FP32; then e^{2 pi i n / 256}.
struct HankelTab {
  const double2* cd;  // [bins][4 functions][2]
  const float4* ct;   // [bins][3]: c4, c5, c6 of the four functions
  const double2* sc;  // [256] cos, sin
};
constexpr size_t kHtBytes = (size_t)kHtBins * (8 * sizeof(double2) + 3 * sizeof(float4)) +
                            kHtTrig * sizeof(double2);

inline HankelTab hankel_tab_at(void* p) {
  HankelTab t;
  t.cd = static_cast<const double2*>(p);
  t.sc = t.cd + (size_t)kHtBins * 8;
  t.ct = reinterpret_cast<const float4*>(t.sc + kHtTrig);
  return t;
}

#ifdef __CUDACC__

// g0, g1 at z = x (ur + i ui), |ur + i ui| = 1: H_nu(z) e^{-iz}.
__device__ __forceinline__ void hankel_scaled(double x, double ur, double ui, cd* g0, cd* g1) {
  if (ui == 0.0) {
    if (x <= 4.0) {
      double j0, y0, j1, y1, s, c;
      hankel01_d(x, &j0, &y0, &j1, &y1);
      sincos(x, &s, &c);
      *g0 = cd{fma(j0, c, y0 * s), fma(y0, c, -j0 * s)};
      *g1 = cd{fma(j1, c, y1 * s), fma(y1, c, -j1 * s)};
      return;
    }
    double p0, q0, p1, q1;
    hankel_pq_d(x, &p0, &q0, &p1, &q1);
    // sqrt(2/(pi x)) (P + iQ) e^{-i pi/4}, e^{-3 i pi/4}
    const double a = sqrt(kInvPi / x);
    *g0 = cd{a * (p0 + q0), a * (q0 - p0)};
    *g1 = cd{a * (q1 - p1), -a * (p1 + q1)};
    return;
  }
  const cd z{x * ur, x * ui};
  if (x <= 1.5) {
    cd h0, h1;
    hankel01_c_series(z, &h0, &h1);
    double s, c;
    sincos(z.re, &s, &c);
    const double e = exp(z.im);
    const cd f{e * c, -e * s};  // e^{-iz}
    *g0 = cd_mul(h0, f);
    *g1 = cd_mul(h1, f);
    return;
  }
  hankel01_c_integral_scaled(z, x, g0, g1);
}

// Direct evaluation outside the table's octaves, of what is wanted: low frequencies
// meet little else (single-layer potential of 1,024 elements at 40,000 points, k =
// 0.05: 45.2 ms with both orders always, 32.1 so).
template <bool H0, bool H1, bool CK>
__device__ __noinline__ void hankel_direct(double d, double kr, double ki, double* h0r,
                                           double* h0i, double* h1r, double* h1i) {
  double a, b, c, e;
  if (CK) {
    cd h0, h1;
    hankel01_c(cd{kr * d, ki * d}, &h0, &h1);
    a = h0.re;
    b = h0.im;
    c = h1.re;
    e = h1.im;
  } else {
    hankel01_d(kr * d, &a, &b, &c, &e);
  }
  if (H0) {
    *h0r = a;
    *h0i = b;
  }
  if (H1) {
    *h1r = c;
    *h1i = e;
  }
}

__device__ __forceinline__ double ht_rsqrt_approx(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// (double)t on the integer pipe (an F2F conversion takes an FP64 slot);
// exact for normal t, an error below 2^-125 for t = 0 or subnormal.
__device__ __forceinline__ double ht_widen(float t) {
  const int b = __float_as_int(t);
  return __hiloint2double((b & 0x80000000) | (((b & 0x7fffffff) >> 3) + 0x38000000), b << 29);
}

// c0 + w (c1 + w (c2 + w (c3 + w t)))
__device__ __forceinline__ double ht_poly(double2 a, double2 b, float t, double w) {
  return fma(fma(fma(fma(ht_widen(t), w, b.y), w, b.x), w, a.y), w, a.x);
}

// H0 (if H0) and H1 (if H1) at z = (kr + i ki) d and 1/d, from the offset
// (wx, wy), d = |(wx, wy)|; ka = |k|.  About 11 FP64 instructions for the
// distance, 15 for e^{iz}, 12 per function order.
template <bool H0, bool H1, bool CK>
__device__ __forceinline__ void hankel_tab_eval(const HankelTab& tb, double wx, double wy,
                                                double kr, double ki, double ka, double* rd,
                                                double* h0r, double* h0i, double* h1r,
                                                double* h1i) {
  // d and 1/d: third-order correction of the 2^-20 seed y of 1/sqrt(d2)
  const double d2 = fma(wx, wx, wy * wy);
  const double y = ht_rsqrt_approx(d2);
  const double h = d2 * y;
  const double e = fma(-h, y, 1.0);
  const double q = e * fma(0.375, e, 0.5);
  const double d = fma(h, q, h);
  *rd = fma(y, q, y);
  const double zr = kr * d;
  const double x = CK ? ka * d : zr;
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const unsigned bin = (unsigned)((hi >> 14) - kHtBase);
  if (bin >= (unsigned)kHtBins) {  // outside the octaves, d = 0, infinite or NaN
    const double ds = sqrt(d2);
    *rd = 1.0 / ds;
    hankel_direct<H0, H1, CK>(ds, kr, CK ? ki : 0.0, h0r, h0i, h1r, h1i);
    return;
  }
  // w in [-1/2, 1/2): the mantissa bits below the interval's, exact
  const double w =
      __hiloint2double(0x3ff00000 | ((hi & 0x3fff) << 6) | ((unsigned)lo >> 26), lo << 6) - 1.5;
  const float wf =
      __int_as_float(0x3f800000 | ((hi & 0x3fff) << 9) | ((unsigned)lo >> 23)) - 1.5f;
  // e^{i zr}
  const double tn = fma(zr, 40.743665431525206, 6755399441055744.0);
  const double n = tn - 6755399441055744.0;
  const int in = __double2loint(tn) & (kHtTrig - 1);
  double r = fma(-n, 0.02454369260617026, zr);   // 2 pi / 256
  r = fma(-n, 9.567553118338697e-19, r);  // and its rounding
  const double r2 = r * r;
  const double sn = fma(r * r2, fma(r2, 1.0 / 120.0, -1.0 / 6.0), r);
  const double cm = r2 * fma(r2, fma(r2, -1.0 / 720.0, 1.0 / 24.0), -0.5);  // cos r - 1
  const double2 cs = __ldg(tb.sc + in);
  double er = cs.x + fma(cs.x, cm, -cs.y * sn), ei = cs.y + fma(cs.y, cm, cs.x * sn);
  if (CK) {
    const double a = exp(-ki * d);
    er *= a;
    ei *= a;
  }
  const double2* c = tb.cd + (size_t)bin * 8;
  const float4* ct = tb.ct + (size_t)bin * 3;
  const float4 t4 = __ldg(ct), t5 = __ldg(ct + 1), t6 = __ldg(ct + 2);
  if (H0) {
    const double a = ht_poly(__ldg(c), __ldg(c + 1), fmaf(wf, fmaf(wf, t6.x, t5.x), t4.x), w);
    const double b = ht_poly(__ldg(c + 2), __ldg(c + 3), fmaf(wf, fmaf(wf, t6.y, t5.y), t4.y), w);
    *h0r = fma(er, a, -ei * b);
    *h0i = fma(er, b, ei * a);
  }
  if (H1) {
    const double a = ht_poly(__ldg(c + 4), __ldg(c + 5), fmaf(wf, fmaf(wf, t6.z, t5.z), t4.z), w);
    const double b = ht_poly(__ldg(c + 6), __ldg(c + 7), fmaf(wf, fmaf(wf, t6.w, t5.w), t4.w), w);
    *h1r = fma(er, a, -ei * b);
    *h1i = fma(er, b, ei * a);
  }
}

#endif  // __CUDACC__

}  // namespace bem2d_gpu
