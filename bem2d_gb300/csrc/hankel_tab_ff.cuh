// Float-float H0 and H1 for 4 <= x < 4096 from a table of short polynomials:
// the evaluator of the mixed-precision far field.
//
// The far field issues FP32 instructions only, so its time is their number.
// With amp = sqrt(2/(pi x)) and E = e^{i(x - pi/4)}
//   H0(x) = E amp (P0 + i Q0),   H1(x)/x = -i E (amp/x) (P1 + i Q1),
// and amp P0, amp Q0, (amp/x) P1, (amp/x) Q1 are algebraic in x: on each of
// 128 equal intervals of every octave a polynomial of degree 5 in x - centre
// carries them to 2^-49 (the nearest singularity, x = 0, lies 128 intervals
// away).  Terms 0..2 are float-float, 3..5 (below 2^-22) FP32.  That is 25
// instructions per function and nothing else: no 1/x, 1/sqrt(x) or branch on
// the range of x as in pq_ff, whose pieces are the general evaluator.
//   E: x = n (2 pi/512) + r, |r| <= 0.52 (2 pi/512); E = T (1 + (cos r - 1) + i
// sin r) with T from a table of 512, sin r to r^5 and cos r - 1 to r^4.
//
// Sums and products here leave the low part unnormalised (up to a few ulps of
// the high one) wherever the consumer takes it so; what that and the
// truncations cost is checked against 50 digits on the CPU.
#pragma once

#include "hankel.cuh"
#include "hankel_ff.cuh"

namespace bem2d_gpu {

constexpr int kFtOct0 = 2;       // x from 2^2 ..
constexpr int kFtOctaves = 10;   // .. up to 2^12
constexpr int kFtPerOct = 128;   // seven mantissa bits
constexpr int kFtBins = kFtOctaves * kFtPerOct;
constexpr int kFtBase = (127 + kFtOct0) * kFtPerOct;  // bin 0's exponent | mantissa bits
constexpr int kFtWords = 36;     // floats of one interval (see ft_build)
constexpr int kFtTrig = 512;
constexpr int kFtFloats = kFtBins * kFtWords + 4 * kFtTrig;

struct FtVec4 {
  float x, y, z, w;
};

__host__ __device__ __forceinline__ int ft_bits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_int(x);
#else
  int i;
  static_assert(sizeof i == sizeof x, "");
  __builtin_memcpy(&i, &x, sizeof i);
  return i;
#endif
}
__host__ __device__ __forceinline__ float ft_float(int i) {
#ifdef __CUDA_ARCH__
  return __int_as_float(i);
#else
  float x;
  __builtin_memcpy(&x, &i, sizeof x);
  return x;
#endif
}

// Interval of x; outside [0, kFtBins) for x outside [4, 4096), infinite or NaN.
__host__ __device__ __forceinline__ int ft_bin(float x) { return (ft_bits(x) >> 16) - kFtBase; }

// Products and a b + c d with the low part left unnormalised.
__host__ __device__ __forceinline__ ff ffu_mul(ff a, ff b) {
  const float p = f_mul_rn(a.hi, b.hi);
  float e = fmaf(a.hi, b.hi, -p);
  e = fmaf(a.hi, b.lo, e);
  return ff_make(p, fmaf(a.lo, b.hi, e));
}
__host__ __device__ __forceinline__ ff ffu_dot2(ff a, ff b, ff c, ff d) {
  const float p = f_mul_rn(a.hi, b.hi);
  const float q = f_mul_rn(c.hi, d.hi);
  float e1 = fmaf(a.hi, b.hi, -p);
  e1 = fmaf(a.hi, b.lo, e1);
  e1 = fmaf(a.lo, b.hi, e1);
  float e2 = fmaf(c.hi, d.hi, -q);
  e2 = fmaf(c.hi, d.lo, e2);
  e2 = fmaf(c.lo, d.hi, e2);
  const ff s = two_sum(p, q);
  return ff_make(s.hi, s.lo + (e1 + e2));
}
__host__ __device__ __forceinline__ ff ffu_add(ff a, ff b) {
  const ff s = two_sum(a.hi, b.hi);
  return ff_make(s.hi, s.lo + (a.lo + b.lo));
}

// sqrt(a): the single-precision root a y, y ~ 1/sqrt(a), corrected once in
// single precision (h within half a unit of its last place and little more),
// then the residual a - h^2, one FMA, as the low part.
__host__ __device__ __forceinline__ ff ff_sqrt(ff a) {
  const float y = f_rsqrt(a.hi);
  const float x0 = f_mul_rn(a.hi, y), hy = 0.5f * y;
  const float h = fmaf(fmaf(-x0, x0, a.hi), hy, x0);
  return ff_make(h, f_mul_rn(fmaf(-h, h, a.hi) + a.lo, hy));
}

// c0 + w (c1 + w (c2 + w (c3 + w (c4 + w c5)))), c0..c2 float-float: each
// coefficient bounds the rest of the sum, so fast two-sums split the heads
__host__ __device__ __forceinline__ ff ft_poly(float c0h, float c0l, float c1h, float c1l,
                                               float c2h, float c2l, float c3, float c4, float c5,
                                               ff w) {
  const float t = f_mul_rn(w.hi, fmaf(fmaf(c5, w.hi, c4), w.hi, c3));
  const float s2 = c2h + t;
  const float e2 = (t - (s2 - c2h)) + c2l;
  const float p1 = f_mul_rn(w.hi, s2);
  float f1 = fmaf(w.hi, s2, -p1);
  f1 = fmaf(w.hi, e2, f1);
  f1 = fmaf(w.lo, s2, f1);
  const float s1 = c1h + p1;
  const float e1 = (p1 - (s1 - c1h)) + (f1 + c1l);
  const float p0 = f_mul_rn(w.hi, s1);
  float f0 = fmaf(w.hi, s1, -p0);
  f0 = fmaf(w.hi, e1, f0);
  f0 = fmaf(w.lo, s1, f0);
  const float s0 = c0h + p0;
  return ff_make(s0, (p0 - (s0 - c0h)) + (f0 + c0l));
}

// amp P0, amp Q0 (if H0), (amp/x) P1, (amp/x) Q1 (if H1) at x from its
// interval's 36 floats (16-byte aligned).
template <bool H0, bool H1, typename V4>
__host__ __device__ __forceinline__ void ft_pq(const V4* c, ff x, ff* p0, ff* q0, ff* p1, ff* q1) {
  // x - centre: the difference of the heads is exact, and 0 or above |x.lo|
  const ff w = fast_two_sum(x.hi - ft_float((ft_bits(x.hi) & ~0xffff) | 0x8000), x.lo);
  if (H0) {
    const V4 a = c[0], b = c[1], d = c[2], e = c[3];
    const float l = c[8].x, m = c[8].y;
    *p0 = ft_poly(a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, l, w);
    *q0 = ft_poly(d.x, d.y, d.z, d.w, e.x, e.y, e.z, e.w, m, w);
  }
  if (H1) {
    const V4 a = c[4], b = c[5], d = c[6], e = c[7];
    const float l = c[8].z, m = c[8].w;
    *p1 = ft_poly(a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, l, w);
    *q1 = ft_poly(d.x, d.y, d.z, d.w, e.x, e.y, e.z, e.w, m, w);
  }
}

// 2 pi/512 = C1 + C2 + C3 (kRedC1 .. kRedC3 of hankel_ff.cuh over 8)
constexpr float kFtC1 = kRedC1 / 8.0f;
constexpr float kFtC2 = kRedC2 / 8.0f;
constexpr float kFtC3 = kRedC3 / 8.0f;

// e^{i(x - pi/4)}, 0 <= x < 4096; trig[n] = (cos, sin)(2 pi n/512 - pi/4) as
// (cos.hi, cos.lo, sin.hi, sin.lo).
template <typename V4>
__host__ __device__ __forceinline__ ffc ft_expi(ff x, const V4* trig) {
  const float magic = 12582912.0f;  // 1.5 2^23: rounds to an integer in the low bits
  const float tn = fmaf(x.hi, 8.0f * kRedInv, magic);
  const float j = tn - magic;
  const V4 T = trig[ft_bits(tn) & (kFtTrig - 1)];
  const float r1 = fmaf(-j, kFtC1, x.hi);  // exact
  // r1 + x.lo - j C2 - j C3
  const float p2 = f_mul_rn(j, -kFtC2), e2 = fmaf(j, -kFtC2, -p2);
  const ff t = two_sum(p2, x.lo);
  ff r = two_sum(r1, t.hi);
  r.lo += fmaf(-j, kFtC3, t.lo + e2);
  const float rr = f_mul_rn(r.hi, r.hi);
  const float re = fmaf(r.hi + r.hi, r.lo, fmaf(r.hi, r.hi, -rr));
  // s = sin r, c = 1 - cos r
  const float sl = fmaf(f_mul_rn(rr, r.hi), fmaf(rr, 1.0f / 120.0f, -1.0f / 6.0f), r.lo);
  const float ch = 0.5f * rr;
  const float cl = fmaf(-1.0f / 24.0f * rr, rr, 0.5f * re);
  // T - T c + i T s: |T.hi| is 0 or above |s|, so fast two-sums split the
  // sums from the largest term down
  ffc e;
  {
    const float p = f_mul_rn(T.z, r.hi), q = f_mul_rn(T.x, ch);
    float f = fmaf(T.z, r.hi, -p);
    f = fmaf(T.z, sl, f);
    f = fmaf(T.w, r.hi, f);
    float h = fmaf(T.x, ch, -q);
    h = fmaf(T.x, cl, h);
    h = fmaf(T.y, ch, h);
    const ff u = fast_two_sum(T.x, -p);
    const ff v = fast_two_sum(u.hi, -q);
    e.re = ff_make(v.hi, (u.lo + v.lo) + (T.y - (f + h)));
  }
  {
    const float p = f_mul_rn(T.x, r.hi), q = f_mul_rn(T.z, ch);
    float f = fmaf(T.x, r.hi, -p);
    f = fmaf(T.x, sl, f);
    f = fmaf(T.y, r.hi, f);
    float h = fmaf(T.z, ch, -q);
    h = fmaf(T.z, cl, h);
    h = fmaf(T.w, ch, h);
    const ff u = fast_two_sum(T.z, p);
    const ff v = fast_two_sum(u.hi, -q);
    e.im = ff_make(v.hi, (u.lo + v.lo) + (T.w + (f - h)));
  }
  return e;
}

// Host-side table: per interval c0 .. c2 as (hi, lo) pairs, c3, c4 of the four
// functions amp P0, amp Q0, (amp/x) P1, (amp/x) Q1 (8 floats each), then their
// c5; after the intervals the 512 values of e^{i(2 pi n/512 - pi/4)}.  The
// coefficients are discrete Chebyshev sums over 16 points of the FP64
// evaluator (least squares: its rounding is averaged, not interpolated).
inline void ft_build(float* tab) {
  const long double pi = 3.14159265358979323846264338327950288L;
  constexpr int kN = 16, kD = 6;
  double v[kN], ct[kD][kN];
  for (int l = 0; l < kN; ++l) {
    v[l] = (double)cosl(pi * (l + 0.5L) / kN);
    for (int j = 0; j < kD; ++j) ct[j][l] = (double)(cosl(pi * j * (l + 0.5L) / kN) * 2 / kN);
  }
  for (int bin = 0; bin < kFtBins; ++bin) {
    const double len = std::ldexp(1.0, kFtOct0 + bin / kFtPerOct) / kFtPerOct;
    const double cen = (kFtPerOct + bin % kFtPerOct + 0.5) * len;
    double a[4][kD] = {};
    for (int l = 0; l < kN; ++l) {
      const double x = cen + 0.5 * len * v[l];
      double p0, q0, p1, q1;
      const double ix = hankel_pq_d(x, &p0, &q0, &p1, &q1);
      const double amp = std::sqrt(kTwoOverPi * ix);
      const double f[4] = {amp * p0, amp * q0, amp * ix * p1, amp * ix * q1};
      for (int fn = 0; fn < 4; ++fn)
        for (int j = 0; j < kD; ++j) a[fn][j] += f[fn] * ct[j][l];
    }
    float* o = tab + (size_t)bin * kFtWords;
    for (int fn = 0; fn < 4; ++fn) {
      const double* b = a[fn];
      const double c[kD] = {0.5 * b[0] - b[2] + b[4], b[1] - 3 * b[3] + 5 * b[5],
                            2 * b[2] - 8 * b[4],      4 * b[3] - 20 * b[5],
                            8 * b[4],                 16 * b[5]};
      double s = 1.0;
      for (int j = 0; j < kD; ++j, s *= 2.0 / len) {
        const double cj = c[j] * s;
        const float h = (float)cj;
        if (j < 3) {
          o[8 * fn + 2 * j] = h;
          o[8 * fn + 2 * j + 1] = (float)(cj - (double)h);
        } else if (j < 5) {
          o[8 * fn + 3 + j] = h;
        } else {
          o[32 + fn] = h;
        }
      }
    }
  }
  float* t = tab + (size_t)kFtBins * kFtWords;
  for (int n = 0; n < kFtTrig; ++n) {
    // exact quarter-turn symmetry is not needed, exact zeros are (n = 192, 448: cos; 64, 320: sin)
    const long double a = 2.0L * pi * n / kFtTrig - pi / 4;
    const long double c = (n % 256 == 192) ? 0.0L : cosl(a), s = (n % 256 == 64) ? 0.0L : sinl(a);
    t[4 * n] = (float)c;
    t[4 * n + 1] = (float)(c - (long double)t[4 * n]);
    t[4 * n + 2] = (float)s;
    t[4 * n + 3] = (float)(s - (long double)t[4 * n + 2]);
  }
}

}  // namespace bem2d_gpu
