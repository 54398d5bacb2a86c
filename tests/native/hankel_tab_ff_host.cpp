// Host build of the far field's float-float table evaluator
// (bem2d_gb300/csrc/hankel_tab_ff.cuh), exported for accuracy tests.
#include <vector>

#include "hankel_tab_ff.cuh"

using namespace bem2d_gpu;

// out[4i..4i+3] = J0, Y0, J1/x, Y1/x at 4 <= x[i] < 4096 (x rounded to
// float-float first); returns how many x lie outside the table
extern "C" int hankel_tab_ff_host(int n, const double* x, double* out) {
  std::vector<FtVec4> tab(kFtFloats / 4);
  ft_build(&tab[0].x);
  int outside = 0;
  for (int i = 0; i < n; ++i) {
    const ff xf = ff_from_double(x[i]);
    const int bin = ft_bin(xf.hi);
    if ((unsigned)bin >= (unsigned)kFtBins) {
      ++outside;
      continue;
    }
    ff p0, q0, p1, q1;
    ft_pq<true, true>(&tab[(size_t)bin * (kFtWords / 4)], xf, &p0, &q0, &p1, &q1);
    const ffc e = ft_expi(xf, &tab[(size_t)kFtBins * (kFtWords / 4)]);
    // H0 = E (P0 + i Q0), H1 = -i E (P1 + i Q1)
    out[4 * i] = ff_to_double(ffu_dot2(e.re, p0, ff_neg(e.im), q0));
    out[4 * i + 1] = ff_to_double(ffu_dot2(e.re, q0, e.im, p0));
    out[4 * i + 2] = ff_to_double(ffu_dot2(e.re, q1, e.im, p1));
    out[4 * i + 3] = -ff_to_double(ffu_dot2(e.re, p1, ff_neg(e.im), q1));
  }
  return outside;
}

// out[i] = sqrt(x[i]) through ff_sqrt
extern "C" void sqrt_ff_host(int n, const double* x, double* out) {
  for (int i = 0; i < n; ++i) out[i] = ff_to_double(ff_sqrt(ff_from_double(x[i])));
}
