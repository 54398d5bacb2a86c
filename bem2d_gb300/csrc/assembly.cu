// Galerkin assembly kernels for sm_103a: node tables, near field, mass matrix
// and right-hand sides (FP64 far field and potentials: far_fp64.cu).
//
//  node_table_kernel  per (unknown, Gauss node): Map, Normal, |J| w phi
//  near_kernel        (near.cuh) one warp per self/adjacent pair: graded rules
//                     (IntegrateIdent :67-109 with AdaptedGauss1; Integrate
//                     with AdaptedGauss3 / AdaptedGauss2 for next / prev,
//                     :271-282), fused  alpha*K + beta*M  epilogue; element
//                     geometry tabulated per warp at the rules' distinct
//                     coordinates; the mixed-precision variant evaluates
//                     the Bessel functions in float-float
//  ident_kernel       EvalIdent (lib/bem2d_quadrature.cpp:79-127)
//  rhs_kernel         DotProdBasFuns (lib/bem2d_quadrature.h:111-156)
#include <algorithm>
#include <type_traits>

#include "near.cuh"

namespace bem2d_gpu {

// ---------------------------------------------------------------------------
// One thread per unknown: Map, Normal and |J| w phi at each Gauss node (FP64
// table); optionally the float-float table relative to the element centre
// Map(1/2).
__global__ void node_table_kernel(DevGeom g, DevRules r, NodeTable t, NodeTableFF tf,
                                  int want_ff) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= g.n_unk) return;
  const int e = g.unk_elem[u];
  const double* prm = g.param + 8 * (size_t)e;
  const ElemPt mid = elem_eval(g.kind[e], prm, 0.5);
  float rad = 0.0f;
  for (int q = 0; q < r.ng; ++q) {
    const size_t idx = (size_t)u * r.ng + q;
    const double tq = r.gx[q];
    const ElemPt p = elem_eval(g.kind[e], prm, tq);
    double nx, ny;
    elem_normal(p, &nx, &ny);
    const double w = elem_jac(p) * r.gw[q] * basis_eval(g.unk_kind[u], g.unk_param[u], tq);
    t.x[idx] = p.mx;
    t.y[idx] = p.my;
    t.nx[idx] = nx;
    t.ny[idx] = ny;
    t.w[idx] = w;
    if (want_ff) {
      const double ox = p.mx - mid.mx, oy = p.my - mid.my;
      const ff fox = ff_from_double(ox), foy = ff_from_double(oy);
      const ff fnx = ff_from_double(nx), fny = ff_from_double(ny), fw = ff_from_double(w);
      tf.ox[idx] = make_float2(fox.hi, fox.lo);
      tf.oy[idx] = make_float2(foy.hi, foy.lo);
      tf.nx[idx] = make_float2(fnx.hi, fnx.lo);
      tf.ny[idx] = make_float2(fny.hi, fny.lo);
      tf.w[idx] = make_float2(fw.hi, fw.lo);
      rad = fmaxf(rad, (float)sqrt(ox * ox + oy * oy));
    }
  }
  if (want_ff) {
    tf.c[u] = make_double2(mid.mx, mid.my);
    tf.rad[u] = rad * (1.0f + 1e-6f);
  }
}

void launch_node_table(const DevGeom& g, const DevRules& r, NodeTable t,
                       const NodeTableFF* tf, cudaStream_t s) {
  NodeTableFF z{};
  node_table_kernel<<<(g.n_unk + 127) / 128, 128, 0, s>>>(g, r, t, tf ? *tf : z, tf ? 1 : 0);
}

// ---- near field, real wavenumbers (near.cuh) ----------------------------------
int launch_near(const DevGeom& g, const DevRules& r, const NearPair* pairs, int npairs, int nb,
                int kernel, double k, double eta, double alpha, double beta, double2* out,
                long long ld, cudaStream_t s, float2* out32, long long ld32) {
  if (npairs == 0) return BEM2D_OK;
  const float* tab = out32 ? expi_table_dev() : nullptr;
  if (out32 && !tab) return BEM2D_ERR_NOMEM;
  auto go = [&](auto mixed, auto n) {
    launch_near_m<decltype(mixed)::value, false, decltype(n)::value>(
        g, r, pairs, npairs, kernel, k, 0.0, eta, alpha, beta, tab, out, ld, out32, ld32, s);
  };
  using One = std::integral_constant<int, 1>;
  using Run = std::integral_constant<int, kNearBasis>;
  if (out32)
    nb > 1 ? go(std::true_type{}, Run{}) : go(std::true_type{}, One{});
  else
    nb > 1 ? go(std::false_type{}, Run{}) : go(std::false_type{}, One{});
  return BEM2D_OK;
}

// ---------------------------------------------------------------------------
__global__ void ident_kernel(DevGeom g, DevRules r, const NearPair* __restrict__ pairs,
                             int npairs, double2* __restrict__ out, long long ld) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= npairs) return;
  const NearPair pr = pairs[p];
  if (!pr.same) return;
  out[(size_t)pr.j * ld + pr.i] = make_double2(mass_entry(g, r, pr.i, pr.j), 0.0);
}

void launch_ident(const DevGeom& g, const DevRules& r, const NearPair* pairs,
                  int npairs, double2* out, long long ld, cudaStream_t s) {
  if (npairs == 0) return;
  ident_kernel<<<(npairs + 127) / 128, 128, 0, s>>>(g, r, pairs, npairs, out, ld);
}

// ---------------------------------------------------------------------------
// b_u = scale * sum_q f(x_q) |J| phi_u w_q, f one of the plane-wave
// functionals (lib/bem2d_fun.h:14-93).  The wavenumber is k + i ki:
// e^{i (k + i ki) d.x} = e^{-ki d.x} e^{i k d.x}.
__global__ void rhs_kernel(int n, NodeTable t, int ng, int fun, double k, double ki,
                           double dx, double dy, double eta, double scale,
                           double2* __restrict__ out) {
  const int u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= n) return;
  double acc_re = 0.0, acc_im = 0.0;
  for (int q = 0; q < ng; ++q) {
    const size_t o = (size_t)u * ng + q;
    const double dd = dx * t.x[o] + dy * t.y[o];
    const double ph = k * dd;
    double fs, fc;
    sincos(ph, &fs, &fc);
    if (ki != 0.0) {
      const double a = exp(-ki * dd);
      fs *= a;
      fc *= a;
    }
    double vr, vi;
    if (fun == BEM2D_FUN_PLANEWAVE) {
      vr = fc;
      vi = fs;
    } else {
      const double nd = t.nx[o] * dx + t.ny[o] * dy;
      vr = -k * fs * nd;  // i k f (n.d)
      vi = k * fc * nd;
      if (ki != 0.0) {  // the i * (i ki) f (n.d) part
        vr -= ki * fc * nd;
        vi -= ki * fs * nd;
      }
      if (fun == BEM2D_FUN_COMBINEDPLANEWAVE) {  // - i eta f
        vr += eta * fs;
        vi -= eta * fc;
      }
    }
    acc_re = fma(vr, t.w[o], acc_re);
    acc_im = fma(vi, t.w[o], acc_im);
  }
  out[u] = make_double2(scale * acc_re, scale * acc_im);
}

void launch_rhs(const DevGeom& g, const NodeTable& t, int ng, int fun, double k,
                double dx, double dy, double eta, double scale, double2* out,
                cudaStream_t s, double ki) {
  rhs_kernel<<<(g.n_unk + 127) / 128, 128, 0, s>>>(g.n_unk, t, ng, fun, k, ki, dx, dy,
                                                   eta, scale, out);
}

}  // namespace bem2d_gpu
