// EulerBeam3D evaluated into arrays: residual and Newton tangent (beam_spin.hpp),
// and the element results.
#pragma once
#include "beam_spin.hpp"

namespace mgpu {

//   X0,X1,X2: element dofs and their first/second time derivatives (X1,X2 ignored if !D)
//   U: U-dof loads per unit length (nullptr if none)
//   out R[12], K[144];  rdir[12] (optional, D): derivative along X₁ += av, X₂ += bv
//   H[36] (optional): ∂R/∂U, column-major 12x3
template <bool D>
MG_HD void beam_element(const BeamConst& c, const double* X0, const double* X1, const double* X2, const double* U,
                        Perturb pt, const double* av, const double* bv, double* R, double* K, double* rdir,
                        double* H) {
  if constexpr (D)
    beam_newmark(c, X0, X1, X2, U, pt, av, bv, R, [&](int i, int j, real v) { K[i + 12 * j] = to_d(v); }, rdir, H);
  else
    beam_static(c, X0, U, R, [&](int i, int j, real v) { K[i + 12 * j] = K[j + 12 * i] = to_d(pt.p0 * v); }, H);
}

// ---- element results of one beam at a state (getresult of the residual's
// requestable values, toolbox/BeamElement.jl:151-189): the element record's
// 69 fields f, the dofs X0[12], the EI scale a (1 without an A-dof); out[50]:
// ε, rₛₘ (9, column-major), then per Gauss point x (3), κ (3), fᵢ = EA ε and
// mᵢ = (GJ κ₁, a EI₃ κ₂, a EI₂ κ₃).  The rotations are the element's own; the
// rest follows kinematics (:177-189): uₗ₂ = rₛₘᵀ d − L/2 e₁ and vₗ₂ = rₛₘᵀΔv.
MG_HD void beam_results(const double* f, const double* X0, double a, double* out) {
  const double* rm = f + 3;
  const double* cm = f;
  const double* zgp = f + 12;
  const double* tgm = f + 18;
  const double* tge = f + 21;
  const double* ya = f + 24;
  const double* yu = f + 28;
  const double* yv = f + 32;
  const double* ka = f + 36;
  const double* ku = f + 40;
  const double* kv = f + 44;
  const double L = f[48];
  const double EA = f[53], EI2 = a * f[54], EI3 = a * f[55], GJ = f[56];
  real r[9], n[3];
  {
    const real v1[3] = {X0[3], X0[4], X0[5]}, v2[3] = {X0[9], X0[10], X0[11]};
    const real s1 = dot3(v1, v1), s2 = dot3(v2, v2);
    real r1[9], r2[9], rd[9], rmr[9], r1m[9];
    rot_matrix(v1, s1, sin_fun(s1), r1);
    rot_matrix(v2, s2, sin_fun(s2), r2);
    half_rotation(r1, r2, n);
    const real s = dot3(n, n);
    rot_matrix(n, s, sin_fun(s), rd);
    for (int k = 0; k < 9; ++k) rmr[k] = rm[k];
    mul33(r1, rmr, r1m);
    mul33(rd, r1m, r);
  }
  real d[3], cs[3], ul2[3], vl2[3];
  for (int i = 0; i < 3; ++i) {
    d[i] = 0.5 * (X0[6 + i] - X0[i]) + 0.5 * tgm[i];
    cs[i] = 0.5 * (X0[i] + X0[6 + i]) + cm[i];
  }
  for (int k = 0; k < 3; ++k) {
    ul2[k] = dot3(r + 3 * k, d);
    vl2[k] = dot3(r + 3 * k, n);
  }
  ul2[0] -= 0.5 * L;
  const real eps = sqrt((ul2[0] + 0.5 * L) * (ul2[0] + 0.5 * L) + ul2[1] * ul2[1] + ul2[2] * ul2[2]) * 2.0 / L - 1.0;
  out[0] = to_d(eps);
  for (int k = 0; k < 9; ++k) out[1 + k] = to_d(r[k]);
  for (int g = 0; g < 4; ++g) {
    double* o = out + 10 + 10 * g;
    const real k0 = ka[g] * vl2[0];
    const real k1 = ku[g] * ul2[1] + kv[g] * vl2[2];
    const real k2 = ku[g] * ul2[2] - kv[g] * vl2[1];
    const real y[3] = {ya[g] * ul2[0], yu[g] * ul2[1] + yv[g] * vl2[2], yu[g] * ul2[2] - yv[g] * vl2[1]};
    real pp[3];
    for (int i = 0; i < 3; ++i) pp[i] = tge[i] * zgp[g] + y[i];
    for (int i = 0; i < 3; ++i) o[i] = to_d(r[i] * pp[0] + r[i + 3] * pp[1] + r[i + 6] * pp[2] + cs[i]);
    o[3] = to_d(k0);
    o[4] = to_d(k1);
    o[5] = to_d(k2);
    o[6] = to_d(EA * eps);
    o[7] = to_d(GJ * k0);
    o[8] = to_d(EI3 * k1);
    o[9] = to_d(EI2 * k2);
  }
}

}  // namespace mgpu
