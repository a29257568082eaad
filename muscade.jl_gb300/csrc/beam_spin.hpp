// EulerBeam3D residual and exact Newton tangent in closed form, for the GB300
// element kernels (host-compilable too).
//
// Reference behaviour (toolbox/BeamElement.jl):
//   residual   :151-174    R = Σ_gp (fᵢ ε∂X₀ + mᵢ·κ∂X₀ + fₑ·x∂X₀ + mₑ·vₛₘ∂X₀) dL
//   kinematics :177-189,  corotated :193-208,  resultants :28-64
//   rotations  toolbox/Rotations.jl:13-182 (scac's Taylor branch mirrored here)
//
// Formulation (mathematically identical to the reference):
//  * r₁ = Rod(v₁), r₂ = Rod(v₂), n = Δv = ½Rod⁻¹(r₂r₁ᵀ), rₛₘ = Rod(n) r₁ rₘ with
//    columns t, n̂, b̂.  With d = ½(u₂−u₁)+½tgₘ the strain measures are
//    ε = 2|d|/L − 1, θ = rₛₘᵀn and w = (n̂·d, b̂·d); a Gauss point lies at
//    x = yᵤ d + (yₐ−yᵤ)(t·d) t + yᵥ n×t + ½(u₁+u₂) + cₘ.
//  * Σ_gp(fᵢ ε∂X₀ + mᵢ·κ∂X₀)dL is the gradient of the quadratic strain energy
//    Π; the external terms are the gradient of ψ = Σ_gp dL f_gp·x_gp +
//    Σ_gp dL mₑ·vₛₘ with the loads held fixed.  R = ∇(Π+ψ) and the tangent is
//    ∇²(Π+ψ) plus Σ_gp dL x∂X₀ᵀ δf_gp + vₛₘ∂X₀ᵀ δmₑ (load variation).
//  * Rotations are varied by spins.  δr_a = [w_a]r_a with w_a = T(v_a)δv_a, and in
//    the frame half way between the nodes (x' = Rod(n) w₁, y' = Rod(n)ᵀ w₂,
//    p = ½(x'+y'), r = y'−x') everything is a function of n alone:
//        δn = D r,          D = (I − c n nᵀ)/(2a)
//        spin of rₛₘ  ω = p + β n×r,   β = b/(2a)
//        δp = β(n×r)×p + p̃,   δr = −r×p + β(n×r)×r + r̃      (second variation)
//    with a = sinθ/θ, b = (1−cosθ)/θ², c = (θ−sinθ)/θ³ at θ = |n| and p̃, r̃ the parts
//    from ẇ_a.  D is even and the odd part of the spin is β[n] because n changes
//    sign, and nothing else does, when the nodes are exchanged.  So the whole
//    second variation of Π+ψ is a 9 × 9 quadratic form in (δd, p, r), summed once
//    with the moments of the frozen stresses, and goes to the dofs with two 3 × 3
//    matrices, Rod(n)T(v₁) and Rod(n)ᵀT(v₂).
//    What bounds the element on GB300 is the number of FP64 instructions (a warp
//    instruction holds a sub-partition's FP64 pipe for 64 cycles), and this form
//    needs a sixth of those of second-order Taylor arithmetic through every
//    rotation matrix (21 Hessian entries of each of nine components), which is
//    how the derivative was taken before; csrc/flopcount.cpp counts them.
// Output layout: R[12], K[i + 12 j] = ∂R_i/∂X_j (column-major, like asm[2]).
#pragma once
#include "tj.hpp"

namespace mgpu {

// ---- functions of a rotation angle θ, by s = θ² ---------------------------
//   a = sinθ/θ, b = (1−cosθ)/θ², c = (θ−sinθ)/θ³ and the two remainders they are
// built from, e = (½−b)/s and f = (1/6−c)/s (so that no difference of nearly
// equal numbers is taken): Taylor series of e and f, Σ(−s)ᵏ/(2k+4)! and
// Σ(−s)ᵏ/(2k+5)!, whose first omitted term is below 2⁻⁵⁶ of the sum (8 terms up
// to s = 1, 15 up to s = 10, |θ| just over π).  The derivatives in s follow:
//   a_s = (c−b)/2,  b_s = e − c/2,  c_s = (3f−e)/2.
struct SinFun {
  real a, b, c, e, f;
};
MG_HD real sin_as(const SinFun& q) { return 0.5 * (q.c - q.b); }
MG_HD real sin_bs(const SinFun& q) { return fma(-0.5, q.c, q.e); }
MG_HD real sin_cs(const SinFun& q) { return 0.5 * fma(3.0, q.f, -q.e); }

// 1/n!
MG_HD constexpr double inv_fact(int n) {
  double r = 1.0;
  for (int k = 2; k <= n; ++k) r *= k;
  return 1.0 / r;
}
template <int K>
MG_HD void sin_series(real s, real& e, real& f) {
  real ee = inv_fact(2 * K + 2), ff = inv_fact(2 * K + 3);
#pragma unroll
  for (int k = K - 2; k >= 0; --k) {
    ee = fma(-s, ee, inv_fact(2 * k + 4));
    ff = fma(-s, ff, inv_fact(2 * k + 5));
  }
  e = ee;
  f = ff;
}
MG_HD SinFun sin_fun(real s) {
  SinFun q;
  if (s < 10.0) {
    if (s < 1.0)
      sin_series<8>(s, q.e, q.f);
    else
      sin_series<15>(s, q.e, q.f);
    q.c = fma(-s, q.f, 1.0 / 6.0);
    q.b = fma(-s, q.e, 0.5);
    q.a = fma(-s, q.c, 1.0);
  } else {  // also NaN
    const real th = sqrt(s);
    real sn, cs;
    sincos(th, &sn, &cs);
    const real is = 1.0 / s;
    q.a = sn / th;
    q.b = (1.0 - cs) * is;
    q.c = (1.0 - q.a) * is;
    q.e = (0.5 - q.b) * is;
    q.f = (1.0 / 6.0 - q.c) * is;
  }
  return q;
}

// 1/scac(x) with scac(x) = sinc1(acos x) and the reference's degree-5 Taylor
// branch near 1 (toolbox/Rotations.jl)
constexpr double kScac1 = 1.0 / 3.0, kScac2 = -2.0 / 90.0, kScac3 = 0.0052911879917544626,
                 kScac4 = -0.0016229317117234072, kScac5 = 0.0005625;
MG_HD real inv_scac(real x) {
  const real dx = x - 1.0;
  if (!(fabs(dx) > 1e-3)) return 1.0 / (1.0 + dx * (kScac1 + dx * (kScac2 + dx * (kScac3 + dx * (kScac4 + dx * kScac5)))));
  const real th = acos(x);
  return 1.0 / sin_fun(th * th).a;
}
// 1/scac and its first two derivatives in x
MG_HD void inv_scac2(real x, real g[3]) {
  const real dx = x - 1.0;
  real f0, f1, f2;
  if (!(fabs(dx) > 1e-3)) {
    f0 = 1.0 + dx * (kScac1 + dx * (kScac2 + dx * (kScac3 + dx * (kScac4 + dx * kScac5))));
    f1 = kScac1 + dx * (2.0 * kScac2 + dx * (3.0 * kScac3 + dx * (4.0 * kScac4 + dx * (5.0 * kScac5))));
    f2 = 2.0 * kScac2 + dx * (6.0 * kScac3 + dx * (12.0 * kScac4 + dx * (20.0 * kScac5)));
  } else {  // dx/ds = −a/2 along x = cosθ, s = θ²
    const real th = acos(x);
    const SinFun q = sin_fun(th * th);
    const real ia = 1.0 / q.a;
    f0 = q.a;
    f1 = (q.b - q.c) * ia;
    f2 = -2.0 * ia * ia * (sin_bs(q) - sin_cs(q) - f1 * sin_as(q));
  }
  const real i0 = 1.0 / f0, i2 = i0 * i0;
  g[0] = i0;
  g[1] = -f1 * i2;
  g[2] = i2 * fma(2.0 * f1 * f1, i0, -f2);
}

// ---- 3-vectors and 3 × 3 matrices (column-major) ---------------------------
MG_HD real dot3(const real a[3], const real b[3]) { return fma(a[2], b[2], fma(a[1], b[1], a[0] * b[0])); }
MG_HD void cross3(const real a[3], const real b[3], real r[3]) {
  r[0] = fma(a[1], b[2], -(a[2] * b[1]));
  r[1] = fma(a[2], b[0], -(a[0] * b[2]));
  r[2] = fma(a[0], b[1], -(a[1] * b[0]));
}
MG_HD void cross3_add(real s, const real a[3], const real b[3], real r[3]) {  // r += s a×b
  real c[3];
  cross3(a, b, c);
  for (int i = 0; i < 3; ++i) r[i] = fma(s, c[i], r[i]);
}
MG_HD void mul33(const real A[9], const real B[9], real C[9]) {  // A B
  for (int j = 0; j < 3; ++j)
    for (int i = 0; i < 3; ++i) C[i + 3 * j] = fma(A[i + 6], B[2 + 3 * j], fma(A[i + 3], B[1 + 3 * j], A[i] * B[3 * j]));
}
MG_HD void mul33t(const real A[9], const real B[9], real C[9]) {  // Aᵀ B
  for (int j = 0; j < 3; ++j)
    for (int i = 0; i < 3; ++i) C[i + 3 * j] = dot3(A + 3 * i, B + 3 * j);
}
MG_HD void mul33nt(const real A[9], const real B[9], real C[9]) {  // A Bᵀ
  for (int j = 0; j < 3; ++j)
    for (int i = 0; i < 3; ++i) C[i + 3 * j] = fma(A[i + 6], B[j + 6], fma(A[i + 3], B[j + 3], A[i] * B[j]));
}
// diag·I + k [v] + m v vᵀ
MG_HD void axis_matrix(real diag, real k, real m, const real v[3], real M[9]) {
  const real m0 = m * v[0], m1 = m * v[1], m2 = m * v[2];
  const real p01 = m0 * v[1], p02 = m0 * v[2], p12 = m1 * v[2];
  const real k0 = k * v[0], k1 = k * v[1], k2 = k * v[2];
  M[0] = fma(m0, v[0], diag);
  M[4] = fma(m1, v[1], diag);
  M[8] = fma(m2, v[2], diag);
  M[1] = p01 + k2;
  M[3] = p01 - k2;
  M[2] = p02 - k1;
  M[6] = p02 + k1;
  M[5] = p12 + k0;
  M[7] = p12 - k0;
}
// Rodrigues(v) = cosθ I + a [v] + b v vᵀ (Rotations.jl:131-135) and its left
// tangent map T(v) = a I + b [v] + c v vᵀ
MG_HD void rot_matrix(const real v[3], real s, const SinFun& q, real R[9]) {
  axis_matrix(fma(-s, q.b, 1.0), q.a, q.b, v, R);
}
MG_HD void tan_matrix(const real v[3], const SinFun& q, real T[9]) { axis_matrix(q.a, q.b, q.c, v, T); }

// Half relative rotation n = ½Rod⁻¹(r₂r₁ᵀ), Rod⁻¹(m) = spin⁻¹(m)/scac((tr m − 1)/2)
// (Rotations.jl:105)
MG_HD void half_rotation(const real r1[9], const real r2[9], real n[3]) {
  real Q[9];
  mul33nt(r2, r1, Q);
  const real h = 0.25 * inv_scac(0.5 * (Q[0] + Q[4] + Q[8] - 1.0));
  n[0] = h * (Q[5] - Q[7]);
  n[1] = h * (Q[6] - Q[2]);
  n[2] = h * (Q[1] - Q[3]);
}

// ---- per-element constants, precomputed at create time ----------------------
struct BeamConst {
  double rm[9];   // as-meshed frame (column-major)
  double tgm[3];  // c₂ − c₁
  double L;
  // strain energy Π = ½kε ε² + ½kt θt² + ½k3v θb² + k3uv wn θb + ½k3u wn²
  //                 + ½k2v θn² − k2uv wb θn + ½k2u wb²
  double ke, kt, k3u, k3uv, k3v, k2u, k2uv, k2v;
  double S0;                                    // Σ dL
  double dL[4], ya[4], yu[4], yv[4];            // Gauss data
  double mu, iota1, w, Ca[3], Cl[3], Cq[3];     // cross section (dynamic part)
};

// Newton variation of the state: X₀ += p0 δ, X₁ += p1 δ, X₂ += p2 δ
// (SweepX{0}: 1,0,0;  Newmark: 1,a₁,b₁;  diffed K/C/M: unit vectors).
struct Perturb {
  double p0, p1, p2;
};

// rotation-dof index (0..5) of element dof j, or -1 for translations
MG_HD int rot_index(int j) { return (j >= 3 && j < 6) ? j - 3 : (j >= 9 ? j - 6 : -1); }

// Geometry of an element at a state: what both the residual and the tangent use.
struct BeamState {
  real n[3], s;      // half relative rotation and |n|²
  SinFun q;          // its functions
  real rd[9];        // Rod(n)
  real rs[9];        // rₛₘ: t, n̂, b̂
  real d[3], dh[3], idn, eps;
  real th[3], wn, wb;
};

MG_HD void beam_state(const BeamConst& c, const double* X0, SinFun& q1, SinFun& q2, BeamState& g) {
  const real v1[3] = {X0[3], X0[4], X0[5]}, v2[3] = {X0[9], X0[10], X0[11]};
  real r1[9], r1m[9];
  {
    real r2[9];
    const real s1 = dot3(v1, v1), s2 = dot3(v2, v2);
    q1 = sin_fun(s1);
    q2 = sin_fun(s2);
    rot_matrix(v1, s1, q1, r1);
    rot_matrix(v2, s2, q2, r2);
    half_rotation(r1, r2, g.n);
  }
  g.s = dot3(g.n, g.n);
  g.q = sin_fun(g.s);
  rot_matrix(g.n, g.s, g.q, g.rd);
  real rm[9];
  for (int k = 0; k < 9; ++k) rm[k] = c.rm[k];
  mul33(r1, rm, r1m);
  mul33(g.rd, r1m, g.rs);
  for (int i = 0; i < 3; ++i) g.d[i] = 0.5 * (X0[6 + i] - X0[i]) + 0.5 * c.tgm[i];
  const real dn = sqrt(dot3(g.d, g.d));
  g.idn = 1.0 / dn;
  for (int i = 0; i < 3; ++i) g.dh[i] = g.d[i] * g.idn;
  g.eps = dn * 2.0 / c.L - 1.0;
  for (int k = 0; k < 3; ++k) g.th[k] = dot3(g.rs + 3 * k, g.n);
  g.wn = dot3(g.rs + 3, g.d);
  g.wb = dot3(g.rs + 6, g.d);
}

// External loads held fixed in the residual: Σ dL yᵤ f, Σ dL (yₐ−yᵤ) f,
// Σ dL yᵥ f, Σ dL f and Σ dL mₑ
struct BeamLoads {
  real u[3], a[3], v[3], o[3], m[3];
};

// The residual, and the second variation with the loads held: the 9 × 9 form in
// (δd, p, r), then its dof entries through out(i, j, v), each pair i <= j of the
// symmetric matrix once.  ROT: with the moment term mₑ·vₛₘ.
template <bool ROT, class Out>
MG_HD void beam_frozen(const BeamConst& c, const double* X0, const SinFun& q1, const SinFun& q2, const BeamState& g,
                       const BeamLoads& f, double* R, Out&& out) {
  const real *t = g.rs, *nn = g.rs + 3, *bb = g.rs + 6, *n = g.n, *d = g.d;
  // stresses σ = ∂Π/∂q, q = (ε, θ, w)
  const real s_e = c.ke * g.eps;
  const real s_t = c.kt * g.th[0];
  const real s_wn = fma(c.k3u, g.wn, c.k3uv * g.th[2]);
  const real s_b = fma(c.k3uv, g.wn, c.k3v * g.th[2]);
  const real s_wb = fma(c.k2u, g.wb, -(c.k2uv * g.th[1]));
  const real s_n = fma(c.k2v, g.th[1], -(c.k2uv * g.wb));
  const real tA = dot3(t, f.a), td = dot3(t, d), tV = dot3(t, f.v);
  // ---- first variation: Φ̇ = P·ḋ + gO·ω + gv·ṅ
  real ps[3], qs[3], P[3];  // Σ σ_θ column, Σ σ_w column, ∂Φ/∂d
  for (int i = 0; i < 3; ++i) {
    ps[i] = fma(s_b, bb[i], fma(s_n, nn[i], s_t * t[i]));
    qs[i] = fma(s_wb, bb[i], s_wn * nn[i]);
    P[i] = fma(tA, t[i], qs[i]);
  }
  const real at[3] = {fma(s_t, n[0], fma(tA, d[0], td * f.a[0])) + fma(f.v[1], n[2], -(f.v[2] * n[1])),
                      fma(s_t, n[1], fma(tA, d[1], td * f.a[1])) + fma(f.v[2], n[0], -(f.v[0] * n[2])),
                      fma(s_t, n[2], fma(tA, d[2], td * f.a[2])) + fma(f.v[0], n[1], -(f.v[1] * n[0]))};
  real an[3], ab[3], gv[3], gO[3];
  for (int i = 0; i < 3; ++i) {
    an[i] = fma(s_n, n[i], s_wn * d[i]);
    ab[i] = fma(s_b, n[i], s_wb * d[i]);
    gv[i] = ps[i];
  }
  cross3_add(1.0, t, f.v, gv);
  cross3(t, at, gO);
  cross3_add(1.0, nn, an, gO);
  cross3_add(1.0, bb, ab, gO);
  // ---- second variation, spin part K6 (packed 00 01 02 11 12 22): sym(Σ a yᵀ) − (Σ a·y) I
  // + sym2(t×d, t×A), and the coupling C = [ps] + V tᵀ − (t·V) I of ω with ṅ
  real K6[6];
  {
    const real tr = dot3(at, t) + dot3(an, nn) + dot3(ab, bb);
    real td_[3], tA_[3];
    cross3(t, d, td_);
    cross3(t, f.a, tA_);
    int k = 0;
    for (int i = 0; i < 3; ++i)
      for (int j = i; j < 3; ++j, ++k) {
        if (i == j) {
          K6[k] = fma(at[i], t[i], fma(an[i], nn[i], fma(ab[i], bb[i], fma(2.0 * td_[i], tA_[i], -tr))));
        } else {
          const real y = fma(at[i], t[j], fma(at[j], t[i], fma(an[i], nn[j], fma(an[j], nn[i], fma(ab[i], bb[j], ab[j] * bb[i])))));
          K6[k] = fma(0.5, y, fma(td_[i], tA_[j], td_[j] * tA_[i]));
        }
      }
  }
  if constexpr (ROT) {  // mₑ·vₛₘ, vₛₘ = Rod⁻¹(rₛₘ) = ι(x) q, with ι = 1/scac, x = (tr−1)/2, q = spin⁻¹
    const real* M = g.rs;
    const real tr = M[0] + M[4] + M[8];
    real io[3];
    inv_scac2(0.5 * (tr - 1.0), io);
    const real q[3] = {0.5 * (M[5] - M[7]), 0.5 * (M[6] - M[2]), 0.5 * (M[1] - M[3])};
    const real uq = dot3(f.m, q);
    real Bu[3], W[9];  // Bᵀ u with B = ½(tr I − M) = ∂q/∂ω;  [u] M
    for (int i = 0; i < 3; ++i) Bu[i] = 0.5 * fma(tr, f.m[i], -dot3(M + 3 * i, f.m));
    for (int j = 0; j < 3; ++j) cross3(f.m, M + 3 * j, W + 3 * j);
    for (int i = 0; i < 3; ++i) gO[i] += fma(io[0], Bu[i], -(io[1] * uq * q[i]));
    int k = 0;
    for (int i = 0; i < 3; ++i)
      for (int j = i; j < 3; ++j, ++k) {
        const real Bij = (i == j ? tr : 0.0) - 0.5 * (M[i + 3 * j] + M[j + 3 * i]);  // 2 sym(B)
        const real w = 0.5 * (W[i + 3 * j] + W[j + 3 * i]);
        K6[k] += io[2] * uq * q[i] * q[j] - io[1] * (q[i] * Bu[j] + Bu[i] * q[j] + 0.5 * uq * Bij) +
                 0.5 * io[0] * (w - q[i] * f.m[j] - f.m[i] * q[j]);
      }
  }
  const real Km[9] = {K6[0], K6[1], K6[2], K6[1], K6[3], K6[4], K6[2], K6[4], K6[5]};
  // ---- to (p, r): ω = p + β n×r, ṅ = κ0 r − κ1 n (n·r)
  const SinFun& q = g.q;
  const real k0 = 0.5 / q.a, k1 = q.c * k0, be = q.b * k0;
  const real as = sin_as(q) / q.a;  // a_s/a
  const real k0s = -k0 * as, k1s = fma(sin_cs(q), k0, -(k1 * as)), bes = fma(sin_bs(q), k0, -(be * as));
  const real bn[3] = {be * n[0], be * n[1], be * n[2]};
  real G[3], h[3];  // G = n×gO, h: moment conjugate to r
  cross3(n, gO, G);
  const real gvn = dot3(gv, n);
  for (int i = 0; i < 3; ++i) h[i] = fma(k0, gv[i], fma(-be, G[i], -(k1 * gvn * n[i])));
  const real hn = dot3(h, n);
  // moments at the nodes: w₁ and w₂
  real G1[3], G2[3];
  {
    real gx[3], gy[3];
    for (int i = 0; i < 3; ++i) {
      gx[i] = fma(0.5, gO[i], -h[i]);
      gy[i] = fma(0.5, gO[i], h[i]);
    }
    for (int i = 0; i < 3; ++i) G1[i] = dot3(g.rd + 3 * i, gx);
    for (int i = 0; i < 3; ++i) G2[i] = fma(g.rd[i + 6], gy[2], fma(g.rd[i + 3], gy[1], g.rd[i] * gy[0]));
  }
  // Hpr = K N + C D + ½[gO]N − ½[h],  N = β[n]
  real Hpr[9], Hrr[6];
  {
    real KN[9];  // K N: row i is (row i of K) × βn
    for (int i = 0; i < 3; ++i) {
      const real ki[3] = {Km[i], Km[i + 3], Km[i + 6]};
      real x[3];
      cross3(ki, bn, x);
      for (int j = 0; j < 3; ++j) KN[i + 3 * j] = x[j];
    }
    // C n and C D = κ0 C − κ1 (C n) nᵀ
    real Cn[3], pn[3];
    cross3(ps, n, pn);
    const real tn = g.th[0];
    for (int i = 0; i < 3; ++i) Cn[i] = pn[i] + fma(f.v[i], tn, -(tV * n[i]));
    real CD[9];
    const real k0ps[3] = {k0 * ps[0], k0 * ps[1], k0 * ps[2]};
    const real sk[9] = {0.0, k0ps[2], -k0ps[1], -k0ps[2], 0.0, k0ps[0], k0ps[1], -k0ps[0], 0.0};
    for (int j = 0; j < 3; ++j)
      for (int i = 0; i < 3; ++i) {
        real v = fma(k0 * f.v[i], t[j], fma(-k1 * Cn[i], n[j], sk[i + 3 * j]));
        if (i == j) v = fma(-k0, tV, v);
        CD[i + 3 * j] = v;
      }
    // ½[gO]β[n] = ½(bn gOᵀ − (gO·bn) I)
    const real gbn = 0.5 * dot3(gO, bn);
    const real hs[9] = {0.0, h[2], -h[1], -h[2], 0.0, h[0], h[1], -h[0], 0.0};
    for (int j = 0; j < 3; ++j)
      for (int i = 0; i < 3; ++i) {
        real v = KN[i + 3 * j] + CD[i + 3 * j];
        v = fma(0.5 * bn[i], gO[j], v);
        if (i == j)
          v -= gbn;
        else
          v = fma(-0.5, hs[i + 3 * j], v);
        Hpr[i + 3 * j] = v;
      }
    // Hrr = Nᵀ K N + 2 sym(Nᵀ C D) + sym(n zᵀ) + iso·I
    real NCD[9], NKN[9];  // Nᵀ X = −bn × columns
    for (int j = 0; j < 3; ++j) {
      cross3(CD + 3 * j, bn, NCD + 3 * j);
      cross3(KN + 3 * j, bn, NKN + 3 * j);
    }
    const real z0 = fma(-k1, k0, k0s), z1 = fma(2.0 * k1, k1, -k1s) * gvn, z2 = -fma(-be, k1, bes);
    real z[3];
    for (int i = 0; i < 3; ++i) z[i] = fma(z0, gv[i], fma(z1, n[i], fma(z2, G[i], be * h[i])));
    const real iso = -fma(k0 * k1, gvn, be * hn);
    int k = 0;
    for (int i = 0; i < 3; ++i)
      for (int j = i; j < 3; ++j, ++k) {
        if (i == j)
          Hrr[k] = NKN[i + 3 * i] + fma(2.0, NCD[i + 3 * i], fma(n[i], z[i], iso));
        else
          Hrr[k] = NKN[i + 3 * j] + (NCD[i + 3 * j] + NCD[j + 3 * i]) + 0.5 * fma(n[i], z[j], n[j] * z[i]);
      }
  }
  // ---- material part and the d blocks
  const real i2L = 2.0 / c.L;
  real Hdd[6], Hdp[9], Hdr[9], Hpp[6];
  {
    // ∂(θ, w)/∂(p, r): θ_k: (col×n, g1 col + g2 θ_k n);  w_k: (col×d, (col×d)×βn)
    const real g1 = fma(-be, g.s, k0), g2 = be - k1;
    real C[3][3], gr[3][3], En[3], Eb[3], Fn[3], Fb[3];
    for (int k = 0; k < 3; ++k) {
      const real* col = g.rs + 3 * k;
      cross3(col, n, C[k]);
      const real w = g2 * g.th[k];
      for (int i = 0; i < 3; ++i) gr[k][i] = fma(g1, col[i], w * n[i]);
    }
    cross3(nn, d, En);
    cross3(bb, d, Eb);
    cross3(En, bn, Fn);
    cross3(Eb, bn, Fb);
    real unp[3], ubp[3], vbp[3], vnp[3], ctp[3], unr[3], ubr[3], vbr[3], vnr[3], ctr[3];
    for (int i = 0; i < 3; ++i) {
      unp[i] = fma(c.k3u, En[i], c.k3uv * C[2][i]);
      ubp[i] = fma(c.k3uv, En[i], c.k3v * C[2][i]);
      vbp[i] = fma(c.k2u, Eb[i], -(c.k2uv * C[1][i]));
      vnp[i] = fma(c.k2v, C[1][i], -(c.k2uv * Eb[i]));
      ctp[i] = c.kt * C[0][i];
      unr[i] = fma(c.k3u, Fn[i], c.k3uv * gr[2][i]);
      ubr[i] = fma(c.k3uv, Fn[i], c.k3v * gr[2][i]);
      vbr[i] = fma(c.k2u, Fb[i], -(c.k2uv * gr[1][i]));
      vnr[i] = fma(c.k2v, gr[1][i], -(c.k2uv * Fb[i]));
      ctr[i] = c.kt * gr[0][i];
    }
    real tA_[3], tAN[3];
    cross3(t, f.a, tA_);
    cross3(tA_, bn, tAN);
    const real Pbn = dot3(P, bn);
    const real sp[9] = {0.0, P[2], -P[1], -P[2], 0.0, P[0], P[1], -P[0], 0.0};  // [P]
    const real se = s_e * i2L * g.idn, kd = fma(c.ke * i2L, i2L, -se);
    int k = 0;
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) {
        const real wi = c.k3u * nn[i], vi = c.k2u * bb[i];
        if (j >= i) {
          real v = fma(wi, nn[j], fma(vi, bb[j], kd * g.dh[i] * g.dh[j]));
          if (i == j) v += se;
          Hdd[k] = v;
          v = fma(En[i], unp[j], fma(C[2][i], ubp[j], fma(Eb[i], vbp[j], fma(C[1][i], vnp[j], fma(C[0][i], ctp[j], K6[k])))));
          Hpp[k] = v;
          Hrr[k] = fma(Fn[i], unr[j], fma(gr[2][i], ubr[j], fma(Fb[i], vbr[j], fma(gr[1][i], vnr[j], fma(gr[0][i], ctr[j], Hrr[k])))));
          ++k;
        }
        const int m = i + 3 * j;
        Hpr[m] = fma(En[i], unr[j], fma(C[2][i], ubr[j], fma(Eb[i], vbr[j], fma(C[1][i], vnr[j], fma(C[0][i], ctr[j], Hpr[m])))));
        Hdp[m] = fma(nn[i], unp[j], fma(bb[i], vbp[j], fma(t[i], tA_[j], -sp[m])));
        real v = fma(nn[i], unr[j], fma(bb[i], vbr[j], fma(t[i], tAN[j], -(bn[i] * P[j]))));
        if (i == j) v += Pbn;
        Hdr[m] = v;
      }
  }
  // ---- to the dofs
  real X1[9], Y2[9];
  const real v1[3] = {X0[3], X0[4], X0[5]}, v2[3] = {X0[9], X0[10], X0[11]};
  {
    real T[9];
    tan_matrix(v1, q1, T);
    mul33(g.rd, T, X1);
    tan_matrix(v2, q2, T);
    mul33t(g.rd, T, Y2);
    real gx[3], gy[3];
    for (int i = 0; i < 3; ++i) {
      gx[i] = fma(0.5, gO[i], -h[i]);
      gy[i] = fma(0.5, gO[i], h[i]);
      const real Pt = 0.5 * fma(s_e * i2L, g.dh[i], P[i] + f.u[i]);
      R[i] = to_d(fma(0.5, f.o[i], -Pt));
      R[6 + i] = to_d(fma(0.5, f.o[i], Pt));
    }
    for (int i = 0; i < 3; ++i) {
      R[3 + i] = to_d(dot3(X1 + 3 * i, gx));
      R[9 + i] = to_d(dot3(Y2 + 3 * i, gy));
    }
  }
  // translations: d = ½(u₂ − u₁)
  {
    int k = 0;
    for (int i = 0; i < 3; ++i)
      for (int j = i; j < 3; ++j, ++k) {
        const real v = 0.25 * Hdd[k];
        out(i, j, v);
        out(6 + i, 6 + j, v);
        out(i, 6 + j, -v);
        if (j != i) out(j, 6 + i, -v);
      }
    real A[9], B[9];
    for (int m = 0; m < 9; ++m) A[m] = 0.5 * fma(0.5, Hdp[m], -Hdr[m]);
    mul33(A, X1, B);
    for (int j = 0; j < 3; ++j)
      for (int i = 0; i < 3; ++i) {
        out(i, 3 + j, -B[i + 3 * j]);
        out(3 + j, 6 + i, B[i + 3 * j]);
      }
    for (int m = 0; m < 9; ++m) A[m] = 0.5 * fma(0.5, Hdp[m], Hdr[m]);
    mul33(A, Y2, B);
    for (int j = 0; j < 3; ++j)
      for (int i = 0; i < 3; ++i) {
        out(i, 9 + j, -B[i + 3 * j]);
        out(6 + i, 9 + j, B[i + 3 * j]);
      }
  }
  // rotations: δᵀ XᵀHX δ and, from w = T(v)v̇, the moment's part
  // ẇ·G = v̇ᵀ(sym(v kᵀ) + c (G·v) I) v̇,  k = (2c−b) G + 2b_s G×v + 2c_s (G·v) v
  {
    real S[9], Z[9], B[9];
    int k = 0;
    real hxx[9], hyy[9], hxy[9];
    for (int i = 0; i < 3; ++i)
      for (int j = i; j < 3; ++j, ++k) {
        const real m = fma(0.25, Hpp[k], Hrr[k]), o = fma(0.25, Hpp[k], -Hrr[k]);
        const real sy = 0.5 * (Hpr[i + 3 * j] + Hpr[j + 3 * i]);
        hxx[i + 3 * j] = hxx[j + 3 * i] = m - sy;
        hyy[i + 3 * j] = hyy[j + 3 * i] = m + sy;
        const real sk = i == j ? real(0.0) : 0.5 * (Hpr[i + 3 * j] - Hpr[j + 3 * i]);
        hxy[i + 3 * j] = o + sk;
        hxy[j + 3 * i] = o - sk;
      }
    mul33(hxx, X1, S);
    mul33(hyy, Y2, Z);
    mul33(hxy, Y2, B);
    const real *va[2] = {v1, v2}, *Ga[2] = {G1, G2}, *Xa[2] = {X1, Y2}, *Sa[2] = {S, Z};
    const SinFun* qa[2] = {&q1, &q2};
    for (int a = 0; a < 2; ++a) {
      const real *v = va[a], *G_ = Ga[a];
      const SinFun& qq = *qa[a];
      const real gv_ = dot3(G_, v), cg = qq.c * gv_, kg = fma(2.0, qq.c, -qq.b), kx = 2.0 * sin_bs(qq), kv = 2.0 * sin_cs(qq) * gv_;
      real gx[3], kk[3];
      cross3(G_, v, gx);
      for (int i = 0; i < 3; ++i) kk[i] = 0.5 * fma(kg, G_[i], fma(kx, gx[i], kv * v[i]));
      for (int i = 0; i < 3; ++i)
        for (int j = i; j < 3; ++j) {
          real w = dot3(Xa[a] + 3 * i, Sa[a] + 3 * j);
          w = i == j ? fma(2.0 * v[i], kk[i], w + cg) : fma(v[i], kk[j], fma(v[j], kk[i], w));
          out(3 + 6 * a + i, 3 + 6 * a + j, w);
        }
    }
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) out(3 + i, 9 + j, dot3(X1 + 3 * i, B + 3 * j));
  }
}


// Columns of ∂m/∂v and ∂(n×t)/∂v over the six rotation dofs, m = (t·d) t
MG_HD void beam_modes(const double* X0, const SinFun& q1, const SinFun& q2, const BeamState& g, real Jm[6][3],
                      real Jw[6][3]) {
  const real *t = g.rs, *n = g.n;
  const real k0 = 0.5 / g.q.a, k1 = g.q.c * k0, be = g.q.b * k0, td = dot3(t, g.d);
  for (int a = 0; a < 2; ++a) {
    const real v[3] = {X0[3 + 6 * a], X0[4 + 6 * a], X0[5 + 6 * a]};
    real T[9], X[9];
    tan_matrix(v, a ? q2 : q1, T);
    if (a)
      mul33t(g.rd, T, X);
    else
      mul33(g.rd, T, X);
    const real sg = a ? 1.0 : -1.0;
    for (int j = 0; j < 3; ++j) {
      const real* x = X + 3 * j;
      real *jm = Jm[3 * a + j], *jw = Jw[3 * a + j], w[3] = {0.5 * x[0], 0.5 * x[1], 0.5 * x[2]}, dn[3], jt[3];
      cross3_add(sg * be, n, x, w);
      const real nx = sg * k1 * dot3(n, x);
      for (int i = 0; i < 3; ++i) dn[i] = fma(sg * k0, x[i], -(nx * n[i]));
      cross3(w, t, jt);
      const real jd = dot3(jt, g.d);
      for (int i = 0; i < 3; ++i) jm[i] = fma(t[i], jd, td * jt[i]);
      cross3(dn, t, jw);
      cross3_add(1.0, n, jt, jw);
    }
  }
}

// ∂R/∂U of loads −U per unit length at the Gauss points, H[i + 12 k]
MG_HD void beam_uload(const BeamConst& c, const double* X0, const SinFun& q1, const SinFun& q2, const BeamState& g,
                      double* H) {
  real Jm[6][3], Jw[6][3], su = 0.0, sa = 0.0, sv = 0.0;
  beam_modes(X0, q1, q2, g, Jm, Jw);
  for (int k = 0; k < 4; ++k) {
    su += c.dL[k] * c.yu[k];
    sa += c.dL[k] * (c.ya[k] - c.yu[k]);
    sv += c.dL[k] * c.yv[k];
  }
  for (int k = 0; k < 3; ++k)
    for (int j = 0; j < 3; ++j) {
      const real m = fma(sa * g.rs[k], g.rs[j], k == j ? su : real(0.0)), o = k == j ? c.S0 : 0.0;
      H[j + 12 * k] = to_d(0.5 * (m - o));
      H[6 + j + 12 * k] = to_d(-0.5 * (m + o));
      H[3 + j + 12 * k] = to_d(-fma(sa, Jm[j][k], sv * Jw[j][k]));
      H[9 + j + 12 * k] = to_d(-fma(sa, Jm[3 + j][k], sv * Jw[3 + j][k]));
    }
}

// SweepX{0}: residual and tangent, loads w and −U per unit length.  out(i, j, v)
// receives each pair i <= j of the symmetric tangent once.
template <class Out>
MG_HD void beam_static(const BeamConst& c, const double* X0, const double* U, double* R, Out&& out, double* H) {
  SinFun q1, q2;
  BeamState g;
  beam_state(c, X0, q1, q2, g);
  BeamLoads f;
  {
    real su = 0.0, sa = 0.0, sv = 0.0;
    for (int k = 0; k < 4; ++k) {
      su += c.dL[k] * c.yu[k];
      sa += c.dL[k] * (c.ya[k] - c.yu[k]);
      sv += c.dL[k] * c.yv[k];
    }
    for (int i = 0; i < 3; ++i) {
      const real q = (i == 2 ? c.w : 0.0) - (U ? U[i] : 0.0);
      f.u[i] = su * q;
      f.a[i] = sa * q;
      f.v[i] = sv * q;
      f.o[i] = c.S0 * q;
      f.m[i] = 0.0;
    }
  }
  beam_frozen<false>(c, X0, q1, q2, g, f, R, out);
  if (H) beam_uload(c, X0, q1, q2, g, H);
}

}  // namespace mgpu
