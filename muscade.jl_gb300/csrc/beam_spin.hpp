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
//    What bounds the element on GB300 is the number of FP64 instructions: a warp
//    instruction holds a sub-partition's FP64 pipe for 64 cycles.  This form needs
//    2,500 flops a beam and 11,700 with time derivatives (csrc/flopcount.cpp);
//    second-order Taylor arithmetic through every rotation matrix, which took the
//    derivative before, needed 16,200 and 44,200 (and spilled 16 KB a thread).
//    Measured: 210,000 static beams 3.70 -> 0.62 ms, 50,000 Newmark beams
//    2.84 -> 0.85 ms, and a model of one warp 350 -> 57 µs and 1,010 -> 282 µs.
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
  const real k0 = k * v[0], k1 = k * v[1], k2 = k * v[2];
  M[0] = fma(m0, v[0], diag);
  M[4] = fma(m1, v[1], diag);
  M[8] = fma(m2, v[2], diag);
  M[1] = fma(m0, v[1], k2);
  M[3] = fma(m0, v[1], -k2);
  M[2] = fma(m0, v[2], -k1);
  M[6] = fma(m0, v[2], k1);
  M[5] = fma(m1, v[2], k0);
  M[7] = fma(m1, v[2], -k0);
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
  // ε = 2|d|/L − 1 as (|2d|² − L²)/(L (2|d| + L)), the numerator from (2d − tgₘ)·(2d + tgₘ)
  // (2d − tgₘ is exact for small strains; |tgₘ|² − L² is rounding only): the
  // difference from 1 would add the rounding of the root and the quotient, EA·2⁻⁵³
  // of axial force, different at every state, which keeps the Newton iterations of
  // stiff beams from settling (5,000 beams of EA = 1e10, Σ Δx² to 1e-14: 8.4
  // iterations a step; 4.1 this way).  d keeps its own rounding, as in the
  // reference: time stepping amplifies it in the rates of the multipliers.
  const real tg[3] = {c.tgm[0], c.tgm[1], c.tgm[2]}, L = c.L;
  real l2 = fma(tg[2], tg[2], fma(tg[1], tg[1], fma(tg[0], tg[0], -(L * L))));
  for (int i = 0; i < 3; ++i) l2 = fma(fma(2.0, g.d[i], -tg[i]), fma(2.0, g.d[i], tg[i]), l2);
  g.eps = l2 / fma(L, 2.0 * dn, L * L);
  for (int k = 0; k < 3; ++k) g.th[k] = dot3(g.rs + 3 * k, g.n);
  g.wn = dot3(g.rs + 3, g.d);
  g.wb = dot3(g.rs + 6, g.d);
}

// External loads held fixed in the residual: Σ dL yᵤ f, Σ dL (yₐ−yᵤ) f,
// Σ dL yᵥ f, Σ dL f and Σ dL mₑ
struct BeamLoads {
  real u[3], a[3], v[3], o[3], m[3];
};

// x' = X₁ δv₁ and y' = Y₂ δv₂
MG_HD void beam_maps(const double* X0, const SinFun& q1, const SinFun& q2, const BeamState& g, real X1[9], real Y2[9]) {
  const real v1[3] = {X0[3], X0[4], X0[5]}, v2[3] = {X0[9], X0[10], X0[11]};
  real T[9];
  tan_matrix(v1, q1, T);
  mul33(g.rd, T, X1);
  tan_matrix(v2, q2, T);
  mul33t(g.rd, T, Y2);
}

// The residual, and the second variation with the loads held: the 9 × 9 form in
// (δd, p, r), then its dof entries through out(i, j, v), each pair i <= j of the
// symmetric matrix once.  ROT and rot: with the moment term mₑ·vₛₘ.
template <bool ROT, class Out>
MG_HD void beam_frozen(const BeamConst& c, const double* X0, const SinFun& q1, const SinFun& q2, const BeamState& g,
                       const BeamLoads& f, bool rot, const real X1[9], const real Y2[9], double* R, Out&& out) {
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
  if (ROT && rot) {  // mₑ·vₛₘ, vₛₘ = Rod⁻¹(rₛₘ) = ι(x) q, with ι = 1/scac, x = (tr−1)/2, q = spin⁻¹
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
    const real s2 = s_e * i2L, kd = fma(c.ke * i2L, i2L, -(s2 * g.idn));
    int k = 0;
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) {
        const real wi = c.k3u * nn[i], vi = c.k2u * bb[i];
        if (j >= i) {
          real v = fma(wi, nn[j], fma(vi, bb[j], kd * g.dh[i] * g.dh[j]));
          if (i == j) v = fma(s2, g.idn, v);
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
  const real v1[3] = {X0[3], X0[4], X0[5]}, v2[3] = {X0[9], X0[10], X0[11]};
  {
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
      const real gv_ = dot3(G_, v), kg = fma(2.0, qq.c, -qq.b), kx = 2.0 * sin_bs(qq), kv = 2.0 * sin_cs(qq) * gv_;
      real gx[3], kk[3];
      cross3(G_, v, gx);
      for (int i = 0; i < 3; ++i) kk[i] = 0.5 * fma(kg, G_[i], fma(kx, gx[i], kv * v[i]));
      for (int i = 0; i < 3; ++i)
        for (int j = i; j < 3; ++j) {
          real w = dot3(Xa[a] + 3 * i, Sa[a] + 3 * j);
          w = i == j ? fma(2.0 * v[i], kk[i], fma(qq.c, gv_, w)) : fma(v[i], kk[j], fma(v[j], kk[i], w));
          out(3 + 6 * a + i, 3 + 6 * a + j, w);
        }
    }
    for (int i = 0; i < 3; ++i)
      for (int j = 0; j < 3; ++j) out(3 + i, 9 + j, dot3(X1 + 3 * i, B + 3 * j));
  }
}


// Spin of rₛₘ and δn along x' = x (sg = −1) or y' = x (sg = 1)
MG_HD void beam_spin(real sg, const real n[3], real k0, real k1, real be, const real x[3], real w[3], real dn[3]) {
  for (int i = 0; i < 3; ++i) w[i] = 0.5 * x[i];
  cross3_add(sg * be, n, x, w);
  const real nx = sg * k1 * dot3(n, x);
  for (int i = 0; i < 3; ++i) dn[i] = fma(sg * k0, x[i], -(nx * n[i]));
}

// ∂R/∂U of loads −U per unit length at the Gauss points, H[i + 12 k]
MG_HD void beam_uload(const BeamConst& c, const BeamState& g, const real X1[9], const real Y2[9], double* H) {
  const real *t = g.rs, *n = g.n;
  const real k0 = 0.5 / g.q.a, k1 = g.q.c * k0, be = g.q.b * k0, td = dot3(t, g.d);
  real su = 0.0, sa = 0.0, sv = 0.0;
  for (int k = 0; k < 4; ++k) {
    su += c.dL[k] * c.yu[k];
    sa += c.dL[k] * (c.ya[k] - c.yu[k]);
    sv += c.dL[k] * c.yv[k];
  }
  for (int j = 0; j < 6; ++j) {
    real w[3], dn[3], jt[3], jw[3];
    beam_spin(j < 3 ? -1.0 : 1.0, n, k0, k1, be, j < 3 ? X1 + 3 * j : Y2 + 3 * (j - 3), w, dn);
    cross3(w, t, jt);
    cross3(dn, t, jw);
    cross3_add(1.0, n, jt, jw);
    const real jd = dot3(jt, g.d);
    for (int k = 0; k < 3; ++k)
      H[(j < 3 ? 3 + j : 6 + j) + 12 * k] = to_d(-fma(sa, fma(t[k], jd, td * jt[k]), sv * jw[k]));
  }
  for (int k = 0; k < 3; ++k)
    for (int j = 0; j < 3; ++j) {
      const real m = fma(sa * t[k], t[j], k == j ? su : real(0.0)), o = k == j ? c.S0 : 0.0;
      H[j + 12 * k] = to_d(0.5 * (m - o));
      H[6 + j + 12 * k] = to_d(-0.5 * (m + o));
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
  real X1[9], Y2[9];
  beam_maps(X0, q1, q2, g, X1, Y2);
  beam_frozen<false>(c, X0, q1, q2, g, f, false, X1, Y2, R, out);
  if (H) beam_uload(c, g, X1, Y2, H);
}

// ---- time derivatives ---------------------------------------------------------
MG_HD void axpy3(real a, const real x[3], real y[3]) {
  for (int i = 0; i < 3; ++i) y[i] = fma(a, x[i], y[i]);
}

// e_s and f_s, from the next remainders (e = 1/24 − s e', f = 1/120 − s f'):
// e_s = 2e' − f/2, f_s = (5f'−e')/2
template <int K>
MG_HD void sin_series_next(real s, real& e, real& f) {
  real ee = inv_fact(2 * K + 4), ff = inv_fact(2 * K + 5);
#pragma unroll
  for (int k = K - 2; k >= 0; --k) {
    ee = fma(-s, ee, inv_fact(2 * k + 6));
    ff = fma(-s, ff, inv_fact(2 * k + 7));
  }
  e = ee;
  f = ff;
}
MG_HD void sin_next(real s, const SinFun& q, real& es, real& fs) {
  if (s < 10.0) {
    real e1, f1;
    if (s < 1.0)
      sin_series_next<7>(s, e1, f1);
    else
      sin_series_next<14>(s, e1, f1);
    es = fma(2.0, e1, -0.5 * q.f);
    fs = 0.5 * fma(5.0, f1, -e1);
  } else {
    const real is = 1.0 / s;
    es = is * fma(0.5, q.c, -2.0 * q.e);
    fs = 0.5 * is * fma(-5.0, q.f, q.e);
  }
}

// T(v) and its first two time derivatives.  Where |v| < 1e-14 the
// reference takes sinc1 for a constant: there Rod = I + S + S²/2, whose third
// derivative is that of T with a = 1, b = c = 1/2 held.
MG_HD void tan_jets(const real v[3], const real v1[3], const real v2[3], real s, const SinFun& q, real T[9],
                    real Td[9], real Tdd[9]) {
  tan_matrix(v, q, T);
  const real s1 = 2.0 * dot3(v, v1), s2 = 2.0 * (dot3(v1, v1) + dot3(v, v2));
  real a1 = 0.0, b1 = 0.0, c1 = 0.0, a2 = 0.0, b2 = 0.0, c2 = 0.0, c0 = 0.5;
  if (!(s < 1e-28)) {
    real es, fs;
    sin_next(s, q, es, fs);
    const real as = sin_as(q), bs = sin_bs(q), cs = sin_cs(q);
    const real bss = fma(-0.5, cs, es), ass = 0.5 * (cs - bs), css = 0.5 * fma(3.0, fs, -es);
    a1 = as * s1;
    b1 = bs * s1;
    c1 = cs * s1;
    a2 = fma(ass * s1, s1, as * s2);
    b2 = fma(bss * s1, s1, bs * s2);
    c2 = fma(css * s1, s1, cs * s2);
    c0 = q.c;
  }
  for (int j = 0; j < 3; ++j)
    for (int i = 0; i < 3; ++i) {
      const real vv = v[i] * v[j], v1v = fma(v1[i], v[j], v[i] * v1[j]);
      const real vx = fma(2.0 * v1[i], v1[j], fma(v2[i], v[j], v[i] * v2[j]));
      Td[i + 3 * j] = fma(c1, vv, c0 * v1v);
      Tdd[i + 3 * j] = fma(c2, vv, fma(2.0 * c1, v1v, c0 * vx));
    }
  const int up[3] = {5, 6, 1}, dw[3] = {7, 2, 3};  // +v_k and −v_k of [v]
  for (int k = 0; k < 3; ++k) {
    Td[4 * k] += a1;
    Tdd[4 * k] += a2;
    const real x = fma(b1, v[k], q.b * v1[k]), y = fma(b2, v[k], fma(2.0 * b1, v1[k], q.b * v2[k]));
    Td[up[k]] += x;
    Td[dw[k]] -= x;
    Tdd[up[k]] += y;
    Tdd[dw[k]] -= y;
  }
}

// SweepX{2}: residual and Newton matrix p0 ∂R/∂X + p1 ∂R/∂X′ + p2 ∂R/∂X″.
// out(i, j, v) receives all 144 entries once, column by column (first the
// rotations' columns).  rdir (optional): ∂R along X′ += av, X″ += bv.
// The loads' variation Σ dL x∂X₀ᵀ δf goes through the modes of a Gauss point's
// position, x = yᵤ d + (yₐ−yᵤ) m + yᵥ w + ½(u₁+u₂), m = (t·d)t, w = n×t: per
// direction the modes' velocity and acceleration vary (∂ẋ/∂X = J̇, ∂ẍ/∂X = J̈,
// ∂ẍ/∂X′ = 2J̇ for a Jacobian J), the forces are summed over the Gauss points per
// mode, and the six rotation rows come from the two sums' moment and couple alone.
// Without drag that needs the modes' Gram sums only.
// PART splits an element over four threads that repeat its state and share the
// rest: 1 the residual and the symmetric part (out receives pairs i <= j), 2 to 4 a
// third of the columns each (out receives the loads' part alone) and of rdir's sums,
// which `sum` adds up: it returns whether this thread goes on with their total.
// 0 is the whole element on one thread.
struct BeamDirSums {
  real Vm[3], Am[3], Vw[3], Aw[3], vi;
};
template <int PART, class Out, class Sum>
MG_HD void beam_newmark_part(const BeamConst& c, const double* X0, const double* X1, const double* X2, const double* U,
                             Perturb pt, const double* av, const double* bv, double* R, Out&& out, Sum&& sum,
                             double* rdir, double* H) {
  SinFun q1, q2;
  BeamState g;
  beam_state(c, X0, q1, q2, g);
  const real *t = g.rs, *n = g.n, *d = g.d;
  const SinFun& q = g.q;
  const real k0 = 0.5 / q.a, k1 = q.c * k0, be = q.b * k0;
  // ---- nodes: maps X = Rod(±n) T of (x', y') and of the derivatives of T
  real X[2][9], Xd[2][9], Xdd[2][9];
  for (int a = 0; a < 2; ++a) {
    const int o = 3 + 6 * a;
    const real v[3] = {X0[o], X0[o + 1], X0[o + 2]}, v1[3] = {X1[o], X1[o + 1], X1[o + 2]},
               v2[3] = {X2[o], X2[o + 1], X2[o + 2]};
    real T[9], Td[9], Tdd[9];
    tan_jets(v, v1, v2, dot3(v, v), a ? q2 : q1, T, Td, Tdd);
    if (a) {
      mul33t(g.rd, T, X[1]);
      mul33t(g.rd, Td, Xd[1]);
      mul33t(g.rd, Tdd, Xdd[1]);
    } else {
      mul33(g.rd, T, X[0]);
      mul33(g.rd, Td, Xd[0]);
      mul33(g.rd, Tdd, Xdd[0]);
    }
  }
  // ---- time derivatives of n and of the spin of rₛₘ
  real n1[3], n2[3], om[3], om1[3], sp[2][3], sp1[2][3];  // ṅ, n̈, ω, ω̇, spins of Rod(±n) and their rates
  {
    real w[2][3], wd[2][3];  // w = X v̇, X v̈ + Ẋ v̇ (the frame's own turn apart)
    for (int a = 0; a < 2; ++a)
      for (int i = 0; i < 3; ++i) {
        const int o = 3 + 6 * a;
        w[a][i] = fma(X[a][i], X1[o], fma(X[a][i + 3], X1[o + 1], X[a][i + 6] * X1[o + 2]));
        wd[a][i] = fma(X[a][i], X2[o], fma(X[a][i + 3], X2[o + 1], X[a][i + 6] * X2[o + 2])) +
                   fma(Xd[a][i], X1[o], fma(Xd[a][i + 3], X1[o + 1], Xd[a][i + 6] * X1[o + 2]));
      }
    real r[3], p[3], o[3], r1[3], p1[3], o1[3], x[3];
    for (int i = 0; i < 3; ++i) {
      r[i] = w[1][i] - w[0][i];
      p[i] = 0.5 * (w[0][i] + w[1][i]);
      r1[i] = wd[1][i] - wd[0][i];
      p1[i] = 0.5 * (wd[0][i] + wd[1][i]);
    }
    cross3(n, r, x);
    for (int i = 0; i < 3; ++i) o[i] = be * x[i];
    cross3_add(1.0, p, r, r1);
    cross3_add(1.0, o, r, r1);
    cross3_add(1.0, o, p, p1);
    const real nr = dot3(n, r), as = sin_as(q) / q.a;
    const real k0d = -k0 * as * nr, k1d = fma(sin_cs(q), k0, -(k1 * as)) * nr, bed = fma(sin_bs(q), k0, -(be * as)) * nr;
    for (int i = 0; i < 3; ++i) n1[i] = fma(k0, r[i], -(k1 * nr * n[i]));
    const real nrd = dot3(n1, r) + dot3(n, r1);
    for (int i = 0; i < 3; ++i)
      n2[i] = fma(k0, r1[i], fma(k0d, r[i], -fma(fma(k1d, nr, k1 * nrd), n[i], k1 * nr * n1[i])));
    for (int i = 0; i < 3; ++i) o1[i] = bed * x[i];
    cross3_add(be, n1, r, o1);
    cross3_add(be, n, r1, o1);
    for (int i = 0; i < 3; ++i) {
      om[i] = p[i] + o[i];
      om1[i] = p1[i] + o1[i];
      sp[0][i] = fma(0.5, r[i], o[i]);
      sp[1][i] = fma(-0.5, r[i], o[i]);
      sp1[0][i] = fma(0.5, r1[i], o1[i]);
      sp1[1][i] = fma(-0.5, r1[i], o1[i]);
    }
  }
  // rates of κ0, κ1, β with n (of their second derivatives in s too)
  real k01, k11, be1, k02, k12, be2;
  {
    real es, fs;
    sin_next(g.s, q, es, fs);
    const real s1 = 2.0 * dot3(n, n1), s2 = 2.0 * (dot3(n1, n1) + dot3(n, n2));
    const real ia = 1.0 / q.a, as = sin_as(q), bs = sin_bs(q), cs = sin_cs(q);
    const real bss = fma(-0.5, cs, es), ass = 0.5 * (cs - bs), css = 0.5 * fma(3.0, fs, -es);
    // z/(2a) for z = 1, c, b: derivative (z_s/2 − as·(z/2a))/a, and again
    const real p = as * ia, k0s = -k0 * p, k1s = fma(0.5 * cs, ia, -(k1 * p)), bes = fma(0.5 * bs, ia, -(be * p));
    const real k0ss = -(2.0 * p * k0s + ass * ia * k0);
    const real k1ss = 0.5 * css * ia - (2.0 * p * k1s + ass * ia * k1);
    const real bess = 0.5 * bss * ia - (2.0 * p * bes + ass * ia * be);
    k01 = k0s * s1;
    k11 = k1s * s1;
    be1 = bes * s1;
    k02 = fma(k0ss * s1, s1, k0s * s2);
    k12 = fma(k1ss * s1, s1, k1s * s2);
    be2 = fma(bess * s1, s1, bes * s2);
  }
  // ---- modes and their rates
  real t1[3], t2[3], d1[3], d2[3], m1[3], m2[3], w1[3], w2[3];
  cross3(om, t, t1);
  cross3(om1, t, t2);
  cross3_add(1.0, om, t1, t2);
  for (int i = 0; i < 3; ++i) {
    d1[i] = 0.5 * (X1[6 + i] - X1[i]);
    d2[i] = 0.5 * (X2[6 + i] - X2[i]);
  }
  const real xi = dot3(t, d), xi1 = dot3(t1, d) + dot3(t, d1),
             xi2 = dot3(t2, d) + fma(2.0, dot3(t1, d1), dot3(t, d2));
  for (int i = 0; i < 3; ++i) {
    m1[i] = fma(xi1, t[i], xi * t1[i]);
    m2[i] = fma(xi2, t[i], fma(2.0 * xi1, t1[i], xi * t2[i]));
  }
  cross3(n1, t, w1);
  cross3_add(1.0, n, t1, w1);
  cross3(n2, t, w2);
  cross3_add(2.0, n1, t1, w2);
  cross3_add(1.0, n, t2, w2);
  const bool rot = c.iota1 != 0.0;
  const bool drag = c.Ca[0] != 0.0 || c.Ca[1] != 0.0 || c.Ca[2] != 0.0 || c.Cl[0] != 0.0 || c.Cl[1] != 0.0 ||
                    c.Cl[2] != 0.0 || c.Cq[0] != 0.0 || c.Cq[1] != 0.0 || c.Cq[2] != 0.0;
  real yd[4], cv[3], ca[3];
  for (int k = 0; k < 4; ++k) yd[k] = c.ya[k] - c.yu[k];
  for (int i = 0; i < 3; ++i) {
    cv[i] = 0.5 * (X1[i] + X1[6 + i]);
    ca[i] = 0.5 * (X2[i] + X2[6 + i]);
  }
  auto point = [&](int k, real xd[3], real xdd[3]) {  // velocity and acceleration of Gauss point k
    for (int i = 0; i < 3; ++i) {
      xd[i] = fma(c.yu[k], d1[i], fma(yd[k], m1[i], fma(c.yv[k], w1[i], cv[i])));
      xdd[i] = fma(c.yu[k], d2[i], fma(yd[k], m2[i], fma(c.yv[k], w2[i], ca[i])));
    }
  };
  // ---- loads and their sums
  const real vi = dot3(om1, t);  // vᵢ₂ of the rotational inertia: the spin acceleration about the axis
  real Ks[PART == 0 ? 78 : 1];  // the symmetric part, packed by columns: (i, j), i <= j at i + j (j + 1)/2
  if constexpr (PART <= 1) {
    BeamLoads f;
    for (int i = 0; i < 3; ++i) {
      f.u[i] = f.a[i] = f.v[i] = f.o[i] = 0.0;
      f.m[i] = rot ? c.S0 * c.iota1 * vi * t[i] : real(0.0);
    }
    for (int k = 0; k < 4; ++k) {
      real xd[3], xdd[3];
      point(k, xd, xdd);
      real fe[3];
      for (int i = 0; i < 3; ++i) fe[i] = fma(c.mu, xdd[i], (i == 2 ? c.w : 0.0) - (U ? U[i] : 0.0));
      if (drag)
        for (int i = 0; i < 3; ++i) {
          const real x1 = dot3(g.rs + 3 * i, xd), x2 = dot3(g.rs + 3 * i, xdd);
          axpy3(fma(c.Ca[i], x2, x1 * fma(c.Cq[i], fabs(x1), c.Cl[i])), g.rs + 3 * i, fe);
        }
      for (int i = 0; i < 3; ++i) {
        const real w = c.dL[k] * fe[i];
        f.u[i] = fma(c.yu[k], w, f.u[i]);
        f.a[i] = fma(yd[k], w, f.a[i]);
        f.v[i] = fma(c.yv[k], w, f.v[i]);
        f.o[i] += w;
      }
    }
    beam_frozen<true>(c, X0, q1, q2, g, f, rot, X[0], X[1], R, [&](int i, int j, real v) {
      if constexpr (PART == 0)
        Ks[i + j * (j + 1) / 2] = pt.p0 * v;
      else
        out(i, j, pt.p0 * v);
    });
    if (H) beam_uload(c, g, X[0], X[1], H);
    if constexpr (PART == 1) return;
  }
  // Dₛᵀ of vₛₘ: ∂vₛₘ = Dₛ ω, Dₛ = ι B − ι' q qᵀ, B = ½(tr I − rₛₘ)
  real io[3] = {0.0, 0.0, 0.0}, vq[3], tau[3];
  const real trs = g.rs[0] + g.rs[4] + g.rs[8];
  if (rot) inv_scac2(0.5 * (trs - 1.0), io);
  vq[0] = 0.5 * (g.rs[5] - g.rs[7]);
  vq[1] = 0.5 * (g.rs[6] - g.rs[2]);
  vq[2] = 0.5 * (g.rs[1] - g.rs[3]);
  auto DsT = [&](const real y[3], real z[3]) {
    const real qy = io[1] * dot3(vq, y);
    for (int i = 0; i < 3; ++i) z[i] = fma(0.5 * io[0], fma(trs, y[i], -dot3(g.rs + 3 * i, y)), -(qy * vq[i]));
  };
  DsT(t, tau);
  // Gram sums over (yᵤ, y_d, yᵥ, 1), with the mass
  real Guu = 0.0, Gud = 0.0, Guv = 0.0, Gu = 0.0, Gdd = 0.0, Gdv = 0.0, Gd = 0.0, Gvv = 0.0, Gv = 0.0;
  for (int k = 0; k < 4; ++k) {
    const real l = c.mu * c.dL[k], lu = l * c.yu[k], ld = l * yd[k], lv = l * c.yv[k];
    Guu = fma(lu, c.yu[k], Guu);
    Gud = fma(lu, yd[k], Gud);
    Guv = fma(lu, c.yv[k], Guv);
    Gu += lu;
    Gdd = fma(ld, yd[k], Gdd);
    Gdv = fma(ld, c.yv[k], Gdv);
    Gd += ld;
    Gvv = fma(lv, c.yv[k], Gvv);
    Gv += lv;
  }
  const real G1 = c.mu * c.S0;
  // forces of a direction with drag, from the point's velocity and acceleration
  // variation mk(k, V, A) and the spin sg of rₛₘ (nullptr: none)
  auto dragsum = [&](auto&& mk, const real* sg, real Fu[3], real Fm[3], real Fv[3], real F1[3]) {
    for (int i = 0; i < 3; ++i) Fu[i] = Fm[i] = Fv[i] = F1[i] = 0.0;
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
      real xd[3], xdd[3], V[3], A[3], df[3];
      point(k, xd, xdd);
      mk(k, V, A);
      for (int i = 0; i < 3; ++i) df[i] = c.mu * A[i];
      if (sg) {
        cross3_add(-1.0, sg, xd, V);
        cross3_add(-1.0, sg, xdd, A);
      }
      for (int i = 0; i < 3; ++i) {
        const real* col = g.rs + 3 * i;
        const real x1 = dot3(col, xd);
        real y = c.Ca[i] * dot3(col, A);
        y = fma(fma(2.0 * c.Cq[i], fabs(x1), c.Cl[i]), dot3(col, V), y);
        axpy3(y, col, df);
        if (sg) {
          const real fl = fma(c.Ca[i], dot3(col, xdd), x1 * fma(c.Cq[i], fabs(x1), c.Cl[i]));
          cross3_add(fl, sg, col, df);
        }
      }
      for (int i = 0; i < 3; ++i) {
        const real w = c.dL[k] * df[i];
        Fu[i] = fma(c.yu[k], w, Fu[i]);
        Fm[i] = fma(yd[k], w, Fm[i]);
        Fv[i] = fma(c.yv[k], w, Fv[i]);
        F1[i] += w;
      }
    }
  };
  // rows of a column from its forces per mode and its couple rho on the spin:
  // col[12], the translations' rows, and x·z of the rotations'
  auto rows = [&](const real Fu[3], const real Fm[3], const real Fv[3], const real F1[3], const real rho[3], real col[12]) {
    const real tF = dot3(t, Fm);
    real y[3], la[3], cp[3], z[3], s[3];
    for (int i = 0; i < 3; ++i) {
      const real a = fma(tF, t[i], Fu[i]);
      col[i] = 0.5 * (F1[i] - a);
      col[6 + i] = 0.5 * (F1[i] + a);
      y[i] = fma(tF, d[i], xi * Fm[i]);
      la[i] = rho[i];
    }
    cross3_add(1.0, Fv, n, y);
    cross3_add(1.0, t, y, la);
    cross3(t, Fv, cp);
    const real nc = k1 * dot3(n, cp);
    for (int i = 0; i < 3; ++i) z[i] = fma(k0, cp[i], -(nc * n[i]));
    cross3_add(be, la, n, z);
    for (int a = 0; a < 2; ++a) {
      for (int i = 0; i < 3; ++i) s[i] = fma(0.5, la[i], a ? z[i] : -z[i]);
      for (int i = 0; i < 3; ++i) col[3 + 6 * a + i] = dot3(X[a] + 3 * i, s);
    }
  };
  auto put = [&](int j, const real col[12]) {
    for (int i = 0; i < 12; ++i) {
      if constexpr (PART == 0)
        out(i, j, Ks[i <= j ? i + j * (j + 1) / 2 : j + i * (i + 1) / 2] + col[i]);
      else
        out(i, j, col[i]);
    }
  };
  BeamDirSums r{};
  const real zero[3] = {0.0, 0.0, 0.0};
  // ---- rotation columns (one thread's whole element keeps the loops: fewer spills)
#pragma unroll (PART == 0 ? 1 : 2)
  for (int a = 0; a < 2; ++a) {
    const real sg = a ? 1.0 : -1.0;
#pragma unroll (PART == 0 ? 1 : 3)
    for (int j = 0; j < 3; ++j) {
      if (PART > 1 && (3 * a + j) / 2 != PART - 2) continue;
      const real* x = X[a] + 3 * j;
      const real* y1 = Xd[a] + 3 * j;
      real x1[3], x2[3];  // ẋ, ẍ of the column: the frame turns with sp
      for (int i = 0; i < 3; ++i) {
        x1[i] = y1[i];
        x2[i] = Xdd[a][3 * j + i];
      }
      cross3_add(1.0, sp[a], x, x1);
      cross3_add(1.0, sp1[a], x, x2);
      cross3_add(1.0, sp[a], x1, x2);
      cross3_add(1.0, sp[a], y1, x2);
      // spin σ = ½x ± β n×x and δn = ±(κ0 x − κ1 n (n·x)), with their rates
      real s0[3], s1[3], s2[3], e0[3], e1[3], e2[3], z[3];
      cross3(n, x, z);
      for (int i = 0; i < 3; ++i) {
        s0[i] = fma(sg * be, z[i], 0.5 * x[i]);
        s1[i] = fma(sg * be1, z[i], 0.5 * x1[i]);
        s2[i] = fma(sg * be2, z[i], 0.5 * x2[i]);
      }
      cross3(n1, x, z);
      cross3_add(1.0, n, x1, z);  // (n×x)˙
      axpy3(sg * be, z, s1);
      axpy3(2.0 * sg * be1, z, s2);
      cross3(n2, x, z);
      cross3_add(2.0, n1, x1, z);
      cross3_add(1.0, n, x2, z);
      axpy3(sg * be, z, s2);
      const real h0 = dot3(n, x), h1 = dot3(n1, x) + dot3(n, x1),
                 h2 = dot3(n2, x) + fma(2.0, dot3(n1, x1), dot3(n, x2));
      const real p0_ = k1 * h0, p1_ = fma(k11, h0, k1 * h1), p2_ = fma(k12, h0, fma(2.0 * k11, h1, k1 * h2));
      for (int i = 0; i < 3; ++i) {
        e0[i] = sg * fma(k0, x[i], -(p0_ * n[i]));
        e1[i] = sg * (fma(k01, x[i], k0 * x1[i]) - fma(p1_, n[i], p0_ * n1[i]));
        e2[i] = sg * (fma(k02, x[i], fma(2.0 * k01, x1[i], k0 * x2[i])) - fma(p2_, n[i], fma(2.0 * p1_, n1[i], p0_ * n2[i])));
      }
      if (g.s < 1e-28) {  // Rod(n) = I + S + S²/2 there (see tan_jets)
        const real a2 = dot3(n1, n1) * (1.0 / 3.0), b2 = dot3(n1, e0) * (2.0 / 3.0);
        for (int i = 0; i < 3; ++i) s2[i] += fma(a2, e0[i], b2 * n1[i]);
      }
      // m and w: Jacobian column and its rates
      real jt[3], jt1[3], jt2[3], jm[3], jm1[3], jm2[3], jw[3], jw1[3], jw2[3];
      cross3(s0, t, jt);
      cross3(s1, t, jt1);
      cross3_add(1.0, s0, t1, jt1);
      cross3(s2, t, jt2);
      cross3_add(2.0, s1, t1, jt2);
      cross3_add(1.0, s0, t2, jt2);
      const real u0 = dot3(jt, d), u1 = dot3(jt1, d) + dot3(jt, d1),
                 u2 = dot3(jt2, d) + fma(2.0, dot3(jt1, d1), dot3(jt, d2));
      for (int i = 0; i < 3; ++i) {
        jm[i] = fma(u0, t[i], xi * jt[i]);
        jm1[i] = fma(u1, t[i], fma(u0, t1[i], fma(xi1, jt[i], xi * jt1[i])));
        jm2[i] = fma(u2, t[i], fma(2.0 * u1, t1[i], fma(u0, t2[i], fma(xi2, jt[i], fma(2.0 * xi1, jt1[i], xi * jt2[i])))));
      }
      cross3(e0, t, jw);
      cross3_add(1.0, n, jt, jw);
      cross3(e1, t, jw1);
      cross3_add(1.0, e0, t1, jw1);
      cross3_add(1.0, n1, jt, jw1);
      cross3_add(1.0, n, jt1, jw1);
      cross3(e2, t, jw2);
      cross3_add(2.0, e1, t1, jw2);
      cross3_add(1.0, e0, t2, jw2);
      cross3_add(1.0, n2, jt, jw2);
      cross3_add(2.0, n1, jt1, jw2);
      cross3_add(1.0, n, jt2, jw2);
      const real ts0 = dot3(t, s0), ts1 = fma(2.0, dot3(t, s1), dot3(t1, s0));
      if (rdir) {
        const real aj = av[3 + 6 * a + j], bj = bv[3 + 6 * a + j];
        axpy3(aj, jm, r.Vm);
        axpy3(2.0 * aj, jm1, r.Am);
        axpy3(bj, jm, r.Am);
        axpy3(aj, jw, r.Vw);
        axpy3(2.0 * aj, jw1, r.Aw);
        axpy3(bj, jw, r.Aw);
        r.vi = fma(aj, ts1, fma(bj, ts0, r.vi));
      }
      real Am[3], Aw[3], Fu[3], Fm[3], Fv[3], F1[3], rho[3] = {0.0, 0.0, 0.0}, col[12];
      for (int i = 0; i < 3; ++i) {
        Am[i] = fma(pt.p0, jm2[i], fma(2.0 * pt.p1, jm1[i], pt.p2 * jm[i]));
        Aw[i] = fma(pt.p0, jw2[i], fma(2.0 * pt.p1, jw1[i], pt.p2 * jw[i]));
      }
      if (drag) {
        real Vm[3], Vw[3];
        const real s[3] = {pt.p0 * s0[0], pt.p0 * s0[1], pt.p0 * s0[2]};
        for (int i = 0; i < 3; ++i) {
          Vm[i] = fma(pt.p0, jm1[i], pt.p1 * jm[i]);
          Vw[i] = fma(pt.p0, jw1[i], pt.p1 * jw[i]);
        }
        dragsum(
            [&](int k, real V[3], real A[3]) {
              for (int i = 0; i < 3; ++i) {
                V[i] = fma(yd[k], Vm[i], c.yv[k] * Vw[i]);
                A[i] = fma(yd[k], Am[i], c.yv[k] * Aw[i]);
              }
            },
            s, Fu, Fm, Fv, F1);
      } else {
        for (int i = 0; i < 3; ++i) {
          Fu[i] = fma(Gud, Am[i], Guv * Aw[i]);
          Fm[i] = fma(Gdd, Am[i], Gdv * Aw[i]);
          Fv[i] = fma(Gdv, Am[i], Gvv * Aw[i]);
          F1[i] = fma(Gd, Am[i], Gv * Aw[i]);
        }
      }
      if (rot) {  // δmₑ = ι₁ (δvᵢ t + vᵢ δt), δvᵢ = p0 (t·σ̈ + ṫ·σ̇) + p1 (2 t·σ̇ + ṫ·σ) + p2 t·σ
        const real dv = fma(pt.p0, dot3(t, s2) + dot3(t1, s1), fma(pt.p1, ts1, pt.p2 * ts0));
        const real sc = c.S0 * c.iota1;
        DsT(jt, z);
        for (int i = 0; i < 3; ++i) rho[i] = sc * fma(dv, tau[i], pt.p0 * vi * z[i]);
      }
      rows(Fu, Fm, Fv, F1, rho, col);
      put(3 + 6 * a + j, col);
    }
  }
  // ---- translation columns: d moves by ∓½, the midpoint by ½
#pragma unroll (PART == 0 ? 1 : 3)
  for (int j = 0; j < 3; ++j) {
    if (PART > 1 && j != PART - 2) continue;
    real Am[3], Fu[3], Fm[3], Fv[3], F1[3], c1[12], c2[12], ca_[12], cb_[12];
    for (int i = 0; i < 3; ++i) {
      const real M = t[i] * t[j], M1 = fma(t1[i], t[j], t[i] * t1[j]),
                 M2 = fma(t2[i], t[j], fma(2.0 * t1[i], t1[j], t[i] * t2[j]));
      Am[i] = fma(pt.p0, M2, fma(2.0 * pt.p1, M1, pt.p2 * M));
    }
    if (rdir) {
      const real aj = 0.5 * (av[6 + j] - av[j]), bj = 0.5 * (bv[6 + j] - bv[j]);
      for (int i = 0; i < 3; ++i) {
        r.Vm[i] = fma(aj * t[j], t[i], r.Vm[i]);
        r.Am[i] = fma(2.0 * aj, fma(t1[i], t[j], t[i] * t1[j]), fma(bj * t[j], t[i], r.Am[i]));
      }
    }
    if (drag) {
      dragsum(
          [&](int k, real V[3], real A[3]) {
            for (int i = 0; i < 3; ++i) {
              const real M = t[i] * t[j], M1 = fma(t1[i], t[j], t[i] * t1[j]);
              V[i] = yd[k] * fma(pt.p0, M1, pt.p1 * M);
              A[i] = yd[k] * Am[i];
              if (i == j) {
                V[i] = fma(c.yu[k], pt.p1, V[i]);
                A[i] = fma(c.yu[k], pt.p2, A[i]);
              }
            }
          },
          nullptr, Fu, Fm, Fv, F1);
      rows(Fu, Fm, Fv, F1, zero, c1);
      dragsum(
          [&](int, real V[3], real A[3]) {
            for (int i = 0; i < 3; ++i) {
              V[i] = i == j ? pt.p1 : 0.0;
              A[i] = i == j ? pt.p2 : 0.0;
            }
          },
          nullptr, Fu, Fm, Fv, F1);
    } else {
      for (int i = 0; i < 3; ++i) {
        const real A = i == j ? pt.p2 : 0.0;
        Fu[i] = fma(Gud, Am[i], Guu * A);
        Fm[i] = fma(Gdd, Am[i], Gud * A);
        Fv[i] = fma(Gdv, Am[i], Guv * A);
        F1[i] = fma(Gd, Am[i], Gu * A);
      }
      rows(Fu, Fm, Fv, F1, zero, c1);
      for (int i = 0; i < 3; ++i) {
        const real A = i == j ? pt.p2 : 0.0;
        Fu[i] = Gu * A;
        Fm[i] = Gd * A;
        Fv[i] = Gv * A;
        F1[i] = G1 * A;
      }
    }
    rows(Fu, Fm, Fv, F1, zero, c2);
    for (int i = 0; i < 12; ++i) {
      ca_[i] = 0.5 * (c2[i] - c1[i]);
      cb_[i] = 0.5 * (c2[i] + c1[i]);
    }
    put(j, ca_);
    put(6 + j, cb_);
  }
  // ---- the direction X′ += av, X″ += bv
  if (rdir && sum(r)) {
    real Fu[3], Fm[3], Fv[3], F1[3], col[12], rho[3], dv1[3], dv2[3], cv1[3], cv2[3];
    for (int i = 0; i < 3; ++i) {
      dv1[i] = 0.5 * (av[6 + i] - av[i]);
      dv2[i] = 0.5 * (bv[6 + i] - bv[i]);
      cv1[i] = 0.5 * (av[i] + av[6 + i]);
      cv2[i] = 0.5 * (bv[i] + bv[6 + i]);
      rho[i] = rot ? c.S0 * c.iota1 * r.vi * tau[i] : real(0.0);
    }
    if (drag) {
      dragsum(
          [&](int k, real V[3], real A[3]) {
            for (int i = 0; i < 3; ++i) {
              V[i] = fma(c.yu[k], dv1[i], fma(yd[k], r.Vm[i], fma(c.yv[k], r.Vw[i], cv1[i])));
              A[i] = fma(c.yu[k], dv2[i], fma(yd[k], r.Am[i], fma(c.yv[k], r.Aw[i], cv2[i])));
            }
          },
          nullptr, Fu, Fm, Fv, F1);
    } else {
      for (int i = 0; i < 3; ++i) {
        Fu[i] = fma(Guu, dv2[i], fma(Gud, r.Am[i], fma(Guv, r.Aw[i], Gu * cv2[i])));
        Fm[i] = fma(Gud, dv2[i], fma(Gdd, r.Am[i], fma(Gdv, r.Aw[i], Gd * cv2[i])));
        Fv[i] = fma(Guv, dv2[i], fma(Gdv, r.Am[i], fma(Gvv, r.Aw[i], Gv * cv2[i])));
        F1[i] = fma(Gu, dv2[i], fma(Gd, r.Am[i], fma(Gv, r.Aw[i], G1 * cv2[i])));
      }
    }
    rows(Fu, Fm, Fv, F1, rho, col);
    for (int i = 0; i < 12; ++i) rdir[i] = to_d(col[i]);
  }
}

template <class Out>
MG_HD void beam_newmark(const BeamConst& c, const double* X0, const double* X1, const double* X2, const double* U,
                        Perturb pt, const double* av, const double* bv, double* R, Out&& out, double* rdir, double* H) {
  beam_newmark_part<0>(c, X0, X1, X2, U, pt, av, bv, R, out, [](BeamDirSums&) { return true; }, rdir, H);
}

}  // namespace mgpu
