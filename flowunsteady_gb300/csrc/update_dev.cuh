// update_dev.cuh — what happens to one particle between two pair passes of a step, as
// device functions: the stretching terms, E_str, C_d, the Runge-Kutta update and the
// packed source records of the next pass.  post_kernel (update.cu) runs them over a
// field, and the reduction of a small field's partial sums (pair_kernel.cuh) runs them
// on each target right after its final values.
//
// State layout (FP64 SoA, leading dimension ld = capacity): X[k*ld+i], Γ[k*ld+i],
// σ[i]; U[k*ld+i]; J[(3a+b)*ld+i] = dU_a/dx_b; E_str[k*ld+i]; C[k*ld+i] with
// k = 0: C_d, 1: <Γ·L>, 2: <Γ·m>; RK registers Q[r*ld+i], r = 0..2 x, 3..5 Γ,
// 6 σ, 7 σ² (core spreading).
//
// Restated from FLOWUnsteady docs/src/theory/rvpm.md:
//   stretching S = (Γ·∇)u (classic) or its transpose (:363, default transposed);
//   dΓ/dt = S - 3Z Γ - C_d/ζ_σ(0) E_str,  dσ/dt = -σ Z,
//   Z = [(f+g)/(1+3f) S·Γ - f/(1+3f) C_d/ζ_σ(0) E_str·Γ]/|Γ|²          (:196-236)
//   (equivalent to Eqs. 7-8: (g+f)/(1/3+f) = 3(g+f)/(1+3f));
//   dynamic C_d = <Γ·L>/<Γ·m> with backscatter clipping                  (:264-297);
//   low-storage RK3 (Williamson 1980) and core spreading d(σ²)/dt = 2ν   (:364-367).
#pragma once

#include "update.h"
#include "vpm_device.cuh"

namespace vpm {

__device__ inline void stretch_dev(const double* J, int64_t ld, int64_t i, double v0, double v1,
                                   double v2, int transposed, double& s0, double& s1,
                                   double& s2) {
  const double j00 = J[0 * ld + i], j01 = J[1 * ld + i], j02 = J[2 * ld + i];
  const double j10 = J[3 * ld + i], j11 = J[4 * ld + i], j12 = J[5 * ld + i];
  const double j20 = J[6 * ld + i], j21 = J[7 * ld + i], j22 = J[8 * ld + i];
  if (transposed) {
    s0 = j00 * v0 + j10 * v1 + j20 * v2;
    s1 = j01 * v0 + j11 * v1 + j21 * v2;
    s2 = j02 * v0 + j12 * v1 + j22 * v2;
  } else {
    s0 = j00 * v0 + j01 * v1 + j02 * v2;
    s1 = j10 * v0 + j11 * v1 + j12 * v2;
    s2 = j20 * v0 + j21 * v1 + j22 * v2;
  }
}

// Non-finite test on the exponent bits (integer pipe; FP64 compares issue on
// the FP64 pipe, 1/64 of the FP32 rate on GB300).
__device__ inline bool finite_bits(double x) {
  return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}

// v = S(J, Γ) into rows V (the per-source term of the E_str pass).
__device__ inline void stretch_at(const double* J, const double* G, int64_t ld, int64_t i,
                                  int transposed, double* V) {
  double s0, s1, s2;
  stretch_dev(J, ld, i, G[i], G[ld + i], G[2 * ld + i], transposed, s0, s1, s2);
  V[i] = s0; V[ld + i] = s1; V[2 * ld + i] = s2;
}

// E_str = S(J_p, Ω_p) - V_p from the raw ζ sums (rows 0..2 Ω, 3..5 V).
__device__ inline void estr_at(const double* raw, const double* J, int64_t ld, int64_t i,
                               int transposed, double* E) {
  double s0, s1, s2;
  stretch_dev(J, ld, i, raw[i], raw[ld + i], raw[2 * ld + i], transposed, s0, s1, s2);
  E[i] = s0 - raw[3 * ld + i];
  E[ld + i] = s1 - raw[4 * ld + i];
  E[2 * ld + i] = s2 - raw[5 * ld + i];
}

// DE = S(DJ, Ω) + S(J, DΩ) - DV from the raw sums of the α-derivative ζ pass (rows
// 0..2 Ω, 6..8 DΩ, 9..11 DV).  For differences (fd) S(DJ, DΩ) belongs to DE too.
__device__ inline void estr_d_at(const double* raw, const double* J, const double* DJ, int64_t ld,
                                 int64_t i, int transposed, int fd, double* DE) {
  const double o0 = raw[i], o1 = raw[ld + i], o2 = raw[2 * ld + i];
  const double d0 = raw[6 * ld + i], d1 = raw[7 * ld + i], d2 = raw[8 * ld + i];
  double s0, s1, s2, t0, t1, t2;
  if (fd) stretch_dev(DJ, ld, i, o0 + d0, o1 + d1, o2 + d2, transposed, s0, s1, s2);
  else stretch_dev(DJ, ld, i, o0, o1, o2, transposed, s0, s1, s2);
  stretch_dev(J, ld, i, d0, d1, d2, transposed, t0, t1, t2);
  DE[i] = s0 + t0 - raw[9 * ld + i];
  DE[ld + i] = s1 + t1 - raw[10 * ld + i];
  DE[2 * ld + i] = s2 + t2 - raw[11 * ld + i];
}

// Pseudo-three-level dynamic coefficient (once per step, first RK stage):
//   nume = (3α-2) Γ·[S(J(ασ)) - S(J(σ))],  deno = σ³/ζ(0) Γ·[E(ασ) - E(σ)],
//   Lagrangian average with rlxf, C_d = nume/deno, |C_d| forced/limited.
__device__ inline void sfs_dynamic_at(int64_t i, int64_t ld, const double* G, const double* S,
                                      const double* J, const double* Jt, const double* E,
                                      const double* Et, double* C, const SfsParams& p) {
  const double g0 = G[i], g1 = G[ld + i], g2 = G[2 * ld + i];
  double a0, a1, a2, b0, b1, b2;
  double nume, deno;
  if (p.analytic) {
    // Jt = DJ, Et = DE: the test-filter differences are (α-1)·D to first order, or
    // (analytic = 2) Jt and Et are the differences.
    const double h = p.analytic == 2 ? 1.0 : p.alpha - 1.0;
    stretch_dev(Jt, ld, i, g0, g1, g2, p.transposed, a0, a1, a2);
    nume = h * (g0 * a0 + g1 * a1 + g2 * a2);
    deno = h * (g0 * Et[i] + g1 * Et[ld + i] + g2 * Et[2 * ld + i]);
  } else {
    stretch_dev(Jt, ld, i, g0, g1, g2, p.transposed, a0, a1, a2);
    stretch_dev(J, ld, i, g0, g1, g2, p.transposed, b0, b1, b2);
    nume = g0 * (a0 - b0) + g1 * (a1 - b1) + g2 * (a2 - b2);
    deno = g0 * (Et[i] - E[i]) + g1 * (Et[ld + i] - E[ld + i]) +
           g2 * (Et[2 * ld + i] - E[2 * ld + i]);
  }
  const double sg = S[i];
  nume *= 3.0 * p.alpha - 2.0;
  deno *= sg * sg * sg * p.inv_zeta0;
  nume = p.rlxf * nume + (1.0 - p.rlxf) * C[ld + i];
  deno = p.rlxf * deno + (1.0 - p.rlxf) * C[2 * ld + i];
  double cd = deno != 0.0 ? nume / deno : 0.0;
  if (p.force_positive) cd = fabs(cd);
  if (p.minC > 0.0 && fabs(cd) < p.minC) cd = copysign(p.minC, cd);
  if (p.maxC > 0.0 && fabs(cd) > p.maxC) cd = copysign(p.maxC, cd);
  C[i] = cd;
  C[ld + i] = nume;
  C[2 * ld + i] = deno;
}

// One RK stage (or an Euler step: a = 0, b = 1) of a free particle, fused:
// backscatter clipping, rVPM right-hand side, low-storage register update,
// state update, core spreading, non-finite detection.  FP64 throughout; the
// FP64 pipe (not HBM) bounds it, so each particle forms the right-hand side
// once, one reciprocal of |Γ|² and (with core spreading) one square root.
__device__ inline void rk_update_at(int64_t i, int64_t ld, double* X, double* G, double* S,
                                    const double* U, const double* J, const double* E, double* C,
                                    double* Q, const UpdateParams& p, int* status) {
  // Everything is read before the first store: the rows may alias for the compiler.
  const double g0 = G[i], g1 = G[ld + i], g2 = G[2 * ld + i];
  const double sg = S[i];
  double x[3], u[3], q[8];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    x[k] = X[k * ld + i];
    u[k] = U[k * ld + i];
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) q[k] = k < 7 || p.nu > 0.0 ? Q[k * ld + i] : 0.0;
  double s0, s1, s2;
  stretch_dev(J, ld, i, g0, g1, g2, p.transposed, s0, s1, s2);
  const double gg = g0 * g0 + g1 * g1 + g2 * g2;
  double Z = p.zs * (s0 * g0 + s1 * g1 + s2 * g2);
  double cz = 0.0, e0 = 0.0, e1 = 0.0, e2 = 0.0;
  if (p.sfs) {
    e0 = E[i]; e1 = E[ld + i]; e2 = E[2 * ld + i];
    double cd = C[i];
    const double ge = g0 * e0 + g1 * e1 + g2 * e2;
    if (p.clip_backscatter && cd * ge < 0.0) {
      cd = 0.0;
      C[i] = 0.0;
    }
    cz = cd * (sg * sg) * (sg * p.inv_zeta0);   // C_d/ζ_σ(0)
    Z -= p.ze * cz * ge;
  }
  Z = gg > 0.0 ? Z * (1.0 / gg) : 0.0;
  const double a = p.a, b = p.b, dt = p.dt;
  // position
  const double q0 = a * q[0] + dt * (u[0] + p.uinf0);
  const double q1 = a * q[1] + dt * (u[1] + p.uinf1);
  const double q2 = a * q[2] + dt * (u[2] + p.uinf2);
  Q[0 * ld + i] = q0; Q[1 * ld + i] = q1; Q[2 * ld + i] = q2;
  const double x0 = x[0] + b * q0, x1 = x[1] + b * q1, x2 = x[2] + b * q2;
  X[i] = x0; X[ld + i] = x1; X[2 * ld + i] = x2;
  // strength
  const double z3 = 3.0 * Z;
  const double r0 = a * q[3] + dt * (s0 - z3 * g0 - cz * e0);
  const double r1 = a * q[4] + dt * (s1 - z3 * g1 - cz * e1);
  const double r2 = a * q[5] + dt * (s2 - z3 * g2 - cz * e2);
  Q[3 * ld + i] = r0; Q[4 * ld + i] = r1; Q[5 * ld + i] = r2;
  const double n0 = g0 + b * r0, n1 = g1 + b * r1, n2 = g2 + b * r2;
  G[i] = n0; G[ld + i] = n1; G[2 * ld + i] = n2;
  // core size: stretching, then core spreading
  const double qs = a * q[6] - dt * sg * Z;
  Q[6 * ld + i] = qs;
  double ns = sg + b * qs;
  if (p.nu > 0.0) {
    const double qn = a * q[7] + dt * 2.0 * p.nu;
    Q[7 * ld + i] = qn;
    ns = sqrt(ns * ns + b * qn);
  }
  S[i] = ns;
  if (!(finite_bits(n0) && finite_bits(n1) && finite_bits(n2) && finite_bits(ns) &&
        finite_bits(x0) && finite_bits(x1) && finite_bits(x2)))
    atomicOr(status, STATUS_NONFINITE);
}

// Packed source records of the FP32 U/J passes, per source
//   (xh, yh, zh, a), (xl, yl, zl, b), (Γx, Γy, Γz, 0)
// with x ≈ xh + xl (split_f32) and (a, b) the kernel constants of σ·scale.
template <int KERNEL>
__device__ inline void uj_record_at(int64_t i, int64_t ld, const double* X, const double* G,
                                    const double* S, double scale, float4* rec) {
  float xh, xl, yh, yl, zh, zl, ka, kb;
  split_f32(X[i], xh, xl);
  split_f32(X[ld + i], yh, yl);
  split_f32(X[2 * ld + i], zh, zl);
  source_consts<KERNEL, float>(S[i] * scale, ka, kb);
  rec[3 * i] = make_float4(xh, yh, zh, ka);
  rec[3 * i + 1] = make_float4(xl, yl, zl, kb);
  rec[3 * i + 2] = make_float4(float(G[i]), float(G[ld + i]), float(G[2 * ld + i]), 0.f);
}

// Packed source records of the FP32 ζ passes, per source
//   (xh, yh, zh, a), (xl, yl, zl, b), (Γx, Γy, Γz, c), (v_q, 0) [, (w_q, 0)]
// with (a, b, c) the ζ constants of σ·scale (zeta_consts_f32) and v_q, w_q
// from the rows V, W (zero when null).  Staging these instead of the FP64
// rows keeps FP64 arithmetic (differences, the constants' divisions, and for
// Winckelmans a pow) out of the pair kernels, where every CTA would repeat it
// for every source it stages.
template <int KERNEL>
__device__ inline void zeta_record_at(int64_t i, int64_t ld, bool d, const double* X,
                                      const double* G, const double* S, const double* V,
                                      const double* W, double scale, float4* rec) {
  float xh, xl, yh, yl, zh, zl, ka, kb, kc;
  split_f32(X[i], xh, xl);
  split_f32(X[ld + i], yh, yl);
  split_f32(X[2 * ld + i], zh, zl);
  zeta_consts_f32<KERNEL>(S[i] * scale, ka, kb, kc);
  float4* r = rec + (d ? 5 : 4) * i;
  r[0] = make_float4(xh, yh, zh, ka);
  r[1] = make_float4(xl, yl, zl, kb);
  r[2] = make_float4(float(G[i]), float(G[ld + i]), float(G[2 * ld + i]), kc);
  r[3] = V ? make_float4(float(V[i]), float(V[ld + i]), float(V[2 * ld + i]), 0.f)
           : make_float4(0.f, 0.f, 0.f, 0.f);
  if (d)
    r[4] = W ? make_float4(float(W[i]), float(W[ld + i]), float(W[2 * ld + i]), 0.f)
             : make_float4(0.f, 0.f, 0.f, 0.f);
}

// The operations of p at particle i, in the order of the flags.
template <int KERNEL>
__device__ inline void post_particle(const PostArgs& p, int64_t i) {
  const int64_t ld = p.ld;
  if (p.flags & POST_STRETCH) stretch_at(p.Js, p.G, ld, i, p.transposed, p.V);
  if (p.flags & POST_STRETCH_D) stretch_at(p.Jt, p.G, ld, i, p.transposed, p.V + 3 * ld);
  if (p.flags & POST_ZETA_REC)
    zeta_record_at<KERNEL>(i, ld, p.flags & POST_STRETCH_D, p.X, p.G, p.S, p.V, p.V + 3 * ld,
                           p.rec_scale, p.rec);
  if (p.flags & POST_ESTR) estr_at(p.raw, p.Js, ld, i, p.transposed, p.Eo);
  if (p.flags & POST_ESTR_D) estr_d_at(p.raw, p.Js, p.Jt, ld, i, p.transposed, p.sfs.analytic == 2, p.Et);
  if (i < p.nv && !(p.stat && p.stat[i])) {
    if (p.flags & POST_CONSTANT) p.C[i] = p.cd;
    if (p.flags & POST_DYNAMIC) sfs_dynamic_at(i, ld, p.G, p.S, p.J, p.Jt, p.E, p.Et, p.C, p.sfs);
    if (p.flags & POST_UPDATE)
      rk_update_at(i, ld, p.X, p.G, p.S, p.U, p.J, p.E, p.C, p.Q, p.up, p.status);
  }
  if (p.flags & POST_UJ_REC) uj_record_at<KERNEL>(i, ld, p.X, p.G, p.S, p.rec_scale, p.rec);
}

}  // namespace vpm
