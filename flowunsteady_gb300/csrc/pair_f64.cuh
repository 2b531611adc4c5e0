// pair_f64.cuh — FP64 pair routines of the direct passes and of the free-vortex
// forces.
//
// GB300 retires about two FP64 operations per SM and cycle, so an FP64 pass costs
// its FP64 operations and nothing else: integer, FP32, shared-memory and branch
// instructions issue in their shadow (a warp's FP64 instruction holds the pipe 16
// cycles).  The routines therefore trade FP64 operations for table reads and
// integer tests:
//   - Gaussian-erf core functions below ρ² = 90 from the expansions of f64_tables.cuh
//     (13 FMAs for q and p together, at any ρ) instead of erf, exp, a square root and
//     two divisions (about 150 operations) or the two 14-term series;
//   - 2^x from a 2,048-entry table and a cubic (7 operations);
//   - the far-field, coincidence and range tests on the bit patterns;
//   - constants of the source staged once per tile.
// Measured on GB300 (FP64 Gaussian-erf, two rings of 7,600 particles): U/J pass
// 5.63 -> 4.19 ms, ζ pass 3.46 -> 2.00 ms; Winckelmans U/J of 4,096 particles 1.45 ->
// 1.23 ms.
#pragma once

#include "f64_tables.cuh"
#include "vpm_device.cuh"

namespace vpm {

static __device__ const CoreTable d_core_table = make_core_table();
static __device__ const Exp2Table d_exp2_table = make_exp2_table();

// Copies `n` doubles of a table to shared memory (all threads of the block; the
// caller synchronises).
__device__ __forceinline__ void stage_table(double* dst, const double* src, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
}

// Constants of a source of core σ, staged once per tile.
//   U/J  Gaussian-erf: a = 1/(2σ²), b = 1/σ³, c = 1/(3σ⁵); with the α-derivative also
//        ea = -2048 log2(e)/(2σ²), dq = √(2/π)/σ³, dp = √(2/π)/σ⁵ (Dq = -dq e^{-ρ²/2},
//        Dp = dp e^{-ρ²/2}), or, for differences to the cores ασ (fd = α > 0), the
//        constants a, b, c of ασ in ea, dq, dp;
//        Winckelmans: a = σ², b = 3/2 σ², c = 5/2 σ²; ea = -15/2 σ⁴, dq = -35/2 σ⁴
//        (Dq = ea s^{-7/2}, Dp = dq s^{-9/2}, s = r² + σ²).
//   ζ    Gaussian-erf: a = -2048 log2(e)/(2σ²), b = ζ(0)/σ³, c = 1/σ², or a of ασ;
//        Winckelmans: as zeta_consts.
template <int KERNEL, bool D>
__device__ __forceinline__ void uj_consts_f64(double sig, double& a, double& b, double& c,
                                              double& ea, double& dq, double& dp, double fd = 0.0) {
  const double s2 = sig * sig;
  if constexpr (KERNEL == VPM_KERNEL_WINCKELMANS) {
    a = s2;
    b = 1.5 * s2;
    c = 2.5 * s2;
    if constexpr (D) {
      ea = -7.5 * s2 * s2;
      dq = -17.5 * s2 * s2;
    }
  } else {
    const double i1 = 1.0 / sig, i2 = 1.0 / s2;
    a = 0.5 * i2;
    b = i2 * i1;
    c = b * i2 * (1.0 / 3.0);
    if (D && fd > 0.0) {
      const double ia = 1.0 / fd, ia2 = ia * ia;
      ea = a * ia2;
      dq = b * (ia2 * ia);
      dp = c * (ia2 * ia2 * ia);
    } else if constexpr (D) {
      ea = -0.5 * kLog2e * double(kExp2Rows) / s2;
      dq = kSqrt2overPi * b;
      dp = dq * i2;
    }
  }
}
template <int KERNEL>
__device__ __forceinline__ void zeta_consts_f64(double sig, double& a, double& b, double& c,
                                                double fd = 0.0) {
  zeta_consts<KERNEL, double>(sig, a, b);
  if constexpr (KERNEL == VPM_KERNEL_GAUSSIANERF) {
    a *= double(kExp2Rows);
    c = fd > 0.0 ? a / (fd * fd) : 1.0 / (sig * sig);
  }
}

// r² == 0, on the bit pattern.
__device__ __forceinline__ bool is_zero_f64(double r2) {
  return ((__double2hiint(r2) & 0x7fffffff) | __double2loint(r2)) == 0;
}

constexpr double kRound52 = 6755399441055744.0;      // 1.5·2^52: adding it rounds to an integer

// F_1 and F_2 at u = x/2 < 45 from the staged core table.
__device__ __forceinline__ void core_f12(double u, const double* __restrict__ tab, double& f1,
                                         double& f2) {
  const double t = fma(u, 16.0, kRound52);
  const double d = fma(t - kRound52, 0.0625, -u);
  const double* c = tab + __double2loint(t);
  double b = c[7 * kCoreRows], bd = b;
  b = fma(b, d, c[6 * kCoreRows]);
#pragma unroll
  for (int k = 5; k >= 0; --k) {
    bd = fma(bd, d, b);
    b = fma(b, d, c[k * kCoreRows]);
  }
  f1 = b;
  f2 = bd;
}

// F_1 alone.
__device__ __forceinline__ double core_f1(double u, const double* __restrict__ tab) {
  const double t = fma(u, 16.0, kRound52);
  const double d = fma(t - kRound52, 0.0625, -u);
  const double* c = tab + __double2loint(t);
  double b = c[7 * kCoreRows];
#pragma unroll
  for (int k = 6; k >= 0; --k) b = fma(b, d, c[k * kCoreRows]);
  return b;
}

// u = x/2 below kFarRho2D/2 = 45 (u >= 0; any NaN counts as far): by the high words.
__device__ __forceinline__ bool core_is_near(double u) {
  return core_near_word(unsigned(__double2hiint(u)));
}

// q = g/r³ and p/(-3), p = q'/r, of a Gaussian-erf pair; h2 = 1/(2σ²), c3 = 1/σ³,
// c5 = 1/(3σ⁵).  The pair is dropped when r² == 0.
__device__ __forceinline__ void uj_f64_gauss(double r2, double h2, double c3, double c5,
                                             const double* __restrict__ tab, double& q, double& p) {
  const double u = r2 * h2;
  if (core_is_near(u)) {
    double f1, f2;
    core_f12(u, tab, f1, f2);
    const bool self = is_zero_f64(r2);
    q = f1 * (self ? 0.0 : c3);
    p = f2 * (self ? 0.0 : c5);
  } else {   // g = 1 to FP64 rounding (see kFarRho2D)
    const double ri = rsqrt(r2);
    const double ri2 = ri * ri;
    q = ri2 * ri;
    p = q * ri2;
  }
}

// 2^(r2·a) with a2048 = 2048·a <= 0: n = the nearest integer to r2·a2048, 2^(n/2048)
// from the table and the exponent field, and 2^(f/2048), |f| <= 1/2, by a cubic whose
// d⁴ term is economised (truncation 4e-18).  r2·a2048 - n is one FMA, so the argument
// is not rounded.  0 below 2^-1100; in the subnormal range by way of 2^128 more.
__device__ __forceinline__ double exp2_f64(double r2, double a2048, const double* __restrict__ tab) {
  constexpr double kL = 0.69314718055994530942 / kExp2Rows;
  constexpr double k1 = kL, k2 = kL * kL / 2 + kL * kL * kL * kL / 96, k3 = kL * kL * kL / 6;
  const double t = fma(r2, a2048, kRound52);
  const int n = __double2loint(t);
  const double f = fma(r2, a2048, kRound52 - t);
  const double g = f * fma(fma(k3, f, k2), f, k1);
  const double s = tab[n & (kExp2Rows - 1)];
  const int ex = n >> 11;
  const bool low = ex < -1000;
  const double v = __hiloint2double(__double2hiint(s) + (low ? ex + 128 : ex) * (1 << 20),
                                    __double2loint(s));
  const double r = fma(v, g, v);
  // In range are n = 0 .. -2^31: the high word of t is that of 1.5·2^52 at n = 0 and one
  // less below it, where the low word is n itself (above 0 for n < -2^31, and 0 again,
  // with that lower high word, at n = -2^32).  A NaN is out of range: 0, as for r = 0.
  // A vote, so that the product by 2^-128 is not formed for every pair (an FP64 ring step
  // 22.2 -> 21.6 ms): all 32 lanes call this together.
  const bool in = n <= 0 && __double2hiint(t) == 0x43380000 + (n >> 31);
  if (!__any_sync(0xffffffffu, low || !in)) return r;
  if (!in || ex < -1100) return 0.0;
  return low ? r * 0x1p-128 : r;
}

// Accumulate one U/J pair: U 0..2, A 3..11, W 12..14.  (A22 is summed like the rest: as
// -(A00 + A11) it saved one operation of 40 to 50 a pair, 2 % of a pass, and carried
// the rounding of both: J22 of nearly planar fields was lost.)
__device__ __forceinline__ void accum_pair_f64(double dx, double dy, double dz, double q, double p,
                                               double gx, double gy, double gz, double* acc) {
  const double c0 = dy * gz - dz * gy, c1 = dz * gx - dx * gz, c2 = dx * gy - dy * gx;
  acc[0] = fma(q, c0, acc[0]); acc[1] = fma(q, c1, acc[1]); acc[2] = fma(q, c2, acc[2]);
  const double p0 = p * c0, p1 = p * c1, p2 = p * c2;
  acc[3] = fma(p0, dx, acc[3]); acc[4] = fma(p0, dy, acc[4]); acc[5] = fma(p0, dz, acc[5]);
  acc[6] = fma(p1, dx, acc[6]); acc[7] = fma(p1, dy, acc[7]); acc[8] = fma(p1, dz, acc[8]);
  acc[9] = fma(p2, dx, acc[9]); acc[10] = fma(p2, dy, acc[10]); acc[11] = fma(p2, dz, acc[11]);
  acc[12] = fma(q, gx, acc[12]); acc[13] = fma(q, gy, acc[13]); acc[14] = fma(q, gz, acc[14]);
}

// All three differences below 2^-537, where r² underflows to 0: the pair counts as
// coincident (Winckelmans forms r² + σ² in one chain and never r² itself).
__device__ __forceinline__ bool coincident_f64(double dx, double dy, double dz) {
  const int hx = __double2hiint(dx) & 0x7fffffff, hy = __double2hiint(dy) & 0x7fffffff,
            hz = __double2hiint(dz) & 0x7fffffff;
  return max(max(hx, hy), hz) < 0x1e600000;
}

}  // namespace vpm
