// f64_tables.cuh — tables of the FP64 pair routines (pair_f64.cuh), computed at
// compile time in double-double arithmetic (Dekker's and Knuth's error-free
// transformations) and rounded once.
//
// Core functions.  With x = ρ²,
//   F_n(x) = √(2/π) ∫_0^1 t^{2n} e^{-x t²/2} dt,
//   g/ρ³ = F_1(x),   (ρg' - 3g)/ρ⁵ = -F_2(x),   F_n' = -F_{n+1}/2
// (the Boys functions of quantum chemistry up to scale; expanding them about a
// grid is Shavitt's method, Methods in Computational Physics 2 (1963)).  About
// x_i = i/8, with d = (x_i - x)/2 and |d| <= 1/32,
//   F_1 = Σ_k T_k d^k,   F_2 = dF_1/dd = Σ_k k T_k d^{k-1},   T_k = F_{1+k}(x_i)/k!.
// Entry k·kCoreRows + i is T_k of x_i, k = 0..7, with the term d^7 of F_2 economised away on |d| <= 1/32
// (Chebyshev: y^7 ≈ (112 y^5 - 56 y^3 + 7 y)/64), so F_2 has degree 6 and its
// truncation stays below 2.4e-17 of F_2.  The F_n come from their positive
// series at the highest order and the stable downward recurrence
//   (2n + 1) F_n = x F_{n+1} + √(2/π) e^{-x/2}.
//
// Exponential.  2^(i/2048), i = 0..2047, from the double-double Taylor series.
#pragma once

#ifdef __CUDACC__
#define VPM_HOST_DEVICE __host__ __device__
#else   // the tables and tests on words are plain C++ for a host compiler
#define VPM_HOST_DEVICE
#endif

namespace vpm {

struct DD {   // hi + lo
  double h, l;
};
constexpr DD dd_sum(double a, double b) {
  const double s = a + b, t = s - a;
  return DD{s, (a - (s - t)) + (b - t)};
}
constexpr DD dd_prod(double a, double b) {
  const double p = a * b;
  const double ta = 134217729.0 * a, ah = ta - (ta - a), al = a - ah;
  const double tb = 134217729.0 * b, bh = tb - (tb - b), bl = b - bh;
  return DD{p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr DD dd_add(DD a, DD b) {
  const DD s = dd_sum(a.h, b.h);
  return dd_sum(s.h, s.l + a.l + b.l);
}
constexpr DD dd_mul(DD a, DD b) {
  const DD p = dd_prod(a.h, b.h);
  return dd_sum(p.h, p.l + (a.h * b.l + a.l * b.h));
}
constexpr DD dd_div(DD a, double b) {
  const double q = a.h / b;
  const DD p = dd_prod(q, b);
  return dd_sum(q, ((a.h - p.h) - p.l + a.l) / b);
}

constexpr int kCoreRows = 721;    // x_i = 0, 1/8, .., 90
constexpr int kCoreCoef = 8;
constexpr int kExp2Rows = 2048;

// Whether u = x/2, given by its high word, is below 45, the end of the core table.  As an
// unsigned number, so that everything with a sign, a NaN's among it (CUDA's own is
// 0xfff8000000000000), is past the end: the low word of a NaN would be the index.
VPM_HOST_DEVICE constexpr bool core_near_word(unsigned hi) { return hi < 0x40468000u; }

struct CoreTable {
  double v[kCoreRows * kCoreCoef];
};
struct Exp2Table {
  double v[kExp2Rows];
};

constexpr CoreTable make_core_table() {
  CoreTable t{};
  // √(2/π) as a double-double, and e^{-1/16} by its series.
  const DD s2pi{0.79788456080286541, -4.9846544045930727e-17};
  DD step{1.0, 0.0}, term{1.0, 0.0};
  for (int k = 1; k < 22; ++k) {
    term = dd_div(term, -16.0 * k);
    step = dd_add(step, term);
  }
  DD e = s2pi;   // √(2/π) e^{-x/2}
  for (int i = 0; i < kCoreRows; ++i) {
    const double x = 0.125 * i;
    // F_9 = √(2/π) e^{-x/2} Σ_k x^k / (19·21···(19 + 2k))
    DD f[10] = {};
    DD c = dd_div(e, 19.0), s = c;
    for (int k = 1; c.h > 1e-24 * s.h; ++k) {
      c = dd_div(dd_mul(c, DD{x, 0.0}), 19.0 + 2.0 * k);
      s = dd_add(s, c);
    }
    f[9] = s;
    for (int n = 8; n >= 1; --n) f[n] = dd_div(dd_add(dd_mul(f[n + 1], DD{x, 0.0}), e), 2.0 * n + 1.0);
    // F_2 = Σ_j p_j d^j with p_j = F_{2+j}/j!; economise p_7, y = 32 d.
    DD p[8] = {};
    double fact = 1.0;
    for (int j = 0; j <= 7; ++j) {
      if (j > 1) fact *= j;
      p[j] = dd_div(f[2 + j], fact);
    }
    const double w = p[7].h / 34359738368.0;   // p_7 / 32^7: the coefficient of y^7
    p[5] = dd_add(p[5], dd_prod(w * 112.0 / 64.0, 33554432.0));
    p[3] = dd_add(p[3], dd_prod(-w * 56.0 / 64.0, 32768.0));
    p[1] = dd_add(p[1], dd_prod(w * 7.0 / 64.0, 32.0));
    t.v[i] = f[1].h;
    for (int k = 1; k < kCoreCoef; ++k) t.v[k * kCoreRows + i] = dd_div(p[k - 1], k).h;
    e = dd_mul(e, step);
  }
  return t;
}

constexpr Exp2Table make_exp2_table() {
  Exp2Table t{};
  const DD ln2{0.69314718055994529, 2.3190468138462996e-17};
  const DD u = dd_div(ln2, double(kExp2Rows));
  DD step{1.0, 0.0}, term{1.0, 0.0};   // 2^(1/2048)
  for (int k = 1; k < 10; ++k) {
    term = dd_div(dd_mul(term, u), k);
    step = dd_add(step, term);
  }
  DD v{1.0, 0.0};
  for (int i = 0; i < kExp2Rows; ++i) {
    t.v[i] = v.h;
    v = dd_mul(v, step);
  }
  return t;
}

}  // namespace vpm
