// rate_math.cuh -- the arithmetic of the generated right-hand sides and of
// their table-driven warp form.  Every operation is written with its
// rounding, so that a cell gets the same bits from both.
#pragma once
#include "mech_dev.cuh"

namespace b200 {
namespace gen {

// x := exp(x) for |x| <= 700 (no overflow or underflow handling; NaN stays
// NaN), K of them side by side: an exponential alone is a chain of 17
// dependent FP64 operations, and at 12 warps per SM four interleaved chains
// are what keeps the pipe busy.
// Argument reduction after Cody and Waite (Software Manual for the Elementary
// Functions, 1980): x = k ln2 + r with ln2 in two parts, the upper one short
// enough that k times it is exact; e^r by its Taylor polynomial of degree 13
// (|r| <= ln2 / 2: the next term is 4e-18), even and odd terms apart.
template <int K>
__device__ __forceinline__ void pexp(double (&x)[K]) {
  double r[K], e[K], o[K];
  int k[K];
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const double t = fma(x[i], 1.4426950408889634, 6755399441055744.0);  // 1.5 * 2^52: rounds to an integer
    k[i] = __double2loint(t);
    const double kd = __dsub_rn(t, 6755399441055744.0);
    r[i] = fma(kd, -0x1.62e42fefa3000p-1, x[i]);
    r[i] = fma(kd, -0x1.3de6af278ece6p-42, r[i]);
  }
#pragma unroll
  for (int i = 0; i < K; ++i) {
    const double s = __dmul_rn(r[i], r[i]);
    e[i] = 1.0 / 479001600.0;
    o[i] = 1.0 / 6227020800.0;
    e[i] = fma(e[i], s, 1.0 / 3628800.0);
    o[i] = fma(o[i], s, 1.0 / 39916800.0);
    e[i] = fma(e[i], s, 1.0 / 40320.0);
    o[i] = fma(o[i], s, 1.0 / 362880.0);
    e[i] = fma(e[i], s, 1.0 / 720.0);
    o[i] = fma(o[i], s, 1.0 / 5040.0);
    e[i] = fma(e[i], s, 1.0 / 24.0);
    o[i] = fma(o[i], s, 1.0 / 120.0);
    e[i] = fma(e[i], s, 0.5);
    o[i] = fma(o[i], s, 1.0 / 6.0);
    // 1 + (r + (r^3 o + r^2 e)): the small terms first
    const double q = fma(__dmul_rn(s, r[i]), o[i], __dmul_rn(s, e[i]));
    const double p = __dadd_rn(1.0, __dadd_rn(r[i], q));
    x[i] = __hiloint2double(__double2hiint(p) + (k[i] << 20), __double2loint(p));
  }
}

// Four exponentials as one out-of-line function: inlined at its 50 (21
// species) or 130 places it is more code than the instruction caches hold.
struct Exp4 {
  double x[4];
};
static __device__ __noinline__ Exp4 pexp4(double a, double b, double c, double d) {
  Exp4 v = {{a, b, c, d}};
  pexp(v.x);
  return v;
}
static __device__ __noinline__ double pexp1(double a) {
  double x[1] = {a};
  pexp(x);
  return x[0];
}

// Argument of an exponential that may underflow (Troe's): e^-690 stands for
// every smaller value, which only adds to terms of order one.
__device__ __forceinline__ double fexp_arg(double x) { return x < -690.0 ? -690.0 : x; }

// NASA-7 polynomials of one species: cp/R, h/RT (b1..b4 = a1/2, a2/3, a3/4,
// a4/5) and g/RT = h/RT - s/R (g1..g4 = a1/-2, a2/-6, a3/-12, a4/-20;
// oml = 1 - ln T).
__device__ __forceinline__ double nasa_cp(double a0, double a1, double a2, double a3, double a4, double T) {
  return fma(T, fma(T, fma(T, fma(T, a4, a3), a2), a1), a0);
}
__device__ __forceinline__ double nasa_h(double a0, double b1, double b2, double b3, double b4, double a5, double T,
                                         double invT) {
  return fma(a5, invT, fma(T, fma(T, fma(T, fma(T, b4, b3), b2), b1), a0));
}
__device__ __forceinline__ double nasa_g(double a0, double g1, double g2, double g3, double g4, double a5, double a6,
                                         double T, double invT, double oml) {
  const double p = fma(T, fma(T, fma(T, g4, g3), g2), g1);
  return __dsub_rn(fma(a0, oml, fma(a5, invT, __dmul_rn(T, p))), a6);
}

// Falloff rate constants from the two limits and the third-body concentration.
__device__ __forceinline__ double lindemann(double kinf, double k0, double M) {
  const double p = __dmul_rn(k0, M);
  return p / __dadd_rn(1.0, p / kinf);
}
__device__ __forceinline__ double troe(double kinf, double k0, double M, double Fc) {
  const double p = __dmul_rn(k0, M), Pr = p / kinf;
  const double lf = log10(fmax(Fc, 1e-300));
  const double u = __dadd_rn(log10(fmax(Pr, 1e-300)), fma(-0.67, lf, -0.4));
  const double f1 = u / fma(-0.14, u, fma(-1.27, lf, 0.75));
  return __dmul_rn(p / __dadd_rn(1.0, Pr), pexp1(__dmul_rn(kLn10, lf) / fma(f1, f1, 1.0)));
}

}  // namespace gen
}  // namespace b200
