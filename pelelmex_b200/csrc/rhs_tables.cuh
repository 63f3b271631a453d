// rhs_tables.cuh -- the table-driven right-hand side (one thread per cell) and
// what the right-hand-side kernels of react_rhs.cu and react_gen.cu share.
#pragma once
#include "bdf_rounds.cuh"
#include "common.cuh"
#include "gen_mechs.cuh"  // mechanism-specific right-hand sides (written by the build)

namespace b200 {
using namespace rounds;

namespace {

// ------------------------------------------------------------ mechanism
// One reaction's rate of progress for the thread's cell; C, g/RT per thread
// in shared memory at [k * ss].  Every thread of the warp evaluates the SAME
// reaction j, so the table reads are broadcasts and the branches uniform.
__device__ __forceinline__ double r_progress(const DevMech& m, int j, double T, double lnT, double invT,
                                             double Ctot, double lnPRT, const double* sC, const double* sG,
                                             int ss) {
  const int R = m.R;
  const double lnA = __ldg(m.arr + j), b = __ldg(m.arr + R + j), ea = __ldg(m.arr + 2 * R + j);
  const double kinf = exp(lnA + b * lnT - ea * invT);
  const int type = __ldg(m.rtype + j);
  const int flags = __ldg(m.rflags + j);
  double M = 0.0;
  if (type != 0) {
    M = Ctot;
    const int e0 = __ldg(m.eff_ptr + j), e1 = __ldg(m.eff_ptr + j + 1);
    for (int q = e0; q < e1; ++q) M += __ldg(m.eff_m1 + q) * sC[__ldg(m.eff_sp + q) * ss];
  }
  double kf = kinf;
  if (type >= 2) {
    const double lnA0 = __ldg(m.arr_lo + j), b0 = __ldg(m.arr_lo + R + j), ea0 = __ldg(m.arr_lo + 2 * R + j);
    const double k0 = exp(lnA0 + b0 * lnT - ea0 * invT);
    const double Pr = k0 * M / kinf;
    double F = 1.0;
    if (type == 3) {
      const double a = __ldg(m.troe + j), i3 = __ldg(m.troe + R + j), i1 = __ldg(m.troe + 2 * R + j);
      const double t2 = __ldg(m.troe + 3 * R + j);
      double Fc = (1.0 - a) * exp(-T * i3) + a * exp(-T * i1);
      if (flags & 4) Fc += exp(-t2 * invT);
      const double logFc = log10(fmax(Fc, 1e-300));
      const double c = -0.4 - 0.67 * logFc, nn = 0.75 - 1.27 * logFc;
      const double u = log10(fmax(Pr, 1e-300)) + c;
      const double f1 = u / (nn - 0.14 * u);
      F = exp(kLn10 * (logFc / (1.0 + f1 * f1)));
    }
    kf = kinf * Pr / (1.0 + Pr) * F;
  }
  // slots 0..3 reactants (nu < 0), 4..7 products (nu > 0)
  double pf = 1.0, pr = 1.0, sg = 0.0;
#pragma unroll
  for (int sl = 0; sl < 8; ++sl) {
    const int k = __ldg(m.sp + sl * R + j);
    if (k >= 0) {
      const int nu = __ldg(m.nu + sl * R + j);
      const int na = nu < 0 ? -nu : nu;
      const double ck = sC[k * ss];
      double p = ck;
      for (int e = 1; e < na; ++e) p *= ck;
      if (sl < 4) pf *= p;
      else pr *= p;
      sg += nu * sG[k * ss];
    }
  }
  double kr = 0.0;
  if (flags & 2) {
    const double lr = __ldg(m.arr_rev + j), br = __ldg(m.arr_rev + R + j), er = __ldg(m.arr_rev + 2 * R + j);
    kr = exp(lr + br * lnT - er * invT);
  } else if (flags & 1) {
    kr = kf * exp(sg - __ldg(m.sdnu + j) * lnPRT);
  }
  double q = kf * pf - kr * pr;
  if (type == 1) q *= M;
  return q;
}

// The cell of the round integrator: its record.
template <int NS>
struct RecView {
  RVec<NS + 1> v;
  __device__ __forceinline__ double yev(int k) const { return v.yev(k); }
  __device__ __forceinline__ double F(int k) const { return v.F(k); }
  __device__ __forceinline__ void set_f(int k, double x) const { v.fv(k) = x; }
};

// HP right-hand side at v.yev (forcing v.F) into v.set_f, thread per cell.  sC,
// sG: scratch of stride ss; sW of stride ws, which may be where set_f writes.
template <int NS, class View, class Stride>
__device__ __forceinline__ void r_rhs(const DevMech& m, const View& v, double* sC, double* sG, int ss, double* sW,
                                      Stride ws) {
  const double T = v.yev(NS);
  const double lnT = log(T), invT = 1.0 / T;
  double Ctot = 0.0, rcp = 0.0;
#pragma unroll 1
  for (int k = 0; k < NS; ++k) {
    double cpR, hRT, sR, dcpR;
    nasa7(m, k, T, lnT, cpR, hRT, sR, dcpR);
    const double iw = __ldg(m.inv_mw + k);
    const double yk = v.yev(k);
    const double Ck = yk * iw;
    sC[k * ss] = Ck;
    sG[k * ss] = hRT - sR;
    sW[k * ws] = 0.0;
    Ctot += Ck;
    rcp += yk * cpR * kRu * iw;
  }
  const double lnPRT = log(kPatm / (kRu * T));
  const int R = m.R;
#pragma unroll 1
  for (int j = 0; j < R; ++j) {
    const double q = r_progress(m, j, T, lnT, invT, Ctot, lnPRT, sC, sG, ss);
#pragma unroll
    for (int sl = 0; sl < 8; ++sl) {
      const int k = __ldg(m.sp + sl * R + j);
      if (k >= 0) {
        sW[k * ws] += (double)__ldg(m.nu + sl * R + j) * q;
      }
    }
  }
  double hs = 0.0;
#pragma unroll 1
  for (int k = 0; k < NS; ++k) {
    double cpR, hRT, sR, dcpR;
    nasa7(m, k, T, lnT, cpR, hRT, sR, dcpR);
    const double yd = sW[k * ws] * __ldg(m.mw + k) + v.F(k);
    v.set_f(k, yd);
    hs += hRT * kRu * T * __ldg(m.inv_mw + k) * yd;
  }
  v.set_f(NS, (v.F(NS) - hs) / rcp);
}

// Right-hand side of a cell outside the generated code's temperatures (never in a
// healthy integration): the table form, out of line and in the caller's scratch,
// because an array of its own would be local memory for every thread the GPU can
// hold (1.2 GB with 53 species).
template <int NS, class View>
__device__ __noinline__ void cold_rhs(const DevMech* m, View v, double* sC, double* sG, int ss, double* sW, long long ws) {
  r_rhs<NS>(*m, v, sC, sG, ss, sW, ws);
}
// The same for a record (vectors at b) by one lane of the warp form, in its scratch
// s.  Few arguments: with those of the other the loop around the call spills (20^3
// dodecane flame: 54.8 ms in right-hand sides, 52.7 so).
template <int NS>
__device__ __noinline__ void cold_rhs_lane(const DevMech* m, double* b, double* s) {
  r_rhs<NS>(*m, RecView<NS>{{b}}, s, s + NS, 1, s + 2 * NS, 1);
}

template <int NS>
__device__ __forceinline__ bool gen_covers(double T) {
  if constexpr (NS == 9) return T >= gen::kGenTlo_synth_h2_9 && T <= gen::kGenThi_synth_h2_9;
  else if constexpr (NS == 21) return T >= gen::kGenTlo_synth_ch4_21 && T <= gen::kGenThi_synth_ch4_21;
  else return T >= gen::kGenTlo_synth_c12_53 && T <= gen::kGenThi_synth_c12_53;
}

// The cell of the rates kernels: MKS state in component-major arrays, no
// forcing, the rate of T not wanted.
template <int NS>
struct InstView {
  const double *rhoY, *T;
  double* dot;
  long long n, c;
  __device__ __forceinline__ double yev(int k) const {
    return k < NS ? rhoY[(long long)k * n + c] * 1.0e-3 : T[c];  // kg/m^3 -> g/cm^3
  }
  __device__ __forceinline__ double F(int) const { return 0.0; }
  __device__ __forceinline__ void set_f(int k, double v) const {
    if (k < NS) dot[(long long)k * n + c] = v * 1.0e3;  // g/cm^3/s -> kg/m^3/s
  }
};

}  // namespace
}  // namespace b200
