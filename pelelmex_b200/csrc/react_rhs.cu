// react_rhs.cu -- right-hand-side kernels of the round-based react path that
// work from the mechanism's tables: f(y) of every cell of a list, one thread per
// cell, and the arithmetic of the generated code (react_gen.cu) by one warp per
// cell for when few cells are left.
#include <algorithm>

#include "bdf_rounds.cuh"
#include "common.cuh"
#include "rate_math.cuh"
#include "rhs_tables.cuh"

namespace b200 {
using namespace rounds;

namespace {

// ------------------------------------------------ constant-memory table
__constant__ __align__(16) unsigned char c_mech[kConstMechBytes];

__device__ __forceinline__ const CMechHeader& cm_hdr() { return *reinterpret_cast<const CMechHeader*>(c_mech); }
__device__ __forceinline__ const double* cm_d(int off) { return reinterpret_cast<const double*>(c_mech + off); }

// NASA-7 cp/R, h/RT, g/RT of species k at T from the constant table.
__device__ __forceinline__ void cm_nasa7(const CMechHeader& H, int k, double T, double lnT, double invT,
                                        double& cpR, double& hRT, double& gRT) {
  const double* nasa = cm_d(H.off_nasa);
  const int N = H.N;
  const int base = (T < nasa[k]) ? 1 : 8;
  const double a0 = nasa[(base + 0) * N + k], a1 = nasa[(base + 1) * N + k], a2 = nasa[(base + 2) * N + k];
  const double a3 = nasa[(base + 3) * N + k], a4 = nasa[(base + 4) * N + k], a5 = nasa[(base + 5) * N + k];
  const double a6 = nasa[(base + 6) * N + k];
  cpR = a0 + T * (a1 + T * (a2 + T * (a3 + T * a4)));
  hRT = a0 + T * (a1 / 2 + T * (a2 / 3 + T * (a3 / 4 + T * a4 / 5))) + a5 * invT;
  const double sR = a0 * lnT + T * (a1 + T * (a2 / 2 + T * (a3 / 3 + T * a4 / 4))) + a6;
  gRT = hRT - sR;
}

// Rate of progress of reaction j from the constant table (same formulas as
// r_progress).
__device__ __forceinline__ double cm_progress(const CMechHeader& H, int j, double T, double lnT, double invT,
                                              double Ctot, double lnPRT, const double* sC, const double* sG,
                                              int ss) {
  const RxnC& r = reinterpret_cast<const RxnC*>(c_mech + H.off_rxn)[j];
  const int type = r.type, flags = r.flags;
  const double kinf = exp(r.lnA + r.b * lnT - r.ea * invT);
  double M = 0.0;
  if (type != 0) {
    M = Ctot;
    const short* esp = reinterpret_cast<const short*>(c_mech + H.off_effsp);
    const double* em1 = cm_d(H.off_effm1);
    for (int q = r.e0; q < r.e1; ++q) M += em1[q] * sC[esp[q] * ss];
  }
  double kf = kinf;
  if (type >= 2) {
    const double k0 = exp(r.lnA0 + r.b0 * lnT - r.ea0 * invT);
    const double Pr = k0 * M / kinf;
    double F = 1.0;
    if (type == 3) {
      double Fc = (1.0 - r.ta) * exp(-T * r.t3i) + r.ta * exp(-T * r.t1i);
      if (flags & 4) Fc += exp(-r.t2 * invT);
      const double logFc = log10(fmax(Fc, 1e-300));
      const double c = -0.4 - 0.67 * logFc, nn = 0.75 - 1.27 * logFc;
      const double u = log10(fmax(Pr, 1e-300)) + c;
      const double f1 = u / (nn - 0.14 * u);
      F = exp(kLn10 * (logFc / (1.0 + f1 * f1)));
    }
    kf = kinf * Pr / (1.0 + Pr) * F;
  }
  double pf = 1.0, pr = 1.0, sg = 0.0;
#pragma unroll
  for (int sl = 0; sl < 8; ++sl) {
    const int k = r.sp[sl];
    if (k >= 0) {
      const int nu = r.nu[sl];
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
  if (flags & 2) kr = exp(r.lr + r.br * lnT - r.er * invT);
  else if (flags & 1) kr = kf * exp(sg - r.sdnu * lnPRT);
  double q = kf * pf - kr * pr;
  if (type == 1) q *= M;
  return q;
}

// HP right-hand side from the constant table (thread per cell).
template <int NS>
__device__ __forceinline__ void cm_rhs(const RVec<NS + 1>& v, double* sC, double* sG, double* sW, int ss) {
  const CMechHeader& H = cm_hdr();
  const double* imw = cm_d(H.off_imw);
  const double* mw = cm_d(H.off_mw);
  const double T = v.yev(NS);
  const double lnT = log(T), invT = 1.0 / T;
  double Ctot = 0.0, rcp = 0.0;
#pragma unroll 1
  for (int k = 0; k < NS; ++k) {
    double cpR, hRT, gRT;
    cm_nasa7(H, k, T, lnT, invT, cpR, hRT, gRT);
    const double yk = v.yev(k);
    const double Ck = yk * imw[k];
    sC[k * ss] = Ck;
    sG[k * ss] = gRT;
    sW[k * ss] = 0.0;
    Ctot += Ck;
    rcp += yk * cpR * kRu * imw[k];
  }
  const double lnPRT = log(kPatm / (kRu * T));
  const int R = H.R;
  const RxnC* rx = reinterpret_cast<const RxnC*>(c_mech + H.off_rxn);
#pragma unroll 1
  for (int j = 0; j < R; ++j) {
    const double q = cm_progress(H, j, T, lnT, invT, Ctot, lnPRT, sC, sG, ss);
#pragma unroll
    for (int sl = 0; sl < 8; ++sl) {
      const int k = rx[j].sp[sl];
      if (k >= 0) sW[k * ss] += (double)rx[j].nu[sl] * q;
    }
  }
  double hs = 0.0;
#pragma unroll 1
  for (int k = 0; k < NS; ++k) {
    double cpR, hRT, gRT;
    cm_nasa7(H, k, T, lnT, invT, cpR, hRT, gRT);
    const double yd = sW[k * ss] * mw[k] + v.F(k);
    v.fv(k) = yd;
    hs += hRT * kRu * T * imw[k] * yd;
  }
  v.fv(NS) = (v.F(NS) - hs) / rcp;
}

// Shared memory of one cell of the warp form, in doubles.
template <int NS>
constexpr int rhs_warp_doubles(int R) { return 5 * NS + R; }

// The generated right-hand side's arithmetic (mechgen.generate), one warp per
// cell from the tables: lane per species, then per reaction, then per species;
// sums over species run in species order on every lane, as the generated code
// adds them.  s: rhs_warp_doubles of the warp's shared memory.
template <int NS, class View>
__device__ __forceinline__ void rhs_warp(const DevMech& m, const View& v, double* s, int lane) {
  using namespace gen;
  const int R = m.R;
  double *sC = s, *sE = s + NS, *sI = s + 2 * NS, *sP = s + 3 * NS, *sH = s + 4 * NS, *sq = s + 5 * NS;
  const double T = v.yev(NS);
  const double lnT = log(T), invT = 1.0 / T;
  const double u = __dmul_rn(T, kRu / kPatm), iu = 1.0 / u;
  const double oml = 1.0 - lnT;
  for (int k = lane; k < NS; k += 32) {
    double a[7];
    const int base = (T < __ldg(m.nasa + k)) ? 1 : 8;
#pragma unroll
    for (int i = 0; i < 7; ++i) a[i] = __ldg(m.nasa + (base + i) * NS + k);
    double x[2];
    x[0] = nasa_g(a[0], a[1] / -2.0, a[2] / -6.0, a[3] / -12.0, a[4] / -20.0, a[5], a[6], T, invT, oml);
    x[1] = -x[0];
    pexp(x);
    sE[k] = x[0];
    sI[k] = x[1];
    sC[k] = __dmul_rn(v.yev(k), __ldg(m.inv_mw + k));
    sP[k] = nasa_cp(a[0], a[1], a[2], a[3], a[4], T);
    sH[k] = __dmul_rn(nasa_h(a[0], a[1] / 2.0, a[2] / 3.0, a[3] / 4.0, a[4] / 5.0, a[5], T, invT), kRu / __ldg(m.mw + k));
  }
  __syncwarp();
  double Ctot = 0.0, rcp = 0.0;
#pragma unroll 9
  for (int k = 0; k < NS; ++k) {
    Ctot = __dadd_rn(Ctot, sC[k]);
    rcp = fma(sC[k], sP[k], rcp);
  }
  for (int j = lane; j < R; j += 32) {
    // a reaction's table entries all at once: one memory latency, not one per slot
    const int type = __ldg(m.rtype + j), flags = __ldg(m.rflags + j);
    int sp[8], nu[8];
#pragma unroll
    for (int sl = 0; sl < 8; ++sl) {
      sp[sl] = __ldg(m.sp + sl * R + j);
      nu[sl] = __ldg(m.nu + sl * R + j);
    }
    auto arrh = [&](const double* p) {
      return fma(-__ldg(p + 2 * R + j), invT, fma(__ldg(p + R + j), lnT, __ldg(p + j)));
    };
    double kf[1] = {arrh(m.arr)};
    const int e0 = __ldg(m.eff_ptr + j), e1 = __ldg(m.eff_ptr + j + 1);
    pexp(kf);
    double M = 0.0;
    if (type != 0) {
      M = Ctot;
      for (int q = e0; q < e1; q += 4) {
        double em[4], c[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          em[t] = q + t < e1 ? __ldg(m.eff_m1 + q + t) : 0.0;
          c[t] = q + t < e1 ? sC[__ldg(m.eff_sp + q + t)] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) M = fma(em[t], c[t], M);  // a padded term adds nothing
      }
    }
    if (type >= 2) {
      double k0[1] = {arrh(m.arr_lo)};
      pexp(k0);
      if (type == 3) {
        const double al = __ldg(m.troe + j);
        double e[3] = {fexp_arg(__dmul_rn(-T, __ldg(m.troe + R + j))), fexp_arg(__dmul_rn(-T, __ldg(m.troe + 2 * R + j))),
                       (flags & 4) ? fexp_arg(__dmul_rn(-__ldg(m.troe + 3 * R + j), invT)) : 0.0};
        pexp(e);
        double Fc = fma(__dsub_rn(1.0, al), e[0], __dmul_rn(al, e[1]));
        if (flags & 4) Fc = __dadd_rn(Fc, e[2]);
        kf[0] = troe(kf[0], k0[0], M, Fc);
      } else {
        kf[0] = lindemann(kf[0], k0[0], M);
      }
    }
    // slots 0..3 reactants (nu < 0), 4..7 products (nu > 0)
    double pf = 1.0, pr = 1.0, fac = 1.0;
#pragma unroll
    for (int sl = 4; sl < 8; ++sl) {
      if (sp[sl] < 0) continue;
      const double c = sC[sp[sl]], x = sE[sp[sl]];
      for (int e = nu[sl]; e > 0; --e) {
        pr = __dmul_rn(pr, c);
        fac = __dmul_rn(fac, x);
      }
    }
#pragma unroll
    for (int sl = 0; sl < 4; ++sl) {
      if (sp[sl] < 0) continue;
      const double c = sC[sp[sl]], x = sI[sp[sl]];
      for (int e = -nu[sl]; e > 0; --e) {
        pf = __dmul_rn(pf, c);
        fac = __dmul_rn(fac, x);
      }
    }
    double q;
    if (flags & 2) {
      double kr[1] = {arrh(m.arr_rev)};
      pexp(kr);
      q = __dsub_rn(__dmul_rn(kf[0], pf), __dmul_rn(kr[0], pr));
    } else if (flags & 1) {
      int sd = (int)__ldg(m.sdnu + j);
      for (; sd > 0; --sd) fac = __dmul_rn(fac, u);
      for (; sd < 0; ++sd) fac = __dmul_rn(fac, iu);
      q = __dmul_rn(kf[0], fma(-fac, pr, pf));
    } else {
      q = __dmul_rn(kf[0], pf);
    }
    if (type == 1) q = __dmul_rn(q, M);
    sq[j] = q;
  }
  __syncwarp();
  for (int k = lane; k < NS; k += 32) {
    double w = 0.0;
    const int p0 = __ldg(m.inc_ptr + k), p1 = __ldg(m.inc_ptr + k + 1);
    for (int p = p0; p < p1; p += 8) {
      double a[8], q[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        a[t] = p + t < p1 ? __ldg(m.inc_nu + p + t) : 0.0;
        q[t] = p + t < p1 ? sq[__ldg(m.inc_rxn + p + t)] : 0.0;
      }
#pragma unroll
      for (int t = 0; t < 8; ++t) w = fma(a[t], q[t], w);
    }
    const double yd = fma(w, __ldg(m.mw + k), v.F(k));
    v.set_f(k, yd);
    sP[k] = yd;
  }
  __syncwarp();
  double hs = 0.0;
#pragma unroll 9
  for (int k = 0; k < NS; ++k) hs = fma(sH[k], sP[k], hs);
  if (lane == 0) v.set_f(NS, fma(-T, hs, v.F(NS)) / __dmul_rn(kRu, rcp));
  __syncwarp();  // the scratch is free again
}

// Right-hand sides from the mechanism's tables (constant bank or global), one
// thread per cell.
template <int NS>
__global__ void __launch_bounds__(kRoundsRhsBlock, 6) rk_rhs(RoundsParams R) {
  constexpr int n = NS + 1;
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ DevMech s_mech;
  if (threadIdx.x == 0) s_mech = R.P.mech;
  __syncthreads();
  const int cnt = *R.cnt_in;
  // counters of the lists this round's later kernels append to
  if (blockIdx.x == 0 && threadIdx.x < kRoundLists) R.cnt_next[threadIdx.x] = 0;
  double* sC = reinterpret_cast<double*>(dsm) + threadIdx.x;
  double* sG = sC + NS * blockDim.x;
  double* sW = sG + NS * blockDim.x;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < cnt; idx += gridDim.x * blockDim.x) {
    const int slot = R.list_in[idx] & ~kSetupFlag;
    const RVec<n> v{reinterpret_cast<double*>(rec_of(R.S, slot) + R.S.L.off_vec)};
    if (R.const_mech) cm_rhs<NS>(v, sC, sG, sW, blockDim.x);
    else r_rhs<NS>(s_mech, RecView<NS>{v}, sC, sG, (int)blockDim.x, sW, (int)blockDim.x);
  }
}

// Generated right-hand sides for few live cells, one warp per cell.  A thread
// takes 60 us (21 species) to 200 us (53) for a cell however few there are, mostly
// waiting for its code; the warp form, a few loops over the tables, 15 to 43.  It
// is bound by the latency of the table reads, so a reaction's entries are read
// together (53 species: 57 us a launch with one read after the other).
constexpr int kRhsWarpBlock = 128;
template <int NS>
__global__ void __launch_bounds__(kRhsWarpBlock, 8) rk_rhs_warp(RoundsParams R) {
  constexpr int n = NS + 1;
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ DevMech s_mech;
  if (threadIdx.x == 0) s_mech = R.P.mech;
  __syncthreads();
  const int cnt = *R.cnt_in;
  if (blockIdx.x == 0 && threadIdx.x < kRoundLists) R.cnt_next[threadIdx.x] = 0;
  const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
  double* sw = reinterpret_cast<double*>(dsm) + (threadIdx.x >> 5) * rhs_warp_doubles<NS>(s_mech.R);
  for (int idx = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; idx < cnt; idx += nw) {
    const int slot = R.list_in[idx] & ~kSetupFlag;
    const RVec<n> v{reinterpret_cast<double*>(rec_of(R.S, slot) + R.S.L.off_vec)};
    if (gen_covers<NS>(v.yev(NS))) {
      rhs_warp<NS>(s_mech, RecView<NS>{v}, sw, lane);
    } else {
      if (lane == 0) cold_rhs_lane<NS>(&s_mech, v.b, sw);
      __syncwarp();
    }
  }
}

// T from (h, Y) by Newton on h(T) = sum Y_k h_k(T) from the given T, one
// thread per cell (MKS, component-major; getTfromHY of the C ABI).
template <int NS>
__global__ void __launch_bounds__(128) rk_t_from_hy(DevMech m, const double* __restrict__ rhoY,
                                                    const double* __restrict__ rhoH, double* __restrict__ T,
                                                    long long ncells) {
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < ncells;
       c += (long long)gridDim.x * blockDim.x) {
    double w[NS];
#pragma unroll
    for (int k = 0; k < NS; ++k) w[k] = rhoY[(long long)k * ncells + c] * __ldg(m.inv_mw + k);
    const double h = rhoH[c] * (1.0e4 / kRu);  // J/m^3 -> erg/g kg/m^3, over Ru
    double t = T[c];
    for (int it = 0; it < 100; ++it) {
      const double invT = 1.0 / t;
      double hs = 0.0, cs = 0.0;
#pragma unroll
      for (int k = 0; k < NS; ++k) {
        const double* a = m.nasa + (t < __ldg(m.nasa + k) ? 1 : 8) * NS + k;
        const double a0 = __ldg(a), a1 = __ldg(a + NS), a2 = __ldg(a + 2 * NS), a3 = __ldg(a + 3 * NS),
                     a4 = __ldg(a + 4 * NS);
        cs += w[k] * (a0 + t * (a1 + t * (a2 + t * (a3 + t * a4))));
        hs += w[k] * (a0 + t * (a1 * 0.5 + t * (a2 * (1.0 / 3.0) + t * (a3 * 0.25 + t * (a4 * 0.2)))) +
                      __ldg(a + 5 * NS) * invT);
      }
      const double dT = (h - hs * t) / cs;
      t += dT;
      // a cell without mass (a covered one, say) has no temperature: its infinite
      // step is not a converged one, and the next is NaN, which ends the loop
      if (!(fabs(dT) >= 1e-12 * t)) break;
    }
    T[c] = t;
  }
}

// The same by a warp, lane per species; sums run in species order on every lane,
// as the thread form adds them.  s: 3 NS doubles of the warp's shared memory.
template <int NS>
__device__ __forceinline__ double t_warp(const DevMech& m, const InstView<NS>& v, const double* rhoH, double* s, int lane) {
  double *sw = s, *sc = s + NS, *sh = s + 2 * NS;
  for (int k = lane; k < NS; k += 32) sw[k] = v.rhoY[(long long)k * v.n + v.c] * __ldg(m.inv_mw + k);
  const double h = rhoH[v.c] * (1.0e4 / kRu);
  double t = v.T[v.c];
  for (int it = 0; it < 100; ++it) {
    const double invT = 1.0 / t;
    for (int k = lane; k < NS; k += 32) {
      const double* a = m.nasa + (t < __ldg(m.nasa + k) ? 1 : 8) * NS + k;
      const double a0 = __ldg(a), a1 = __ldg(a + NS), a2 = __ldg(a + 2 * NS), a3 = __ldg(a + 3 * NS),
                   a4 = __ldg(a + 4 * NS);
      sc[k] = a0 + t * (a1 + t * (a2 + t * (a3 + t * a4)));
      sh[k] = a0 + t * (a1 * 0.5 + t * (a2 * (1.0 / 3.0) + t * (a3 * 0.25 + t * (a4 * 0.2)))) + __ldg(a + 5 * NS) * invT;
    }
    __syncwarp();
    double hs = 0.0, cs = 0.0;
#pragma unroll 9
    for (int k = 0; k < NS; ++k) {
      cs += sw[k] * sc[k];
      hs += sw[k] * sh[k];
    }
    __syncwarp();
    const double dT = (h - hs * t) / cs;
    t += dT;
    if (!(fabs(dT) >= 1e-12 * t)) break;
  }
  return t;
}

// InstView of the warp form, which has its T at hand.
template <int NS>
struct InstViewT : InstView<NS> {
  double t;
  __device__ __forceinline__ double yev(int k) const { return k < NS ? InstView<NS>::yev(k) : t; }
};

// Mass production rates at (rhoY, T) with the generated right-hand side
// (reactionRateRhoY of the C ABI): one thread per cell, and for few cells one
// warp per cell with the same bits, which solves for T first when rhoH is given.
// dot = nullptr: T only.
template <int NS>
__global__ void __launch_bounds__(kRhsWarpBlock, 8) rk_rates_warp(DevMech m, InstView<NS> view, const double* rhoH, double* T) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ DevMech s_mech;
  if (threadIdx.x == 0) s_mech = m;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  double* sw = reinterpret_cast<double*>(dsm) + (threadIdx.x >> 5) * rhs_warp_doubles<NS>(s_mech.R);
  InstViewT<NS> v{view, 0.0};
  for (v.c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v.c < v.n; v.c += (gridDim.x * blockDim.x) >> 5) {
    if (rhoH) {
      v.t = t_warp<NS>(s_mech, v, rhoH, sw, lane);
      if (lane == 0) T[v.c] = v.t;
    } else {
      v.t = v.T[v.c];
    }
    if (!v.dot) continue;
    if (gen_covers<NS>(v.t)) {
      rhs_warp<NS>(s_mech, v, sw, lane);
    } else {
      if (lane == 0) cold_rhs<NS>(&s_mech, v, sw, sw + NS, 1, sw + 2 * NS, 1);
      __syncwarp();
    }
  }
}

// Dynamic shared memory of a CTA: the columns of the table forms; the warp
// form's scratch.
template <int NS>
int rhs_smem() { return 3 * NS * kRoundsRhsBlock * (int)sizeof(double); }
template <int NS>
int rhs_warp_smem(int R) { return kRhsWarpBlock / 32 * rhs_warp_doubles<NS>(R) * (int)sizeof(double); }

// Most cells for which the warp form is used, in cells per warp of a grid that
// fills the GPU (4736 warps).  2 for the smaller mechanisms: 32^3 H2 spends
// 1.37 ms in right-hand sides with it, 1.64 with 4 and 3.6 with 8; 61x43x37 CH4
// 12.7 and 12.9 ms with 2 and 4.  8 for 53 species, whose thread form spills: six
// boxes of 571,824 cells take 18 ms (26 with one that took the thread form from
// 3500 cells on).
constexpr int rhs_warp_waves(int NS) { return NS <= 32 ? 2 : 8; }

template <int NS>
cudaError_t rhs_grid_t(int sm_count, int R, int gen, RhsGrid* G) {
  cudaError_t e = cudaFuncSetAttribute(rk_rhs<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, rhs_smem<NS>());
  if (e != cudaSuccess) return e;
  int b = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, rk_rhs<NS>, kRoundsRhsBlock, rhs_smem<NS>());
  G->thread = std::max(1, b) * sm_count;
  if (e == cudaSuccess && gen) e = gen_rhs_grid(NS, sm_count, &G->thread);
  G->warp = G->warp_cells = 0;
  if (e != cudaSuccess || !gen) return e;
  const int smem = rhs_warp_smem<NS>(R);
  if ((e = cudaFuncSetAttribute(rk_rhs_warp<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess)
    return e;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, rk_rhs_warp<NS>, kRhsWarpBlock, smem);
  G->warp = std::max(1, b) * sm_count;
  G->warp_cells = rhs_warp_waves(NS) * G->warp * (kRhsWarpBlock / 32);
  return e;
}

template <int NS>
cudaError_t rhs_launch_t(const RoundsParams& R, int grid, int by_warp, cudaStream_t st) {
  if (by_warp) rk_rhs_warp<NS><<<grid, kRhsWarpBlock, rhs_warp_smem<NS>(R.P.mech.R), st>>>(R);
  else if (R.gen_mech) return gen_rhs_launch(NS, R, grid, st);
  else rk_rhs<NS><<<grid, kRoundsRhsBlock, rhs_smem<NS>(), st>>>(R);
  return cudaGetLastError();
}

// Most cells whose T and rates one launch takes, a warp per cell: about a wave of
// the GPU's 4736 warps for the smaller mechanisms, half of one for 53 species.  A
// call (T and rates, host included) takes 16 / 19 / 37 us at 512 cells of 9 / 21 /
// 53 species, 20 / 29 / 50 with T by thread in a launch of its own; 20 / 29 against
// 23 / 35 at 4096 cells of 9 and 21, where T alone of 9000 cells of 21 species
// already takes 21 against 15; 46 against 56 at 2048 of 53, 64 and 66 at 4096.
constexpr int inst_warp_cells(int NS) { return NS <= 32 ? 4096 : 2048; }

template <int NS>
cudaError_t inst_launch_t(const DevMech& m, const double* rhoY, const double* rhoH, double* T, double* dot,
                          long long ncells, int sm_count, cudaStream_t st) {
  const InstView<NS> v{rhoY, T, dot, ncells, 0};
  const int smem = rhs_warp_smem<NS>(m.R), per = kRhsWarpBlock / 32;
  cudaError_t e = cudaFuncSetAttribute(rk_rates_warp<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  if (ncells <= inst_warp_cells(NS)) {
    rk_rates_warp<NS><<<(int)((ncells + per - 1) / per), kRhsWarpBlock, smem, st>>>(m, v, rhoH, T);
    return cudaGetLastError();
  }
  const long long need = (ncells + 127) / 128;
  rk_t_from_hy<NS><<<(int)std::min<long long>(need, 8LL * sm_count), 128, 0, st>>>(m, rhoY, rhoH, T, ncells);
  e = cudaGetLastError();
  if (e != cudaSuccess || dot == nullptr) return e;
  RhsGrid G;
  if ((e = rhs_grid_t<NS>(sm_count, m.R, 1, &G)) != cudaSuccess) return e;
  if (ncells > G.warp_cells) return gen_rates_launch(NS, m, rhoY, T, dot, ncells, G.thread, st);
  rk_rates_warp<NS><<<(int)std::min<long long>((ncells + per - 1) / per, G.warp), kRhsWarpBlock, smem, st>>>(m, v, nullptr, T);
  return cudaGetLastError();
}

}  // namespace

cudaError_t inst_launch_gen(const DevMech& m, const double* rhoY, const double* rhoH, double* T, double* dot,
                            long long ncells, int sm_count, cudaStream_t st) {
  return m.N == 9 ? inst_launch_t<9>(m, rhoY, rhoH, T, dot, ncells, sm_count, st)
         : m.N == 21 ? inst_launch_t<21>(m, rhoY, rhoH, T, dot, ncells, sm_count, st)
         : m.N == 53 ? inst_launch_t<53>(m, rhoY, rhoH, T, dot, ncells, sm_count, st)
                     : cudaErrorInvalidValue;
}

cudaError_t rounds_upload_const(const void* blob, int bytes, cudaStream_t st) {
  if (bytes > kConstMechBytes) return cudaErrorInvalidValue;
  return cudaMemcpyToSymbolAsync(c_mech, blob, (size_t)bytes, 0, cudaMemcpyHostToDevice, st);
}

cudaError_t rhs_grid(int N, int R, int gen, int sm_count, RhsGrid* G) {
  return N == 9 ? rhs_grid_t<9>(sm_count, R, gen, G)
         : N == 21 ? rhs_grid_t<21>(sm_count, R, gen, G)
         : N == 53 ? rhs_grid_t<53>(sm_count, R, gen, G)
                   : cudaErrorInvalidValue;
}

cudaError_t rhs_launch(int N, const RoundsParams& R, int grid, int by_warp, cudaStream_t st) {
  return N == 9 ? rhs_launch_t<9>(R, grid, by_warp, st)
         : N == 21 ? rhs_launch_t<21>(R, grid, by_warp, st)
         : N == 53 ? rhs_launch_t<53>(R, grid, by_warp, st)
                   : cudaErrorInvalidValue;
}

}  // namespace b200
