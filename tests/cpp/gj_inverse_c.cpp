// C entry to the round integrator's register inverses (gj_inverse.cuh), run by a
// warp on the CPU, for tests/test_gj_inverse.py.
#include "warp_host.h"

#include "gj_inverse.cuh"

using namespace b200;

namespace {

// Inverse of D (I - gamma J) D^-1 (FP32) or I - gamma J (FP64, dsc = 1), dense
// row-major J and out; form 0: one row per lane, 1: two rows per lane, 2: lane
// groups, of which the last has no cell.
template <int n, typename LUT, int form>
int invert(const double* J, const double* dsc, double gamma, int order, double* out) {
  constexpr int G = ctrl_group(n), V = vec_of<LUT>(), GPW = 32 / G, ldl = n | 1;
  constexpr int CPL = (n + G - 1) / G;
  alignas(16) static double Jr[n * n], rds[GPW][n], dl[64];
  alignas(16) static LUT Xs[GPW][(n * ldl + 3) / 4 * 4], Ar[GPW][n * ((n + V - 1) / V) * V];
  static int prow[GPW][64], pinv[GPW][64], ier[32];
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) Jr[mat_idx<n, G, kVJ>(i, j)] = J[i * n + j];
  for (int i = 0; i < n; ++i) dl[i] = dsc[i];
  for (int g = 0; g < GPW; ++g) std::fill(Ar[g], Ar[g] + n * ((n + V - 1) / V) * V, (LUT)0);
  warp_host::run([&](int lane) {
    if constexpr (form == 0) {
      ier[lane] = reg_gj_inverse<n>(Jr, gamma, Xs[0], ldl, prow[0], pinv[0], Ar[0], lane);
    } else if constexpr (form == 1) {
      ier[lane] = reg_gj_inverse2<n>(Jr, dl, gamma, Xs[0], ldl, prow[0], pinv[0], Ar[0], lane);
    } else {
      const int gi = lane / G, gl = lane % G;
      const bool live = gi + 1 < GPW;
      double di[CPL];
      for (int cc = 0; cc < CPL; ++cc) di[cc] = live && gl + G * cc < n ? dl[gl + G * cc] : 1.0;
      ier[lane] = grp_reg_gj_inverse<n, G>(Jr, live, di, rds[gi], live ? gamma : 0.0, Xs[gi], prow[gi], pinv[gi], Ar[gi], gl);
    }
  }, order);
  for (int l = 1; l < 32 && form != 2; ++l)
    if (ier[l] != ier[0]) return -1;
  for (int g = 1; g + 1 < GPW && form == 2; ++g)  // every group has the same cell
    if (memcmp(Ar[g], Ar[0], sizeof(Ar[0])) != 0) return -2;
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) out[i * n + j] = (double)Ar[0][mat_idx<n, G, V>(i, j)];
  return ier[0];
}

}  // namespace

extern "C" int gj_invert(int n, int fp64, const double* J, const double* dsc, double gamma, int order, double* out) {
  if (n == 10) return fp64 ? invert<10, double, 0>(J, dsc, gamma, order, out) : invert<10, float, 2>(J, dsc, gamma, order, out);
  if (n == 22) return fp64 ? invert<22, double, 0>(J, dsc, gamma, order, out) : invert<22, float, 2>(J, dsc, gamma, order, out);
  if (n == 54 && !fp64) return invert<54, float, 1>(J, dsc, gamma, order, out);
  return -3;
}
