// C entry to the Jacobian table's builder (jac_table.h) for tests/test_jac_table.py.
#include <cstring>

#include "jac_table.h"

extern "C" int jac_table_apply(int N, int R, const int* rtype, const int* sp, const int* nu, const int* eff_ptr,
                               const int* eff_sp, const double* eff_m1, int ld, const double* D, int* nd, double* out) {
  b200::JacTable T;
  if (!b200::build_jac_table(N, R, rtype, sp, nu, eff_ptr, eff_sp, eff_m1, ld, 12, &T)) return 1;
  *nd = T.nd;
  if (!D) return 0;
  memset(out, 0, sizeof(double) * ((N + 1) * ld + 2 * N));
  for (int s = 0; s < T.slices; ++s)
    for (int l = 0; l < 32; ++l) {
      double v = 0.0;
      for (int t = T.off[s]; t < T.off[s + 1]; ++t) {
        const unsigned term = T.term[(size_t)t * 32 + l];
        v += T.coef[term & 4095u] * D[term >> 12];
      }
      const int tgt = T.tgt[(size_t)s * 32 + l];
      if (tgt >= 0) out[tgt] = v;
      else if (v != 0.0) return 2;
    }
  return 0;
}
