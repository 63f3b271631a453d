// jac_table.h -- host side of the Jacobian kernel's table: which derivatives
// of the reaction rates add to which entry of d(wdot)/d(C, T).
//
// Derivatives of reaction j, from dptr[j]: one per species slot (by that
// slot's concentration, reactants 0..3 then products 4..7), one by T, the rate
// itself, and for third-body and falloff reactions the derivative by the
// third-body concentration.
// Entry (k, l): sum over the reactions of nu_k times the derivative by slot l
// or T, plus nu_k (eff_l - 1) times the third-body one where the efficiency of
// l differs from 1.  The default efficiency's part, nu_k times the third-body
// derivative for every l, is kept once per k (the row u); the production rates
// themselves, nu_k times the rates, follow it (the row w).
#pragma once
#include <algorithm>
#include <cstdint>
#include <map>
#include <utility>
#include <vector>

namespace b200 {

struct JacTable {
  int nd = 0, slices = 0;
  std::vector<int> dptr, off, tgt;
  std::vector<unsigned> term;
  std::vector<double> coef;
};

// sp, nu: [8][R] species (-1 empty) and signed stoichiometry; eff_m1:
// efficiency - 1.  ld: column stride of the kernel's Jacobian; the row u lies
// at (N + 1) ld, the row w behind it.  False when the table's index fields cannot hold the
// mechanism (coef_bits of 32 for the coefficient).
inline bool build_jac_table(int N, int R, const int* rtype, const int* sp, const int* nu, const int* eff_ptr,
                            const int* eff_sp, const double* eff_m1, int ld, int coef_bits, JacTable* T) {
  struct Entry {
    int tgt;
    std::vector<std::pair<int, double>> terms;
  };
  std::map<int, std::vector<std::pair<int, double>>> sums;  // target -> (derivative, coefficient)
  const int u0 = (N + 1) * ld;
  T->dptr.resize(R);
  T->nd = 0;
  for (int j = 0; j < R; ++j) {
    T->dptr[j] = T->nd;
    int cols[8], ncol = 0;
    std::map<int, double> net;
    for (int s = 0; s < 8; ++s) {
      const int k = sp[(size_t)s * R + j];
      if (k < 0) continue;
      cols[ncol++] = k;
      net[k] += nu[(size_t)s * R + j];
    }
    for (const auto& r : net) {
      if (r.second == 0.0) continue;
      for (int c = 0; c < ncol; ++c) sums[cols[c] * ld + r.first].push_back({T->nd + c, r.second});
      sums[N * ld + r.first].push_back({T->nd + ncol, r.second});
      sums[u0 + N + r.first].push_back({T->nd + ncol + 1, r.second});
      if (rtype[j] != 0) {
        const int d = T->nd + ncol + 2;
        sums[u0 + r.first].push_back({d, r.second});
        for (int q = eff_ptr[j]; q < eff_ptr[j + 1]; ++q)
          if (eff_m1[q] != 0.0) sums[eff_sp[q] * ld + r.first].push_back({d, r.second * eff_m1[q]});
      }
    }
    T->nd += ncol + 2 + (rtype[j] != 0 ? 1 : 0);
  }
  if (T->nd >= (1 << (32 - coef_bits))) return false;
  std::vector<Entry> e;
  for (auto& s : sums) e.push_back({s.first, std::move(s.second)});
  std::stable_sort(e.begin(), e.end(), [](const Entry& a, const Entry& b) { return a.terms.size() > b.terms.size(); });
  std::map<double, unsigned> cidx;
  T->coef.assign(1, 0.0);  // coefficient 0: padding
  cidx[0.0] = 0;
  T->slices = (int)((e.size() + 31) / 32);
  T->off.assign(1, 0);
  T->tgt.assign((size_t)T->slices * 32, -1);
  for (int s = 0; s < T->slices; ++s) {
    const size_t rows = e[(size_t)s * 32].terms.size();
    const size_t base = T->term.size();
    T->term.resize(base + rows * 32, 0u);
    for (int l = 0; l < 32 && (size_t)s * 32 + l < e.size(); ++l) {
      const Entry& x = e[(size_t)s * 32 + l];
      T->tgt[(size_t)s * 32 + l] = x.tgt;
      for (size_t t = 0; t < x.terms.size(); ++t) {
        const auto at = cidx.insert({x.terms[t].second, (unsigned)T->coef.size()});
        if (at.second) T->coef.push_back(x.terms[t].second);
        T->term[base + t * 32 + l] = ((unsigned)x.terms[t].first << coef_bits) | at.first->second;
      }
    }
    T->off.push_back((int)((base + rows * 32) / 32));
  }
  return T->coef.size() <= (size_t)1 << coef_bits;
}

}  // namespace b200
