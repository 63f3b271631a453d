// gj_inverse.cuh -- Newton-matrix inverses of the round-based react path, with
// the matrices in registers.
#pragma once
#include "rec_matrix.cuh"

namespace b200 {
using namespace rounds;

constexpr unsigned kAllLanes = 0xffffffffu;

// Shared memory of one cell of the lane-group inversion: 1 / dsc [n], the
// matrix [n][n | 1] (FP32) and two index arrays [n].
__host__ __device__ constexpr int gj_cell_bytes(int n) {
  return 8 * n + 4 * ((n * (n | 1) + 3) / 4 * 4) + (8 * n + 15) / 16 * 16;
}

// Row i of the inverse into the record, 16 bytes a store: entry j is
// src[pinv[j]] (the pivot permutation of the columns; pinv = nullptr: none).
template <int n, typename LUT>
__device__ __forceinline__ void store_inverse_row(const LUT* src, const int* pinv, LUT* Ar, int i) {
  constexpr int G = ctrl_group(n), V = vec_of<LUT>();
#pragma unroll
  for (int jb = 0; jb < (n + V - 1) / V; ++jb) {
    __align__(16) LUT t[V];
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const int j = jb * V + e;
      t[e] = j < n ? src[pinv ? pinv[j] : j] : (LUT)0;
    }
    *reinterpret_cast<uint4*>(Ar + mat_vec<n, G, V>(i / G, i % G, jb)) = *reinterpret_cast<const uint4*>(t);
  }
}

// In-place Gauss-Jordan inverse of the Newton matrix I - gamma J with partial
// pivoting, in FP64 (n <= 32): one warp per cell, lane i holding row i in
// registers.  Rows are never exchanged: step k takes as pivot the unused row p_k
// with the largest |a[., k]|, and at the end the inverse is (A^-1)[k][j] =
// X[p_k][q_j] with q_j the step at which row j was the pivot; that permutation is
// applied while the result is written to Ar (mat_idx order).  Xs, prow, pinv:
// per-warp shared scratch.  Returns 0, or k+1 when no usable pivot is left at
// step k.
template <int n>
__device__ __forceinline__ int reg_gj_inverse(const double* J, double gamma, double* Xs, int ldl, int* prow, int* pinv,
                                              double* Ar, int lane) {
  constexpr int G = ctrl_group(n);
  static_assert(n <= 32 && n % 2 == 0, "one row per lane, no column padding");
  const bool row = lane < n;
  double a[n];
#pragma unroll
  for (int jb = 0; jb < n / kVJ; ++jb) {
    double2 jv = make_double2(0.0, 0.0);
    if (row) jv = *reinterpret_cast<const double2*>(J + mat_vec<n, G, kVJ>(lane / G, lane % G, jb));
#pragma unroll
    for (int e = 0; e < kVJ; ++e) {
      const int j = jb * kVJ + e;
      a[j] = row ? ((lane == j) ? 1.0 : 0.0) - gamma * (e ? jv.y : jv.x) : 0.0;
    }
  }
  // Pivot search by one warp reduction: key = the high word of |a[k]| with the
  // low 5 bits replaced by (31 - lane), so the maximum picks the largest
  // magnitude (to 2^-15 relative) and, among equals, the lowest lane.
  // The pivot row goes through shared memory (two buffers, alternating per
  // step, 16-byte chunks) and every row, the pivot row included, is updated
  // by one FMA per column: a_ij -= g_i * a_pj with g_i = a_ik / a_pk off the
  // pivot row and g_p = 1 - 1 / a_pk on it (which scales the pivot row by
  // 1 / a_pk); column k is set last (1 / a_pk on the pivot row, -g_i off it).
  // The columns rotate by one register per step, so that column k is always
  // a[0] and the loop needs no unrolling.
  constexpr int kBuf = 32;  // entries per row buffer
  unsigned used = 0;
  int mystep = -1;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    double* buf = Xs + (k & 1) * kBuf;
    unsigned key = 0u;
    if (row && !((used >> lane) & 1u)) key = ((unsigned)__double2hiint(fabs(a[0])) & ~31u) | (unsigned)(31 - lane);
    const unsigned kmax = __reduce_max_sync(kAllLanes, key);
    if ((kmax >> 5) == 0u) return k + 1;  // no nonzero candidate: singular (warp-uniform)
    const int p = 31 - (int)(kmax & 31u);
    used |= 1u << p;
    if (lane == p) {
      mystep = k;
#pragma unroll
      for (int c = 0; c < n / 2; ++c) reinterpret_cast<double2*>(buf)[c] = make_double2(a[2 * c], a[2 * c + 1]);
    }
    __syncwarp();
    double pr[n];
#pragma unroll
    for (int c = 0; c < n / 2; ++c) {
      const double2 t = reinterpret_cast<const double2*>(buf)[c];
      pr[2 * c] = t.x;
      pr[2 * c + 1] = t.y;
    }
    const double pv = pr[0];
    if (!(fabs(pv) > 0.0) || isnan(pv)) return k + 1;  // zero or NaN pivot (warp-uniform)
    const double inv = 1.0 / pv;
    const double gi = (lane == p) ? 1.0 - inv : a[0] * inv;
#pragma unroll
    for (int j = 1; j < n; ++j) a[j - 1] = fma(-gi, pr[j], a[j]);
    a[n - 1] = (lane == p) ? inv : -gi;
  }
  __syncwarp();  // the pivot-row buffers lie in Xs
  if (row) {
#pragma unroll
    for (int j = 0; j < n; ++j) Xs[lane * ldl + j] = a[j];
    pinv[lane] = mystep;
    prow[mystep] = lane;
  }
  __syncwarp();
  if (row) store_inverse_row<n, double>(Xs + prow[lane] * ldl, pinv, Ar, lane);
  __syncwarp();
  return 0;
}

// The inverse of the scaled matrix D (I - gamma J) D^-1, D = diag(dsc), the same
// way for n <= 32 in FP32 by a group of G lanes per cell, lane g holding rows g,
// g + G, ... in registers: a pivot step costs its search, its
// exchange and its reciprocal once for the 32 / G cells of a warp, and a row
// chunk read from shared memory feeds every row of the lane.  All lanes of the
// warp call it; a group without a cell (live false) works on zeros.  Xs: two
// alternating pivot-row buffers, then the n x ldl result; rds: 1 / dsc [n].
// Bound by the latency of a pivot step (16 warps per SM, three quarters of the
// stalls wait for the previous one): 17.4 M inverses of 22 x 22 take 58 ms, 73
// with one warp and 32 unrolled steps per cell.
// Returns 0, or k+1 when no usable pivot is left at step k.
template <int n, int G>
__device__ __forceinline__ int grp_reg_gj_inverse(const double* J, bool live, const double (&di)[(n + G - 1) / G],
                                                  double* rds, double gamma, float* Xs, int* prow, int* pinv,
                                                  float* Ar, int gl) {
  static_assert(n <= 32, "the pivot key holds five bits of the row");
  constexpr int CPL = (n + G - 1) / G;
  constexpr int ldl = n | 1;
  constexpr int kChunks = (n + 3) / 4, kBuf = 4 * kChunks;
#pragma unroll
  for (int cc = 0; cc < CPL; ++cc) {
    const int i = gl + G * cc;
    if (i < n) rds[i] = 1.0 / di[cc];
  }
  __syncwarp();
  float a[CPL][n];
#pragma unroll
  for (int cc = 0; cc < CPL; ++cc) {
    const int i = gl + G * cc;
#pragma unroll
    for (int jb = 0; jb < n / kVJ; ++jb) {
      double2 jv = make_double2(0.0, 0.0);
      if (live && i < n) jv = *reinterpret_cast<const double2*>(J + mat_vec<n, G, kVJ>(cc, gl, jb));
#pragma unroll
      for (int e = 0; e < kVJ; ++e) {
        const int j = jb * kVJ + e;
        const double mij = ((i == j) ? 1.0 : 0.0) - gamma * (e ? jv.y : jv.x);
        a[cc][j] = (i < n) ? (float)(mij * di[cc] * rds[j]) : 0.0f;
      }
    }
  }
  unsigned used = 0;  // bit cc: this lane's row cc was a pivot
  int step[CPL], ier = 0;
#pragma unroll
  for (int cc = 0; cc < CPL; ++cc) step[cc] = 0;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    float* buf = Xs + (k & 1) * kBuf;
    unsigned key = 0u;
#pragma unroll
    for (int cc = 0; cc < CPL; ++cc) {
      const int i = gl + G * cc;
      if (i < n && !((used >> cc) & 1u)) {
        const unsigned kk = (__float_as_uint(fabsf(a[cc][0])) & ~31u) | (unsigned)(31 - i);
        key = key > kk ? key : kk;
      }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      const unsigned t = __shfl_xor_sync(kAllLanes, key, o, G);
      key = key > t ? key : t;
    }
    if (ier == 0 && (key >> 5) == 0u) ier = k + 1;  // no nonzero candidate: singular (group-uniform)
    const int p = 31 - (int)(key & 31u);
#pragma unroll
    for (int cc = 0; cc < CPL; ++cc) {
      if (p == gl + G * cc) {
        used |= 1u << cc;
        step[cc] = k;
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          float4 t;
          t.x = a[cc][4 * c];
          t.y = (4 * c + 1 < n) ? a[cc][4 * c + 1 < n ? 4 * c + 1 : 0] : 0.f;
          t.z = (4 * c + 2 < n) ? a[cc][4 * c + 2 < n ? 4 * c + 2 : 0] : 0.f;
          t.w = (4 * c + 3 < n) ? a[cc][4 * c + 3 < n ? 4 * c + 3 : 0] : 0.f;
          reinterpret_cast<float4*>(buf)[c] = t;
        }
      }
    }
    __syncwarp();
    const float pv = buf[0];
    if (ier == 0 && (!(fabsf(pv) > 0.f) || isnan(pv))) ier = k + 1;  // zero or NaN pivot (group-uniform)
    const float inv = 1.f / pv;
    float gf[CPL];
#pragma unroll
    for (int cc = 0; cc < CPL; ++cc) gf[cc] = (p == gl + G * cc) ? 1.f - inv : a[cc][0] * inv;
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      const float4 q = reinterpret_cast<const float4*>(buf)[c];
      const float qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = 4 * c + e;
        if (j < n && j > 0) {
#pragma unroll
          for (int cc = 0; cc < CPL; ++cc) a[cc][j - 1] = fmaf(-gf[cc], qv[e], a[cc][j]);
        }
      }
    }
#pragma unroll
    for (int cc = 0; cc < CPL; ++cc) a[cc][n - 1] = (p == gl + G * cc) ? inv : -gf[cc];
  }
  __syncwarp();  // the pivot-row buffers lie in Xs
#pragma unroll
  for (int cc = 0; cc < CPL; ++cc) {
    const int i = gl + G * cc;
    if (i < n) {
#pragma unroll
      for (int j = 0; j < n; ++j) Xs[i * ldl + j] = a[cc][j];
      pinv[i] = step[cc];
      prow[step[cc]] = i;
    }
  }
  __syncwarp();
  if (live && ier == 0) {
#pragma unroll
    for (int cc = 0; cc < CPL; ++cc) {
      const int i = gl + G * cc;
      if (i < n) store_inverse_row<n, float>(Xs + prow[i] * ldl, pinv, Ar, i);
    }
  }
  __syncwarp();
  return ier;
}

// The inverse of the scaled matrix for 32 < n <= 64 in FP32: lane l of a warp
// holds rows l and l + 32 in registers.  The pivot key carries the row index (6
// bits) instead of the lane; the pivot row's owner writes it to shared memory and
// every lane updates both of its rows from 16-byte reads of it.  Unrolled, the 54
// steps are 150 KB of code that waits for instructions: 766,122 inverses took 38
// ms and take 26 in the rolled loop.
template <int n>
__device__ __forceinline__ int reg_gj_inverse2(const double* J, const double* dsc, double gamma, float* Xs, int ldl,
                                               int* prow, int* pinv, float* Ar, int lane) {
  constexpr int G = ctrl_group(n);
  static_assert(n > 32 && n <= 64, "two rows per lane");
  const int r1 = lane + 32;
  const bool row1 = r1 < n;
  const double d0 = dsc[lane], d1 = row1 ? dsc[r1] : 1.0;
  const double rd0 = 1.0 / d0, rd1 = 1.0 / d1;
  float a0[n], a1[n];
#pragma unroll
  for (int jb = 0; jb < n / kVJ; ++jb) {
    const double2 j0 = *reinterpret_cast<const double2*>(J + mat_vec<n, G, kVJ>(lane / G, lane % G, jb));
    double2 j1 = make_double2(0.0, 0.0);
    if (row1) j1 = *reinterpret_cast<const double2*>(J + mat_vec<n, G, kVJ>(r1 / G, r1 % G, jb));
#pragma unroll
    for (int e = 0; e < kVJ; ++e) {
      const int j = jb * kVJ + e;
      const double rdj = (j < 32) ? __shfl_sync(kAllLanes, rd0, j) : __shfl_sync(kAllLanes, rd1, j - 32);
      const double m0 = ((lane == j) ? 1.0 : 0.0) - gamma * (e ? j0.y : j0.x);
      const double m1 = row1 ? ((r1 == j) ? 1.0 : 0.0) - gamma * (e ? j1.y : j1.x) : 0.0;
      a0[j] = (float)(m0 * d0 * rdj);
      a1[j] = row1 ? (float)(m1 * d1 * rdj) : 0.f;
    }
  }
  constexpr int kChunks = (n + 3) / 4;
  constexpr int kBuf = 64;
  unsigned used0 = 0, used1 = 0;
  int step0 = -1, step1 = -1;
#pragma unroll 1
  for (int k = 0; k < n; ++k) {
    float* buf = Xs + (k & 1) * kBuf;
    unsigned key = 0u;
    if (!((used0 >> lane) & 1u)) key = (__float_as_uint(fabsf(a0[0])) & ~63u) | (unsigned)(63 - lane);
    if (row1 && !((used1 >> lane) & 1u)) {
      const unsigned k1 = (__float_as_uint(fabsf(a1[0])) & ~63u) | (unsigned)(63 - r1);
      key = key > k1 ? key : k1;
    }
    const unsigned kmax = __reduce_max_sync(kAllLanes, key);
    if ((kmax >> 6) == 0u) return k + 1;  // no nonzero candidate: singular (warp-uniform)
    const int p = 63 - (int)(kmax & 63u);
    const int pl = p & 31;
    if (p < 32) used0 |= 1u << pl;
    else used1 |= 1u << pl;
    if (lane == pl) {
      if (p < 32) {
        step0 = k;
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          float4 t;
          t.x = a0[4 * c];
          t.y = (4 * c + 1 < n) ? a0[4 * c + 1] : 0.f;
          t.z = (4 * c + 2 < n) ? a0[4 * c + 2] : 0.f;
          t.w = (4 * c + 3 < n) ? a0[4 * c + 3] : 0.f;
          reinterpret_cast<float4*>(buf)[c] = t;
        }
      } else {
        step1 = k;
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
          float4 t;
          t.x = a1[4 * c];
          t.y = (4 * c + 1 < n) ? a1[4 * c + 1] : 0.f;
          t.z = (4 * c + 2 < n) ? a1[4 * c + 2] : 0.f;
          t.w = (4 * c + 3 < n) ? a1[4 * c + 3] : 0.f;
          reinterpret_cast<float4*>(buf)[c] = t;
        }
      }
    }
    __syncwarp();
    const float pv = buf[0];
    if (!(fabsf(pv) > 0.f) || isnan(pv)) return k + 1;  // zero or NaN pivot (warp-uniform)
    const float inv = 1.f / pv;
    const float g0 = (p == lane) ? 1.f - inv : a0[0] * inv;
    const float g1 = (p == r1) ? 1.f - inv : a1[0] * inv;
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      const float4 q = reinterpret_cast<const float4*>(buf)[c];
      const float qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = 4 * c + e;
        if (j < n && j > 0) {
          a0[j - 1] = fmaf(-g0, qv[e], a0[j]);
          a1[j - 1] = fmaf(-g1, qv[e], a1[j]);
        }
      }
    }
    a0[n - 1] = (p == lane) ? inv : -g0;
    a1[n - 1] = (p == r1) ? inv : -g1;
  }
  __syncwarp();  // the row buffers live in Xs
#pragma unroll
  for (int j = 0; j < n; ++j) Xs[lane * ldl + j] = a0[j];
  if (row1) {
#pragma unroll
    for (int j = 0; j < n; ++j) Xs[r1 * ldl + j] = a1[j];
  }
  pinv[lane] = step0;
  prow[step0] = lane;
  if (row1) {
    pinv[r1] = step1;
    prow[step1] = r1;
  }
  __syncwarp();
  for (int h = 0; h < 2; ++h) {
    const int i = lane + 32 * h;
    if (i < n) store_inverse_row<n, float>(Xs + prow[i] * ldl, pinv, Ar, i);
  }
  __syncwarp();
  return 0;
}

}  // namespace b200
