// rec_matrix.cuh -- where the entries of a cell record's matrices lie (round-based
// react path).
#pragma once

namespace b200 {
namespace rounds {

// Lanes per cell of the step and control kernels.
#ifndef B200_CTRL_LANES
#define B200_CTRL_LANES 8
#endif
__host__ __device__ constexpr int ctrl_group(int n) { return n <= 32 ? B200_CTRL_LANES : 16; }

// A matrix of the record for lane groups of G: lane g owns rows g, g + G, ...
// and reads V consecutive columns of one of its rows as one 16-byte vector;
// the lanes of a group read consecutive vectors.  Rows come in blocks of G
// (the last one as many as are left, so no row is padded), columns are padded
// to a multiple of V.
// mat_vec: offset of the vector of columns jb V .. jb V + V - 1 of row
// cc G + g; mat_idx: offset of element (i, j).
template <int n, int G, int V>
__host__ __device__ __forceinline__ constexpr int mat_vec(int cc, int g, int jb) {
  constexpr int JB = (n + V - 1) / V;
  const int rows = (n - cc * G < G) ? n - cc * G : G;
  return (cc * G * JB + jb * rows + g) * V;
}
template <int n, int G, int V>
__host__ __device__ __forceinline__ constexpr int mat_idx(int i, int j) {
  return mat_vec<n, G, V>(i / G, i % G, j / V) + j % V;
}
// columns per 16-byte vector of the Jacobian and of the inverse
constexpr int kVJ = 2;
template <typename LUT>
__host__ __device__ constexpr int vec_of() { return 16 / (int)sizeof(LUT); }

}  // namespace rounds
}  // namespace b200
