// split_rule.h -- which GEMMs split K over a cluster of CTAs (gemm_bf16_splitk in
// mlp_tc.cu), and how.
#pragma once

namespace b200 {
namespace mlp {

constexpr int kSplit = 8;        // CTAs that share a tile
constexpr int kSplitStages = 4;  // ring of staged chunks
constexpr int kSplitKC = 64;     // K of a chunk
constexpr int kSplitTileM = 128;

// N tile: the largest multiple of 16 up to 64 that divides N.
inline int split_nt(int N) {
  for (int nt = 64; nt > 16; nt -= 16)
    if (N % nt == 0) return nt;
  return 16;
}
inline int split_smem(int NT) { return kSplitStages * (kSplitTileM + NT) * kSplitKC * 2; }

// Whether to split K: where 128 x 256 tiles would leave most SMs idle (fewer than
// half of them have one), K has two chunks for each CTA of a cluster (the ranges
// are rounded up, so that the last CTAs may have fewer or none), and the waves of
// split CTAs take less time than the one wave of whole tiles.  In us, with c chunks
// of K: a whole tile (240 + N) / 160 a chunk plus two and a half of them, a wave of
// split CTAs 0.27 (26 + c) whatever their N.  Whole against split: 256 x 256, K
// 16384 807 and 44; 4096 x 256, K 1024 58 and 40; 8192 x 128, K 1024 41 and 40, K
// 1088 45 and 48; 8192 x 256, K 1024 58 and 78, K 4096 211 and 167; 9344 x 80, K
// 4096 131 and 161, K 16384 647 and 559.
inline bool split_pays(int M, int N, int K, int sms) {
  const int c = K / kSplitKC, rows = M / kSplitTileM;
  if (K % kSplitKC != 0 || c < 2 * kSplit || 2 * rows * ((N + 255) / 256) >= sms) return false;
  const int nt = split_nt(N), per = (c + kSplit - 1) / kSplit;
  const int ctas = rows * (N / nt) * kSplit, per_sm = 228 * 1024 / (split_smem(nt) + 2048);
  const double waves = (double)ctas / ((double)per_sm * sms);
  const double split = (waves > 1.0 ? waves : 1.0) * 0.27 * (26 + kSplit * per);
  return split < (240 + (N < 256 ? N : 256)) / 160.0 * (c + 2.5);
}

}  // namespace mlp
}  // namespace b200
