// react_gen.cu -- kernels of the generated right-hand sides (mechgen.py), one
// thread per cell: f(y) of the round integrator's cells, and mass production
// rates.  A module of its own: the mechanisms' coefficients fill half of its
// constant memory.
#include <algorithm>

#define B200_GEN_FUNCTIONS
#include "rate_math.cuh"
#include "rhs_tables.cuh"

namespace b200 {
namespace {

// Resident CTAs (of 64 threads) per SM of the right-hand-side kernel, which
// bound its registers: 6 (168 registers) where the concentrations and rates
// of a cell (4 N registers) fit beside the exponentials in flight, 3 (255) for
// the 53-species mechanism.
#ifndef B200_RHS_MIN_CTAS
#define B200_RHS_MIN_CTAS 6
#endif
constexpr int rhs_min_ctas(int NS) { return NS <= 32 ? B200_RHS_MIN_CTAS : 3; }

template <int NS>
__global__ void __launch_bounds__(kRoundsRhsBlock, rhs_min_ctas(NS)) rk_rhs_gen(const __grid_constant__ RoundsParams R) {
  constexpr int n = NS + 1;
  extern __shared__ __align__(16) unsigned char dsm[];
  const int cnt = *R.cnt_in;
  // counters of the lists this round's later kernels append to
  if (blockIdx.x == 0 && threadIdx.x < kRoundLists) R.cnt_next[threadIdx.x] = 0;
  double* sE = reinterpret_cast<double*>(dsm) + threadIdx.x;
  double* sI = sE + NS * kRoundsRhsBlock;
  for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < cnt; idx += gridDim.x * blockDim.x) {
    const int slot = R.list_in[idx] & ~kSetupFlag;
    const RVec<n> v{reinterpret_cast<double*>(rec_of(R.S, slot) + R.S.L.off_vec)};
    if (!gen_covers<NS>(v.yev(NS))) cold_rhs<NS>(&R.P.mech, RecView<NS>{v}, sE, sI, kRoundsRhsBlock, &v.fv(0), 1);
    else if constexpr (NS == 9) gen::gen_rhs_synth_h2_9(&v.yev(0), &v.F(0), &v.fv(0), sE, sI, kRoundsRhsBlock);
    else if constexpr (NS == 21) gen::gen_rhs_synth_ch4_21(&v.yev(0), &v.F(0), &v.fv(0), sE, sI, kRoundsRhsBlock);
    else if constexpr (NS == 53) gen::gen_rhs_synth_c12_53(&v.yev(0), &v.F(0), &v.fv(0), sE, sI, kRoundsRhsBlock);
  }
}

// Mass production rates at (rhoY, T), one thread per cell.
template <int NS>
__global__ void __launch_bounds__(kRoundsRhsBlock, rhs_min_ctas(NS)) rk_rates(const __grid_constant__ DevMech m, InstView<NS> v) {
  extern __shared__ __align__(16) unsigned char dsm[];
  double* sd = reinterpret_cast<double*>(dsm);
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
  double* sE = sd + threadIdx.x;
  double* sI = sE + NS * kRoundsRhsBlock;
  for (v.c = t0; v.c < v.n; v.c += nt) {
    if (!gen_covers<NS>(v.T[v.c])) {
      cold_rhs<NS>(&m, v, sE, sI, kRoundsRhsBlock, v.dot + v.c, v.n);
      continue;
    }
    double y[NS + 1], f[NS + 1];
    const double F[NS + 1] = {};
#pragma unroll
    for (int k = 0; k <= NS; ++k) y[k] = v.yev(k);
    if constexpr (NS == 9) gen::gen_rhs_synth_h2_9(y, F, f, sE, sI, kRoundsRhsBlock);
    else if constexpr (NS == 21) gen::gen_rhs_synth_ch4_21(y, F, f, sE, sI, kRoundsRhsBlock);
    else if constexpr (NS == 53) gen::gen_rhs_synth_c12_53(y, F, f, sE, sI, kRoundsRhsBlock);
#pragma unroll
    for (int k = 0; k < NS; ++k) v.set_f(k, f[k]);
  }
}

template <int NS>
constexpr int gen_smem() { return 2 * NS * kRoundsRhsBlock * (int)sizeof(double); }

template <int NS>
cudaError_t grid_t(int sm_count, int* grid) {
  cudaError_t e = cudaFuncSetAttribute(rk_rhs_gen<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, gen_smem<NS>());
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(rk_rates<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, gen_smem<NS>());
  int b = 0;
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, rk_rhs_gen<NS>, kRoundsRhsBlock, gen_smem<NS>());
  *grid = std::max(1, b) * sm_count;
  return e;
}

template <int NS>
cudaError_t launch_t(const RoundsParams& R, int grid, cudaStream_t st) {
  rk_rhs_gen<NS><<<grid, kRoundsRhsBlock, gen_smem<NS>(), st>>>(R);
  return cudaGetLastError();
}

template <int NS>
cudaError_t rates_t(const DevMech& m, const double* rhoY, const double* T, double* dot, long long ncells, int grid,
                    cudaStream_t st) {
  const long long need = (ncells + kRoundsRhsBlock - 1) / kRoundsRhsBlock;
  rk_rates<NS><<<(int)std::min<long long>(need, grid), kRoundsRhsBlock, gen_smem<NS>(), st>>>(
      m, InstView<NS>{rhoY, T, dot, ncells, 0});
  return cudaGetLastError();
}

}  // namespace

cudaError_t gen_rhs_grid(int N, int sm_count, int* grid) {
  return N == 9 ? grid_t<9>(sm_count, grid) : N == 21 ? grid_t<21>(sm_count, grid) : grid_t<53>(sm_count, grid);
}

cudaError_t gen_rhs_launch(int N, const RoundsParams& R, int grid, cudaStream_t st) {
  return N == 9 ? launch_t<9>(R, grid, st) : N == 21 ? launch_t<21>(R, grid, st) : launch_t<53>(R, grid, st);
}

cudaError_t gen_rates_launch(int N, const DevMech& m, const double* rhoY, const double* T, double* dot,
                             long long ncells, int grid, cudaStream_t st) {
  return N == 9 ? rates_t<9>(m, rhoY, T, dot, ncells, grid, st)
         : N == 21 ? rates_t<21>(m, rhoY, T, dot, ncells, grid, st)
                   : rates_t<53>(m, rhoY, T, dot, ncells, grid, st);
}

}  // namespace b200

namespace b200 {
// Generated right-hand side matching a mechanism digest: 0 none, else the
// species count of the generated code.
int rounds_generated_for(unsigned long long digest) {
  if (digest == gen::kGenDigest_synth_h2_9) return 9;
  if (digest == gen::kGenDigest_synth_ch4_21) return 21;
  if (digest == gen::kGenDigest_synth_c12_53) return 53;
  return 0;
}
}  // namespace b200
