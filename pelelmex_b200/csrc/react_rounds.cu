// react_rounds.cu -- round-based react path: rhs / ctrl / setup kernels over
// compacted cell lists, and their host-side launch sequence.
//
// A react call is processed in chunks of cells (as many as the state buffer
// holds).  For one chunk:
//   start                     load every cell, mask / validity checks, list A
//   repeat until A is empty (S, SJ: the cells of A whose Newton matrix is
//   rebuilt, and those of them whose Jacobian is recomputed):
//     rhs   (A)               f(y) for every cell of A (thread per cell)
//     step  (A without S)     Newton correction and step; next f -> B (S', SJ'
//                             as the prediction needs), anything rarer -> W
//     jac   (SJ), gj (S)      Jacobian, inverse (warp per cell)
//     step  (S)               the same for the set-up cells
//     ctrl  (W)               the rare paths; finished cells -> outputs
//     swap A, B and the setup lists
// Lists are appended with warp-aggregated atomics, so a warp's slots stay in
// order and the interleaved state accesses stay coalesced as cells drop out.
#include <algorithm>

#include "bdf_rounds.cuh"
#include "common.cuh"
#include "gj_inverse.cuh"

namespace b200 {
using namespace rounds;

namespace {

// (box, i, j, k) of a global cell index of the react call.
struct CellLoc {
  const DevBox* bx;
  int i, j, k;
};

__device__ __forceinline__ CellLoc locate(const ReactParams& P, long long cell) {
  int lo = 0, hi = P.nbox - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (P.boxes[mid].off <= cell) lo = mid;
    else hi = mid - 1;
  }
  CellLoc L;
  L.bx = P.boxes + lo;
  const long long loc = cell - L.bx->off;
  L.i = L.bx->lo0 + (int)(loc % L.bx->nx);
  L.j = L.bx->lo1 + (int)((loc / L.bx->nx) % L.bx->ny);
  L.k = L.bx->lo2 + (int)(loc / ((long long)L.bx->nx * L.bx->ny));
  return L;
}

// Append `val` of the lanes with pred to one list of counter cnt, or of the
// lanes whose bit k of `which` is set to list k (all 32 lanes call it): one
// atomic per warp and list.
__device__ __forceinline__ void warp_append(bool pred, int val, int* list, int* cnt) {
  const unsigned m = __ballot_sync(kFull, pred);
  if (m == 0) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(cnt, __popc(m));
  base = __shfl_sync(kFull, base, leader);
  if (pred) list[base + __popc(m & ((1u << lane) - 1u))] = val;
}

// The lists' atomics are issued together by lanes 0..kRoundLists - 1, so a
// warp waits for one of them and not for their sum.
__device__ __forceinline__ void warp_append_lists(int which, int slot, int rhs_val, const RoundsParams& R) {
  const int lane = threadIdx.x & 31;
  unsigned m[kRoundLists], mine = 0;
#pragma unroll
  for (int k = 0; k < kRoundLists; ++k) {
    m[k] = __ballot_sync(kFull, (which >> k) & 1);
    if (lane == k) mine = m[k];
  }
  int base = 0;
  if (mine) base = atomicAdd(R.cnt_next + lane, __popc(mine));
#pragma unroll
  for (int k = 0; k < kRoundLists; ++k) {
    const int b = __shfl_sync(kFull, base, k);
    if ((which >> k) & 1) R.list[k][b + __popc(m[k] & ((1u << lane) - 1u))] = (k == kRlRhs) ? rhs_val : slot;
  }
}

// Lists a cell with this need goes to.
__device__ __forceinline__ int lists_of(int need) {
  return need == kNeedRhs ? 1 << kRlRhs
         : need == kNeedSetup ? (1 << kRlRhs) | (1 << kRlSetup)
         : need == kNeedSetupJac ? (1 << kRlRhs) | (1 << kRlSetup) | (1 << kRlJac)
                                 : 0;
}

// Warp-aggregated statistics of the lanes with `done` (all 32 lanes call it).
__device__ __forceinline__ void warp_stats(long long* stats, bool done, bool failed, bool masked,
                                           const CellCounters& cnt) {
  if (!stats || __ballot_sync(kFull, done || masked) == 0) return;
  long long v[kStMaxNfe];
  v[kStCells] = done;
  v[kStMasked] = masked;
  v[kStFailed] = done && failed;
  v[kStNst] = done ? cnt.nst : 0;
  v[kStNfe] = done ? cnt.nfe : 0;
  v[kStNje] = done ? cnt.nje : 0;
  v[kStNlu] = done ? cnt.nlu : 0;
  v[kStNetf] = done ? cnt.netf : 0;
  v[kStNcfn] = done ? cnt.ncfn : 0;
  long long mx = done ? cnt.nfe : 0, ms = done ? cnt.nst : 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int s = 0; s < kStMaxNfe; ++s) v[s] += __shfl_xor_sync(kFull, v[s], o);
    mx = max(mx, __shfl_xor_sync(kFull, mx, o));
    ms = max(ms, __shfl_xor_sync(kFull, ms, o));
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int s = 0; s < kStMaxNfe; ++s)
      if (v[s]) atomicAdd(reinterpret_cast<unsigned long long*>(stats + s), (unsigned long long)v[s]);
    if (mx) atomicMax(stats + kStMaxNfe, mx);
    if (ms) atomicMax(stats + kStMaxNst, ms);
  }
}

}  // namespace

// ---------------------------------------------------------------- kernels
template <int NS>
__global__ void __launch_bounds__(128) rk_start(RoundsParams R) {
  constexpr int n = NS + 1;
  const ReactParams& P = R.P;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long base = (long long)blockIdx.x * blockDim.x; base < R.nchunk; base += stride) {
    const long long slot = base + threadIdx.x;
    const bool live = slot < R.nchunk;
    bool go = false, done = false, masked = false;
    // the FP64 retry pass integrates only the cells the FP32 pass flagged
    const bool skip = live && P.retry_pass && P.retry[R.chunk0 + slot] == 0;
    if (live && !skip) {
      const long long cell = R.chunk0 + slot;
      const CellLoc L = locate(P, cell);
      const DevBox& bx = *L.bx;
      if (bx.mask.p)
        masked = bx.mask.p[(long long)(L.i - bx.mask.lo0) + (long long)(L.j - bx.mask.lo1) * bx.mask.js +
                           (long long)(L.k - bx.mask.lo2) * bx.mask.ks] == 0;
      int code = 0;
      if (masked) {
        code = B200CHEM_CELL_MASKED;
        if (bx.fc.p) *elem(bx.fc, L.i, L.j, L.k) = 0.0;
      } else {
        unsigned char* rec = rec_of(R.S, slot);
        const RVec<n> v{reinterpret_cast<double*>(rec + R.S.L.off_vec)};
        const double* yp = elem(bx.rhoY, L.i, L.j, L.k);
        const double* fp = elem(bx.fY, L.i, L.j, L.k);
        double rho = 0.0;
        bool bad = false;
#pragma unroll 4
        for (int q = 0; q < NS; ++q) {
          const double y = yp[q * bx.rhoY.ns], f = fp[q * bx.fY.ns];
          v.zn(0, q) = y;
          v.F(q) = f;
          rho += y;
          bad |= !isfinite(y) || !isfinite(f);
        }
        const double T = *elem(bx.T, L.i, L.j, L.k), fH = *elem(bx.fH, L.i, L.j, L.k);
        v.zn(0, NS) = T;
        v.F(NS) = fH;
        bad |= !(T > 0.0) || !isfinite(T) || !isfinite(fH) || !(rho > 0.0);
        if (bad) {
          code = B200CHEM_CELL_NONFINITE;
          if (bx.fc.p) *elem(bx.fc, L.i, L.j, L.k) = 0.0;
          done = true;
        } else {
          RCell c;
          r_begin<n>(c, v, P.atol, P.rtol, P.dt, P.qmax, P.max_steps);
          store_cell(c, rec);
          go = true;
        }
      }
      if (!go && P.status) P.status[cell] = code;
    }
    warp_append(go, (int)slot, R.list[kRlRhs], R.cnt_next + kRlRhs);
    warp_stats(P.stats, done, true, masked, CellCounters{0, 0, 0, 0, 0, 0, 0});
  }
}

// Minimum resident CTAs (of 128 threads) per SM requested for the step
// kernel: bounds its registers per thread.  The kernel is bound by the cells'
// records (8 KB at 22 components) from HBM, and more cells in flight do not
// help it: the matrices prefetched for them drop out of L2 before they are read
// (9500 cells hold 78 MB), and loads that the registers of 2 CTAs keep in flight
// hide the latency as well.  128^3 CH4, per react: 168 ms at 2 CTAs, 186 at 3,
// 201 at 4, 250 at 5.  A small record (2.3 KB at 10 components) leaves the
// arithmetic, for which more warps are better (32^3 H2: 2.1 ms at 4, 2.2 at 3,
// 2.6 at 2).
constexpr int step_min_ctas(int n) { return n <= 16 ? 4 : 2; }

// Bulk prefetch of [p, p + bytes) into L2 (p and bytes multiples of 16; a
// hint: no completion to wait for).
__device__ __forceinline__ void l2_prefetch(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}

// Shared memory of one cell of the step kernel: the scalars and the vectors
// it reads, as they lie in the record, n doubles of scratch, and 16 bytes
// that spread the cells of a warp over the banks.
template <int n>
constexpr int step_read_bytes() { return (int)sizeof(RCell) + 8 * kVecsRead * n; }
template <int n>
constexpr int step_cell_bytes() { return step_read_bytes<n>() + 8 * ((n + 1) / 2 * 2) + 16; }
template <int n>
constexpr int step_smem() { return 128 / ctrl_group(n) * step_cell_bytes<n>(); }

// One cell of the step kernel, G lanes per cell: the Newton correction with
// the f just evaluated, then the next Newton iterate or, after a converged
// iteration that passes the error test, the next prediction.  Anything else
// (the start of a cell, failures, its last step) goes to the control kernel,
// with the label it resumes at.  Every lane of the warp calls it (the appends
// are warp-collective); `live` marks the groups with a cell; sm: the cell's
// shared memory.
template <int NS, int G, typename LUT>
__device__ __forceinline__ void step_cell(const RoundsParams& R, bool live, int slot, unsigned char* sm, int gl,
                                          unsigned gm) {
  constexpr int n = NS + 1;
  constexpr int CPL = (n + G - 1) / G;
  const ReactParams& P = R.P;
  int which = 0, rhs_val = slot;
  if (live) {
    unsigned char* rec = rec_of(R.S, slot);
    // the matrices stream into L2 while the scalars and vectors are copied
    if (gl == 0) l2_prefetch(rec + R.S.L.off_j, (uint32_t)(R.S.L.stride - R.S.L.off_j));
    for (int b = gl * 16; b < step_read_bytes<n>(); b += G * 16) cp_async16(sm + b, rec + b);
    cp_async_wait();
    __syncwarp(gm);
    RCell& c = *reinterpret_cast<RCell*>(sm);
    const RVec<n> s{reinterpret_cast<double*>(sm + sizeof(RCell))};
    const RVec<n> g{reinterpret_cast<double*>(rec + sizeof(RCell))};
    const int label = c.label;
    which = 1 << kRlCtrl;
    if (label == kLAfterNStart || label == kLAfterNIter || (label == kLAfterSetup && c.setup_ier == 0)) {
      const bool iter = label == kLAfterNIter;
      const int mnewt = iter ? c.mnewt : 0;
      double ac[CPL];
#pragma unroll
      for (int cc = 0; cc < CPL; ++cc) {
        const int i = gl + G * cc;
        ac[cc] = (iter && i < n) ? s.acor(i) : 0.0;
      }
      double del, anrm;
      bool stall = false;
      float ratio = (label == kLAfterSetup) ? kRefineUnknown : c.refine_ratio;
      // the FP64 refinement runs on the first correction with a new matrix,
      // and again on every later one unless that first measurement showed
      // the FP32 solve alone accurate to refine_keep
      const bool refine = !(P.refine_keep > 0.0 && ratio <= P.refine_keep);
      g_newton<n, G, LUT>(s, reinterpret_cast<const double*>(rec + R.S.L.off_j),
                          reinterpret_cast<const LUT*>(rec + R.S.L.off_a),
                          reinterpret_cast<double*>(sm + step_read_bytes<n>()), c.rl1, c.gamma, c.gamma_lu, c.gamrat,
                          gl, gm, ac, &del, &anrm, sizeof(LUT) == 4 ? P.refine_stall : 0.0, &stall, refine, &ratio);
      const double crate = (mnewt > 0) ? fmax(kCRDOWN * c.crate, del / c.delp) : c.crate;
      const double dcon = del * fmin(1.0, crate) / c.tq[4];
      const double acnrm = (mnewt == 0) ? del : anrm;
      const double dsm = acnrm * c.tq[2];
      const bool conv = dcon <= 1.0;
      const bool step = !stall && conv && dsm <= 1.0 && !(c.tn - c.dt >= 0.0) && c.nstloc + 1 < c.max_steps;
      const bool again = !stall && !conv &&
                         !((mnewt >= 1 && del > kRDIV * c.delp) || !(del == del) || mnewt + 1 >= kMAXCOR);
      RCell o;
      if (step) {
        const int need = g_finish_step<n, G>(c, o, s, g, ac, dsm, P.atol, P.rtol, gl, gm);
        which = lists_of(need);
        if (need != kNeedRhs) rhs_val |= kSetupFlag;
      } else {
#pragma unroll
        for (int cc = 0; cc < CPL; ++cc) {
          const int i = gl + G * cc;
          if (i < n) {
            g.acor(i) = ac[cc];
            if (again) g.yev(i) = s.zn(0, i) + ac[cc];
          }
        }
        if (again) which = 1 << kRlRhs;
      }
      __syncwarp(gm);  // every lane is done reading c
      if (gl == 0) {
        c.cnt.nfe++;
        c.cnt.nni++;
        c.crate = crate;
        c.refine_ratio = ratio;
        if (step) {
#define B200_ST(f) c.f = o.f;
          B200_ST(h) B200_ST(hscale) B200_ST(eta) B200_ST(etamax) B200_ST(tn) B200_ST(gamma)
          B200_ST(gamrat) B200_ST(rl1) B200_ST(saved_tq5) B200_ST(saved_t) B200_ST(q) B200_ST(L)
          B200_ST(qwait) B200_ST(nstlj) B200_ST(jcur) B200_ST(ncf) B200_ST(nef) B200_ST(nflag) B200_ST(convfail)
          B200_ST(callSetup) B200_ST(jbad) B200_ST(attempt) B200_ST(nstloc) B200_ST(setup_conv) B200_ST(label)
          B200_ST(cnt.nst) B200_ST(cnt.nje)
#undef B200_ST
#pragma unroll
          for (int i = 1; i < kZn + 2; ++i) c.tau[i] = o.tau[i];
#pragma unroll
          for (int i = 1; i < 6; ++i) c.tq[i] = o.tq[i];
#pragma unroll
          for (int i = 0; i < kZn; ++i) c.l[i] = o.l[i];
        } else if (again) {
          c.delp = del;
          c.mnewt = mnewt + 1;
          c.label = kLAfterNIter;
        } else {
          c.acnrm = acnrm;
          c.mnewt = mnewt;
          if (conv) c.jcur = 0;
          c.label = stall ? kLStall : conv ? kLNlsSuccess : kLNlsRecover;
        }
      }
      __syncwarp(gm);
      for (int b = gl * 16; b < (int)sizeof(RCell); b += G * 16)
        *reinterpret_cast<uint4*>(rec + b) = *reinterpret_cast<const uint4*>(sm + b);
    }
  }
  __syncwarp();  // the shared copies are free again
  warp_append_lists(gl == 0 ? which : 0, slot, rhs_val, R);
}

// Newton correction and step of the cells of list_in, G lanes per cell.  pass
// kStepKept: the cells that keep their Newton matrix (the flagged entries of the
// others are passed over); kStepSetup: a list of those this round's setup
// kernels rebuilt it for; kStepAll: both kinds from the first list.
template <int NS, typename LUT>
__global__ void __launch_bounds__(128, step_min_ctas(NS + 1)) rk_step(RoundsParams R, int pass) {
  constexpr int n = NS + 1;
  constexpr int G = ctrl_group(n);
  constexpr int GPW = 32 / G;  // cells per warp
  extern __shared__ __align__(16) unsigned char dsm[];
  const int cnt = *R.cnt_in;
  const int lane = threadIdx.x & 31, gl = lane % G, gi = lane / G;
  const unsigned gm = (G == 32) ? kFull : (((1u << G) - 1u) << (gi * G));
  unsigned char* sm = dsm + (threadIdx.x / G) * step_cell_bytes<n>();
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int base = wid * GPW; base < cnt; base += nw * GPW) {
    const int idx = base + gi;
    const int entry = idx < cnt ? R.list_in[idx] : 0;
    const bool live = idx < cnt && (pass != kStepKept || !(entry & kSetupFlag));
    step_cell<NS, G, LUT>(R, live, entry & ~kSetupFlag, sm, gl, gm);
  }
}

// Minimum resident CTAs (of 128 threads) per SM requested for the control
// kernel: bounds its registers per thread.
#ifndef B200_CTRL_MIN_CTAS
#define B200_CTRL_MIN_CTAS 3
#endif

// One cell of the control kernel, G lanes per cell: resume the CVODE state
// machine, write the outputs of a finished cell, and append the cell to the
// lists of its next need.  Every lane of the warp calls it (the appends are
// warp-collective); `live` marks the groups with a cell.
template <int NS, int G>
__device__ __forceinline__ void ctrl_cell(const RoundsParams& R, bool live, int slot, int gl, unsigned gm) {
  constexpr int n = NS + 1;
  const ReactParams& P = R.P;
  int need = kDone, status = 0;
  RCell c;
  if (live) {
    unsigned char* rec = rec_of(R.S, slot);
    load_cell(c, rec);
    // a cell the step kernel passed on as it was consumes its f here
    if (c.label <= kLAfterSetup) c.cnt.nfe++;
    const RVec<n> v{reinterpret_cast<double*>(rec + R.S.L.off_vec)};
    need = r_advance<n, G>(c, v, c.label, P.atol, P.rtol, gl, gm, &status);
    __syncwarp(gm);
    if (gl == 0) store_cell(c, rec);
    if (need == kDone) {
      const long long cell = R.chunk0 + slot;
      const CellLoc L = locate(P, cell);
      const DevBox& bx = *L.bx;
      if (status == 0) {
        // y(dt) from the Nordsieck array (Horner in s = (dt - tn) / h)
        const double s = (P.dt - c.tn) / c.h;
        double* yp = elem(bx.rhoY, L.i, L.j, L.k);
        const int q = c.q;
        each<n, G>(gl, [&](int k) {
          double y = v.zn(q, k);
          for (int jj = q - 1; jj >= 0; --jj) y = v.zn(jj, k) + s * y;
          if (k < NS) yp[k * bx.rhoY.ns] = y;
          else *elem(bx.T, L.i, L.j, L.k) = y;
        });
        if (gl == 0) {
          double* hp = elem(bx.rhoH, L.i, L.j, L.k);
          *hp = *hp + P.dt * v.F(NS);
        }
      }
      if (gl == 0) {
        if (status == kStatusRefineStall) {
          // untouched: no outputs, no status; the FP64 pass writes them
          P.retry[cell] = 1;
          if (P.stats) atomicAdd(reinterpret_cast<unsigned long long*>(P.stats + kStStall), 1ull);
        } else {
          if (bx.fc.p) *elem(bx.fc, L.i, L.j, L.k) = (double)c.cnt.nfe;
          if (P.status) P.status[cell] = status;
        }
      }
    }
  }
  const bool lead = live && gl == 0;
  warp_append_lists(lead ? lists_of(need) : 0, slot, need == kNeedRhs ? slot : (slot | kSetupFlag), R);
  warp_stats(P.stats, lead && need == kDone && status != kStatusRefineStall, status != 0, false, c.cnt);
}

// The cells of list_in through the state machine, G lanes per cell.
template <int NS>
__global__ void __launch_bounds__(128, B200_CTRL_MIN_CTAS) rk_ctrl(RoundsParams R) {
  constexpr int n = NS + 1;
  constexpr int G = ctrl_group(n);
  constexpr int GPW = 32 / G;  // cells per warp
  const int cnt = *R.cnt_in;
  const int lane = threadIdx.x & 31, gl = lane % G, gi = lane / G;
  const unsigned gm = (G == 32) ? kFull : (((1u << G) - 1u) << (gi * G));
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int base = wid * GPW; base < cnt; base += nw * GPW) {
    const int idx = base + gi;
    const bool live = idx < cnt;
    ctrl_cell<NS, G>(R, live, live ? R.list_in[idx] : 0, gl, gm);
  }
}

// Warps that work on one cell in the Jacobian kernel: one where a warp covers
// the reactions in two or three strides, a CTA of four for the large
// mechanism, whose Jacobian and rates (38 KB of shared memory) would leave
// five warps on an SM and whose few refreshes per round are a matter of
// latency.
constexpr int jac_warps(int n) { return n <= 32 ? 1 : 4; }
// Leading dimension of the shared Jacobian: odd, so that the lanes of a row
// hit different banks.
constexpr int jac_ld(int n) { return n | 1; }

// Analytic Jacobian of one cell by a team of W warps.  1. lane per reaction:
// the derivatives of its rate by the concentration of each of its slots, by T,
// and by the third-body concentration (D).  2. lane per entry of the Jacobian:
// the sum of nu D over the reactions that reach it, from the mechanism's
// table (jt_*: entries in slices of 32 of about equal length, so that a term
// is one coalesced load and no two lanes write the same entry; the shared
// atomics this replaces were retry loops: 286,308 Jacobians of 53 species took
// 28 ms and take 15; with 21 species both take 15 ns a cell, the reactions).  The default third-body efficiency 1 of every
// species is a row vector u added to all columns, the non-default ones are
// terms.  3. the temperature row; 4. mass units, and the matrix into the cell
// record (mat_idx order, consecutive 16-byte stores).  The rates come along, so
// the kernel needs no f and runs beside the right-hand sides.
// s: C, g/RT, h/RT, hm [Npad]; Js: [n][ld] column-major, then u [N], w [N] and
// the temperature row [n]; entries outside the table stay zero.
template <int n, int CPL, int W>
__device__ __forceinline__ void team_jac(const DevMech& m, const GrpScratch& s, double* hm, double* Js, double* D,
                                         const Vec<CPL>& y, const Vec<CPL>& F, double* J, int tid) {
  constexpr int N = n - 1, ld = jac_ld(n), TS = 32 * W;
  const int lane = tid & 31;
  const Grp<32> g(lane);
  const int R = m.R;
  double* u = Js + n * ld;
  double* w = u + N;
  double* tr = w + N;
  auto sync = [] {
    if constexpr (W == 1) __syncwarp();
    else __syncthreads();
  };
  const double T = grp_get_T<32, CPL>(g, y, N);
  const double lnT = log(T), invT = 1.0 / T;
  double cpk[CPL], hk[CPL], dcpk[CPL];
  grp_species<32, CPL>(m, s, g, y, T, lnT, cpk, hk, dcpk);  // every warp writes the same values
  double csum = 0.0, rcp = 0.0, drcp = 0.0;
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    const int k = lane + 32 * c;
    if (k < N) {
      csum += y.v[c] * __ldg(m.inv_mw + k);
      rcp += y.v[c] * cpk[c];
      drcp += y.v[c] * dcpk[c];
      hm[k] = hk[c] * __ldg(m.mw + k);
    }
  }
  const double Ctot = g.sum(csum);
  rcp = g.sum(rcp);
  drcp = g.sum(drcp);
  const double lnPRT = log(kPatm / (kRu * T));
  sync();
  for (int j = tid; j < R; j += TS) {
    const RxnEval e = eval_reaction<true>(m, SpView{s.C, s.gRT, s.hRT}, j, T, lnT, invT, Ctot, lnPRT);
    const int type = __ldg(m.rtype + j);
    const double mult = (type == 1) ? e.M : 1.0;
    double ceff = 0.0;
    if (type == 1) ceff = e.kf * e.pf - e.kr * e.pr;
    else if (type >= 2) ceff = e.dkf_dM * (e.pf - (e.kf > 0.0 ? e.kr / e.kf : 0.0) * e.pr);
    const double kfm = mult * e.kf, krm = mult * e.kr;
    double c[8];
    int nu[8];
#pragma unroll
    for (int sl = 0; sl < 8; ++sl) {
      const int k = __ldg(m.sp + sl * R + j), v = __ldg(m.nu + sl * R + j);
      nu[sl] = k >= 0 ? (v < 0 ? -v : v) : 0;
      c[sl] = k >= 0 ? s.C[k] : 1.0;
    }
    double* d = D + __ldg(m.jt_dptr + j);
    // derivative by each slot's concentration: reactants forward, products reverse
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      if (nu[a] == 0) continue;
      double p = nu[a] * ipow(c[a], nu[a] - 1);
#pragma unroll
      for (int o = (a < 4 ? 0 : 4); o < (a < 4 ? 4 : 8); ++o)
        if (o != a) p *= ipow(c[o], nu[o]);
      *d++ = (a < 4) ? kfm * p : -krm * p;
    }
    *d++ = mult * (e.kf * e.dlnkf_dT * e.pf - e.dkr_dT * e.pr);
    *d++ = mult * (e.kf * e.pf - e.kr * e.pr);
    if (type != 0) *d = ceff;
  }
  sync();
  for (int sl = tid >> 5; sl < m.jt_slices; sl += W) {
    const int t0 = __ldg(m.jt_off + sl), t1 = __ldg(m.jt_off + sl + 1);
    double v = 0.0;
#pragma unroll 8
    for (int t = t0; t < t1; ++t) {
      const unsigned term = __ldg(m.jt_term + t * 32 + lane);
      v += __ldg(m.jt_coef + (term & (kJtCoefs - 1))) * D[term >> kJtCoefBits];
    }
    const int tgt = __ldg(m.jt_tgt + sl * 32 + lane);
    if (tgt >= 0) Js[tgt] = v;
  }
  sync();
  // dT/dt and sum cp_k d(rhoY_k)/dt, by every warp
  double hdot = 0.0, cpdot = 0.0, FH = 0.0;
#pragma unroll
  for (int c = 0; c < CPL; ++c) {
    const int k = lane + 32 * c;
    if (k < N) {
      const double yd = w[k] * __ldg(m.mw + k) + F.v[c];
      hdot += hk[c] * yd;
      cpdot += cpk[c] * yd;
    } else if (k == N) {
      FH = F.v[c];
    }
  }
  const double Tdot = (g.sum(FH) - g.sum(hdot)) / rcp;
  cpdot = g.sum(cpdot);
  for (int l = tid; l < n; l += TS) {
    const double* col = Js + l * ld;
    double sum = 0.0;
    double extra = 0.0;
    if (l < N) {
      for (int k = 0; k < N; ++k) sum += hm[k] * (col[k] + u[k]);
      sum *= __ldg(m.inv_mw + l);
    } else {
      for (int k = 0; k < N; ++k) sum += hm[k] * col[k];
      extra = cpdot + Tdot * drcp;
    }
    // Tdot * cp of the column's species: the lane that holds species l has it
    tr[l] = -(sum + extra) / rcp;
  }
  sync();
  if (tid < 32) {
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      const int l = lane + 32 * c;
      if (l < N) tr[l] -= Tdot * cpk[c] / rcp;
    }
  }
  sync();
  constexpr int G = ctrl_group(n), JB = n / kVJ;
  static_assert(n % kVJ == 0, "no column padding in J");
#pragma unroll
  for (int cc = 0; cc < (n + G - 1) / G; ++cc) {
    const int rows = (n - cc * G < G) ? n - cc * G : G;
    double2* dst = reinterpret_cast<double2*>(J + mat_vec<n, G, kVJ>(cc, 0, 0));
    for (int t = tid; t < rows * JB; t += TS) {
      const int jb = t / rows, i = cc * G + t % rows;
      double v[kVJ];
#pragma unroll
      for (int e = 0; e < kVJ; ++e) {
        const int j = jb * kVJ + e;
        if (i == N) v[e] = tr[j];
        else if (j < N) v[e] = (Js[j * ld + i] + u[i]) * __ldg(m.mw + i) * __ldg(m.inv_mw + j);
        else v[e] = Js[j * ld + i] * __ldg(m.mw + i);
      }
      dst[t] = make_double2(v[0], v[1]);
    }
  }
  sync();
}

// Jacobian refresh for the cells of the setup list whose matrix CVODE's
// jbad rule marks stale: the analytic FP64 Jacobian into the cell record.
// Minimum resident CTAs (of 128 threads) per SM requested for the Jacobian
// kernel (bounds its registers per thread).
#ifndef B200_JAC_MIN_CTAS
#define B200_JAC_MIN_CTAS 5
#endif

template <int NS>
__global__ void __launch_bounds__(128, B200_JAC_MIN_CTAS) rk_jac(RoundsParams R) {
  constexpr int n = NS + 1, CPL = (n + 31) / 32, W = jac_warps(n), ld = jac_ld(n);
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ DevMech s_mech;
  if (threadIdx.x == 0) s_mech = R.P.mech;
  __syncthreads();
  const int cnt = *R.cnt_in;
  if ((long long)blockIdx.x * (4 / W) >= cnt) return;
  const RoundsSetupLayout& SL = R.SL;
  const int team = threadIdx.x / (32 * W), tid = threadIdx.x % (32 * W), lane = tid & 31;
  const int gt = blockIdx.x * (4 / W) + team, nteams = gridDim.x * (4 / W);
  double* d = reinterpret_cast<double*>(dsm + (size_t)team * SL.jac_smem_per_team);
  GrpScratch ms;
  ms.C = d;
  ms.gRT = d + SL.Npad;
  ms.hRT = d + 2 * SL.Npad;
  ms.q = ms.r1 = ms.r2 = ms.r3 = ms.r4 = nullptr;
  double* hm = d + 3 * SL.Npad;
  double* Js = d + 4 * SL.Npad;
  double* D = SL.jac_d_global ? reinterpret_cast<double*>(R.wscratch) + (size_t)gt * SL.jac_nd : Js + n * ld + 2 * NS + n;
  for (int e = tid; e < n * ld + 2 * NS; e += 32 * W) Js[e] = 0.0;
  const RLayout RL = R.S.L;
  for (int idx = gt; idx < cnt; idx += nteams) {
    const int slot = R.list_in[idx];
    unsigned char* rec = rec_of(R.S, slot);
    // the cells were chosen by CVODE's jbad rule at their prediction, which
    // already counted the refresh
    const RVec<n> v{reinterpret_cast<double*>(rec + RL.off_vec)};
    Vec<CPL> y, F;
#pragma unroll
    for (int cc = 0; cc < CPL; ++cc) {
      const int i = lane + 32 * cc;
      y.v[cc] = (i < n) ? v.yev(i) : 0.0;
      F.v[cc] = (i < n) ? v.F(i) : 0.0;
    }
    team_jac<n, CPL, W>(s_mech, ms, hm, Js, D, y, F, reinterpret_cast<double*>(rec + RL.off_j), tid);
  }
}

// Minimum resident CTAs (of 128 threads) per SM requested for the inversion
// kernel (bounds its registers per thread): 4 for the lane groups (three rows
// of 22 FP32 entries per lane), 6 for one row per lane, 2 for two rows.
#ifndef B200_GJ_MIN_CTAS
#define B200_GJ_MIN_CTAS 4
#endif
template <int n, typename LUT>
constexpr bool gj_by_groups() { return n <= 32 && sizeof(LUT) == 4; }
template <int n, typename LUT>
constexpr int gj_min_ctas() { return gj_by_groups<n, LUT>() ? B200_GJ_MIN_CTAS : n <= 32 ? 6 : 2; }

// Bookkeeping of a setup in the cell's scalars.
__device__ __forceinline__ void gj_done(RCell* cp, double gamma, int ier) {
  cp->cnt.nlu++;
  cp->gamma_lu = gamma;
  cp->gamrat = 1.0;
  cp->gammap = gamma;
  cp->crate = 1.0;
  cp->nstlp = cp->cnt.nst;
  cp->setup_ier = ier;
}

// Newton-matrix inverse of the cells of the setup list: Gauss-Jordan inverse
// of D (I - gamma J) D^-1 with D = diag(ewt) (FP32) or of I - gamma J (FP64),
// written into the cell record.  One warp per cell, or (n <= 32 in FP32) the
// lane groups of the step kernel, whose rows are the ones it reads and writes.
template <int NS, typename LUT>
__global__ void __launch_bounds__(128, gj_min_ctas<NS + 1, LUT>()) rk_gj(RoundsParams R) {
  constexpr int n = NS + 1;
  constexpr int WCPL = (n + 31) / 32;  // rows per lane of the warp forms
  extern __shared__ __align__(16) unsigned char dsm[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const RoundsSetupLayout& SL = R.SL;
  const int cnt = *R.cnt_in;
  const RLayout RL = R.S.L;
  const int gw = blockIdx.x * (blockDim.x >> 5) + w;
  const int nwarps = gridDim.x * (blockDim.x >> 5);
  if constexpr (gj_by_groups<n, LUT>()) {
    constexpr int G = ctrl_group(n), GPW = 32 / G, CPL = (n + G - 1) / G;
    const int gl = lane % G, gi = lane / G;
    double* rds = reinterpret_cast<double*>(dsm + (size_t)(threadIdx.x / G) * gj_cell_bytes(n));
    float* Xs = reinterpret_cast<float*>(rds + n);
    int* prow = reinterpret_cast<int*>(Xs + (n * (n | 1) + 3) / 4 * 4);
    int* pinv = prow + n;
    for (int base = gw * GPW; base < cnt; base += nwarps * GPW) {
      const bool live = base + gi < cnt;
      unsigned char* rec = rec_of(R.S, live ? R.list_in[base + gi] : 0);
      RCell* cp = reinterpret_cast<RCell*>(rec);
      const RVec<n> v{reinterpret_cast<double*>(rec + RL.off_vec)};
      const double gamma = live ? cp->gamma : 0.0;
      double di[CPL];
#pragma unroll
      for (int cc = 0; cc < CPL; ++cc) {
        const int i = gl + G * cc;
        di[cc] = (live && i < n) ? v.ewt(i) : 1.0;
        if (live && i < n) v.dsc(i) = di[cc];
      }
      const int ier = grp_reg_gj_inverse<n, G>(reinterpret_cast<const double*>(rec + RL.off_j), live, di, rds, gamma,
                                               Xs, prow, pinv, reinterpret_cast<float*>(rec + RL.off_a), gl);
      if (live && gl == 0) gj_done(cp, gamma, ier);
    }
  } else {
    unsigned char* sb = dsm + (size_t)w * SL.gj_smem_per_warp;
    double* Dsc = reinterpret_cast<double*>(sb);
    LUT* A = reinterpret_cast<LUT*>(Dsc + SL.Npad);
    LUT* fcol = A + (size_t)n * SL.ldl;
    int* ipiv = reinterpret_cast<int*>(fcol + SL.Npad);
    int* ipiv2 = ipiv + SL.Npad;
    for (int idx = gw; idx < cnt; idx += nwarps) {
      const int slot = R.list_in[idx];
      unsigned char* rec = rec_of(R.S, slot);
      RCell* cp = reinterpret_cast<RCell*>(rec);
      const RVec<n> v{reinterpret_cast<double*>(rec + RL.off_vec)};
      const double* J = reinterpret_cast<const double*>(rec + RL.off_j);
      LUT* Ar = reinterpret_cast<LUT*>(rec + RL.off_a);
      const double gamma = cp->gamma;
#pragma unroll
      for (int cc = 0; cc < WCPL; ++cc) {
        const int i = lane + 32 * cc;
        if (i < n) {
          const double ds = (sizeof(LUT) == 4) ? v.ewt(i) : 1.0;
          Dsc[i] = ds;
          v.dsc(i) = ds;
        }
      }
      __syncwarp();
      int ier;
      if constexpr (WCPL == 1) {
        ier = reg_gj_inverse<n>(J, gamma, A, SL.ldl, ipiv, ipiv2, Ar, lane);
      } else if constexpr (WCPL == 2 && sizeof(LUT) == 4) {
        ier = reg_gj_inverse2<n>(J, Dsc, gamma, A, SL.ldl, ipiv, ipiv2, Ar, lane);
      } else {
        static_assert(sizeof(LUT) == 8, "the unscaled matrix");
        constexpr int G = ctrl_group(n);
        for (int e = lane; e < n * n; e += 32) {
          const int i = e / n, j = e % n;
          A[i * SL.ldl + j] = ((i == j) ? 1.0 : 0.0) - gamma * J[mat_idx<n, G, kVJ>(i, j)];
        }
        __syncwarp();
        ier = grp_gj_eliminate<32, LUT>(A, SL.ldl, ipiv, fcol, n, lane);
        __syncwarp();
        if (ier == 0)
          for (int i = lane; i < n; i += 32) store_inverse_row<n, LUT>(A + i * SL.ldl, nullptr, Ar, i);
      }
      __syncwarp();
      if (lane == 0) gj_done(cp, gamma, ier);
      __syncwarp();
    }
  }
}

// ------------------------------------------------------------ host side
namespace {

// Most shared memory of a Jacobian CTA that keeps two of them on an SM; the
// teams' parts are rounded up to 16 bytes each.
constexpr int kJacSmemCta = 100 * 1024, kJacSmemMax = kJacSmemCta + 4 * 16;

// The limit of dynamic shared memory is a property of the function and not of a
// handle: it is what any mechanism of this species count may need, so that
// handles of different mechanisms do not take it from one another.
template <int NS, typename LUT>
cudaError_t rounds_setup_attrs(const RoundsSetupLayout& SL) {
  constexpr int n = NS + 1;
  cudaError_t e = cudaFuncSetAttribute(rk_jac<NS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kJacSmemMax);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(rk_step<NS, LUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, step_smem<n>());
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(rk_gj<NS, LUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              4 * SL.gj_smem_per_warp);
}

template <int NS, typename LUT>
cudaError_t rounds_grids(int R, int gen, const RoundsSetupLayout& SL, int sm_count, RoundsGrids* G) {
  constexpr int n = NS + 1;
  cudaError_t e = rounds_setup_attrs<NS, LUT>(SL);
  if (e != cudaSuccess) return e;
  int b = 0;
  if ((e = rhs_grid(NS, R, gen, sm_count, &G->rhs)) != cudaSuccess) return e;
  G->rhs_by_warp = 0;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, rk_step<NS, LUT>, 128, step_smem<n>())) !=
      cudaSuccess)
    return e;
  G->step = std::max(1, b) * sm_count;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, rk_ctrl<NS>, 128, 0)) != cudaSuccess) return e;
  G->ctrl = std::max(1, b) * sm_count;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, rk_jac<NS>, 128, SL.jac_smem)) !=
      cudaSuccess)
    return e;
  G->jac = std::max(1, b) * sm_count;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, rk_gj<NS, LUT>, 128, 4 * SL.gj_smem_per_warp)) !=
      cudaSuccess)
    return e;
  G->gj = std::max(1, b) * sm_count;
  G->start = 4 * sm_count;
  return cudaSuccess;
}

template <int NS, typename LUT>
cudaError_t rounds_launch_t(int what, const RoundsParams& R, const RoundsGrids& G, int pass, cudaStream_t st) {
  constexpr int n = NS + 1;
  switch (what) {
    case kRoundsStart:
      rk_start<NS><<<G.start, 128, 0, st>>>(R);
      break;
    case kRoundsRhs:
      return rhs_launch(NS, R, G.rhs_by_warp ? G.rhs.warp : G.rhs.thread, G.rhs_by_warp, st);
    case kRoundsStep:
      rk_step<NS, LUT><<<G.step, 128, step_smem<n>(), st>>>(R, pass);
      break;
    case kRoundsCtrl:
      rk_ctrl<NS><<<G.ctrl, 128, 0, st>>>(R);
      break;
    case kRoundsJac:
      rk_jac<NS><<<G.jac, 128, R.SL.jac_smem, st>>>(R);
      break;
    case kRoundsGj:
      rk_gj<NS, LUT><<<G.gj, 128, 4 * R.SL.gj_smem_per_warp, st>>>(R);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

}  // namespace

bool rounds_supported(int N) { return N == 9 || N == 21 || N == 53; }

RoundsSetupLayout rounds_setup_layout(int N, int lut_bytes, int jac_nd) {
  RoundsSetupLayout L;
  const int n = N + 1;
  L.Npad = ((n + 31) / 32) * 32;
  L.ldl = n | 1;
  // scratch of a Jacobian team; the reactions' derivatives move to device
  // memory where they would leave fewer than two CTAs on an SM (what is left,
  // 8 to 27 KB a CTA, fits)
  const int teams = 4 / jac_warps(n);
  const long long fixed = 8LL * (4 * L.Npad + n * jac_ld(n) + 2 * N + n), dbytes = 8LL * jac_nd;
  L.jac_nd = jac_nd;
  L.jac_d_global = teams * (fixed + dbytes) > kJacSmemCta;
  L.jac_smem_per_team = (int)((fixed + (L.jac_d_global ? 0 : dbytes) + 15) & ~15LL);
  L.jac_smem = teams * L.jac_smem_per_team;
  L.gbytes_per_cta = L.jac_d_global ? teams * dbytes : 0;
  long long b = 8LL * L.Npad + (long long)lut_bytes * ((long long)n * L.ldl + L.Npad) + 4LL * 2 * L.Npad;
  if (n <= 32 && lut_bytes == 4) b = 32LL / ctrl_group(n) * gj_cell_bytes(n);
  L.gj_smem_per_warp = (int)((b + 15) & ~15LL);
  return L;
}

long long rounds_state_bytes_per_cell(int N, int lut_bytes) {
  return rounds_record_layout(N + 1, lut_bytes).stride + 4LL * kRoundSlotLists;  // record + slot lists
}

RState rounds_carve(void* base, long long cap, int N, int lut_bytes) {
  RState S;
  S.rec = static_cast<unsigned char*>(base);
  S.L = rounds_record_layout(N + 1, lut_bytes);
  S.cap = cap;
  return S;
}

cudaError_t rounds_grids_for(int N, int R, int gen, int lut_bytes, const RoundsSetupLayout& SL, int sm_count,
                             RoundsGrids* G) {
  if (N == 9)
    return lut_bytes == 4 ? rounds_grids<9, float>(R, gen, SL, sm_count, G) : rounds_grids<9, double>(R, gen, SL, sm_count, G);
  if (N == 21)
    return lut_bytes == 4 ? rounds_grids<21, float>(R, gen, SL, sm_count, G)
                          : rounds_grids<21, double>(R, gen, SL, sm_count, G);
  if (N == 53)
    return lut_bytes == 4 ? rounds_grids<53, float>(R, gen, SL, sm_count, G)
                          : rounds_grids<53, double>(R, gen, SL, sm_count, G);
  return cudaErrorInvalidValue;
}

cudaError_t rounds_launch(int N, int lut_bytes, int what, const RoundsParams& R, const RoundsGrids& G, int pass,
                          cudaStream_t st) {
  if (N == 9)
    return lut_bytes == 4 ? rounds_launch_t<9, float>(what, R, G, pass, st)
                          : rounds_launch_t<9, double>(what, R, G, pass, st);
  if (N == 21)
    return lut_bytes == 4 ? rounds_launch_t<21, float>(what, R, G, pass, st)
                          : rounds_launch_t<21, double>(what, R, G, pass, st);
  if (N == 53)
    return lut_bytes == 4 ? rounds_launch_t<53, float>(what, R, G, pass, st)
                          : rounds_launch_t<53, double>(what, R, G, pass, st);
  return cudaErrorInvalidValue;
}

}  // namespace b200
