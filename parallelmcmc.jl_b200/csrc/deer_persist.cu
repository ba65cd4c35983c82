// deer_persist.cu -- a whole DEER solve of a Gaussian device target in one
// cooperative launch: tape, every Newton sweep and the verification pass.
//
// Same iteration as the per-sweep kernel (deer_sweep.cu, DEER.jl:553-581),
// restructured so that nothing between sweeps leaves the SM:
//  - CTA j owns the trajectory columns [t0, t0 + ncols) (t0 = j * TT) and keeps
//    them in shared memory from the first sweep to the last, together with
//    its tape (xi, log u) for columns t0 .. t0 + ncols, generated once.
//  - Its scan group is the columns t0 + 1 .. t0 + ncols.  Column t of the
//    Newton system depends on S_{t-1} only, so the group is evaluated from the
//    CTA's own columns (no halo from the neighbour).  The group's aggregate
//    maps S_{t0} to S_{t0 + ncols}, the first column of the next CTA.
//  - Column 0 depends on x0 alone: S_0 = f(x0) in every sweep; CTA 0 forms it
//    once and it seeds the scan over the group aggregates.
//  - Per sweep: evaluate and compose the group, grid barrier, the previous sweep's
//    convergence test (DEER.jl:567-578) read by every CTA alike, per-coordinate
//    scan of the group aggregates (state entering every CTA), grid barrier,
//    replay with damping in shared memory, max|dS| / max|S| atomics.  Testing a
//    sweep after the next sweep's first barrier saves a barrier a sweep; the
//    evaluation after the last sweep is discarded.  Sweep 0 is tested at once
//    after a third barrier, so a one-sweep solve evaluates once.
//  - After the last sweep every CTA verifies its columns (exact MALA step from
//    S_{t-1}, FP64 log-acceptance), writes S, logp(S_t) and the accept flags
//    (_trajectory_logps, interface.jl:517-524), as the finalize kernel does.
// The kernel is used when every CTA is co-resident (cooperative launch), the
// block has no sliding window and the target is a diagonal or dense Gaussian.
// Its parameters come by value in the launch, so a solve is one launch and
// the state readback.
#include <cuda_runtime.h>

#include <cstdint>

#include "deer_column.cuh"
#include "deer_device.cuh"
#include "deer_launch.h"
#include "persist_column.cuh"

namespace pmcmc {

// Shared memory: the sweep plan (columns, A, B, carry, dense-target vectors)
// followed by the CTA's tape, TT + 1 columns of xi (float) and log u (double).
template <typename Real>
__host__ __device__ inline PersistPlan plan_persist_smem(int64_t Dp, int TT, bool dense) {
  auto al = [](size_t x) { return (x + 15) & ~size_t(15); };
  PersistPlan p{};
  p.sweep = plan_sweep_smem<Real>(Dp, TT, dense);
  size_t off = al(p.sweep.total);
  p.xi = off;
  off = al(off + sizeof(float) * (TT + 1) * Dp);
  p.lu = off;
  off = al(off + sizeof(double) * (TT + 1));
  p.x0 = off;
  off = al(off + sizeof(Real) * Dp);
  p.tab = off;
  if (dense) off = al(off + sizeof(double) * Dp);
  else if (Dp <= 256) off = al(off + diag_tab_bytes<Real>(Dp));
  p.total = off;
  return p;
}

PersistPlan persist_smem(bool f64, int64_t Dp, int TT, bool dense) {
  return f64 ? plan_persist_smem<double>(Dp, TT, dense) : plan_persist_smem<float>(Dp, TT, dense);
}

// State entering every CTA (column t0 of CTA j), from the group aggregates: one warp a
// coordinate.  Each lane composes kCarryGroup groups, the lanes' maps are applied to the state in
// turn, and each lane replays its groups (the same association in every run).  One
// warp instead of a CTA needs no CTA barrier, and its first maps are loaded ahead of the
// convergence test: 3.3 -> 2.7 us a sweep with the test at 293 CTAs.
constexpr int kCarryGroup = 10;
template <typename Real>
struct CarryMaps {
  Real a[kCarryGroup], b[kCarryGroup];
  // this lane's groups j0 .. j0 + grp - 1 (identity past the last)
  __device__ __forceinline__ void load(int n, int grp, int j0, int d, int Dp, const Real* agg_a,
                                       const Real* agg_b) {
#pragma unroll
    for (int k = 0; k < kCarryGroup; ++k) {
      const bool in = k < grp && j0 + k < n;
      a[k] = in ? __ldcg(agg_a + static_cast<size_t>(j0 + k) * Dp + d) : Real(1);
      b[k] = in ? __ldcg(agg_b + static_cast<size_t>(j0 + k) * Dp + d) : Real(0);
    }
  }
};
__device__ __forceinline__ int carry_group(int n) { return min(kCarryGroup, (n + 31) / 32); }
// m holds the maps of the first 32 grp groups, loaded ahead.
template <typename Real>
__device__ __forceinline__ void carry_warp(int n, int d, int Dp, const Real* agg_a,
                                           const Real* agg_b, Real s, Real* incl, Real* wa,
                                           Real* wb, CarryMaps<Real>& m) {
  const int lane = threadIdx.x & 31;
  const int grp = carry_group(n);
  for (int base = 0; base < n; base += 32 * grp) {
    const int j0 = base + lane * grp;
    if (base > 0) m.load(n, grp, j0, d, Dp, agg_a, agg_b);
    Real a = 1, b = 0;
#pragma unroll
    for (int k = 0; k < kCarryGroup; ++k)
      if (k < grp && j0 + k < n) {
        b = m.a[k] * b + m.b[k];
        a = m.a[k] * a;
      }
    __syncwarp();
    wa[lane] = a;
    wb[lane] = b;
    __syncwarp();
    Real mine = s;  // state entering this lane's groups
#pragma unroll 8
    for (int l = 0; l < 32; ++l) {
      const Real al = wa[l], bl = wb[l];
      s = al * s + bl;
      if (l < lane) mine = s;
    }
#pragma unroll
    for (int k = 0; k < kCarryGroup; ++k)
      if (k < grp && j0 + k < n) {
        incl[static_cast<size_t>(j0 + k) * Dp + d] = mine;
        mine = m.a[k] * mine + m.b[k];
      }
  }
}

// Two CTAs per SM (at most 128 registers a thread) where that costs few spills: FP32 state
// with up to two quads a lane, FP64 with one on a diagonal target.  Dense targets above 64
// coordinates take one CTA an SM whatever the precision: the loads of P that their products
// keep in flight spill under 128 registers (FP32, D = 128, T = 1024: 76 us a sweep, 46 without;
// D = 256: 234 and 132), and their columns and P leave no more room for a second CTA's columns
// than one has.  kTwo asks for two all the
// same (persist_two_tile in capi.cu says where).
template <typename Real, int TK, int QPL, int LPC, bool kTwo>
constexpr int kPersistMinBlocks =
    kTwo || (sizeof(Real) * QPL <= 8 && !(TK == kDenseGauss && (sizeof(Real) == 8 || LPC == 32)))
        ? 2
        : 1;

// Columns of a diagonal target are evaluated by LPC lanes each (32 / LPC columns per
// warp), those of a dense one by a warp, LPC lanes for its quads and the rest for shares of
// the sums over the coordinates; QPL quads per lane cover Dp / 4 <= LPC * QPL.
template <typename Real, int TK, int JAC, int QPL, int LPC, bool kTwo, bool kTables>
__global__ void __launch_bounds__(kThreads, kPersistMinBlocks<Real, TK, QPL, LPC, kTwo>)
    deer_persist_kernel(const DevParams Pv, DevState* __restrict__ st) {
  __shared__ DevParams P;
  __shared__ Real s_sa[kThreads], s_sb[kThreads];
  __shared__ double s_red[3][kWarps];
  __shared__ unsigned long long s_acc[kWarps];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (threadIdx.x == 0) P = Pv;  // parameters by value: no upload before the launch
  __syncthreads();
  // One CTA (small blocks): its own barrier.  A wait that gives up is noted in grid_bar[1],
  // which every CTA's stop test and the final state read: the phases pair wrongly from there
  // on, but each wait ends at its bound and no result leaves without the timeout status.
  auto all_sync = [&]() {
    if (gridDim.x == 1) __syncthreads();
    else grid_barrier_noted(P.grid_bar, gridDim.x);
  };
  const uint32_t* const note = P.grid_bar + 1;
  auto timed_out = [&]() { return __ldcg(note) != 0u; };
  // this sweep's maxima max|dS|, max|S| and the non-finite flag, as ordered
  // bits of non-negative doubles, in two slots by sweep parity (P.part[0..5])
  unsigned long long* red = reinterpret_cast<unsigned long long*>(P.part);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr bool kDense = TK == kDenseGauss;
  constexpr bool kWhole = kTwo || kWholeColumn<Real, TK, JAC, QPL>;
  constexpr int CPW = kDense ? 1 : 32 / LPC;          // columns per warp
  const int lq = lane & (LPC - 1);                    // quad lane
  const int half = kDense ? 0 : lane / LPC;           // column slot
  const bool stores = !kDense || lane < LPC;          // of several lanes with the same quad
  const int cta = static_cast<int>(blockIdx.x), nctas = static_cast<int>(gridDim.x);
  const int TT = P.tile_cols;
  const int D = static_cast<int>(P.D), Dp = static_cast<int>(P.Dp);
  const int64_t T = P.T;
  const int64_t t0 = static_cast<int64_t>(cta) * TT;
  const int ncols = static_cast<int>(imin64(TT, T - t0));  // >= 1: one CTA per tile
  const bool has_next = t0 + ncols < T;
  const int ng = has_next ? ncols : ncols - 1;  // columns of the scan group
  Smem<Real> sm = carve<Real>(smem_raw, P, TT, kDense, !kWhole);
  const PersistPlan pp = plan_persist_smem<Real>(Dp, TT, kDense);
  float* xis = reinterpret_cast<float*>(smem_raw + pp.xi);
  double* lus = reinterpret_cast<double*>(smem_raw + pp.lu);
  Real* agg_a = static_cast<Real*>(P.agg_a);
  Real* agg_b = static_cast<Real*>(P.agg_b);
  Real* incl = static_cast<Real*>(P.incl);
  Real* carry0 = incl + static_cast<size_t>(nctas) * Dp;  // S_0 = f(x0)
  Real* Sb = static_cast<Real*>(P.S[0]);                   // last column of every CTA

  Real* x0s = reinterpret_cast<Real*>(smem_raw + pp.x0);
  DiagTab<Real> tab{};
  [[maybe_unused]] double* mud = reinterpret_cast<double*>(smem_raw + pp.tab);
  constexpr bool kTab = kTables && QPL <= 2;
  if constexpr (kDense)
    for (int d = tid; d < Dp; d += kThreads) mud[d] = d < D ? P.mean_d[d] : 0.0;
  if constexpr (!kDense && kTab) tab = fill_diag_tab<Real>(smem_raw + pp.tab, P);
  const int nblk = P.nblk > 1 ? static_cast<int>(P.nblk) : 1;
  for (int bi = 0; bi < nblk; ++bi) {  // blocks of one call, back to back
    const int64_t ncols_out = bi + 1 < nblk ? T : P.ncols_out;
    Real* const S_out = static_cast<Real*>(P.S_out) + static_cast<size_t>(bi) * T * D;
    Real* const logp_out =
        P.logp_out ? static_cast<Real*>(P.logp_out) + static_cast<size_t>(bi) * T : nullptr;
    uint8_t* const accept_out = P.accept_out ? P.accept_out + static_cast<size_t>(bi) * T : nullptr;
    DevState* const st_host = P.st_host ? P.st_host + bi : nullptr;
    // totals of the verification pass, folded in by every CTA as it finishes,
    // the arrival counter and the sweep maxima (the grid barriers in between
    // order these resets before every update, and after the previous block's reads)
    if (cta == 0 && tid == 0) {
      for (int i = 0; i < 6; ++i) red[i] = 0ull;
      st->fin_counter = 0;
      st->n_accept = 0;
      st->min_margin_bits = dbits(INFINITY);
      st->max_defect_bits = 0;
    }
    // start state, zero-padded to Dp: the call's x0, or the previous block's last
    // column; loaded here, stored to shared memory after the tape work below
    const Real* x0src = static_cast<const Real*>(bi > 0 ? P.x_next : P.x0_src ? P.x0_src : P.x0);
    const Real x0r = tid < D ? x0src[tid] : Real(0);

    // ---- tape (interface.jl:334-358) of the CTA's columns, drawn once a block ----
    const TapeKey key(P.seed, P.block + static_cast<uint64_t>(bi));
    // the tape of columns t0 .. t0 + ng (the CTA's own and its scan group's), one
    // (column, quad) pair a thread at a time: every lane busy, however D splits
    {
      const int nq = Dp / 4;
      for (int i = tid; i < (ng + 1) * nq; i += kThreads) {
        const int c = i / nq, q = i - c * nq;
        float n[4];
        tape_xi4(key, static_cast<uint32_t>(q), static_cast<uint32_t>(t0 + c + P.t_off), n);
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (4 * q + e >= D) n[e] = 0.f;
        store4(xis + c * Dp + 4 * q, n);
      }
    }
    for (int d = tid; d < Dp; d += kThreads)
      x0s[d] = d == tid ? x0r : d < D ? x0src[d] : Real(0);
    __syncthreads();
    // log u - 0.5 |xi|^2 of the columns t0 .. t0 + ng (the CTA's own and its scan
    // group's), in FP64, one column a thread: what the evaluation compares its part of
    // log alpha with
    for (int c = tid; c <= ng; c += kThreads) {
      double h = 0.0;  // (kWhole: log alpha has the tape term itself)
      const float* n = xis + c * Dp;
#pragma unroll 4
      for (int d = 0; d < (kWhole ? 0 : Dp); d += 4) {
        float v[4];
        load4(n + d, v);
#pragma unroll
        for (int e = 0; e < 4; ++e) h = fma(static_cast<double>(v[e]), static_cast<double>(v[e]), h);
      }
      lus[c] = log(static_cast<double>(tape_u(key, static_cast<uint32_t>(t0 + c + P.t_off)))) - 0.5 * h;
    }
    for (int i = tid; i < ncols * (Dp / 4); i += kThreads) {
      const int nq = Dp / 4, c = i / nq, k = 4 * (i - c * nq);
      Real v[4];
      load4(x0s + k, v);
      store4(sm.Xs + c * Dp + k, v);
    }

    __syncthreads();

    // ---- S_0 = f(x0): the same in every sweep ----
    if (cta == 0 && warp == 0) {  // every column slot of warp 0 forms it; slot 0 stores
      Col<Real, QPL> col;
      if constexpr (kWhole) {
        persist_forward_whole<Real, QPL>(P, sm, key, x0s, xis, col);
      } else if constexpr (kDense) {
        Real z[QPL][4], w[QPL][4], hv[QPL][4];
        persist_forward_dense<Real, JAC, QPL, LPC, false>(P, sm, mud, key, x0s, xis, 0, 0, col, z, w, hv);
      } else {
        persist_forward_diag<Real, QPL, LPC, JAC == kJacDiag, kTab>(P, tab, x0s, xis, col);
      }
      const bool acc = lus[0] < seg_sum<LPC>(col.la);
#pragma unroll
      for (int q = 0; q < QPL; ++q) {
        const int j = lq + LPC * q;
        if (lane < LPC && 4 * j < D) {
          Real f[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            f[e] = 4 * j + e < D ? (acc ? col.y[q][e] : col.x[q][e]) : Real(0);
          store4(carry0 + 4 * j, f);
        }
      }
    }

    const Real dmp = static_cast<Real>(P.damping), omd = static_cast<Real>(1.0 - P.damping);
    const Real big = sizeof(Real) == 4 ? Real(3.402823466e+38f) : Real(1.7976931348623157e308);
    // runs of the scan: nsub runs of Ls columns a coordinate (above 256 coordinates: one run,
    // several coordinates a thread)
    constexpr bool kRuns = 4 * QPL * LPC <= kThreads;
    int nsub = 1, Ls = ng;
    if constexpr (kRuns) {
      nsub = max(1, min(min(kThreads / Dp, 8), ng));
      Ls = (ng + nsub - 1) / nsub;
      nsub = Ls > 0 ? max(1, (ng + Ls - 1) / Ls) : 1;
    }
    int iter = 0, converged = 0, status = 0;
    Real sprev = 0;
    double metric = 0.0;
    // the test of sweep k from its maxima (slot k & 1), after a grid barrier that
    // follows sweep k's apply; on a stop, S_{t0 - 1} (the previous CTA's last
    // column) is read for the verification
    auto stop_test = [&](int k) {
      const unsigned long long* sl = red + 3 * (k & 1);
      const unsigned long long b0 = __ldcg(sl), b1 = __ldcg(sl + 1), b2 = __ldcg(sl + 2);
      const bool late = nctas > 1 && timed_out();
      const double dmax = __longlong_as_double(static_cast<long long>(b0));
      const double smax = __longlong_as_double(static_cast<long long>(b1));
      const bool nonfinite = b2 != 0ull;
      metric = dmax / (P.tol_abs + P.tol_rel * smax);
      converged = metric <= 1.0;
      status = late        ? static_cast<int>(kStTimeout)
               : nonfinite ? static_cast<int>(kStNonfinite)
                           : 0;
      const bool stop = converged || iter >= P.maxiter || status != 0;
      if (stop && cta > 0 && tid < Dp) sprev = __ldcg(Sb + (t0 - 1) * Dp + tid);
      return stop;
    };
    for (;;) {
      // ---- evaluate the scan group: column t0 + c + 1 from S_{t0 + c} ----
      // (warp-uniform loop over groups of CPW columns; a slot past the end
      // repeats the group's first column and stores nothing).  The previous
      // sweep's convergence test comes after the next grid barrier, so this
      // evaluation runs before it is known whether another sweep is needed: a
      // solve of more than one sweep evaluates once more than it sweeps, and a
      // sweep has two grid barriers instead of three.  At maxiter nothing is
      // evaluated.
      const bool sweep = iter < P.maxiter;
      for (int cb = warp * CPW; sweep && cb < ng; cb += kWarps * CPW) {
        const bool valid = cb + half < ng;
        const int c = valid ? cb + half : cb;
        const int t = static_cast<int>(t0 + c + 1);
        const double logu = lus[c + 1];
        const float* xic = xis + (c + 1) * Dp;
        const Real* xcol = sm.Xs + c * Dp;
        Col<Real, QPL> col;
        Real A[QPL][4];
        bool acc;
        if constexpr (kWhole) {
          persist_forward_whole<Real, QPL>(P, sm, key, xcol, xic, col);
          col.la = seg_sum<LPC>(col.la);
          acc = logu < col.la;
          column_jacobian<Real, TK, JAC, QPL, LPC>(P, sm, key, t + P.t_off, iter, acc,
                                                   sigmoid_slope<Real>(col.la - logu), col, A);
        } else if constexpr (kDense) {
          Real z[QPL][4], w[QPL][4], hv[QPL][4];
          persist_forward_dense<Real, JAC, QPL, LPC, true>(P, sm, mud, key, xcol, xic,
                                                           t + P.t_off, iter, col, z, w, hv);
          col.la = seg_sum<LPC>(col.la);
          acc = logu < col.la;
          persist_jacobian_dense<Real, JAC, QPL, LPC>(P, sm, key, t + P.t_off, iter, acc,
                                                      sigmoid_slope<Real>(col.la - logu), col, z,
                                                      w, hv, A);
        } else {
          persist_forward_diag<Real, QPL, LPC, JAC == kJacDiag, kTab>(P, tab, xcol, xic, col);
          col.la = seg_sum<LPC>(col.la);
          acc = logu < col.la;
          const Real gp = sigmoid_slope<Real>(col.la - logu);
          if constexpr (JAC == kJacDiag) {
#pragma unroll
            for (int q = 0; q < QPL; ++q)
#pragma unroll
              for (int e = 0; e < 4; ++e)
                A[q][e] = fma(gp, col.gx[q][e], acc ? Real(1) - col.gy[q][e] : Real(1));
          } else {
            column_jacobian<Real, TK, JAC, QPL, LPC>(P, sm, key, t + P.t_off, iter, acc, gp, col,
                                                     A);
          }
        }
#pragma unroll
        for (int q = 0; q < QPL; ++q) {
          const int j = lq + LPC * q;
          if (valid && stores && 4 * j < D) {
            Real a4[4], b4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              // (past D the state is zero, and stays zero under any A)
              const Real f = acc ? col.y[q][e] : col.x[q][e];
              a4[e] = A[q][e];
              b4[e] = f - A[q][e] * col.x[q][e];
            }
            store4(sm.As + c * Dp + 4 * j, a4);
            store4(sm.Bs + c * Dp + 4 * j, b4);
          }
        }
      }
      // ---- the group's map of every coordinate: runs of consecutive columns, one a
      // thread, composed and joined (the maps stay as they are for the replay below) ----
      Real ea = 1, eb = 0;  // this thread's earlier runs
      if (sweep) {
        __syncthreads();  // evaluated
        if constexpr (kRuns) {
          const int d = tid % Dp, sub = tid / Dp;
          // (the same trip count in every lane: runs of two lengths would diverge)
          const int g0 = sub * Ls, n = sub < nsub ? min(Ls, ng - g0) : 0;
          const Real *pa = sm.As + g0 * Dp + d, *pb = sm.Bs + g0 * Dp + d;
          Real a = 1, b = 0;
          for (int i = 0; i < Ls; i += 4, pa += 4 * Dp, pb += 4 * Dp) {
            Real va[4], vb[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              va[k] = i + k < n ? pa[k * Dp] : Real(1);
              vb[k] = i + k < n ? pb[k * Dp] : Real(0);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              b = va[k] * b + vb[k];
              a = va[k] * a;
            }
          }
          s_sa[tid] = a;
          s_sb[tid] = b;
          __syncthreads();
          for (int j = 0; j < sub; ++j) {
            const Real aj = s_sa[j * Dp + d], bj = s_sb[j * Dp + d];
            eb = aj * eb + bj;
            ea = aj * ea;
          }
          if (sub == nsub - 1 && nctas > 1) {
            agg_a[static_cast<size_t>(cta) * Dp + d] = a * ea;
            agg_b[static_cast<size_t>(cta) * Dp + d] = a * eb + b;
          }
        } else {  // more coordinates than threads: one run each
          for (int d = tid; d < Dp; d += kThreads) {
            Real a = 1, b = 0;
            for (int g = 0; g < ng; ++g) {
              const Real ag = sm.As[g * Dp + d], bg = sm.Bs[g * Dp + d];
              b = ag * b + bg;
              a = ag * a;
            }
            agg_a[static_cast<size_t>(cta) * Dp + d] = a;
            agg_b[static_cast<size_t>(cta) * Dp + d] = b;
          }
        }
      }
      all_sync();

      // ---- convergence test of the previous sweep (DEER.jl:567-578), the same in
      // every CTA: its maxima are complete, every CTA having applied it.  Sweep 0
      // was tested at once, after a barrier of its own (below) ----
      // (the maps of this warp's first coordinate are fetched beside the maxima)
      const int dw = warp * nctas + cta;
      Real s0w = 0;
      CarryMaps<Real> maps;
      if (nctas > 1 && dw < D) {
        maps.load(nctas, carry_group(nctas), lane * carry_group(nctas), dw, Dp, agg_a, agg_b);
        s0w = __ldcg(carry0 + dw);
      }
      if (iter >= 2 && stop_test(iter - 1)) break;
      // this sweep's slot was last read in the test of sweep iter - 2, which
      // every CTA finished before the previous sweep's second barrier: clear it
      // (the next barrier orders the clear before this sweep's atomics)
      if (cta == 0 && tid == 0)
        for (int i = 0; i < 3; ++i) red[3 * (iter & 1) + i] = 0ull;

      // ---- state entering every CTA: the group aggregates per coordinate ----
      if (nctas > 1) {
        for (int d = dw; d < D; d += kWarps * nctas) {
          if (d != dw) {
            maps.load(nctas, carry_group(nctas), lane * carry_group(nctas), d, Dp, agg_a, agg_b);
            s0w = __ldcg(carry0 + d);
          }
          carry_warp<Real>(nctas, d, Dp, agg_a, agg_b, s0w, incl, s_sa + 32 * warp,
                           s_sb + 32 * warp, maps);
        }
        all_sync();
      }

      // ---- apply: every thread replays its run from the state entering it; damping and
      // maxima (exact in the state's precision) ----
      Real my_dmax = 0, my_smax = 0;
      bool bad = false;
      const Real* in = nctas > 1 ? incl + static_cast<size_t>(cta) * Dp : carry0;
      // column c's value v from its Newton state s and its old value o
      auto damp = [&](Real s, Real o) {
        const Real v = omd * o + dmp * s;
        my_dmax = max(my_dmax, fabs(v - o));
        my_smax = max(my_smax, fabs(v));
        bad |= !(fabs(v) <= big);
        return v;
      };
      // n columns of coordinate d after column c0, from its state s; four columns' loads go
      // ahead of their stores
      auto replay = [&](int d, int c0, int n, Real s) {
        const Real *pa = sm.As + c0 * Dp + d, *pb = sm.Bs + c0 * Dp + d;
        Real* px = sm.Xs + (c0 + 1) * Dp + d;
        int i = 0;
        for (; i + 4 <= n; i += 4, pa += 4 * Dp, pb += 4 * Dp, px += 4 * Dp) {
          Real va[4], vb[4], vo[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) va[k] = pa[k * Dp], vb[k] = pb[k * Dp], vo[k] = px[k * Dp];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            s = va[k] * s + vb[k];
            px[k * Dp] = damp(s, vo[k]);
          }
        }
        for (; i < n; ++i, pa += Dp, pb += Dp, px += Dp) {
          s = *pa * s + *pb;
          *px = damp(s, *px);
        }
      };
      if constexpr (kRuns) {
        const int d = tid % Dp, sub = tid / Dp;
        const bool on = sub < nsub && d < D;
        const int c0 = sub * Ls, n = on ? min(Ls, ncols - 1 - c0) : 0;
        const Real cr = on ? __ldcg(in + d) : Real(0);
        if (on && sub == 0) sm.Xs[d] = damp(cr, sm.Xs[d]);
        __syncwarp();
        replay(d, c0, n, ea * cr + eb);
      } else {
        for (int d = tid; d < D; d += kThreads) {
          const Real cr = __ldcg(in + d);
          sm.Xs[d] = damp(cr, sm.Xs[d]);
          replay(d, 0, ncols - 1, cr);
        }
      }
      // this CTA's maxima into the sweep's slot (max is exact in any order; the
      // CTAs arrive spread over the apply phase, so the atomics rarely meet)
      my_dmax = warp_max(my_dmax);
      my_smax = warp_max(my_smax);
      bad = __any_sync(0xffffffffu, bad);
      if (lane == 0) {
        s_red[0][warp] = static_cast<double>(my_dmax);
        s_red[1][warp] = static_cast<double>(my_smax);
        s_red[2][warp] = bad ? 1.0 : 0.0;
      }
      __syncthreads();
      if (has_next)  // the next CTA's verification starts from this column
        for (int d = tid; d < Dp; d += kThreads)
          Sb[(t0 + ncols - 1) * Dp + d] = sm.Xs[(ncols - 1) * Dp + d];
      unsigned long long* slot = red + 3 * (iter & 1);
      if (tid == 0) {
        double a = 0, b = 0, c = 0;
        for (int w = 0; w < kWarps; ++w)
          a = max(a, s_red[0][w]), b = max(b, s_red[1][w]), c = max(c, s_red[2][w]);
        atomicMax(slot, dbits(a));
        atomicMax(slot + 1, dbits(b));
        if (c != 0.0) atomicMax(slot + 2, 1ull);
      }
      __syncwarp();  // warp 0 evaluates together again
      ++iter;
      // the first sweep is tested at once: a block that converges in one sweep
      // (no accepted move) then evaluates nothing more
      if (iter == 1) {
        all_sync();
        if (stop_test(0)) break;
      }
    }

    // ---- verification pass and outputs on the CTA's columns ----
    // S_{t0 - 1}, the previous CTA's last column, into shared memory
    for (int d = tid; d < Dp; d += kThreads)
      sm.carry[d] = cta == 0 ? x0s[d] : d == tid ? sprev : __ldcg(Sb + (t0 - 1) * Dp + d);
    // the CTA's rows of S_out (row t = column t, D entries) in one coalesced copy
    {
      const int64_t nrows = imin64(ncols, ncols_out - t0);
      if (nrows > 0) {
        Real* dst = S_out + t0 * D;
        const int64_t n = nrows * D;
        if (D == Dp && reinterpret_cast<uintptr_t>(dst) % (4 * sizeof(Real)) == 0) {
          for (int64_t i = tid; i < n / 4; i += kThreads) {
            Real v[4];
            load4(sm.Xs + 4 * i, v);
            store4(dst + 4 * i, v);
          }
        } else {
          for (int64_t i = tid; i < n; i += kThreads) {
            const int64_t r = i / D;
            dst[i] = sm.Xs[r * Dp + (i - r * D)];
          }
        }
      }
    }
    __syncthreads();
    unsigned long long nacc = 0;
    double min_margin = __longlong_as_double(0x7ff0000000000000ll), max_def = 0.0;
    for (int cb = warp * CPW; cb < ncols; cb += kWarps * CPW) {
      const bool valid = cb + half < ncols;
      const int c = valid ? cb + half : cb;
      const int64_t t = t0 + c;
      const Real* xcol = c == 0 ? sm.carry : sm.Xs + (c - 1) * Dp;
      const Real* scol = sm.Xs + c * Dp;
      Col<Real, QPL> col;
      // log alpha reduced below with the log density and the defect (one pass)
      if constexpr (kWhole) {
        persist_forward_whole<Real, QPL>(P, sm, key, xcol, xis + c * Dp, col);
      } else if constexpr (kDense) {
        Real z[QPL][4], w[QPL][4], hv[QPL][4];
        persist_forward_dense<Real, JAC, QPL, LPC, false>(P, sm, mud, key, xcol, xis + c * Dp,
                                                          static_cast<int>(t), 0, col, z, w, hv);
      } else {
        persist_forward_diag<Real, QPL, LPC, JAC == kJacDiag, kTab>(P, tab, xcol, xis + c * Dp, col);
      }
      const double logu = lus[c];
      const bool out = valid && t < ncols_out;
      // the recursion defect max|S_t - f_t| for both outcomes, selected after the
      // reductions (which then run alongside the log-density's)
      Real dx = 0, dy = 0;  // exact maxima
      double lp = 0.0;
      double* vd = kDense ? sm.Vd + warp * Dp : nullptr;
#pragma unroll
      for (int q = 0; q < QPL; ++q) {
        const int j = lq + LPC * q;
        if (4 * j < D) {
          Real s4[4];
          load4(scol + 4 * j, s4);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (4 * j + e >= D) continue;
            dx = max(dx, fabs(s4[e] - col.x[q][e]));
            dy = max(dy, fabs(s4[e] - col.y[q][e]));
            const double sd = static_cast<double>(s4[e]) - (kDense ? mud[4 * j + e] : P.mean_d[4 * j + e]);
            if constexpr (TK == kDiagGauss) lp += -0.5 * P.prec_d[4 * j + e] * sd * sd;
            else if (stores) vd[4 * j + e] = sd;
            if (out && stores && t == ncols_out - 1) static_cast<Real*>(P.x_next)[4 * j + e] = s4[e];
          }
        }
      }
      if constexpr (kDense) {
        __syncwarp();
        double o[QPL][4];
        Real none[QPL][4];
        dense_products<Real, QPL, LPC, true, false>(sm, D, Dp, o, none);
#pragma unroll
        for (int q = 0; q < QPL; ++q) {
          const int j = lq + LPC * q;
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (4 * j + e < D) lp += -0.5 * vd[4 * j + e] * o[q][e];
        }
        __syncwarp();
      }
#pragma unroll
      for (int o = LPC / 2; o > 0; o >>= 1) {
        col.la += __shfl_xor_sync(0xffffffffu, col.la, o);
        lp += __shfl_xor_sync(0xffffffffu, lp, o);
        dx = max(dx, __shfl_xor_sync(0xffffffffu, dx, o));
        dy = max(dy, __shfl_xor_sync(0xffffffffu, dy, o));
      }
      const bool acc = logu < col.la;
      if (valid && stores && lq == 0) {
        if (out) {
          if (logp_out) logp_out[t] = static_cast<Real>(lp);
          if (accept_out) accept_out[t] = acc ? 1 : 0;
        }
        nacc += acc ? 1 : 0;
        min_margin = min(min_margin, fabs(col.la - logu));
        max_def = max(max_def, static_cast<double>(acc ? dy : dx));
      }
    }
    // per warp: the column slots' totals
    nacc = warp_sum(nacc);
    max_def = warp_max(max_def);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      min_margin = min(min_margin, __shfl_xor_sync(0xffffffffu, min_margin, o));
    __syncthreads();  // s_red was last read in the convergence test
    if (lane == 0) {
      s_acc[warp] = nacc;
      s_red[0][warp] = min_margin;
      s_red[2][warp] = max_def;
    }
    __syncthreads();
    if (tid == 0) {
      unsigned long long a = 0;
      double mm = s_red[0][0], md = 0.0;
      for (int w = 0; w < kWarps; ++w) {
        a += s_acc[w];
        mm = min(mm, s_red[0][w]);
        md = max(md, s_red[2][w]);
      }
      // accepted count, smallest margin and largest defect into the totals
      // (margins and defects are non-negative: their bits order like the values,
      // and a NaN defect sorts above every number); the last CTA to arrive writes
      // the final state, the others leave without waiting at a grid barrier
      atomicAdd(&st->n_accept, a);
      atomicMin(&st->min_margin_bits, dbits(mm));
      atomicMax(&st->max_defect_bits, dbits(md));
      __threadfence();
      const bool last = atomicAdd(&st->fin_counter, 1u) == static_cast<unsigned>(nctas - 1);
      if (last) {
        __threadfence();

        // ---- last CTA: the final state ----
        const unsigned long long* tot = &st->n_accept;
        DevState f{};
        f.epoch = st->epoch;  // look-back epochs of the per-sweep path continue
        f.iter = iter;
        f.converged = converged;
        f.status = timed_out() ? static_cast<int>(kStTimeout) : status;
        f.metric = metric;
        f.n_accept = __ldcg(tot);
        f.min_margin_bits = __ldcg(&st->min_margin_bits);
        f.max_defect_bits = __ldcg(&st->max_defect_bits);
        *st = f;
        if (st_host) {
          *st_host = f;
          __threadfence_system();
        }
      }
    }
    // the next block starts from this block's last column (x_next) once every
    // CTA has finished this one.  After a wait that gave up, the note stops every CTA at a
    // stop test and here, and the states of the blocks that never ran keep the timeout status
    // that the host put there.
    if (bi + 1 < nblk) {
      if (status == static_cast<int>(kStTimeout)) break;
      all_sync();
    }
  }  // blocks
}

namespace {

template <typename Real, int TK, int JAC, int QPL, int LPC, bool kTwo = false, bool kTables = true>
const void* persist_fn() {
  return reinterpret_cast<const void*>(
      &deer_persist_kernel<Real, TK, JAC, QPL, LPC, kTwo, kTables>);
}

// Lanes a column: as many as it has quads, rounded up to a power of two, so that a small
// state fills the warp with columns (diagonal) or shares of its products (dense).
template <typename Real, int TK, int JAC, bool kTables>
const void* pick_persist(int64_t D) {
  if constexpr (TK == kDiagGauss) {
    if (D <= 4) return persist_fn<Real, TK, JAC, 1, 1, false, kTables>();
    if (D <= 8) return persist_fn<Real, TK, JAC, 1, 2, false, kTables>();
    if (D <= 16) return persist_fn<Real, TK, JAC, 1, 4, false, kTables>();
    if (D <= 32) return persist_fn<Real, TK, JAC, 1, 8, false, kTables>();
    if (D <= 64) return persist_fn<Real, TK, JAC, 1, 16, false, kTables>();
    if (D <= 128) return persist_fn<Real, TK, JAC, 2, 16, false, kTables>();
    if (D <= 256) return persist_fn<Real, TK, JAC, 2, 32, false, kTables>();
    return persist_fn<Real, TK, JAC, 4, 32>();
  } else {
    if (D <= 32) return persist_fn<Real, TK, JAC, 1, 8>();
    if (D <= 64) return persist_fn<Real, TK, JAC, 1, 16>();
    if (D <= 128) return persist_fn<Real, TK, JAC, 1, 32>();
    return D <= 256 ? persist_fn<Real, TK, JAC, 2, 32>() : persist_fn<Real, TK, JAC, 4, 32>();
  }
}

template <typename Real, bool kTables>
const void* pick_persist_t(int tk, int jac, int64_t D) {
  if (tk == kDiagGauss)
    return jac == kJacStoch ? pick_persist<Real, kDiagGauss, kJacStoch, kTables>(D)
                            : pick_persist<Real, kDiagGauss, kJacDiag, kTables>(D);
  return jac == kJacStoch ? pick_persist<Real, kDenseGauss, kJacStoch, kTables>(D)
                          : pick_persist<Real, kDenseGauss, kJacDiag, kTables>(D);
}

}  // namespace

const void* persist_kernel_two(bool f64, int tk, int jac, int64_t D) {
  if (tk != kDenseGauss || D <= 64) return nullptr;
  if (f64)
    return jac == kJacStoch || D > 128 ? nullptr
                                       : persist_fn<double, kDenseGauss, kJacDiag, 1, 32, true>();
  if (D > 256) return nullptr;
  if (jac == kJacStoch)
    return D <= 128 ? persist_fn<float, kDenseGauss, kJacStoch, 1, 32, true>()
                    : persist_fn<float, kDenseGauss, kJacStoch, 2, 32, true>();
  return D <= 128 ? persist_fn<float, kDenseGauss, kJacDiag, 1, 32, true>()
                  : persist_fn<float, kDenseGauss, kJacDiag, 2, 32, true>();
}

const void* persist_kernel(bool f64, int tk, int jac, int64_t D, bool tables) {
  if (tk != kDiagGauss && tk != kDenseGauss) return nullptr;
  if (tables)
    return f64 ? pick_persist_t<double, true>(tk, jac, D) : pick_persist_t<float, true>(tk, jac, D);
  return f64 ? pick_persist_t<double, false>(tk, jac, D)
             : pick_persist_t<float, false>(tk, jac, D);
}

}  // namespace pmcmc
