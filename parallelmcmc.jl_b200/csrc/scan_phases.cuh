// scan_phases.cuh -- the two phases that the chunked scans share (affine_scan_kernel in
// tape_scan.cu, lg_scan_kernel in logistic_sweep.cu): a thread's run of columns composed into
// one affine map, and one coordinate's state carried over the chunks by a warp.
//
// A composition starts from its first map, not from the identity: where a map is infinite
// (200^148 columns of growth overflow FP64), inf * 0 from the identity's offset would make
// NaN of states that the recurrence itself takes to infinity.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace pmcmc {

// (a, b) of n consecutive columns, `stride` apart, kLoads of them in flight.
template <typename Real, int kLoads>
__device__ __forceinline__ void scan_compose_run(const Real* pa, const Real* pb, int n, int stride,
                                                 Real& a, Real& b) {
  a = 1, b = 0;
  for (bool first = true; n > 0; n -= kLoads, pa += kLoads * stride, pb += kLoads * stride) {
    Real va[kLoads], vb[kLoads];
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
      va[k] = k < n ? pa[k * stride] : Real(1);
      vb[k] = k < n ? pb[k * stride] : Real(0);
    }
    b = first ? vb[0] : va[0] * b + vb[0];
    a = first ? va[0] : va[0] * a;
    first = false;
#pragma unroll
    for (int k = 1; k < kLoads; ++k)
      if (k < n) {
        b = va[k] * b + vb[k];
        a = va[k] * a;
      }
  }
}

// The maps of a chunk's earlier runs, composed (sub > 0); s_a, s_b hold run j's at
// j * blk_d + dl.
template <typename Real>
__device__ __forceinline__ void scan_earlier_runs(const Real* s_a, const Real* s_b, int blk_d,
                                                  int dl, int sub, Real& ea, Real& eb) {
  ea = s_a[dl], eb = s_b[dl];
  for (int j = 1; j < sub; ++j) {
    const Real aj = s_a[j * blk_d + dl], bj = s_b[j * blk_d + dl];
    eb = aj * eb + bj;
    ea = aj * ea;
  }
}

// State of coordinate dd entering every chunk (into carry), from `st` entering the first; one
// warp: each lane composes `group` chunks, the lanes' maps are applied to the state in turn
// and each lane replays its group.  w_a, w_b: the warp's 32 entries of shared memory.  Returns
// the state that leaves the last chunk.
template <typename Real, int kG>
__device__ __forceinline__ Real scan_carry(int nch, int group, const Real* agg_a,
                                           const Real* agg_b, int64_t D, int64_t dd, Real st,
                                           Real* carry, Real* w_a, Real* w_b) {
  const int lane = threadIdx.x & 31;
  for (int base = 0; base < nch; base += 32 * group) {
    const int j0 = base + lane * group;
    Real ra[kG], rb[kG];
#pragma unroll
    for (int k = 0; k < kG; ++k) {
      const bool in = k < group && j0 + k < nch;
      ra[k] = in ? __ldcg(agg_a + (j0 + k) * D + dd) : Real(1);
      rb[k] = in ? __ldcg(agg_b + (j0 + k) * D + dd) : Real(0);
    }
    Real ga = ra[0], gb = rb[0];
#pragma unroll
    for (int k = 1; k < kG; ++k)
      if (k < group && j0 + k < nch) {
        gb = ra[k] * gb + rb[k];
        ga = ra[k] * ga;
      }
    __syncwarp();
    w_a[lane] = ga;
    w_b[lane] = gb;
    __syncwarp();
    Real mine = st;  // state entering this lane's group
#pragma unroll 8
    for (int l = 0; l < 32; ++l) {  // identity maps past the last group
      const Real al = w_a[l], bl = w_b[l];
      st = al * st + bl;
      if (l < lane) mine = st;
    }
#pragma unroll
    for (int k = 0; k < kG; ++k)
      if (k < group && j0 + k < nch) {
        carry[dd * nch + j0 + k] = mine;
        mine = ra[k] * mine + rb[k];
      }
  }
  return st;
}

}  // namespace pmcmc
