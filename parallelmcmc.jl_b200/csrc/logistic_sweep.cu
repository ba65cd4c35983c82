// logistic_sweep.cu -- the Newton sweep of the logistic target on the tensor-core path
// with one Hutchinson probe, after its two contraction passes: every column's affine map
// (lg_finish_kernel), then S_t = A_t .* S_{t-1} + B_t with damping and the convergence
// test (lg_scan_kernel; DEER.jl:398-475, 567-578).
//
// At T = 65536, D = 256 every array of a sweep (67 MB) is larger than its share of L2,
// so the sweep is bound by HBM, and each quantity is formed where it costs no array of
// its own: g_y and H(y) w go straight from the pass's G into A and B, log alpha and the
// near-tie list come from the same read.
#include <cuda_runtime.h>

#include <cstdint>

#include "deer_device.cuh"
#include "deer_launch.h"
#include "logistic.h"
#include "logistic_column.cuh"
#include "scan_phases.cuh"

namespace pmcmc {

// One warp a column (finish_column); lpy from the pass's parts.
template <int QPL>
__global__ void __launch_bounds__(kThreads)
    lg_finish_kernel(const DevParams* __restrict__ Pg, const DevState* __restrict__ st, PassG G,
                     const double* __restrict__ lp_parts, int np, double* __restrict__ la_ref,
                     TieList list, int guard) {
  __shared__ DevParams P;
  if (guard && solve_ended(st, Pg->maxiter)) return;
  load_params(Pg, P);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int iter = st->iter;
  const float* S = static_cast<const float*>(P.S[st->cur]);
  const float* x0 = static_cast<const float*>(P.x0);
  const TapeKey key(P.seed, P.block);
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * kWarps + warp; t < P.T;
       t += static_cast<int64_t>(gridDim.x) * kWarps) {
    double ly = 0.0;
    for (int p = 0; p < np; ++p) ly += lp_parts[p * P.T + t];
    const float* x = (iter == 0 || t == 0) ? x0 : S + (t - 1) * P.Dp;
    const double la = finish_column<QPL>(P, key, x, t, iter, G, ly - P.lpx[t], nullptr);
    if (lane == 0) {
      P.lpy[t] = ly;
      la_ref[t] = la;
      tie_note(list, t, la - P.logu[t]);
    }
  }
}

// The scan of affine_scan_kernel (tape_scan.cu) over one launch's columns [c_lo, c_hi),
// with the state S_new = (1 - damping) S_old + damping s written in place of s and its
// maxima taken.  `entry` holds the undamped state entering the launch's first column and
// gets the one leaving its last; the launch with the block's last column tests.
__global__ void __launch_bounds__(kThreads, 3)
    lg_scan_kernel(const DevParams* __restrict__ Pg, DevState* __restrict__ st, int64_t c_lo,
                   int64_t c_hi, ScanPlan pl, float* __restrict__ scratch,
                   float* __restrict__ entry, DevState* st_host) {
  __shared__ float s_a[kThreads], s_b[kThreads];
  __shared__ float s_red[2][kWarps];
  __shared__ int s_bad, s_last;
  const DevParams& P = *Pg;
  // (a launch after the sweep's first goes on whatever status that one set)
  if (c_lo == 0 && solve_ended(st, P.maxiter)) return;
  if (c_lo > 0 && (st->converged || st->iter >= P.maxiter)) return;
  constexpr int kLoads = 16, kG = 8;
  const int tid = threadIdx.x, lane = tid & 31;
  const int iter = st->iter, cur = st->cur;
  const int Dp = static_cast<int>(P.Dp);
  const int64_t T = c_hi - c_lo;
  const float* A = static_cast<const float*>(P.lg[3]) + c_lo * Dp;
  const float* B = static_cast<const float*>(P.lg[4]) + c_lo * Dp;
  const float* x0 = static_cast<const float*>(P.x0);
  const float* So = static_cast<const float*>(P.S[cur]) + c_lo * Dp;
  float* Sn = static_cast<float*>(P.S[cur ^ 1]) + c_lo * Dp;
  const int nch = pl.nchunks;
  float *agg_a = scratch, *agg_b = scratch + static_cast<size_t>(nch) * Dp,
        *carry = agg_b + static_cast<size_t>(nch) * Dp;
  const int db = static_cast<int>(blockIdx.x) % pl.nblk_d;
  const int ch = static_cast<int>(blockIdx.x) / pl.nblk_d;
  const int sub = tid / pl.blk_d, dl = tid - sub * pl.blk_d;
  const int d = db * pl.blk_d + dl;
  const bool active = sub < pl.nsub && d < Dp;
  const int64_t c0 = static_cast<int64_t>(ch) * pl.L, c1 = imin64(T, c0 + pl.L);
  const int64_t u0 = imin64(c1, c0 + static_cast<int64_t>(sub) * pl.Ls);
  const int64_t u1 = imin64(c1, u0 + pl.Ls);
  if (tid == 0) s_bad = 0;
  float a = 1.f, b = 0.f;
  if (active)
    scan_compose_run<float, kLoads>(A + u0 * Dp + d, B + u0 * Dp + d, static_cast<int>(u1 - u0),
                                    Dp, a, b);
  s_a[tid] = a;
  s_b[tid] = b;
  __syncthreads();
  float ea = 1.f, eb = 0.f;  // the chunk's earlier runs, composed
  if (active) {
    if (sub > 0) scan_earlier_runs<float>(s_a, s_b, pl.blk_d, dl, sub, ea, eb);
    if (sub == pl.nsub - 1) {
      agg_a[ch * Dp + d] = sub > 0 ? a * ea : a;
      agg_b[ch * Dp + d] = sub > 0 ? a * eb + b : b;
    }
  }
  const bool one = gridDim.x == 1;  // one chunk: its state is the entering one, no barrier
  if (!one && !grid_barrier(P.grid_bar, gridDim.x))
    atomicCAS(&st->status, 0, static_cast<int>(kStTimeout));
  for (int dd = one ? Dp : (tid >> 5) * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x); dd < Dp;
       dd += static_cast<int>(blockDim.x >> 5) * static_cast<int>(gridDim.x)) {
    const float s = scan_carry<float, kG>(nch, pl.group, agg_a, agg_b, Dp, dd,
                                          c_lo ? __ldcg(entry + dd) : x0[dd], carry,
                                          s_a + (tid & ~31), s_b + (tid & ~31));
    if (lane == 0) entry[dd] = s;
  }
  if (!one && !grid_barrier(P.grid_bar, gridDim.x))
    atomicCAS(&st->status, 0, static_cast<int>(kStTimeout));
  const float dmp = static_cast<float>(P.damping), omd = static_cast<float>(1.0 - P.damping);
  const bool undamped = P.damping == 1.0;
  float dmax = 0.f, smax = 0.f;  // exact in the state's precision
  bool bad = false;
  if (active && u0 < u1) {
    float s = one ? x0[d] : __ldcg(carry + d * nch + ch);
    if (sub > 0) s = ea * s + eb;
    const float xd = x0[d];
    const float *pa = A + u0 * Dp + d, *pb = B + u0 * Dp + d, *po = So + u0 * Dp + d;
    float* pn = Sn + u0 * Dp + d;
    constexpr int kL = 8;
    for (int n = static_cast<int>(u1 - u0); n > 0;
         n -= kL, pa += kL * Dp, pb += kL * Dp, po += kL * Dp, pn += kL * Dp) {
      float va[kL], vb[kL], vo[kL];
#pragma unroll
      for (int k = 0; k < kL; ++k) {
        va[k] = k < n ? pa[k * Dp] : 1.f;
        vb[k] = k < n ? pb[k * Dp] : 0.f;
        vo[k] = k >= n ? 0.f : iter == 0 ? xd : po[k * Dp];  // sweep 0: S_old = x0
      }
#pragma unroll
      for (int k = 0; k < kL; ++k)
        if (k < n) {
          s = va[k] * s + vb[k];
          const float v = undamped ? s : omd * vo[k] + dmp * s;
          dmax = fmaxf(dmax, fabsf(v - vo[k]));
          smax = fmaxf(smax, fabsf(v));
          bad |= !isfinite(v);
          pn[k * Dp] = v;
        }
    }
  }
  dmax = warp_max(dmax);
  smax = warp_max(smax);
  if (__any_sync(0xffffffffu, bad) && lane == 0) s_bad = 1;
  if (lane == 0) {
    s_red[0][tid >> 5] = dmax;
    s_red[1][tid >> 5] = smax;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w)
      dmax = fmaxf(dmax, s_red[0][w]), smax = fmaxf(smax, s_red[1][w]);
    if (s_bad) atomicCAS(&st->status, 0, static_cast<int>(kStNonfinite));
    if (one) {
      s_last = 1;
    } else {
      if (dmax > 0.f) atomicMax(&st->dmax_bits, dbits(static_cast<double>(dmax)));
      if (smax > 0.f) atomicMax(&st->smax_bits, dbits(static_cast<double>(smax)));
      __threadfence();
      s_last = atomicAdd(&st->done_counter, 1u) == gridDim.x - 1;
      if (s_last) st->done_counter = 0;
    }
    if (s_last && c_hi == P.T) {  // convergence test (DEER.jl:567-578), the last CTA to arrive
      double dm = static_cast<double>(dmax), sm = static_cast<double>(smax);
      if (!one) {
        __threadfence();
        dm = bitsd(atomicAdd(&st->dmax_bits, 0ull));
        sm = bitsd(atomicAdd(&st->smax_bits, 0ull));
      }
      // a tensor-core pass of this sweep gave up a wait: its results are not to be used
      if (P.tc_err && *reinterpret_cast<const volatile int*>(P.tc_err))
        atomicCAS(&st->status, 0, static_cast<int>(kStTimeout));
      DevState f = *st;
      f.status = atomicAdd(&st->status, 0);
      f.metric = dm / (P.tol_abs + P.tol_rel * sm);
      f.iter = iter + 1;
      f.cur = cur ^ 1;
      f.converged = f.metric <= 1.0;
      f.dmax_bits = f.smax_bits = 0;
      f.done_counter = 0;
      *st = f;
      *st_host = f;
      __threadfence_system();
    }
  }
}

cudaError_t lg_finish(cudaStream_t s, const DevParams* dP, const DevState* dS, int64_t D,
                      int64_t T, const float* G, int nsplit, const double* lp_parts, int np,
                      double* la_ref, const TieBufs& b, float band, bool guard, int num_sms) {
  const PassG g{G, nsplit};
  const TieList list{band, b.kmax, b.mg, b.list, b.count};
  const int grid = static_cast<int>(imin64((T + kWarps - 1) / kWarps, int64_t(num_sms) * 8));
  const auto fn = D <= 128 ? lg_finish_kernel<1> : D <= 256 ? lg_finish_kernel<2>
                                                            : lg_finish_kernel<4>;
  fn<<<grid, kThreads, 0, s>>>(dP, dS, g, lp_parts, np, la_ref, list, guard ? 1 : 0);
  return cudaGetLastError();
}

// One CTA for a block whose runs are then at most 32 columns (two rounds of loads): the two
// barriers, the carries' trip through L2 and the maxima's atomics cost more than the
// longer runs (D = 24, T = 256: 8.9 us against 11.6).
static bool lg_scan_one(int64_t Dp, int64_t T) {
  return Dp <= kThreads && T <= 32 * (kThreads / Dp);
}

// Columns of a chunk, at least: a launch of few CTAs is co-resident sooner beside other
// streams' kernels (eight chains of a fleet: 144 ms with 4, 131 with 16, 126 with 64), and
// a solve alone is as fast (5.9 ms at N = 3001, D = 101, T = 4099 with 16, 32 and 64).
constexpr int kScanMinCols = 64;

// Columns of one launch: whole chunks within the composition window.
static int64_t lg_scan_cols(int64_t Dp, int64_t T, int num_sms) {
  const int64_t most = 3 * num_sms / ((Dp + kThreads - 1) / kThreads);
  const int64_t seg = imax64(1, most) * (kScanWindow / 8);
  const int64_t nseg = (T + seg - 1) / seg;
  return (T + nseg - 1) / nseg;
}

size_t lg_scan_ws_bytes(int64_t Dp, int64_t T, int num_sms) {
  const int64_t Tn = lg_scan_cols(Dp, T, num_sms);
  const ScanPlan pl = scan_plan(Dp, Tn, 3 * num_sms, kScanMinCols, 8);
  return 4 * static_cast<size_t>(Dp) * (3 * static_cast<size_t>(pl.nchunks) + 1) + 64;
}

cudaError_t lg_scan(cudaStream_t s, const DevParams* dP, DevState* dS, int64_t Dp, int64_t T,
                    void* scratch, DevState* st_host, int num_sms) {
  const int64_t Tn = lg_scan_cols(Dp, T, num_sms);
  float* entry = static_cast<float*>(scratch);
  float* rest = entry + Dp;
  for (int64_t t0 = 0; t0 < T; t0 += Tn) {
    int64_t lo = t0, hi = imin64(T, t0 + Tn);
    ScanPlan pl = scan_plan(Dp, Tn, 3 * num_sms, kScanMinCols, 8);
    pl.nchunks = static_cast<int>((hi - lo + pl.L - 1) / pl.L);
    void* args[] = {&dP, &dS, &lo, &hi, &pl, &rest, &entry, &st_host};
    if (lg_scan_one(Dp, T)) {
      pl.nblk_d = 1;
      pl.blk_d = static_cast<int>(Dp);
      pl.nsub = kThreads / static_cast<int>(Dp);
      pl.Ls = static_cast<int>((T + pl.nsub - 1) / pl.nsub);
      pl.L = static_cast<int>(T);
      pl.nchunks = 1;
      return cudaLaunchKernel(reinterpret_cast<const void*>(lg_scan_kernel), dim3(1),
                              dim3(kThreads), args, 0, s);
    }
    const cudaError_t e = cudaLaunchCooperativeKernel(
        reinterpret_cast<const void*>(lg_scan_kernel), dim3(pl.nchunks * pl.nblk_d),
        dim3(pl.threads), args, 0, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace pmcmc
