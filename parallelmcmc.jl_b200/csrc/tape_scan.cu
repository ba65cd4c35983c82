// tape_scan.cu -- tape materialisation and the standalone diagonal affine scan.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <unordered_map>

#include "deer_device.cuh"
#include "deer_launch.h"
#include "scan_phases.cuh"

namespace pmcmc {

// Tape block of (seed, block): Xi (D x T, column-major) and u (T)
// (counterpart of _make_mala_tape_block, interface.jl:334-358).
__global__ void tape_kernel(int64_t D, int64_t T, uint64_t seed, uint64_t block, float* Xi,
                            float* u) {
  const int64_t nq = (D + 3) / 4;
  const int64_t n = nq * T;
  const TapeKey key(seed, block);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / nq, j = i % nq;
    float v[4];
    tape_xi4(key, static_cast<uint32_t>(j), static_cast<uint32_t>(t), v);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (4 * j + e < D) Xi[t * D + 4 * j + e] = v[e];
    if (j == 0 && u) u[t] = tape_u(key, static_cast<uint32_t>(t));
  }
}

cudaError_t launch_tape(cudaStream_t s, int64_t D, int64_t T, uint64_t seed, uint64_t block,
                        float* Xi, float* u) {
  const int64_t n = ((D + 3) / 4) * T;
  if (n == 0) return cudaSuccess;
  const int grid = static_cast<int>(imin64((n + 255) / 256, 148 * 16));
  tape_kernel<<<grid, 256, 0, s>>>(D, T, seed, block, Xi, u);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// S[:,t] = A[:,t] .* S[:,t-1] + B[:,t] (solve_affine_scan_diag!, DEERScan.jl:102-173)
// in one cooperative launch.  The columns are cut into chunks, one a CTA (and a
// block of up to 256 coordinates); inside it `nsub` runs of consecutive columns a
// coordinate, one a thread:
//   1. every thread composes its run, 64 bytes of A and of B in flight; the runs'
//      maps are composed in shared memory into the chunk's;
//   2. after a grid barrier, one warp a coordinate carries the state over the
//      chunks: each lane composes `group` chunks, the lanes' maps are applied to
//      the state in turn, and each lane replays its group;
//   3. after a second barrier every thread replays the recurrence over its run.
// Bound: HBM, one read of A and B and one write of S; phase 3's second read of A
// and B comes from L2, which a launch's columns fit (scan_plan).  The look-back over
// 64-column tiles that this replaces was a serial chain of T / 2048 hops: 471 us at
// D = 100, T = 65536 in FP32 (78.6 MB), against 21 us here (3.7 TB/s; the floor is
// 12 us, phase 2 and the barriers take most of the rest).
// States are carried by composition over at most 2048 columns at a time, as the
// look-back did, so a coordinate that stays at zero under growing maps stays at
// zero.  A cooperative launch's CTAs are co-resident, so the barriers end.
// ---------------------------------------------------------------------------
// CTAs an SM and chunks a lane composes at a time, without spills: a spilled value in
// phase 2 is read from L2 each time, because the CTAs that already wait at the barrier
// invalidate the SM's L1 with every poll
constexpr int kScanCtas = 3;
// Columns of a chunk, at least (us with 8, 16, 32, 64: D = 64, T = 2048 in FP64 8.8, 6.9, 7.1,
// 7.9; D = 100, T = 8192 in FP32 10.6, 10.5, 8.5, 8.7; D = 256, T = 8192 13.2, 13.3, 10.6, 11.8).
constexpr int kScanMinCols = 32;
template <typename Real>
constexpr int kScanLoads = 64 / sizeof(Real);  // columns of loads in flight a thread
template <typename Real>
constexpr int kScanGroup = sizeof(Real) == 4 ? 8 : 4;

template <typename Real>
__global__ void __launch_bounds__(kThreads, kScanCtas)
    affine_scan_kernel(int64_t D, int64_t T, ScanPlan pl, const Real* __restrict__ A,
                       const Real* __restrict__ B, const Real* s0, Real* __restrict__ S,
                       Real* __restrict__ agg_a, Real* __restrict__ agg_b,
                       Real* __restrict__ carry, uint32_t* bar, int* err) {
  __shared__ Real s_a[kThreads], s_b[kThreads];
  constexpr int kScanUnroll = kScanLoads<Real>;
  const int tid = threadIdx.x;
  const int nch = pl.nchunks;
  const int db = static_cast<int>(blockIdx.x) % pl.nblk_d;
  const int ch = static_cast<int>(blockIdx.x) / pl.nblk_d;
  const int sub = tid / pl.blk_d, dl = tid - sub * pl.blk_d;
  const int64_t d = static_cast<int64_t>(db) * pl.blk_d + dl;
  const bool active = sub < pl.nsub && d < D;
  const int64_t c0 = static_cast<int64_t>(ch) * pl.L, c1 = imin64(T, c0 + pl.L);
  const int64_t u0 = imin64(c1, c0 + static_cast<int64_t>(sub) * pl.Ls);
  const int64_t u1 = imin64(c1, u0 + pl.Ls);
  // columns past the run load the identity map, which changes nothing
  const int Di = static_cast<int>(D);
  auto load = [&](const Real* pa, const Real* pb, int n, Real (&va)[kScanUnroll],
                   Real (&vb)[kScanUnroll]) {
#pragma unroll
    for (int k = 0; k < kScanUnroll; ++k) {
      va[k] = k < n ? pa[k * Di] : Real(1);
      vb[k] = k < n ? pb[k * Di] : Real(0);
    }
  };
  // One chunk: its entering state is s0, nothing to carry and no other CTA to wait for (one
  // warp a coordinate carried 256 of them in turn: 62 us a call at D = 256, T = 8, 35 so).
  const bool one = nch == 1;
  const Real st0 = one && active ? s0[d] : Real(0);
  Real a = 1, b = 0;
  if (active)
    scan_compose_run<Real, kScanUnroll>(A + u0 * D + d, B + u0 * D + d,
                                        static_cast<int>(u1 - u0), Di, a, b);
  s_a[tid] = a;
  s_b[tid] = b;
  __syncthreads();
  Real ea = 1, eb = 0;  // the maps of the chunk's earlier runs, composed
  if (active) {
    if (sub > 0) scan_earlier_runs<Real>(s_a, s_b, pl.blk_d, dl, sub, ea, eb);
    if (sub == pl.nsub - 1 && !one) {
      agg_a[ch * D + d] = sub > 0 ? a * ea : a;
      agg_b[ch * D + d] = sub > 0 ? a * eb + b : b;
    }
  }
  if (!one) {
    if (!grid_barrier(bar, gridDim.x)) atomicExch(err, 1);
    // (the runs' maps in s_a and s_b were last read before the barrier)
    const int w0 = tid & ~31, nw = static_cast<int>(blockDim.x) >> 5;
    for (int64_t dd = static_cast<int64_t>(tid >> 5) * gridDim.x + blockIdx.x; dd < D;
         dd += static_cast<int64_t>(nw) * gridDim.x)
      scan_carry<Real, kScanGroup<Real>>(nch, pl.group, agg_a, agg_b, D, dd, s0[dd], carry,
                                         s_a + w0, s_b + w0);
    if (!grid_barrier(bar, gridDim.x)) atomicExch(err, 1);
  }
  if (active && u0 < u1) {
    Real st = one ? st0 : __ldcg(carry + d * nch + ch);
    if (sub > 0) st = ea * st + eb;
    const Real *pa = A + u0 * D + d, *pb = B + u0 * D + d;
    Real* ps = S + u0 * D + d;
    for (int n = static_cast<int>(u1 - u0); n > 0; n -= kScanUnroll, pa += kScanUnroll * Di,
             pb += kScanUnroll * Di, ps += kScanUnroll * Di) {
      Real va[kScanUnroll], vb[kScanUnroll];
      load(pa, pb, n, va, vb);
#pragma unroll
      for (int k = 0; k < kScanUnroll; ++k)
        if (k < n) {
          st = va[k] * st + vb[k];
          ps[k * Di] = st;
        }
    }
  }
}

// Split of a scan over T columns (a launch's share of them) and D coordinates.
// Up to 3 CTAs an SM, 96 KB of loads in flight an SM; chunks of
// min_cols columns at least (scan_tile_cols of the whole scan), so that the chunks
// fit the scratch.
ScanPlan scan_plan(int64_t D, int64_t T, int max_ctas, int min_cols,
                          int max_group) {
  ScanPlan p{};
  p.nblk_d = static_cast<int>((D + kThreads - 1) / kThreads);
  p.blk_d = static_cast<int>((D + p.nblk_d - 1) / p.nblk_d);
  const int64_t most = imax64(1, max_ctas / p.nblk_d);
  p.L = static_cast<int>(imax64((T + most - 1) / most, min_cols));
  p.nchunks = static_cast<int>((T + p.L - 1) / p.L);
  p.nsub = static_cast<int>(imin64(imin64(kThreads / p.blk_d, 16), p.L));
  p.Ls = (p.L + p.nsub - 1) / p.nsub;
  p.nsub = (p.L + p.Ls - 1) / p.Ls;
  p.threads = (p.nsub * p.blk_d + 31) / 32 * 32;
  p.group = static_cast<int>(imax64(1, imin64(max_group, kScanWindow / p.L)));
  return p;
}

cudaError_t raise_smem_limit(const void* fn, size_t bytes) {
  static std::mutex mu;
  static std::unordered_map<const void*, size_t> limit;
  // (also below 48 KB: static plus dynamic shared memory above 48 KB needs the
  // opt-in even when the dynamic part alone is under it)
  if (bytes == 0) return cudaSuccess;
  std::lock_guard<std::mutex> lk(mu);
  size_t& cur = limit[fn];
  if (bytes <= cur) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(bytes));
  if (e == cudaSuccess) cur = bytes;
  return e;
}

int scan_tile_cols(int64_t D, int64_t T) {
  // Fewest columns a chunk of the scan has, which sizes its scratch: a power of
  // two in 8 .. 64 (fewer for D > 768) that leaves about 2 chunks per SM.
  int TT = 64;
  while (TT > 1 && static_cast<int64_t>(2 * TT + 1) * D * 8 > 96 * 1024) TT >>= 1;
  while (TT > 8 && (T + TT - 1) / TT < 296) TT >>= 1;
  return TT;
}

size_t scan_scratch_bytes(bool f64, int64_t D, int64_t T) {
  const int TT = scan_tile_cols(D, T);
  const int64_t nt = (T + TT - 1) / TT;
  return kScanBarBytes + 3 * (f64 ? 8 : 4) * static_cast<size_t>(nt * D);
}

template <typename Real>
static cudaError_t scan_launches(cudaStream_t s, int64_t D, int64_t T, const Real* A,
                                 const Real* B, const Real* s0, Real* S, void* scratch,
                                 int* err) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const void* fn = reinterpret_cast<const void*>(affine_scan_kernel<Real>);
  const int max_ctas = kScanCtas * sms;  // co-resident by the launch bounds
  const int64_t nblk_d = (D + kThreads - 1) / kThreads;
  if (nblk_d > max_ctas) return cudaErrorInvalidValue;
  // Columns of a launch: chunks within the composition window, and A and B of
  // the launch inside L2 for phase 3's read (about 64 MB of its 126).
  const int64_t by_window = (max_ctas / nblk_d) * (kScanWindow / 8);
  const int64_t by_l2 = (int64_t(64) << 20) / (2 * static_cast<int64_t>(sizeof(Real)) * D);
  const int64_t seg = imin64(by_window, imax64(by_l2, 4096));
  const int64_t nseg = (T + seg - 1) / seg, Tseg = (T + nseg - 1) / nseg;
  for (int64_t t0 = 0; t0 < T; t0 += Tseg) {
    int64_t Tn = imin64(Tseg, T - t0), Dn = D;
    ScanPlan pl = scan_plan(D, Tn, max_ctas, std::max(kScanMinCols, scan_tile_cols(D, T)),
                            kScanGroup<Real>);
    const Real *An = A + t0 * D, *Bn = B + t0 * D, *sn = t0 ? S + (t0 - 1) * D : s0;
    uint32_t* bar = static_cast<uint32_t*>(scratch);
    Real* Sn = S + t0 * D;
    Real* aa = reinterpret_cast<Real*>(static_cast<unsigned char*>(scratch) + kScanBarBytes);
    Real *ab = aa + static_cast<size_t>(pl.nchunks) * D,
         *ca = ab + static_cast<size_t>(pl.nchunks) * D;
    void* args[] = {&Dn, &Tn, &pl, &An, &Bn, &sn, &Sn, &aa, &ab, &ca, &bar, &err};
    const dim3 grid(pl.nchunks * pl.nblk_d), threads(pl.threads);
    e = pl.nchunks == 1 ? cudaLaunchKernel(fn, grid, threads, args, 0, s)
                        : cudaLaunchCooperativeKernel(fn, grid, threads, args, 0, s);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

cudaError_t launch_affine_scan(cudaStream_t s, bool f64, int64_t D, int64_t T, const void* A,
                               const void* B, const void* s0, void* S, void* scratch, int* err) {
  if (T == 0 || D == 0) return cudaSuccess;
  return f64 ? scan_launches(s, D, T, static_cast<const double*>(A), static_cast<const double*>(B),
                             static_cast<const double*>(s0), static_cast<double*>(S), scratch, err)
             : scan_launches(s, D, T, static_cast<const float*>(A), static_cast<const float*>(B),
                             static_cast<const float*>(s0), static_cast<float*>(S), scratch, err);
}

// ---------------------------------------------------------------------------
// Plain path: Hillis-Steele doubling scan, one launch per level
// (DEERScan.jl:135-171), then damping and the metric reductions.
// ---------------------------------------------------------------------------
template <typename Real>
__global__ void doubling_level_kernel(int64_t Dp, int64_t T, int64_t off,
                                      const Real* __restrict__ al, const Real* __restrict__ be,
                                      Real* __restrict__ aln, Real* __restrict__ ben) {
  const int64_t n = T * Dp;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / Dp;
    if (t >= off) {
      const Real a2 = al[i];
      aln[i] = a2 * al[i - off * Dp];
      ben[i] = a2 * be[i - off * Dp] + be[i];
    } else {
      aln[i] = al[i];
      ben[i] = be[i];
    }
  }
}

template <typename Real>
__global__ void doubling_apply_kernel(int64_t Dp, int64_t T, const Real* __restrict__ al,
                                      const Real* __restrict__ be, const Real* __restrict__ s0,
                                      Real* __restrict__ S) {
  const int64_t n = T * Dp;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    S[i] = al[i] * s0[i % Dp] + be[i];
}

template <typename Real>
__global__ void damp_metric_kernel(int64_t D, int64_t Dp, int64_t T, const Real* __restrict__ So,
                                   Real* __restrict__ Sn, double damping,
                                   unsigned long long* red) {
  const int64_t n = T * Dp;
  double dm = 0, sm = 0;
  bool bad = false;
  const Real dmp = static_cast<Real>(damping), omd = static_cast<Real>(1.0 - damping);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    if (i % Dp >= D) continue;
    Real v = Sn[i];
    if (damping != 1.0) {
      v = omd * So[i] + dmp * v;
      Sn[i] = v;
    }
    dm = max(dm, static_cast<double>(fabs(v - So[i])));
    sm = max(sm, static_cast<double>(fabs(v)));
    bad |= !isfinite(v);
  }
  dm = warp_max(dm);
  sm = warp_max(sm);
  if ((threadIdx.x & 31) == 0) {
    if (dm > 0) atomicMax(red, dbits(dm));
    if (sm > 0) atomicMax(red + 1, dbits(sm));
    if (bad) atomicExch(red + 2, 1ull);
  }
}

cudaError_t launch_doubling_scan(cudaStream_t s, bool f64, int64_t Dp, int64_t T, const void* A,
                                 const void* B, const void* s0, void* S, void* al0, void* be0,
                                 void* al1, void* be1) {
  const int64_t n = T * Dp;
  const int grid = static_cast<int>(imin64((n + 255) / 256, 148 * 8));
  const void* al = A;
  const void* be = B;
  void* bufs[2][2] = {{al0, be0}, {al1, be1}};
  int which = 0;
  for (int64_t off = 1; off < T; off <<= 1, which ^= 1) {
    if (f64)
      doubling_level_kernel<double><<<grid, 256, 0, s>>>(
          Dp, T, off, static_cast<const double*>(al), static_cast<const double*>(be),
          static_cast<double*>(bufs[which][0]), static_cast<double*>(bufs[which][1]));
    else
      doubling_level_kernel<float><<<grid, 256, 0, s>>>(
          Dp, T, off, static_cast<const float*>(al), static_cast<const float*>(be),
          static_cast<float*>(bufs[which][0]), static_cast<float*>(bufs[which][1]));
    al = bufs[which][0];
    be = bufs[which][1];
  }
  if (f64)
    doubling_apply_kernel<double><<<grid, 256, 0, s>>>(Dp, T, static_cast<const double*>(al),
                                                       static_cast<const double*>(be),
                                                       static_cast<const double*>(s0),
                                                       static_cast<double*>(S));
  else
    doubling_apply_kernel<float><<<grid, 256, 0, s>>>(Dp, T, static_cast<const float*>(al),
                                                      static_cast<const float*>(be),
                                                      static_cast<const float*>(s0),
                                                      static_cast<float*>(S));
  return cudaGetLastError();
}

cudaError_t launch_damp_metric(cudaStream_t s, bool f64, int64_t D, int64_t Dp, int64_t T,
                               const void* S_old, void* S_new, double damping,
                               unsigned long long* red) {
  const int64_t n = T * Dp;
  const int grid = static_cast<int>(imin64((n + 255) / 256, 148 * 8));
  cudaError_t e = cudaMemsetAsync(red, 0, 3 * sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  if (f64)
    damp_metric_kernel<double><<<grid, 256, 0, s>>>(D, Dp, T, static_cast<const double*>(S_old),
                                                    static_cast<double*>(S_new), damping, red);
  else
    damp_metric_kernel<float><<<grid, 256, 0, s>>>(D, Dp, T, static_cast<const float*>(S_old),
                                                   static_cast<float*>(S_new), damping, red);
  return cudaGetLastError();
}

template <typename Real>
__global__ void broadcast_kernel(int64_t Dp, int64_t T, const Real* __restrict__ x0,
                                 Real* __restrict__ S) {
  const int64_t n = T * Dp;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    S[i] = x0[i % Dp];
}

cudaError_t launch_broadcast(cudaStream_t s, bool f64, int64_t Dp, int64_t T, const void* x0,
                             void* S) {
  const int64_t n = T * Dp;
  const int grid = static_cast<int>(imin64((n + 255) / 256, 148 * 8));
  if (f64)
    broadcast_kernel<double><<<grid, 256, 0, s>>>(Dp, T, static_cast<const double*>(x0),
                                                  static_cast<double*>(S));
  else
    broadcast_kernel<float><<<grid, 256, 0, s>>>(Dp, T, static_cast<const float*>(x0),
                                                 static_cast<float*>(S));
  return cudaGetLastError();
}

// Bound check of the look-back wait: one warp looks back from tile 1 over a
// flag array that nothing publishes (all zeros: no epoch, no state), so lane 0
// spins on tile 0 until kMaxSpins and the warp reports the give-up in err[0].  The same
// routine guards the per-sweep kernel.
__global__ void lookback_bound_kernel(const uint32_t* flags, int* err) {
  int e = 0;
  lookback_fixed(1, 1u, flags, &e);
  if (threadIdx.x == 0) err[0] = e;
}

cudaError_t launch_lookback_bound(cudaStream_t s, const uint32_t* flags, int* err) {
  lookback_bound_kernel<<<1, 32, 0, s>>>(flags, err);
  return cudaGetLastError();
}

// Bound check of the grid barrier (the persistent solve, the scans, the near ties): one CTA
// arrives at a barrier of two.
__global__ void barrier_bound_kernel(uint32_t* bar, int* err) {
  grid_barrier_noted(bar, 2);
  if (threadIdx.x == 0) err[0] = __ldcg(bar + 1) != 0u ? 1 : 0;
}

cudaError_t launch_barrier_bound(cudaStream_t s, uint32_t* bar, int* err) {
  barrier_bound_kernel<<<1, kThreads, 0, s>>>(bar, err);
  return cudaGetLastError();
}

}  // namespace pmcmc
