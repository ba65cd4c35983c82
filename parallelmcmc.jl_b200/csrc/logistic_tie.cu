// logistic_tie.cu -- FP64 decisions for near-tie columns of the logistic target,
// and the verification pass at a returned trajectory.
//
// The accept decision of column t compares log u_t with log alpha_t
// (MALA.jl:402-404, strict <).  With FP32 state and the 22-bit tensor-core
// contractions, log alpha carries an absolute error of about 1e-5 .. 1e-4:
// each of the N log-likelihood terms of lp(x) and lp(y) is rounded on its own,
// and their errors add up over the rows.  A column whose margin
// |log alpha - log u| lies inside that band can change its decision from one
// Newton sweep to the next while the iterate moves only by rounding-level
// amounts; every change moves the trajectory after the column, and the solve
// stalls (N = 10000, D = 256, T = 65536: 369 sweeps where the FP64 solve takes
// 49, and accept flags that differ from the FP64 sequential chain).
//
// The sequential FP64 chain (MALA.jl:377-411, bayes_logreg.jl:37-58) decides
// such a column by its exact log alpha.
// So after the contraction passes of a
// sweep:
//   1. log alpha_t of every column from the sweep's quantities and |margin_t|; the
//      columns inside a band are counted and listed (the finish kernel, or
//      tie_margin_kernel on the paths without it);
//   2. tie_solve_kernel, one cooperative launch that ends at once when the list is
//      empty: at most kmax columns (the widest of four nested bands whose count fits),
//      in FP64 from the FP64 design matrix: the gradient at x_bar_t = S_{t-1}, the
//      proposal y_t = x_bar + eps g + sqrt(2 eps) xi_t, lp(x_bar), lp(y), the gradient
//      at y and both log proposal densities (logq_mala, MALA.jl:172-193); log alpha_t
//      in FP64 replaces the sweep's value, and the column's (A, B) is formed again.
// The sweep takes log alpha from la_ref for every column.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "deer_device.cuh"
#include "deer_launch.h"
#include "logistic.h"
#include "logistic_column.cuh"

namespace pmcmc {
namespace tie {

constexpr int kTieThreads = 256;
constexpr int kTieWarps = kTieThreads / 32;
constexpr int kTieCtas = 2;    // an SM
constexpr int kTieParts = 32;  // of the rows, most

// log alpha_t as the sweep computes it (column_logistic in deer_sweep.cu):
//   sum_d [-tau/2 (y^2 - x^2) + (r1^2 - r2^2) / (4 eps)] + lpy_t - lpx_t,
//   r1 = sqrt(2 eps) xi, r2 = (x - y) - eps g_y, in FP64 from the state's
// precision.  One warp a column.
template <typename Real>
__global__ void tie_margin_kernel(const DevParams* __restrict__ Pg,
                                  const DevState* __restrict__ st, double* __restrict__ la_ref,
                                  TieList list) {
  const DevParams& P = *Pg;
  const int lane = threadIdx.x & 31;
  const int64_t D = P.D, Dp = P.Dp;
  const bool from_x0 = st->iter == 0;
  const Real* S = static_cast<const Real*>(P.S[st->cur]);
  const Real* x0 = static_cast<const Real*>(P.x0);
  const Real* yv = static_cast<const Real*>(P.lg[1]);
  const Real* gyv = static_cast<const Real*>(P.lg[3]);
  const int64_t nw = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
       t < P.T; t += nw) {
    const Real* xb = (from_x0 || t == 0) ? x0 : S + (t - 1) * Dp;
    double la = 0.0;
    for (int64_t d = lane; d < D; d += 32) {
      const double xd = static_cast<double>(xb[d]);
      const double yd = static_cast<double>(yv[t * Dp + d]);
      const double r1 = P.sqrt2eps * static_cast<double>(P.xi[t * Dp + d]);
      const double r2 = (xd - yd) - P.eps * static_cast<double>(gyv[t * Dp + d]);
      la += -0.5 * P.tau * (yd * yd - xd * xd) + (r1 * r1 - r2 * r2) * P.inv4eps;
    }
    la = warp_sum(la) + (P.lpy[t] - P.lpx[t]);
    if (lane == 0) {
      la_ref[t] = la;
      if (list.count) tie_note(list, t, la - P.logu[t]);
    }
  }
}

// Two FP64 MMAs (8 x 8, k = 4) with the same A: lane l holds A[l / 4][l % 4], B[l % 4][l / 4]
// and C[l / 4][2 (l % 4) .. + 1].
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// Four values another CTA of this launch may have written (FP64), or of the state (FP32,
// not written here).
__device__ __forceinline__ void load_cg4(const double* p, double (&v)[4]) {
  const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
  const double2 b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
  v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}
__device__ __forceinline__ void load_cg4(const float* p, double (&v)[4]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
}

struct TieArgs {
  TieList list;
  const double* X;   // N x Dp
  const double* y;   // N
  int64_t N;
  double *By, *GX;   // [kmax x Dp] proposals, gradients at x_bar
  int64_t Nr;        // N rounded up to 8
  double* R;         // [kmax x Nr] y - sigmoid
  double* lpP;       // [ceil(N / 8) x kmax] log-likelihood sums of 8 rows
  double* lpx;       // [kmax]
  double* GP;        // parts of the gradients (tie_gp_elems)
  double* la_ref;
  PassG G;           // g = NULL: no (A, B) to form again
  int qpl;
};

// The work below is bound by L2 (X is read four times, 8 rows or 16 values of d by up to
// 16 columns a warp), by the five grid barriers where the list is short and by the FP64
// rate where it is long.  Against the eleven launches around four DGEMMs over all kmax columns
// that it replaces: 129 us instead of 400 at N = 10000, D = 256 and 65 columns, 45 instead
// of 80 at N = 3001, D = 101 and 4 columns, 3 instead of 45 with an empty list (N = 400, D = 24);
// each row's log1p by itself adds 10 and 1.5 us to the first two.
__global__ void __launch_bounds__(kTieThreads, kTieCtas)
    tie_solve_kernel(const DevParams* __restrict__ Pg, DevState* __restrict__ st, TieArgs a) {
  __shared__ int s_base[kTieWarps], s_pos;
  __shared__ double s_sum[kTieWarps];
  const DevParams& P = *Pg;
  auto all_sync = [&]() {
    if (!grid_barrier(P.grid_bar, gridDim.x))
      atomicCAS(&st->status, 0, static_cast<int>(kStTimeout));
  };
  const int tid = threadIdx.x, lane = tid & 31;
  const int kmax = a.list.kmax;
  int cnt = static_cast<int>(*reinterpret_cast<const volatile uint32_t*>(a.list.count));
  if (cnt == 0) return;
  if (cnt > kmax) {
    // more columns than fit: the widest band that does, or the first kmax columns of the
    // narrowest, in column order, from the margins
    if (blockIdx.x == 0) {
      if (tid == 0) s_pos = 0;
      int bi = 1;
      float b = a.list.band * 0.25f;
      while (bi < kTieBands - 1 && __ldcg(a.list.count + bi) > static_cast<uint32_t>(kmax)) ++bi, b *= 0.25f;
      __syncthreads();
      for (int64_t t0 = 0; t0 < P.T && s_pos < kmax; t0 += kTieThreads) {
        const bool in = t0 + tid < P.T && a.list.mg[t0 + tid] < b;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) s_base[tid >> 5] = __popc(m);
        __syncthreads();
        int pos = s_pos;
        for (int w = 0; w < (tid >> 5); ++w) pos += s_base[w];
        pos += __popc(m & ((1u << lane) - 1u));
        if (in && pos < kmax) a.list.list[pos] = static_cast<int32_t>(t0 + tid);
        __syncthreads();
        if (tid == 0)
          for (int w = 0; w < kTieWarps; ++w) s_pos += s_base[w];
        __syncthreads();
      }
      if (tid == 0) a.list.count[1] = min(s_pos, kmax);
    }
    all_sync();
    cnt = static_cast<int>(__ldcg(a.list.count + 1));
  }
  const int64_t N = a.N, D = P.D, Dp = P.Dp;
  const int64_t gw = static_cast<int64_t>(blockIdx.x) * kTieWarps + (tid >> 5);
  const int64_t nw = static_cast<int64_t>(gridDim.x) * kTieWarps;
  const int ct = (cnt + 15) / 16;              // tiles of 16 columns
  const int64_t rt = (N + 7) / 8, dt = (Dp + 15) / 16;
  // parts of the gradients' sums over the rows (each is read again, in order)
  const int ns = static_cast<int>(imax64(1, imin64(kTieParts, nw / (dt * ct))));
  const int64_t per = ((N + ns - 1) / ns + 15) / 16 * 16;
  const bool from_x0 = st->iter == 0;
  const float* S = static_cast<const float*>(P.S[st->cur]);
  const float* x0 = static_cast<const float*>(P.x0);
  const int r8 = lane >> 2, k4 = lane & 3;
  auto xbar = [&](int k) {
    const int64_t t = __ldcg(a.list.list + min(k, cnt - 1));
    return (from_x0 || t == 0) ? x0 : S + (t - 1) * Dp;
  };
  // Logits of 8 rows x 16 columns a warp; R and the rows' log-likelihood terms.  The MMAs'
  // k runs over the coordinates in an order of its own: lane k4 of a row or column holds
  // four consecutive ones, loaded 16 bytes at a time (one value a load is bound by the
  // load unit, 37 us instead of 14 at N = 10000, D = 256, 65 columns).
  auto logits = [&](auto x_of) {
    for (int64_t w = gw; w < rt * ct; w += nw) {
      const int64_t row0 = w / ct * 8;
      const int c0 = static_cast<int>(w % ct) * 16;
      const int64_t row = row0 + r8;
      const double* xr = a.X + (row < N ? row : N - 1) * Dp;
      const auto* f0 = x_of(min(c0 + r8, cnt - 1));
      const auto* f1 = x_of(min(c0 + 8 + r8, cnt - 1));
      const bool two = c0 + 8 < cnt;
      double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 2
      for (int k = 4 * k4; k - 4 * k4 < Dp; k += 16) {
        double av[4] = {0.0, 0.0, 0.0, 0.0}, b0[4] = {0.0, 0.0, 0.0, 0.0},
               b1[4] = {0.0, 0.0, 0.0, 0.0};
        if (k < Dp) {
          load4(xr + k, av);
          load_cg4(f0 + k, b0);
          if (two) load_cg4(f1 + k, b1);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          dmma(c[0], av[i], b0[i]);
          if (two) dmma(c[1], av[i], b1[i]);
        }
      }
      const double lab = row < N ? a.y[row] : 0.0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h && !two) break;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int col = c0 + 8 * h + 2 * k4 + i;
          const double z = c[h][i];
          const double e = exp(-fabs(z));
          const double p = (z >= 0.0 ? 1.0 : e) / (1.0 + e);
          // lab z - softplus(z), without the cancellation where lab = 1 and z > 0
          const double zn = lab != 0.0 ? -z : z;
          double term = row < N ? -((zn > 0.0 ? zn : 0.0) + log1p(e)) : 0.0;
#pragma unroll
          for (int o = 4; o < 32; o <<= 1) term += __shfl_xor_sync(0xffffffffu, term, o);
          if (col < cnt) {
            a.R[static_cast<int64_t>(col) * a.Nr + row] = row < N ? lab - p : 0.0;
            if (r8 == 0) a.lpP[row0 / 8 * kmax + col] = term;
          }
        }
      }
    }
  };
  // Parts of X'R: 16 values of d (lane r8 holds two) x 16 columns a warp, over `per` rows
  // (lane k4 holds four consecutive ones of 16)
  auto gradients = [&]() {
    for (int64_t w = gw; w < dt * ct * ns; w += nw) {
      const int64_t part = w / (dt * ct), q = w % (dt * ct);
      const int64_t d = q / ct * 16 + 2 * r8;
      const int c0 = static_cast<int>(q % ct) * 16;
      const int64_t n0 = part * per, n1 = imin64(N, n0 + per);
      const double* xc = a.X + (d < Dp ? d : Dp - 2);
      const double* q0 = a.R + static_cast<int64_t>(min(c0 + r8, cnt - 1)) * a.Nr;
      const double* q1 = a.R + static_cast<int64_t>(min(c0 + 8 + r8, cnt - 1)) * a.Nr;
      const bool two = c0 + 8 < cnt;
      double c[2][2][2] = {};  // [d][columns]
#pragma unroll 2
      for (int64_t n = n0 + 4 * k4; n - 4 * k4 < n1; n += 16) {
        double2 av[4];
        double b0[4] = {0.0, 0.0, 0.0, 0.0}, b1[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 0; i < 4; ++i)  // a row past N is read as the last one, times R = 0
          av[i] = *reinterpret_cast<const double2*>(xc + imin64(n + i, N - 1) * Dp);
        if (n < n1) {  // (R is zero from N to its stride)
          load_cg4(q0 + n, b0);
          if (two) load_cg4(q1 + n, b1);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          dmma(c[0][0], av[i].x, b0[i]);
          dmma(c[1][0], av[i].y, b0[i]);
          if (two) {
            dmma(c[0][1], av[i].x, b1[i]);
            dmma(c[1][1], av[i].y, b1[i]);
          }
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int col = c0 + 8 * h + 2 * k4 + i;
          if (col < cnt && d < Dp)
            *reinterpret_cast<double2*>(a.GP + (part * cnt + col) * Dp + d) =
                make_double2(c[0][h][i], c[1][h][i]);
        }
    }
  };
  auto grad_at = [&](int64_t k, int64_t d) {
    double g = 0.0;
#pragma unroll 8
    for (int p = 0; p < ns; ++p) g += __ldcg(a.GP + (p * cnt + k) * Dp + d);
    return g;
  };
  // sums over the CTA, the same in every thread
  auto cta_sum = [&](double v) {
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) s_sum[tid >> 5] = v;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kTieWarps; ++w) t += s_sum[w];
    return t;
  };
  auto loglik = [&](int64_t k) {
    double l = 0.0;
#pragma unroll 4
    for (int64_t r = tid; r < rt; r += kTieThreads) l += __ldcg(a.lpP + r * kmax + k);
    return cta_sum(l);
  };

  logits([&](int k) { return xbar(k); });
  all_sync();
  gradients();
  all_sync();
  // gx = X'r - tau x_bar (bayes_logreg.jl:48-58), y = x_bar + eps gx + sqrt(2 eps) xi
  // (MALA.jl:221-222); one CTA a column
  for (int64_t k = blockIdx.x; k < cnt; k += gridDim.x) {
    const int64_t t = __ldcg(a.list.list + k);
    const float* x = xbar(static_cast<int>(k));
    for (int64_t d = tid; d < Dp; d += kTieThreads) {
      double gx = 0.0, y = 0.0;
      if (d < D) {
        const double xd = static_cast<double>(x[d]);
        gx = grad_at(k, d) - P.tau * xd;
        y = xd + P.eps * gx + P.sqrt2eps * static_cast<double>(P.xi[t * Dp + d]);
      }
      a.GX[k * Dp + d] = gx;
      a.By[k * Dp + d] = y;
    }
    const double l = loglik(k);
    if (tid == 0) a.lpx[k] = l;
  }
  all_sync();
  logits([&](int k) { return static_cast<const double*>(a.By) + static_cast<int64_t>(k) * Dp; });
  all_sync();
  gradients();
  all_sync();
  // log alpha_t = [lp(y) + logq(x|y)] - [lp(x) + logq(y|x)] (MALA.jl:172-193, 402), and
  // the column's affine map by it; one CTA a column
  for (int64_t k = blockIdx.x; k < cnt; k += gridDim.x) {
    const int64_t t = __ldcg(a.list.list + k);
    const float* x = xbar(static_cast<int>(k));
    double xx = 0.0, yy = 0.0, q1 = 0.0, q2 = 0.0;
    for (int64_t d = tid; d < D; d += kTieThreads) {
      const double xd = static_cast<double>(x[d]), yd = __ldcg(a.By + k * Dp + d);
      const double gx = __ldcg(a.GX + k * Dp + d);
      const double gy = grad_at(k, d) - P.tau * yd;
      const double u = yd - (xd + P.eps * gx);
      const double v = xd - (yd + P.eps * gy);
      xx += xd * xd;
      yy += yd * yd;
      q1 += u * u;
      q2 += v * v;
    }
    xx = cta_sum(xx);
    yy = cta_sum(yy);
    q1 = cta_sum(q1);
    q2 = cta_sum(q2);
    const double lp_x = __ldcg(a.lpx + k) - 0.5 * P.tau * xx;
    const double lp_y = loglik(k) - 0.5 * P.tau * yy;
    const double la = (lp_y - q2 * P.inv4eps) - (lp_x - q1 * P.inv4eps);
    if (tid == 0) a.la_ref[t] = la;
    if (a.G.g && tid < 32) {
      const TapeKey key(P.seed, P.block);
      const int iter = st->iter;
      if (a.qpl == 1) finish_column<1>(P, key, x, t, iter, a.G, 0.0, &la);
      else if (a.qpl == 2) finish_column<2>(P, key, x, t, iter, a.G, 0.0, &la);
      else finish_column<4>(P, key, x, t, iter, a.G, 0.0, &la);
    }
  }
  if (blockIdx.x == 0 && tid < kTieBands) a.list.count[tid] = 0;  // every CTA has read them
}

// Verification at a returned trajectory S (after the contraction passes at
// x_bar_t = S_{t-1}): the decision by la_ref, f_t = accept ? y_t : x_bar_t,
// the defect max_d |S_t - f_t| (max into the state), the accept flag and the
// signed margin of every column.
template <typename Real>
__global__ void lg_verify_kernel(const DevParams* __restrict__ Pg, DevState* __restrict__ st,
                                 const double* __restrict__ la_ref) {
  __shared__ double red[32];
  const DevParams& P = *Pg;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t D = P.D, Dp = P.Dp;
  const Real* S = static_cast<const Real*>(P.S[st->cur]);
  const Real* x0 = static_cast<const Real*>(P.x0);
  const Real* yv = static_cast<const Real*>(P.lg[1]);
  const int64_t nw = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
  double def = 0.0;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + warp; t < P.T;
       t += nw) {
    const Real* xb = t == 0 ? x0 : S + (t - 1) * Dp;
    const double la = la_ref[t], logu = P.logu[t];
    const bool acc = logu < la;
    for (int64_t d = lane; d < D; d += 32) {
      const Real f = acc ? yv[t * Dp + d] : xb[d];
      def = fmax(def, fabs(static_cast<double>(S[t * Dp + d]) - static_cast<double>(f)));
    }
    if (lane == 0) {
      P.acc_col[t] = acc ? 1 : 0;
      P.la_col[t] = la - logu;
    }
  }
  def = warp_max(def);
  if (lane == 0) red[warp] = def;
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = 0.0;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) m = fmax(m, red[w]);
    if (m > 0) atomicMax(&st->max_defect_bits, dbits(m));
  }
}

}  // namespace tie

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {
size_t up256(size_t b) { return (b + 255) & ~size_t(255); }
}  // namespace

// Parts of the gradients: more than one only while every part's tile has a warp of its
// own, so at most 256 entries a warp of the largest grid, or one part of all columns.
static size_t tie_gp_elems(int64_t Dp, int kmax) {
  const size_t warps = size_t(256) * tie::kTieCtas * tie::kTieWarps;  // up to 256 SMs
  return std::max(warps * 256, static_cast<size_t>(Dp) * kmax);
}

size_t lg_tie_ws_bytes(const LogisticDev& X, int64_t T, int kmax) {
  const size_t K = static_cast<size_t>(kmax), Dp = static_cast<size_t>(X.Dp);
  const size_t rt = static_cast<size_t>((X.N + 7) / 8);
  return up256(4 * static_cast<size_t>(T)) + up256(4 * K) + up256(16) + 2 * up256(8 * Dp * K) +
         up256(8 * 8 * rt * K) + up256(8 * rt * K) + up256(8 * K) +
         up256(8 * tie_gp_elems(X.Dp, kmax));
}

TieBufs lg_tie_carve(void* ws, const LogisticDev& X, int64_t T, int kmax) {
  TieBufs b{};
  const size_t K = static_cast<size_t>(kmax), Dp = static_cast<size_t>(X.Dp);
  const size_t rt = static_cast<size_t>((X.N + 7) / 8);
  unsigned char* p = static_cast<unsigned char*>(ws);
  auto take = [&](size_t bytes) {
    unsigned char* q = p;
    p += up256(bytes);
    return q;
  };
  b.kmax = kmax;
  b.mg = reinterpret_cast<float*>(take(4 * static_cast<size_t>(T)));
  b.list = reinterpret_cast<int32_t*>(take(4 * K));
  b.count = reinterpret_cast<uint32_t*>(take(16));
  b.By = reinterpret_cast<double*>(take(8 * Dp * K));
  b.GX = reinterpret_cast<double*>(take(8 * Dp * K));
  b.R = reinterpret_cast<double*>(take(8 * 8 * rt * K));
  b.lpP = reinterpret_cast<double*>(take(8 * rt * K));
  b.lpx = reinterpret_cast<double*>(take(8 * K));
  b.GP = reinterpret_cast<double*>(take(8 * tie_gp_elems(X.Dp, kmax)));
  return b;
}

cudaError_t lg_tie_reset(cudaStream_t s, const TieBufs& b) {
  return cudaMemsetAsync(b.count, 0, 16, s);
}

static TieList tie_list(const TieBufs& b, float band) {
  return TieList{band, b.kmax, b.mg, b.list, b.count};
}

cudaError_t lg_margin(cudaStream_t s, bool f64, const DevParams* dP, const DevState* dS,
                      int64_t T, double* la_ref, const TieBufs* b, float band) {
  const int g = static_cast<int>((T + 7) / 8 < 148 * 16 ? (T + 7) / 8 : 148 * 16);
  const TieList list = b ? tie_list(*b, band) : TieList{};
  if (f64) tie::tie_margin_kernel<double><<<g, 256, 0, s>>>(dP, dS, la_ref, list);
  else tie::tie_margin_kernel<float><<<g, 256, 0, s>>>(dP, dS, la_ref, list);
  return cudaGetLastError();
}

cudaError_t lg_tie_solve(cudaStream_t s, const LogisticDev& X, const DevParams* dP,
                         DevState* dS, double* la_ref, const TieBufs& b, float band,
                         const float* G, int nsplit, int64_t T, int num_sms) {
  tie::TieArgs a{};
  a.list = tie_list(b, band);
  a.X = X.X64;
  a.y = X.y64;
  a.N = X.N;
  a.Nr = (X.N + 7) / 8 * 8;
  a.By = b.By;
  a.GX = b.GX;
  a.R = b.R;
  a.lpP = b.lpP;
  a.lpx = b.lpx;
  a.GP = b.GP;
  a.la_ref = la_ref;
  a.G = PassG{G, nsplit};
  a.qpl = X.D <= 128 ? 1 : X.D <= 256 ? 2 : 4;
  void* args[] = {&dP, &dS, &a};
  // A warp a tile of 8 rows and 16 columns, with a near tie in 1024 columns (65 in 65536 at
  // N = 10000, D = 256).  More CTAs only wait at the barriers, and a cooperative launch
  // waits until the other streams' kernels leave room for all of it: with two CTAs on every SM
  // whatever the work, seven chains side by side (N up to 3000, T up to 4900) took 37 ms instead of 26.
  const int64_t want = ((X.N + 7) / 8 * (T / (16 * 1024) + 1) + tie::kTieWarps - 1) / tie::kTieWarps;
  const int grid = static_cast<int>(
      imin64(imax64(want, 16), int64_t(std::min(num_sms, 256)) * tie::kTieCtas));
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(tie::tie_solve_kernel),
                                     dim3(grid), dim3(tie::kTieThreads), args, 0, s);
}

cudaError_t lg_verify(cudaStream_t s, bool f64, const DevParams* dP, DevState* dS, int64_t T,
                      const double* la_ref) {
  const int g = static_cast<int>((T + 7) / 8 < 148 * 16 ? (T + 7) / 8 : 148 * 16);
  if (f64) tie::lg_verify_kernel<double><<<g, 256, 0, s>>>(dP, dS, la_ref);
  else tie::lg_verify_kernel<float><<<g, 256, 0, s>>>(dP, dS, la_ref);
  return cudaGetLastError();
}

}  // namespace pmcmc
