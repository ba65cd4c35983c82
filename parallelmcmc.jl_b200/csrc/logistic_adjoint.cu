// logistic_adjoint.cu -- gradient of a trajectory objective with respect to
// epsilon for the logistic target, at a returned trajectory with its accept
// decisions held fixed.
//
// The objectives are those of the Gaussian adjoint:
//   esjd    = (1/T) sum_t min(1, alpha_t) |y_t - x_{t-1}|^2
//   mean_sq = (1/T) sum_t |x_t|^2
// with the MALA step of src/MALA/MALA.jl:207-229, 377-411 and the logistic
// model of bayes_logreg.jl:30-86.  The derivative is the reverse recurrence
//   lambda_t = c_t + J_{t+1}^T lambda_{t+1},  J_{t+1} = I + eps H(x_t) (accepted) or I,
//   dL/deps  = direct + sum_{t accepted} lambda_t . (g(x_{t-1}) + xi_t / sqrt(2 eps)),
// where c_t (the objective's gradient in x_t) and `direct` (its partial in eps)
// come from per-step terms.  Those need Hessian-vector products at x_{t-1} and
// y_t for every t, batched over the columns (hvp_kernel, GEMMs above 128 coordinates):
//   H(z) V = -X^T (p(1 - p) .* (X V)) - tau V,  p = sigmoid(X z).
// J_{t+1} is dense and changes with t, so the recurrence is not one affine scan
// of diagonal maps.  It is solved by Jacobi iterations on its diagonal part:
//   lambda^{k+1}_t = D_{t+1} lambda^{k+1}_{t+1} + c_t + (J_{t+1} - D_{t+1}) lambda^k_{t+1},
// D_{t+1} = 1 + eps diag H(x_t) = 1 - eps (X.*X)^T p(1 - p) - eps tau; each
// iteration is one batched HVP and one diagonal affine scan (the standalone
// scan, run on the time-reversed arrays).  The fixed point is the
// exact recurrence; the iterations stop when max|lambda^{k+1} - lambda^k| <=
// 1e-12 max|lambda^{k+1}|.
//
// Everything runs in FP64 (FP64 MMAs, and cuBLAS DGEMM with pedantic math) whatever the
// state's type.  Layouts: D-vectors of column t at t * Dp (zero-padded to Dp); N x T
// matrices column-major (column t at t * N).
#include <cublas_v2.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "deer_device.cuh"
#include "deer_launch.h"
#include "logistic.h"
#include "pmcmc_rng.cuh"

namespace pmcmc {
namespace lga {

constexpr int kTh = 256;

__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return s;  // valid in thread 0
}

// XB column t = x_{t-1} (x0 for t = 0) from S (T x D rows of Real) and x0; XI
// column t = xi_t and LU[t] = log u_t of the tape (seed, block).
template <typename Real>
__global__ void setup_kernel(const Real* __restrict__ S, const Real* __restrict__ x0, int D,
                             int Dp, int64_t T, uint64_t seed, uint64_t block,
                             double* __restrict__ XB, double* __restrict__ XI,
                             double* __restrict__ LU) {
  const TapeKey key(seed, block);
  const int nq = Dp / 4;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < T * nq;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / nq;
    const int j = static_cast<int>(i - t * nq);
    float n[4];
    tape_xi4(key, static_cast<uint32_t>(j), static_cast<uint32_t>(t), n);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = 4 * j + e;
      const bool in = d < D;
      XI[t * Dp + d] = in ? static_cast<double>(n[e]) : 0.0;
      XB[t * Dp + d] = in ? static_cast<double>(t == 0 ? x0[d] : S[(t - 1) * D + d]) : 0.0;
    }
    if (j == 0) LU[t] = log(static_cast<double>(tape_u(key, static_cast<uint32_t>(t))));
  }
}

// Per column t of L = X Z (N x T): R = y - p in place, W = p (1 - p), and the
// log-likelihood sum_n y_n L - softplus(L) into ll[t].  One block a column.
__global__ void lik_kernel(double* __restrict__ L, const double* __restrict__ ylab, int64_t N,
                           double* __restrict__ W, double* __restrict__ ll) {
  __shared__ double sh[kTh / 32];
  const int64_t t = blockIdx.x;
  double* col = L + t * N;
  double* wc = W + t * N;
  double s = 0.0;
  for (int64_t n = threadIdx.x; n < N; n += blockDim.x) {
    const double l = col[n];
    const double e = exp(-fabs(l));
    const double p = l >= 0 ? 1.0 / (1.0 + e) : e / (1.0 + e);
    s += ylab[n] * l - (fmax(l, 0.0) + log1p(e));
    col[n] = ylab[n] - p;
    wc[n] = p * (1.0 - p);
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) ll[t] = s;
}

// An FP64 MMA (16 x 8, k = 8): with r = l / 4 and q = l % 4, lane l holds A[r + 8 (i % 2)]
// [q + 4 (i / 2)], B[q + 4 i][r] and C[r + 8 (i / 2)][2 q + i % 2].
__device__ __forceinline__ void dmma(double (&c)[4], const double (&a)[4], const double (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// 16 bytes into shared memory, zeros unless `in`.
__device__ __forceinline__ void cp16(double* dst, const double* src, bool in) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src),
               "r"(in ? 16 : 0)
               : "memory");
}

// X^T (W .* (X V)) over the rows of split blockIdx.y, 32 columns a CTA, into P + split *
// Dp * n.  Per chunk of 64 rows: the logits' derivative tile L = (X V) .* W (a warp: 16
// rows, 16 columns), then acc += X^T L (a warp: every fourth tile of 16 coordinates) -- X
// is read once, L stays in shared memory and the sums over the rows in registers.  The FP64
// tensor rate bounds it (2 N Dp n products; a warp loads 1 byte of shared memory a product,
// half of what an MMA's time allows).  Row strides of 4 mod 16 doubles keep the fragments
// conflict-free.  N = 2000, D = 64, n = 2048: 52 us (20 TFLOP/s; 55 with 8 x 8 x 4 MMAs),
// against 62 for two DGEMMs, their split-k reduction, the product with W between them
// and the axpby after.
constexpr int kHvRows = 64, kHvCols = 32, kHvMaxDp = 128, kHvSL = kHvRows + 4;
__host__ __device__ inline int hv_stride(int Dp) { return ((Dp + 15) / 16 * 16 + 11) / 16 * 16 + 4; }
inline size_t hv_smem(int Dp) {
  return 8 * (static_cast<size_t>(2 * kHvRows + kHvCols) * hv_stride(Dp) + kHvCols * kHvSL);
}
template <int ND>  // tiles of 16 coordinates a warp
__global__ void __launch_bounds__(kTh)
    hvp_kernel(const double* __restrict__ X, const double* __restrict__ W,
               const double* __restrict__ V, int64_t N, int Dp, int64_t n,
               double* __restrict__ P) {
  extern __shared__ __align__(16) double sh[];
  const int SX = hv_stride(Dp);
  double* Xs = sh;                         // two chunks of rows
  double* Vs = Xs + 2 * kHvRows * SX;      // the columns
  double* Ls = Vs + kHvCols * SX;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r8 = lane >> 2, k4 = lane & 3;
  const int64_t c0 = static_cast<int64_t>(blockIdx.x) * kHvCols;
  const int64_t chunks = (N + kHvRows - 1) / kHvRows;
  const int64_t ch0 = chunks * blockIdx.y / gridDim.y, ch1 = chunks * (blockIdx.y + 1) / gridDim.y;
  const int h = Dp / 2;  // pairs a row
  auto fetch = [&](int64_t ch) {
    if (ch < ch1)
      for (int i = tid; i < kHvRows * h; i += kTh) {
        const int r = i / h, k = 2 * (i - r * h);
        const int64_t row = ch * kHvRows + r;
        cp16(Xs + ((ch & 1) * kHvRows + r) * SX + k, X + (row < N ? row : 0) * Dp + k, row < N);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = tid; i < kHvCols * h; i += kTh) {
    const int c = i / h, k = 2 * (i - c * h);
    cp16(Vs + c * SX + k, V + (c0 + c < n ? c0 + c : 0) * Dp + k, c0 + c < n);
  }
  fetch(ch0);
  fetch(ch0 + 1);
  const int m = warp % 4, cw = 16 * (warp / 4);  // the warp's 16 rows (and coordinates), 16 columns
  double acc[ND][2][4] = {};
  for (int64_t ch = ch0; ch < ch1; ++ch) {
    double w[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int64_t row = ch * kHvRows + 16 * m + 8 * (e / 2) + r8;
        const int64_t c = c0 + cw + 8 * j + 2 * k4 + e % 2;
        w[j][e] = row < N && c < n ? __ldg(W + c * N + row) : 0.0;
      }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // the chunk has arrived, the last one's L is read
    const double* Xc = Xs + (ch & 1) * kHvRows * SX;
    double l[2][4] = {};
    {
      const double* a = Xc + (16 * m + r8) * SX + k4;
      const double* b = Vs + (cw + r8) * SX + k4;
#pragma unroll 2
      for (int k = 0; k < Dp; k += 8) {  // (Dp a multiple of 4: the last half step multiplies zeros)
        const bool two = k + 4 < Dp;
        double av[4], bv[2][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) av[i] = i < 2 || two ? a[8 * (i % 2) * SX + k + 4 * (i / 2)] : 0.0;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < 2; ++i) bv[j][i] = i == 0 || two ? b[8 * j * SX + k + 4 * i] : 0.0;
        dmma(l[0], av, bv[0]);
        dmma(l[1], av, bv[1]);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        Ls[(cw + 8 * j + 2 * k4 + e % 2) * kHvSL + 16 * m + 8 * (e / 2) + r8] = l[j][e] * w[j][e];
    __syncthreads();
    {
      const double* a = Xc + k4 * SX + 16 * m + r8;
      const double* b = Ls + (cw + r8) * kHvSL + k4;
#pragma unroll 2
      for (int k = 0; k < kHvRows; k += 8) {
        double bv[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int i = 0; i < 2; ++i) bv[j][i] = b[8 * j * kHvSL + k + 4 * i];
#pragma unroll
        for (int t = 0; t < ND; ++t)
          if (16 * (m + 4 * t) < Dp) {
            double av[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) av[i] = a[(k + 4 * (i / 2)) * SX + 64 * t + 8 * (i % 2)];
            dmma(acc[t][0], av, bv[0]);
            dmma(acc[t][1], av, bv[1]);
          }
      }
    }
    __syncthreads();  // this chunk's slot is free
    fetch(ch + 2);
  }
  double* out = P + static_cast<size_t>(blockIdx.y) * Dp * n;
#pragma unroll
  for (int t = 0; t < ND; ++t)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = 16 * (m + 4 * t) + 8 * (e / 2) + r8;
        const int64_t c = c0 + cw + 8 * j + 2 * k4 + e % 2;
        if (d < Dp && c < n) out[c * Dp + d] = acc[t][j][e];
      }
}

// A Hessian-vector product whose sum over the rows is in ns parts, `stride` apart:
// -(P_0 + ... ) - tau v (ns = 0: the product itself).
struct HvSum {
  const double* P;
  int ns;
  size_t stride;
  double tau;
  __device__ __forceinline__ double at(size_t i, double v) const {
    if (ns == 0) return P[i];
    double s = P[i];
    for (int k = 1; k < ns; ++k) s += P[k * stride + i];
    return -s - tau * v;
  }
};
__global__ void hvsum_kernel(HvSum h, const double* V, double* out, int64_t n) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[i] = h.at(i, V[i]);
}

// L .* W elementwise (N x T).
__global__ void mulw_kernel(double* __restrict__ L, const double* __restrict__ W, int64_t n) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    L[i] *= W[i];
}

// out = a * out + b * V over Dp x T (padded rows stay zero: V and out are zero there).
__global__ void axpby_kernel(double* __restrict__ out, double a, const double* __restrict__ V,
                             double b, int64_t n) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[i] = a * out[i] + b * V[i];
}

// GX = G - tau XB;  Y = XB + eps GX + sqrt(2 eps) XI.
__global__ void propose_kernel(const double* __restrict__ XB, const double* __restrict__ XI,
                               double* __restrict__ GX, double* __restrict__ Y, double eps,
                               double tau, int64_t n) {
  const double c = sqrt(2.0 * eps);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double g = GX[i] - tau * XB[i];
    GX[i] = g;
    Y[i] = XB[i] + eps * g + c * XI[i];
  }
}

// Per column t: Q = XB - Y - eps GY, DY = GX + XI / sqrt(2 eps), E = Y - XB; log
// alpha (FP64, the sequential chain's formula), the accept flag, alpha, its
// derivative in log alpha and |E|^2.  One warp a column.
__global__ void local1_kernel(const double* __restrict__ XB, const double* __restrict__ Y,
                              const double* __restrict__ GX, const double* __restrict__ GY,
                              const double* __restrict__ XI, const double* __restrict__ LU,
                              const double* __restrict__ llx, const double* __restrict__ lly,
                              int Dp, int64_t T, double eps, double tau, double* __restrict__ Q,
                              double* __restrict__ DY, double* __restrict__ E,
                              double* __restrict__ sc) {
  const int lane = threadIdx.x & 31;
  const int64_t t = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (t >= T) return;
  const double rs = 1.0 / sqrt(2.0 * eps);
  double xx = 0, yy = 0, qq = 0, ii = 0, ee = 0;
  for (int d = lane; d < Dp; d += 32) {
    const int64_t k = t * Dp + d;
    const double x = XB[k], y = Y[k], xi = XI[k];
    const double q = x - y - eps * GY[k];
    const double e = y - x;
    Q[k] = q;
    DY[k] = GX[k] + xi * rs;
    E[k] = e;
    xx += x * x;
    yy += y * y;
    qq += q * q;
    ii += xi * xi;
    ee += e * e;
  }
  for (int o = 16; o > 0; o >>= 1) {
    xx += __shfl_xor_sync(0xffffffffu, xx, o);
    yy += __shfl_xor_sync(0xffffffffu, yy, o);
    qq += __shfl_xor_sync(0xffffffffu, qq, o);
    ii += __shfl_xor_sync(0xffffffffu, ii, o);
    ee += __shfl_xor_sync(0xffffffffu, ee, o);
  }
  if (lane == 0) {
    const double la = (lly[t] - 0.5 * tau * yy) - (llx[t] - 0.5 * tau * xx) - qq / (4.0 * eps) +
                      0.5 * ii;
    const bool acc = LU[t] < la;
    const double alpha = la < 0.0 ? exp(la) : 1.0;
    double* s = sc + 8 * t;
    s[0] = la;
    s[1] = acc ? 1.0 : 0.0;
    s[2] = alpha;
    s[3] = la < 0.0 ? alpha : 0.0;  // d alpha / d log alpha
    s[4] = ee;
    s[5] = qq;
  }
}

// Per column t (esjd): dq = -(DY + eps H(y) DY) - GY, the partial of log alpha
// in eps, and the direct term s[6] = dalpha dla e2 + alpha 2 E . DY; the vector
// w = Q + eps H(y) Q in place of HQ.  One warp a column.
__global__ void local2_kernel(const double* __restrict__ GY, const double* __restrict__ DY,
                              const double* __restrict__ Q, const double* __restrict__ E,
                              const double* __restrict__ HyDY, double* __restrict__ HyQ, int Dp,
                              int64_t T, double eps, double* __restrict__ sc) {
  const int lane = threadIdx.x & 31;
  const int64_t t = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (t >= T) return;
  double gd = 0, qdq = 0, edy = 0;
  for (int d = lane; d < Dp; d += 32) {
    const int64_t k = t * Dp + d;
    const double dy = DY[k], q = Q[k];
    const double dq = -(dy + eps * HyDY[k]) - GY[k];
    gd += GY[k] * dy;
    qdq += q * dq;
    edy += E[k] * dy;
    HyQ[k] = q + eps * HyQ[k];
  }
  for (int o = 16; o > 0; o >>= 1) {
    gd += __shfl_xor_sync(0xffffffffu, gd, o);
    qdq += __shfl_xor_sync(0xffffffffu, qdq, o);
    edy += __shfl_xor_sync(0xffffffffu, edy, o);
  }
  if (lane == 0) {
    double* s = sc + 8 * t;
    const double dla = gd - qdq / (2.0 * eps) + s[5] / (4.0 * eps * eps);
    s[6] = s[3] * dla * s[4] + s[2] * 2.0 * edy;
  }
}

// c_{t-1} (esjd) for t >= 1: (dalpha e2 v + alpha 2 eps H(x) E) / T with
// v = J_x GY - GX - (Q - J_x w) / (2 eps), J_x = I + eps H(x_{t-1}); c_{T-1} = 0.
__global__ void cvec_esjd_kernel(const double* __restrict__ GY, const double* __restrict__ GX,
                                 const double* __restrict__ Q, const double* __restrict__ Wv,
                                 const double* __restrict__ HxGY, const double* __restrict__ HxW,
                                 const double* __restrict__ HxE, const double* __restrict__ sc,
                                 int Dp, int64_t T, double eps, double* __restrict__ C) {
  const double invT = 1.0 / static_cast<double>(T);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < T * Dp;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / Dp + 1;  // the step whose terms land on column t - 1
    if (t >= T) {
      C[i] = 0.0;
      continue;
    }
    const int64_t k = i + Dp;  // column t
    const double* s = sc + 8 * t;
    const double jgy = GY[k] + eps * HxGY[k];
    const double jw = Wv[k] + eps * HxW[k];
    const double v = jgy - GX[k] - (Q[k] - jw) / (2.0 * eps);
    C[i] = (s[3] * s[4] * v + s[2] * 2.0 * eps * HxE[k]) * invT;
  }
}

// c_t (mean_sq) = 2 S_t / T: S_t is XB column t + 1, and the last row of S for t = T - 1.
template <typename Real>
__global__ void cvec_msq_kernel(const double* __restrict__ XB, const Real* __restrict__ S, int D,
                                int Dp, int64_t T, double* __restrict__ C) {
  const double k2 = 2.0 / static_cast<double>(T);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < T * Dp;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / Dp;
    const int d = static_cast<int>(i - t * Dp);
    const double st = t + 1 < T ? XB[i + Dp]
                      : d < D   ? static_cast<double>(S[(T - 1) * D + d])
                                : 0.0;
    C[i] = k2 * st;
  }
}

// DJ = 1 + eps (G - tau), G = -(X.*X)^T W computed by the caller.
__global__ void diagj_kernel(double* __restrict__ DJ, int D, int Dp, int64_t T, double eps,
                             double tau) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < T * Dp;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int d = static_cast<int>(i % Dp);
    DJ[i] = d < D ? 1.0 + eps * (-DJ[i] - tau) : 0.0;
  }
}

// The diagonal affine maps of one Jacobi iteration, time-reversed (row s holds
// step t = T - 1 - s): lambda_t = a_t lambda_{t+1} + b_t.  HL column t is
// H(x_t) lambda^k_{t+1} (t < T - 1), its parts summed here.
__global__ void revmaps_kernel(const double* __restrict__ C, const double* __restrict__ LAM,
                               const HvSum HL, const double* __restrict__ DJ,
                               const double* __restrict__ sc, int Dp, int64_t T, double eps,
                               double* __restrict__ Ar, double* __restrict__ Br) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < T * Dp;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / Dp, d = i - t * Dp;
    const int64_t r = (T - 1 - t) * Dp + d;
    double a = 0.0, b = C[i];
    if (t + 1 < T) {
      if (sc[8 * (t + 1) + 1] != 0.0) {
        const double dj = DJ[i + Dp], lk = LAM[i + Dp];
        a = dj;
        b += lk + eps * HL.at(i, lk) - dj * lk;
      } else {
        a = 1.0;
      }
    }
    Ar[r] = a;
    Br[r] = b;
  }
}

// LAM_new column t = Sr row T - 1 - t; per-block maxima of |new - old| and
// |new| into part[2 * block .. ], and over the blocks (in the last one to end, `left`
// counts them and is 0 again after) into out.
__global__ void revgather_kernel(const double* __restrict__ Sr, double* __restrict__ LAM,
                                 int Dp, int64_t T, double* __restrict__ part,
                                 unsigned* __restrict__ left, double* __restrict__ out) {
  __shared__ double sd[kTh], sm[kTh];
  __shared__ bool last;
  double md = 0.0, mx = 0.0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < T * Dp;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / Dp, d = i - t * Dp;
    const double v = Sr[(T - 1 - t) * Dp + d];
    md = fmax(md, fabs(v - LAM[i]));
    mx = fmax(mx, fabs(v));
    LAM[i] = v;
  }
  sd[threadIdx.x] = md;
  sm[threadIdx.x] = mx;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      sd[threadIdx.x] = fmax(sd[threadIdx.x], sd[threadIdx.x + o]);
      sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = sd[0];
    part[2 * blockIdx.x + 1] = sm[0];
    __threadfence();
    last = atomicAdd(left, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  md = mx = 0.0;
  for (int b = threadIdx.x; b < static_cast<int>(gridDim.x); b += kTh) {
    const double d = __ldcg(part + 2 * b), m = __ldcg(part + 2 * b + 1);
    md = fmax(md, d);
    mx = fmax(mx, m);
  }
  sd[threadIdx.x] = md;
  sm[threadIdx.x] = mx;
  __syncthreads();
  for (int o = kTh / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      sd[threadIdx.x] = fmax(sd[threadIdx.x], sd[threadIdx.x + o]);
      sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = sd[0];
    out[1] = sm[0];
    *left = 0;
  }
}

// sc[8 t + 7] = LAM_t . DY_t of the accepted columns (one warp a column; in the one block
// that sums them, a thread a column, the uncoalesced reads took 130 us at T = 2048, D = 64).
__global__ void lamdy_kernel(const double* __restrict__ LAM, const double* __restrict__ DY,
                             double* __restrict__ sc, int Dp, int64_t T) {
  const int lane = threadIdx.x & 31;
  const int64_t t = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  if (t >= T) return;
  double v = 0.0;
  if (sc[8 * t + 1] != 0.0)
    for (int d = lane; d < Dp; d += 32) v += LAM[t * Dp + d] * DY[t * Dp + d];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) sc[8 * t + 7] = v;
}

// out[0] = sum_t direct_t / T (esjd) + sum_{t accepted} LAM_t . DY_t, in a
// fixed order (one block).
__global__ void final_kernel(const double* __restrict__ sc, int64_t T, int esjd,
                             double* __restrict__ out) {
  __shared__ double sh[kTh / 32];
  double s = 0.0;
  for (int64_t t = threadIdx.x; t < T; t += blockDim.x) {
    const double* st = sc + 8 * t;
    if (esjd) s += st[6] / static_cast<double>(T);
    s += st[7];
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) out[0] = s;
}

inline int grid_for(int64_t n) {
  const int64_t g = (n + kTh - 1) / kTh;
  return static_cast<int>(g < 148 * 8 ? (g > 0 ? g : 1) : 148 * 8);
}

}  // namespace lga

namespace {

// The workspace carve of lg_adjoint, in doubles: every array rounded up to 32
// (256 bytes).  The size and the carve both come from here.
struct AdjLayout {
  size_t v, m;  // one Dp x T and one N x T array
  int gpart;
  size_t total;  // doubles
};

inline size_t r32(size_t n) { return (n + 31) & ~size_t(31); }

AdjLayout adj_layout(const LogisticDev& X, int64_t T) {
  const int64_t N = X.N, Dp = X.Dp;
  AdjLayout a{};
  a.v = static_cast<size_t>(Dp) * T;
  a.m = static_cast<size_t>(N) * T;
  a.gpart = std::min(X.num_sms, lga::grid_for(Dp * T));  // (each ends with an atomic)
  const size_t t = static_cast<size_t>(T);
  a.total = 16 * r32(a.v) + 3 * r32(a.m) + 3 * r32(t) + r32(8 * t) +
            r32(2 * static_cast<size_t>(a.gpart)) + r32(8) + r32(static_cast<size_t>(Dp));
  return a;
}

}  // namespace

size_t lg_adjoint_ws_bytes(const LogisticDev& X, int64_t T) {
  return 8 * adj_layout(X, T).total;
}

namespace {

// -X^T (W .* (X V)) - tau V for n columns, `sum` its parts: up to kHvMaxDp coordinates by
// hvp_kernel, the rows in as many splits as fill the chip and fit L (N x n), or in one into
// `out`; above, where the products dominate, by two DGEMMs over L into `out`.
int hvp_parts(cudaStream_t s, cublasHandle_t cb, const LogisticDev& X, const double* W,
              const double* V, int64_t n, double* L, double* out, lga::HvSum* sum) {
  const double one = 1.0, zero = 0.0, mone = -1.0;
  const int N = static_cast<int>(X.N), dp = static_cast<int>(X.Dp), nc = static_cast<int>(n);
  if (dp <= lga::kHvMaxDp) {
    const int64_t tiles = (n + lga::kHvCols - 1) / lga::kHvCols;
    const int64_t chunks = (X.N + lga::kHvRows - 1) / lga::kHvRows;
    const int64_t slots = X.num_sms * (dp <= 64 ? 2 : 1);
    const int64_t ns =
        std::max<int64_t>(1, std::min({slots / tiles, chunks, X.N / X.Dp, int64_t(16)}));
    double* P = ns > 1 ? L : out;
    const size_t smem = lga::hv_smem(dp);
    auto k = dp <= 64 ? lga::hvp_kernel<1> : lga::hvp_kernel<2>;
    if (raise_smem_limit(reinterpret_cast<const void*>(k), smem) != cudaSuccess) return 3;
    k<<<dim3(static_cast<unsigned>(tiles), static_cast<unsigned>(ns)), lga::kTh, smem, s>>>(
        X.X64, W, V, X.N, dp, n, P);
    *sum = lga::HvSum{P, static_cast<int>(ns), static_cast<size_t>(X.Dp) * n, X.tau};
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
  }
  if (cublasDgemm(cb, CUBLAS_OP_T, CUBLAS_OP_N, N, nc, dp, &one, X.X64, dp, V, dp, &zero, L, N) !=
      CUBLAS_STATUS_SUCCESS)
    return 3;
  lga::mulw_kernel<<<lga::grid_for(X.N * n), lga::kTh, 0, s>>>(L, W, X.N * n);
  if (cublasDgemm(cb, CUBLAS_OP_N, CUBLAS_OP_N, dp, nc, N, &mone, X.X64, dp, L, N, &zero, out,
                  dp) != CUBLAS_STATUS_SUCCESS)
    return 3;
  lga::axpby_kernel<<<lga::grid_for(X.Dp * n), lga::kTh, 0, s>>>(out, 1.0, V, -X.tau, X.Dp * n);
  *sum = lga::HvSum{out, 0, 0, 0.0};
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

// H(z) V in one array.
int hvp(cudaStream_t s, cublasHandle_t cb, const LogisticDev& X, const double* W, const double* V,
        int64_t n, double* L, double* out) {
  lga::HvSum h{};
  const int rc = hvp_parts(s, cb, X, W, V, n, L, out, &h);
  if (rc || h.ns == 0) return rc;
  lga::hvsum_kernel<<<lga::grid_for(X.Dp * n), lga::kTh, 0, s>>>(h, V, out, X.Dp * n);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

}  // namespace

int lg_adjoint(cudaStream_t s, cublasHandle_t cb, const LogisticDev& X, bool f64,
               const void* x0, const void* S, uint64_t seed, uint64_t block, int64_t T,
               double eps, int esjd, void* ws, int max_iter, double* grad_eps, int* iters,
               ScanFn scan, void* scan_ctx) {
  using namespace lga;
  const int64_t Dp = X.Dp, N = X.N;
  const int D = static_cast<int>(X.D);
  const AdjLayout Ly = adj_layout(X, T);
  const size_t v = Ly.v, m = Ly.m;
  double* p = static_cast<double*>(ws);
  double* const end = p + Ly.total;
  auto take = [&](size_t n) {
    double* r = p;
    p += r32(n);
    return r;
  };
  double *XB = take(v), *XI = take(v), *GX = take(v), *Y = take(v), *GY = take(v), *Q = take(v),
         *DY = take(v), *E = take(v), *V1 = take(v), *V2 = take(v), *V3 = take(v), *V4 = take(v),
         *C = take(v), *LAM = take(v), *Ar = take(v), *Br = take(v);
  double *Lb = take(m), *Wx = take(m), *Wy = take(m);
  double *LU = take(T), *llx = take(T), *lly = take(T), *sc = take(8 * T);
  const int gpart = Ly.gpart;
  double* part = take(2 * static_cast<size_t>(gpart));
  double* out = take(8);
  double* s0 = take(static_cast<size_t>(Dp));
  if (p > end) return 3;  // the carve must fit the layout it was sized from
  const double one = 1.0, zero = 0.0;
  const int n = static_cast<int>(N), dp = static_cast<int>(Dp), Tc = static_cast<int>(T);
  const int gv = grid_for(static_cast<int64_t>(v));
  if (f64)
    setup_kernel<double><<<gv, kTh, 0, s>>>(static_cast<const double*>(S),
                                            static_cast<const double*>(x0), D, dp, T, seed, block,
                                            XB, XI, LU);
  else
    setup_kernel<float><<<gv, kTh, 0, s>>>(static_cast<const float*>(S),
                                           static_cast<const float*>(x0), D, dp, T, seed, block,
                                           XB, XI, LU);
  // ---- forward quantities at x_{t-1} and y_t ----
  if (cublasDgemm(cb, CUBLAS_OP_T, CUBLAS_OP_N, n, Tc, dp, &one, X.X64, dp, XB, dp, &zero, Lb,
                  n) != CUBLAS_STATUS_SUCCESS)
    return 3;
  lik_kernel<<<Tc, kTh, 0, s>>>(Lb, X.y64, N, Wx, llx);
  if (cublasDgemm(cb, CUBLAS_OP_N, CUBLAS_OP_N, dp, Tc, n, &one, X.X64, dp, Lb, n, &zero, GX,
                  dp) != CUBLAS_STATUS_SUCCESS)
    return 3;
  propose_kernel<<<gv, kTh, 0, s>>>(XB, XI, GX, Y, eps, X.tau, static_cast<int64_t>(v));
  if (cublasDgemm(cb, CUBLAS_OP_T, CUBLAS_OP_N, n, Tc, dp, &one, X.X64, dp, Y, dp, &zero, Lb, n) !=
      CUBLAS_STATUS_SUCCESS)
    return 3;
  lik_kernel<<<Tc, kTh, 0, s>>>(Lb, X.y64, N, Wy, lly);
  if (cublasDgemm(cb, CUBLAS_OP_N, CUBLAS_OP_N, dp, Tc, n, &one, X.X64, dp, Lb, n, &zero, GY,
                  dp) != CUBLAS_STATUS_SUCCESS)
    return 3;
  axpby_kernel<<<gv, kTh, 0, s>>>(GY, 1.0, Y, -X.tau, static_cast<int64_t>(v));
  const int gw = static_cast<int>((32 * T + kTh - 1) / kTh);
  local1_kernel<<<gw, kTh, 0, s>>>(XB, Y, GX, GY, XI, LU, llx, lly, dp, T, eps, X.tau, Q, DY, E,
                                   sc);
  if (cudaGetLastError() != cudaSuccess) return 3;
  // ---- c_t and the direct term ----
  if (esjd) {
    if (hvp(s, cb, X, Wy, DY, T, Lb, V1)) return 3;  // H(y) DY
    if (hvp(s, cb, X, Wy, Q, T, Lb, V2)) return 3;   // H(y) Q
    local2_kernel<<<gw, kTh, 0, s>>>(GY, DY, Q, E, V1, V2, dp, T, eps, sc);  // V2 <- w
    if (hvp(s, cb, X, Wx, GY, T, Lb, V1)) return 3;  // H(x) GY
    if (hvp(s, cb, X, Wx, V2, T, Lb, V3)) return 3;  // H(x) w
    if (hvp(s, cb, X, Wx, E, T, Lb, V4)) return 3;   // H(x) E
    cvec_esjd_kernel<<<gv, kTh, 0, s>>>(GY, GX, Q, V2, V1, V3, V4, sc, dp, T, eps, C);
  } else if (f64) {
    cvec_msq_kernel<double><<<gv, kTh, 0, s>>>(XB, static_cast<const double*>(S), D, dp, T, C);
  } else {
    cvec_msq_kernel<float><<<gv, kTh, 0, s>>>(XB, static_cast<const float*>(S), D, dp, T, C);
  }
  // ---- D_t = diag J_t: 1 + eps diag H(x_{t-1}) ----
  double* DJ = V4;  // H(x) E is consumed
  if (cublasDgemm(cb, CUBLAS_OP_N, CUBLAS_OP_N, dp, Tc, n, &one, X.X2_64, dp, Wx, n, &zero, DJ,
                  dp) != CUBLAS_STATUS_SUCCESS)
    return 3;
  diagj_kernel<<<gv, kTh, 0, s>>>(DJ, D, dp, T, eps, X.tau);
  // ---- Jacobi iterations on lambda_t = c_t + J_{t+1} lambda_{t+1} ----
  if (cudaMemcpyAsync(LAM, C, 8 * v, cudaMemcpyDeviceToDevice, s) != cudaSuccess) return 3;
  if (cudaMemsetAsync(s0, 0, 8 * Dp, s) != cudaSuccess) return 3;
  double* HL = V1;
  double* Sr = V3;
  int k = 0;
  bool done = false;
  unsigned* left = reinterpret_cast<unsigned*>(out + 4);
  if (cudaMemsetAsync(left, 0, 8, s) != cudaSuccess) return 3;
  for (; k < max_iter && !done; ++k) {
    // HL column t = H(x_t) lambda^k_{t+1}: W column t + 1 (x_t = XB column t + 1)
    HvSum hl{HL, 0, 0, 0.0};
    if (T > 1 && hvp_parts(s, cb, X, Wx + N, LAM + Dp, T - 1, Lb, HL, &hl)) return 3;
    revmaps_kernel<<<gv, kTh, 0, s>>>(C, LAM, hl, DJ, sc, dp, T, eps, Ar, Br);
    if (cudaGetLastError() != cudaSuccess) return 3;
    const int rc = scan(scan_ctx, Dp, T, Ar, Br, s0, Sr);
    if (rc) return rc;
    revgather_kernel<<<gpart, kTh, 0, s>>>(Sr, LAM, dp, T, part, left, out);
    double mm[2];
    if (cudaMemcpyAsync(mm, out, sizeof mm, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
      return 3;
    const double md = mm[0], mx = mm[1];
    if (!std::isfinite(md) || !std::isfinite(mx)) return 4;
    done = md <= 1e-12 * mx || mx == 0.0;
  }
  lamdy_kernel<<<gw, kTh, 0, s>>>(LAM, DY, sc, dp, T);
  final_kernel<<<1, kTh, 0, s>>>(sc, T, esjd, out);
  if (cudaMemcpyAsync(grad_eps, out, 8, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return 3;
  *iters = k;
  return done ? 0 : 5;
}

}  // namespace pmcmc
