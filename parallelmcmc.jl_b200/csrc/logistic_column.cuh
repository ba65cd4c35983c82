// logistic_column.cuh -- one column's finish on the tensor-core path of the logistic
// target: from the second pass's G to log alpha, the accept decision and the column's
// affine map (A, B).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "deer_column.cuh"
#include "deer_device.cuh"

namespace pmcmc {

// The second pass's G (nsplit parts of 2T x Dp: value block, then tangent block).
struct PassG {
  const float* g;
  int nsplit;
};

// Rest of the batched fwd + JVP (MALA.jl:592-625) for column t, one warp, one Hutchinson
// probe: g_y = X'r - tau y, H(y) w = -X's - tau w from G; log alpha in FP64 (the
// likelihood part dlp = loglik(y) - loglik(x) given), or la_fixed where it is not NULL;
// A = z .* J z and B = f - A .* x_bar into lg[3] and lg[4].  Returns log alpha.
template <int QPL>
__device__ __forceinline__ double finish_column(const DevParams& P, const TapeKey& key,
                                                const float* xcol, int64_t t, int iter,
                                                const PassG& G, double dlp,
                                                const double* la_fixed) {
  const int lane = threadIdx.x & 31;
  const int D = static_cast<int>(P.D), Dp = static_cast<int>(P.Dp);
  const float eps = static_cast<float>(P.eps), inv2eps = static_cast<float>(P.inv2eps);
  const float tau = static_cast<float>(P.tau);
  const size_t off = static_cast<size_t>(t) * Dp;
  const size_t half = static_cast<size_t>(P.T) * Dp;
  float x[QPL][4], gx[QPL][4], y[QPL][4], gy[QPL][4], w[QPL][4], hvy[QPL][4], z[QPL][4];
  double la = 0.0;
#pragma unroll
  for (int q = 0; q < QPL; ++q) {
    const int j = lane + 32 * q;
    if (4 * j < D) {
      float xi[4];
      load4(xcol + 4 * j, x[q]);
      load4(static_cast<const float*>(P.lg[0]) + off + 4 * j, gx[q]);
      load4(static_cast<const float*>(P.lg[1]) + off + 4 * j, y[q]);
      load4(static_cast<const float*>(P.lg[2]) + off + 4 * j, w[q]);
      load4(P.xi + off + 4 * j, xi);
      const float* gp = G.g + off + 4 * j;
      load4(gp, gy[q]);
      load4(gp + half, hvy[q]);
      for (int p = 1; p < G.nsplit; ++p) {  // the pass's parts, in order
        float a[4], b[4];
        load4(gp + 2 * half * p, a);
        load4(gp + 2 * half * p + half, b);
#pragma unroll
        for (int e = 0; e < 4; ++e) gy[q][e] += a[e], hvy[q][e] += b[e];
      }
      const U4 pb = probe_bits(key, static_cast<uint32_t>(j >> 5),
                               static_cast<uint32_t>(t + P.t_off), 0, iter);
      const uint32_t wv = u4_word(pb, (j >> 3) & 3);
      const int sh = (j & 7) * 4;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool in = 4 * j + e < D;
        gy[q][e] = in ? gy[q][e] - tau * y[q][e] : 0.f;
        hvy[q][e] = in ? -hvy[q][e] - tau * w[q][e] : 0.f;
        z[q][e] = in ? (((wv >> (sh + e)) & 1u) ? 1.f : -1.f) : 0.f;
        if (in) {
          const double xd = static_cast<double>(x[q][e]), yd = static_cast<double>(y[q][e]);
          const double r1 = P.sqrt2eps * static_cast<double>(xi[e]);
          const double r2 = (xd - yd) - P.eps * static_cast<double>(gy[q][e]);
          la += -0.5 * P.tau * (yd * yd - xd * xd) + (r1 * r1 - r2 * r2) * P.inv4eps;
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        x[q][e] = gx[q][e] = y[q][e] = gy[q][e] = w[q][e] = hvy[q][e] = z[q][e] = 0.f;
    }
  }
  la = warp_sum(la) + dlp;
  if (la_fixed) la = *la_fixed;
  const double logu = P.logu[t];
  const bool acc = logu < la;
  const float gs = sigmoid_slope<float>(la - logu);
  float dla = 0.f;
#pragma unroll
  for (int q = 0; q < QPL; ++q)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float r = x[q][e] - y[q][e] - eps * gy[q][e];
      const float dr = z[q][e] - w[q][e] - eps * hvy[q][e];
      dla += gy[q][e] * w[q][e] - gx[q][e] * z[q][e] - inv2eps * r * dr;
    }
  const float dg = gs * warp_sum(dla);
#pragma unroll
  for (int q = 0; q < QPL; ++q) {
    const int j = lane + 32 * q;
    if (4 * j < Dp) {
      float a[4], b[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float jz = (acc ? w[q][e] : z[q][e]) + (y[q][e] - x[q][e]) * dg;
        a[e] = z[q][e] * jz;
        b[e] = (acc ? y[q][e] : x[q][e]) - a[e] * x[q][e];
      }
      store4(static_cast<float*>(P.lg[3]) + off + 4 * j, a);
      store4(static_cast<float*>(P.lg[4]) + off + 4 * j, b);
    }
  }
  if (lane == 0) {
    P.acc_col[t] = acc ? 1 : 0;
    P.la_col[t] = la - logu;
  }
  return la;
}

// Columns whose margin lies within the near-tie band (logistic_tie.cu): counted in the
// nested bands band / 4^i, those of the widest listed while they fit.  count[0..3] start
// at zero and are cleared by the kernel that takes the list.
struct TieList {
  float band;
  int kmax;
  float* mg;         // [T] |margin|
  int32_t* list;     // [kmax]
  uint32_t* count;   // [4]
};
constexpr int kTieBands = 4;
__device__ __forceinline__ void tie_note(const TieList& L, int64_t t, double margin) {
  const float m = static_cast<float>(fabs(margin));
  L.mg[t] = m;
  float b = L.band;
  for (int i = 0; i < kTieBands && m < b; ++i, b *= 0.25f) {
    const uint32_t k = atomicAdd(L.count + i, 1u);
    if (i == 0 && k < static_cast<uint32_t>(L.kmax)) L.list[k] = static_cast<int32_t>(t);
  }
}

}  // namespace pmcmc
