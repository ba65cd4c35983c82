// persist_column.cuh -- one column of the persistent solve (deer_persist.cu): the forward
// MALA half and the Jacobian diagonal, for a group of lanes.
//
// The quantities are those of column_forward / column_jacobian (deer_column.cuh) with two
// differences.  (1) log alpha is taken without its tape term 0.5 |xi|^2, which is added
// once a block to the threshold (lu = log u - 0.5 |xi|^2): with u = (y - x) - eps lam (y - mu)
// the rest is sum -lam/2 (y - x)(x + y - 2 mu) - u^2 / (4 eps), 9 FP64 operations and two
// conversions a coordinate instead of 16 and three.  (2) Dense targets: the product with P of
// the state (FP64) and of the probe (state's precision) run together, over all 32 lanes
// (below).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "deer_column.cuh"
#include "deer_device.cuh"

namespace pmcmc {

// Diagonal target.  Per-coordinate constants, in shared memory (zero-padded to Dp) for
// D <= 256 where they fit beside the columns; else, formed where they are used.
template <typename Real>
struct DiagTab {
  const Real *lam, *mu, *el, *k2;      // precision, mean, eps lam, eps lam^2 / 2
  // -lam / 2, -eps lam, mean (FP32 state): coordinates 4j, 4j + 1 of every quad, then
  // 4j + 2, 4j + 3 (a quad's 32 bytes in one place would be read with bank conflicts)
  const double2 *hl, *nel, *mud;
  int nq;
};
template <typename Real>
__host__ __device__ constexpr size_t diag_tab_bytes(int64_t Dp) {
  return (4 * sizeof(Real) + 3 * sizeof(double)) * static_cast<size_t>(Dp);
}
template <typename Real>
__device__ __forceinline__ DiagTab<Real> fill_diag_tab(unsigned char* base, const DevParams& P) {
  const int D = static_cast<int>(P.D), Dp = static_cast<int>(P.Dp);
  double* hl = reinterpret_cast<double*>(base);
  double *nel = hl + Dp, *mud = nel + Dp;
  const int nq = Dp / 4;
  Real* lam = reinterpret_cast<Real*>(mud + Dp);
  Real *mu = lam + Dp, *el = mu + Dp, *k2 = el + Dp;
  const Real eps = static_cast<Real>(P.eps);
  for (int i = threadIdx.x; i < Dp; i += blockDim.x) {
    const bool in = i < D;
    const double ld = in ? P.prec_d[i] : 0.0;
    const Real l = in ? prec_of<Real>(P)[i] : Real(0);
    const int k = ((i & 2) ? 2 * nq : 0) + 2 * (i >> 2) + (i & 1);
    hl[k] = -0.5 * ld;
    nel[k] = -P.eps * ld;
    mud[k] = in ? P.mean_d[i] : 0.0;
    lam[i] = l;
    mu[i] = in ? mean_of<Real>(P)[i] : Real(0);
    el[i] = eps * l;
    k2[i] = Real(0.5) * (eps * l) * l;
  }
  return DiagTab<Real>{lam, mu, el, k2, reinterpret_cast<const double2*>(hl),
                       reinterpret_cast<const double2*>(nel),
                       reinterpret_cast<const double2*>(mud), nq};
}

// LPC lanes a column, lane owns quads j = lane + LPC q.  c.la is this lane's part of
// log alpha - 0.5 |xi|^2.  Padded coordinates are zero throughout.  With kExact (the
// exact Jacobian diagonal) c.gx holds v = eps lam^2 / 2 r (y - x), r = x - y - eps g_y: for
// a diagonal Gaussian the gradient of log alpha in coordinate i (column_jacobian) is
// (1 - eps lam) g_y - g_x - lam r (1 - eps lam / 2) = eps lam^2 r / 2, because
// (1 - eps lam)(y - mu) - (x - mu) = -r; and c.gy holds eps lam.
template <typename Real, int QPL, int LPC, bool kExact, bool kTab>
__device__ __forceinline__ void persist_forward_diag(const DevParams& P, const DiagTab<Real>& tab,
                                                     const Real* xcol, const float* xic,
                                                     Col<Real, QPL>& c) {
  const int lane = threadIdx.x & (LPC - 1);
  const int D = static_cast<int>(P.D);
  const Real eps = static_cast<Real>(P.eps), c2 = static_cast<Real>(P.sqrt2eps);
  double la = 0.0;
#pragma unroll
  for (int q = 0; q < QPL; ++q) {
    const int j = lane + LPC * q;
    if (4 * j >= D) {
#pragma unroll
      for (int e = 0; e < 4; ++e) c.x[q][e] = c.gx[q][e] = c.y[q][e] = c.gy[q][e] = Real(0);
      continue;
    }
    Real lam[4], mu[4], el[4], k2[4];
    double hl[4], nel[4], mud[4];
    float n[4];
    load4(xcol + 4 * j, c.x[q]);
    load4(xic + 4 * j, n);
    if constexpr (kTab) {
      load4(tab.lam + 4 * j, lam);
      load4(tab.mu + 4 * j, mu);
      if constexpr (sizeof(Real) == 4) {
        auto get = [&](const double2* t, double (&v)[4]) {
          const double2 a = t[j], b = t[tab.nq + j];
          v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
        };
        get(tab.hl, hl);
        get(tab.nel, nel);
        get(tab.mud, mud);
      }
      if constexpr (kExact || sizeof(Real) == 8) load4(tab.el + 4 * j, el);
      if constexpr (kExact) load4(tab.k2 + 4 * j, k2);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool in = 4 * j + e < D;
        const double ld = in ? P.prec_d[4 * j + e] : 0.0;
        lam[e] = in ? prec_of<Real>(P)[4 * j + e] : Real(0);
        mu[e] = in ? mean_of<Real>(P)[4 * j + e] : Real(0);
        hl[e] = -0.5 * ld;
        nel[e] = -P.eps * ld;
        mud[e] = in ? P.mean_d[4 * j + e] : 0.0;
        el[e] = eps * lam[e];
        k2[e] = Real(0.5) * el[e] * lam[e];
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if constexpr (kTab && sizeof(Real) == 8) hl[e] = -0.5 * lam[e], nel[e] = -el[e], mud[e] = mu[e];
      const Real x = c.x[q][e];
      const Real gx = -lam[e] * (x - mu[e]);
      const Real y = fma(c2, static_cast<Real>(n[e]), fma(eps, gx, x));
      c.y[q][e] = y;
      if constexpr (kExact) {
        const Real d = y - x;
        c.gx[q][e] = k2[e] * fma(el[e], y - mu[e], -d) * d;
        c.gy[q][e] = el[e];
      } else {
        c.gx[q][e] = gx;
        c.gy[q][e] = -lam[e] * (y - mu[e]);
      }
      const double xd = static_cast<double>(x) - mud[e];
      const double yd = static_cast<double>(y) - mud[e];
      const double dl = yd - xd;
      const double u = fma(nel[e], yd, dl);
      la = fma(hl[e], dl * (xd + yd), la);
      la = fma(-P.inv4eps * u, u, la);
    }
  }
  c.la = la;
}

// Dense target: lanes of a quad group.  G = 8, 16 or 32 lanes hold the column's quads (one a
// lane for D <= 128, QPL with G = 32), and the 32 / G groups hold the same values; a product
// with P splits its sum over the groups and adds the parts by shuffles.
template <int G>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = G; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int G>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = G; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// o = P vd (FP64) and, with kZ, h = P vf (state's precision), vectors of the warp in shared
// memory.
template <typename Real, int QPL, int G, bool kV, bool kZ>
__device__ __forceinline__ void dense_products(const Smem<Real>& sm, int D, int Dp,
                                               double (&o)[QPL][4], Real (&h)[QPL][4]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane / G, jl = lane & (G - 1);
  constexpr int KS = 32 / G;
  const int kper = (D + KS - 1) / KS, k0 = g * kper, k1 = min(D, k0 + kper);
  const double* vd = sm.Vd + warp * Dp;
  const Real* vf = sm.Vf + warp * Dp;
#pragma unroll
  for (int q = 0; q < QPL; ++q) {
    const int j = jl + G * q;
    double a[4] = {0, 0, 0, 0};
    Real b[4] = {0, 0, 0, 0};
    if (4 * j < D) {
      // (the copy in shared memory keeps a quad's halves apart: 16-byte reads at a stride of
      // 32 would meet in their banks)
      const double* pd = sm.Pd + (sm.split ? 2 * j : 4 * j);
      const int up = sm.split ? Dp / 2 : 2;
      [[maybe_unused]] const Real* pf = sm.Pf + 4 * j;
#pragma unroll 4
      for (int k = k0; k < k1; ++k) {
        double m[4];
        Real n[4];
        if constexpr (kV || sizeof(Real) == 8) {
          const double2 lo = *reinterpret_cast<const double2*>(pd + static_cast<size_t>(k) * Dp);
          const double2 hi = *reinterpret_cast<const double2*>(pd + static_cast<size_t>(k) * Dp + up);
          m[0] = lo.x, m[1] = lo.y, m[2] = hi.x, m[3] = hi.y;
        }
        if constexpr (kV) {
          const double v = vd[k];
#pragma unroll
          for (int e = 0; e < 4; ++e) a[e] = fma(m[e], v, a[e]);
        }
        if constexpr (kZ) {
          if constexpr (sizeof(Real) == 8) {  // one read of P for both
#pragma unroll
            for (int e = 0; e < 4; ++e) n[e] = m[e];
          } else {
            load4(pf + static_cast<size_t>(k) * Dp, n);
          }
          const Real v = vf[k];
#pragma unroll
          for (int e = 0; e < 4; ++e) b[e] = fma(n[e], v, b[e]);
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if constexpr (kV) o[q][e] = group_sum<G>(a[e]);
      if constexpr (kZ) h[q][e] = group_sum<G>(b[e]);
    }
  }
}

// A vector of the column into the warp's FP64 or state-precision vector.
template <typename Real, int QPL, int G, typename V>
__device__ __forceinline__ void put_column(V* v, const Real (&s)[QPL][4], const double* sub, int D) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < QPL; ++q) {
    const int j = lane + G * q;
    if (lane < G && 4 * j < D)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (4 * j + e < D)
          v[4 * j + e] = static_cast<V>(s[q][e]) - (sub ? static_cast<V>(sub[4 * j + e]) : V(0));
  }
}

// Rademacher probe k of the column in this lane's quads (zero past D).
template <typename Real, int QPL, int G>
__device__ __forceinline__ void column_probe(const DevParams& P, const TapeKey& key, int t, int k,
                                             int iter, Real (&z)[QPL][4]) {
  const int jl = threadIdx.x & (G - 1);
  const int D = static_cast<int>(P.D);
#pragma unroll
  for (int q = 0; q < QPL; ++q) {
    const int j = jl + G * q;
    const U4 pb = probe_bits(key, static_cast<uint32_t>(j >> 5), static_cast<uint32_t>(t), k, iter);
    const uint32_t wv = u4_word(pb, (j >> 3) & 3) >> ((j & 7) * 4);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      z[q][e] = 4 * j + e < D ? (((wv >> e) & 1u) ? Real(1) : Real(-1)) : Real(0);
  }
}

// (mud: the mean in shared memory; after a grid barrier a global load misses L1.)
// Forward half of a dense column and, for JAC = stoch, the products of the first probe:
// z, w = z - eps P z and hvy = -P w, two rounds of products instead of four.
template <typename Real, int JAC, int QPL, int G, bool kProbe>
__device__ __forceinline__ void persist_forward_dense(const DevParams& P, const Smem<Real>& sm,
                                                      const double* mud, const TapeKey& key,
                                                      const Real* xcol, const float* xic, int t,
                                                      int iter,
                                                      Col<Real, QPL>& c, Real (&z)[QPL][4],
                                                      Real (&w)[QPL][4], Real (&hvy)[QPL][4]) {
  constexpr bool kZ = kProbe && JAC == kJacStoch;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, jl = lane & (G - 1);
  const int D = static_cast<int>(P.D), Dp = static_cast<int>(P.Dp);
  const Real eps = static_cast<Real>(P.eps), c2 = static_cast<Real>(P.sqrt2eps);
  double* vd = sm.Vd + warp * Dp;
  Real* vf = sm.Vf + warp * Dp;
  float n[QPL][4];
#pragma unroll
  for (int q = 0; q < QPL; ++q) {
    const int j = jl + G * q;
#pragma unroll
    for (int e = 0; e < 4; ++e) c.x[q][e] = Real(0), n[q][e] = 0.f;
    if (4 * j < D) {
      load4(xcol + 4 * j, c.x[q]);
      load4(xic + 4 * j, n[q]);
    }
  }
  if constexpr (kZ) {
    column_probe<Real, QPL, G>(P, key, t, 0, iter, z);
    put_column<Real, QPL, G>(vf, z, nullptr, D);
  }
  put_column<Real, QPL, G>(vd, c.x, mud, D);
  __syncwarp();
  double o[QPL][4];
  Real h[QPL][4];
  dense_products<Real, QPL, G, true, kZ>(sm, D, Dp, o, h);
  __syncwarp();
  double la = 0.0;
#pragma unroll
  for (int q = 0; q < QPL; ++q) {
    const int j = jl + G * q;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const bool in = 4 * j + e < D;
      c.gx[q][e] = in ? static_cast<Real>(-o[q][e]) : Real(0);
      c.y[q][e] = in ? fma(c2, static_cast<Real>(n[q][e]), fma(eps, c.gx[q][e], c.x[q][e])) : Real(0);
      if (in) la += 0.5 * (static_cast<double>(c.x[q][e]) - mud[4 * j + e]) * o[q][e];
      if constexpr (kZ) w[q][e] = in ? z[q][e] - eps * h[q][e] : Real(0);
    }
  }
  put_column<Real, QPL, G>(vd, c.y, mud, D);
  if constexpr (kZ) put_column<Real, QPL, G>(vf, w, nullptr, D);
  __syncwarp();
  dense_products<Real, QPL, G, true, kZ>(sm, D, Dp, o, h);
  __syncwarp();
#pragma unroll
  for (int q = 0; q < QPL; ++q) {
    const int j = jl + G * q;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const bool in = 4 * j + e < D;
      c.gy[q][e] = in ? static_cast<Real>(-o[q][e]) : Real(0);
      if (in) {
        const double yd = static_cast<double>(c.y[q][e]) - mud[4 * j + e];
        const double r2 = (static_cast<double>(c.x[q][e]) - static_cast<double>(c.y[q][e])) +
                          P.eps * o[q][e];
        la = fma(-0.5 * yd, o[q][e], la);
        la = fma(-P.inv4eps * r2, r2, la);
      }
      if constexpr (kZ) hvy[q][e] = -h[q][e];
    }
  }
  c.la = la;
}

// Dense columns that the per-sweep kernel's code (column_forward, column_jacobian) evaluates
// faster: many quads a lane, P read from L2, the exact diagonal, whose three products of P
// have no pair to share a read with (FP32, D = 300, T = 200: 214 us a sweep, 310 by the code
// below; FP64, D = 256, T = 64: 150 and 210).  Their log alpha includes the tape term.
template <typename Real, int TK, int JAC, int QPL>
constexpr bool kWholeColumn =
    TK == kDenseGauss && JAC == kJacDiag && QPL >= (sizeof(Real) == 8 ? 2 : 4);
template <typename Real, int QPL>
__device__ __forceinline__ void persist_forward_whole(const DevParams& P, const Smem<Real>& sm,
                                                      const TapeKey& key, const Real* xcol,
                                                      const float* xic, Col<Real, QPL>& c) {
  const int lane = threadIdx.x & 31, D = static_cast<int>(P.D);
  float n[QPL][4];
#pragma unroll
  for (int q = 0; q < QPL; ++q) {
#pragma unroll
    for (int e = 0; e < 4; ++e) n[q][e] = 0.f;
    if (4 * (lane + 32 * q) < D) load4(xic + 4 * (lane + 32 * q), n[q]);
  }
  column_forward<Real, kDenseGauss, QPL, 32, false>(P, sm, key, xcol, 0, c, n);
}

// -P v for a vector of the column, all groups.
template <typename Real, int QPL, int G>
__device__ __forceinline__ void dense_neg(const Smem<Real>& sm, int D, int Dp,
                                          const Real (&v)[QPL][4], Real (&out)[QPL][4]) {
  Real* vf = sm.Vf + (threadIdx.x >> 5) * Dp;
  put_column<Real, QPL, G>(vf, v, nullptr, D);
  __syncwarp();
  double none[QPL][4];
  dense_products<Real, QPL, G, false, true>(sm, D, Dp, none, out);
  __syncwarp();
#pragma unroll
  for (int q = 0; q < QPL; ++q)
#pragma unroll
    for (int e = 0; e < 4; ++e) out[q][e] = -out[q][e];
}

// Jacobian diagonal of a dense column; z, w, hvy: the first probe's, from the forward half.
template <typename Real, int JAC, int QPL, int G>
__device__ __forceinline__ void persist_jacobian_dense(const DevParams& P, const Smem<Real>& sm,
                                                       const TapeKey& key, int t, int iter,
                                                       bool acc, Real gp, const Col<Real, QPL>& c,
                                                       Real (&z)[QPL][4], Real (&w)[QPL][4],
                                                       Real (&hvy)[QPL][4], Real (&A)[QPL][4]) {
  const int jl = threadIdx.x & (G - 1);
  const int D = static_cast<int>(P.D), Dp = static_cast<int>(P.Dp);
  const Real eps = static_cast<Real>(P.eps), inv2eps = static_cast<Real>(P.inv2eps);
  if constexpr (JAC == kJacStoch) {
#pragma unroll
    for (int q = 0; q < QPL; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) A[q][e] = Real(0);
    for (int k = 0; k < P.probes; ++k) {
      if (k > 0) {
        column_probe<Real, QPL, G>(P, key, t, k, iter, z);
        dense_neg<Real, QPL, G>(sm, D, Dp, z, w);
#pragma unroll
        for (int q = 0; q < QPL; ++q)
#pragma unroll
          for (int e = 0; e < 4; ++e) w[q][e] = z[q][e] + eps * w[q][e];
        dense_neg<Real, QPL, G>(sm, D, Dp, w, hvy);
      }
      Real dla = 0;
#pragma unroll
      for (int q = 0; q < QPL; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const Real r = c.x[q][e] - c.y[q][e] - eps * c.gy[q][e];
          const Real dr = z[q][e] - w[q][e] - eps * hvy[q][e];
          dla += c.gy[q][e] * w[q][e] - c.gx[q][e] * z[q][e] - inv2eps * r * dr;
        }
      const Real dg = gp * seg_sum<G>(dla);
#pragma unroll
      for (int q = 0; q < QPL; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const Real jz = (acc ? w[q][e] : z[q][e]) + (c.y[q][e] - c.x[q][e]) * dg;
          A[q][e] += z[q][e] * jz;
        }
    }
    if (P.probes > 1) {
      const Real inv = Real(1) / static_cast<Real>(P.probes);
#pragma unroll
      for (int q = 0; q < QPL; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) A[q][e] *= inv;
    }
  } else {
    // as in column_jacobian, from -P g_y, -P r and P P r
    Real r[QPL][4], pgy[QPL][4], pr[QPL][4], ppr[QPL][4];
#pragma unroll
    for (int q = 0; q < QPL; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) r[q][e] = c.x[q][e] - c.y[q][e] - eps * c.gy[q][e];
    dense_neg<Real, QPL, G>(sm, D, Dp, c.gy, pgy);
    dense_neg<Real, QPL, G>(sm, D, Dp, r, pr);
    dense_neg<Real, QPL, G>(sm, D, Dp, pr, ppr);
#pragma unroll
    for (int q = 0; q < QPL; ++q) {
      const int j = jl + G * q;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 4 * j + e;
        const Real pii = i < D ? sm.Pf[static_cast<size_t>(i) * Dp + i] : Real(0);
        const Real dl = c.gy[q][e] + eps * pgy[q][e] - c.gx[q][e] + pr[q][e] +
                        Real(0.5) * eps * ppr[q][e];
        A[q][e] = (acc ? Real(1) - eps * pii : Real(1)) + (c.y[q][e] - c.x[q][e]) * gp * dl;
      }
    }
  }
}

}  // namespace pmcmc
