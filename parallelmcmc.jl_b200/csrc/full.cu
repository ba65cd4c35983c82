// full.cu -- the dense-Jacobian (:full) Newton sweep and the adjoint pass for
// the Gaussian device targets.
//
// The reference rejects :full (DEER.jl:465-466, interface.jl:274-275).  Here
// it is Newton with the exact Jacobian of the surrogate step, the matrix whose
// action is the JVP of MALA.jl:768-795.  For a Gaussian with precision
// P = Q diag(lam) Q^T the Hessian is the constant -P, so with M = I - eps P
//     J_t = C_t + u_t v_t^T,   C_t = M (accepted) or I (rejected),
//     u_t = g(1-g) (y_t - x_t),  v_t = grad_x log alpha_t
//         = M g_y - g_x - P r + (eps/2) P^2 r,  r = x - y - eps g_y.
// MALA on N(mu, P^-1) is equivariant under x' = Q^T (x - mu), xi' = Q^T xi:
// in the eigenbasis the target is the diagonal Gaussian N(0, diag(1/lam)) and
//     J'_t = diag(c_t) + u'_t v'_t^T,   c_t = 1 - a_t eps lam.
// The Newton iterate is therefore carried in the eigenbasis (S', with the
// original-basis S kept alongside for the convergence test and the outputs),
// and the step is taken in update form (the same iterates in exact
// arithmetic as the reference's S-form B_t = f_t - J_t x_bar_t, DEER.jl:419):
//     delta'_t = J'_t delta'_{t-1} + (f'_t - S'_t),   S' += damping delta',
//     S += damping Q delta',
// so rounding in the chunk products slows convergence at worst and never
// moves the fixed point.  All sweep buffers use the stride DQ (16, 32, 64 or
// 128, zero-padded) so that the per-step loops have compile-time trip counts.
// Per solve, `rotate` forms xi' and x0'.  A sweep is five launches (four with few chunks):
//   eval   one warp per column: the diagonal-target forward step in the
//          eigenbasis, u', v', r' = f'_t - S'_t and the accept flag
//   chunk  one CTA per chunk of L columns: the chunk's map [Phi'|beta'] as an
//          augmented DQ x (DQ+1) matrix in registers; four or eight lanes own a few
//          columns, whose recursions need no barrier (column sums by shuffles)
//   group  a few CTAs per group of chunks: the group's map, and each chunk's prefix
//   carry  one CTA: updates entering each group, the maps read two steps ahead
//   apply  one CTA per chunk: exact replay of the chunk from its entering
//          update (the old iterates arrive by cp.async meanwhile), the
//          rotation Q delta' as a warp-tiled product, damping, max|dS| and
//          max|S| in the original basis, and the convergence test +
//          CUDA-graph loop control in the last CTA.
//
// Adjoint (no counterpart in the reference): at a returned trajectory, with
// the accept decisions held fixed, f_t(x) = a_t y_t(x) + (1 - a_t) x has
// Jacobian C_t, so for an objective L(x_1..x_T) the adjoint is the diagonal
// (primed) reverse scan lambda'_t = c'_t + diag(c_{t+1}) lambda'_{t+1} and
//     dL/deps     = explicit + sum_t a_t lambda_t . (g(x_bar_t) + xi_t / sqrt(2 eps)),
//     dL/dlog s_i = sum_t a_t eps lam_i lambda'_{t,i} x_bar'_{t,i}     (s_i = 1 / lam_i).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "deer_column.cuh"
#include "deer_device.cuh"
#include "deer_launch.h"
#include "f32x2.cuh"
#include "full.h"

namespace pmcmc {

namespace {

template <typename S>
__device__ __forceinline__ void load_struct(const S* g, S& s) {
  static_assert(sizeof(S) % 8 == 0, "struct size must be a multiple of 8 bytes");
  constexpr int n = sizeof(S) / 8;
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    reinterpret_cast<unsigned long long*>(&s)[i] = reinterpret_cast<const unsigned long long*>(g)[i];
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// out = rows 4*lane .. 4*lane+3 of M v for one warp (M in shared memory in
// matvec4's layout, v a shared vector of D entries); zeros past Dp.
__device__ __forceinline__ void warp_rotate(const float* Ms, const float* v, int D, int Dp,
                                            float out[4]) {
  const int lane = threadIdx.x & 31;
  if (4 * lane < Dp) {
    matvec4<float, float, float>(Ms, v, D, Dp, lane, out);
  } else {
    out[0] = out[1] = out[2] = out[3] = 0.f;
  }
}

// Writes the warp's quad of v (masked to D) into a warp-private shared vector.
__device__ __forceinline__ void put_vec(float* vs, const float v[4], int D) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int e = 0; e < 4; ++e)
    if (4 * lane + e < D) vs[4 * lane + e] = v[e];
}

// Rotates a warp quad in place through the warp-private vector vw.
__device__ __forceinline__ void rotate_quad(const float* Qs, float* vw, int D, int Dp, float q[4]) {
  put_vec(vw, q, D);
  __syncwarp();
  warp_rotate(Qs, vw, D, Dp, q);
  __syncwarp();
}

// Warp-tiled product for up to 8 columns at once: acc[c][e] = sum_{k<K}
// Ms(4*lane+e, k) X[c*ldx + k] (Ms column-major at stride DQ, X columns in
// shared memory); each matrix element read serves 8 columns.  Lanes past DQ
// return zeros.
template <int DQ>
__device__ __forceinline__ void warp_tile8(const float* Ms, const float* X, int ldx, int nc, int K,
                                          float acc[8][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int c = 0; c < 8; ++c)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[c][e] = 0.f;
  if (4 * lane >= DQ) return;
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    float q[4];
    load4(Ms + k * DQ + 4 * lane, q);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float x = c < nc ? X[c * ldx + k] : 0.f;
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[c][e] = fmaf(q[e], x, acc[c][e]);
    }
  }
}

// Shared memory of the per-column kernels of the adjoint: the column plan
// (TT = 1), then Q (Dp x Dp, dense target) and kWarps warp-private vectors.
__host__ __device__ inline size_t eval_smem_bytes(int64_t Dp, bool dense) {
  const SmemPlan pl = plan_sweep_smem<float>(Dp, 1, dense);
  return pl.total + sizeof(float) * ((dense ? Dp * Dp : 0) + kWarps * Dp);
}

// Eager mode (no graph): sweeps launched after convergence, maxiter or an
// error are no-ops, like the fused sweep's.
__device__ __forceinline__ bool sweep_done(const DevState* st, int use_cond, int maxiter) {
  if (use_cond) return false;
  return *reinterpret_cast<const volatile int32_t*>(&st->converged) ||
         *reinterpret_cast<const volatile int32_t*>(&st->iter) >= maxiter ||
         *reinterpret_cast<const volatile int32_t*>(&st->status) != 0;
}

}  // namespace

// ---------------------------------------------------------------------------
// rotate (once per solve): xi'_t = Q^T xi_t, x0' = Q^T (x0 - mu), at stride DQ
// ---------------------------------------------------------------------------
template <int DQ>
__global__ void __launch_bounds__(kThreads)
    full_rotate_kernel(const DevParams* __restrict__ Pg, const FullArgs* __restrict__ Fg,
                       DevState* __restrict__, cudaGraphConditionalHandle, int) {
  __shared__ DevParams P;
  __shared__ FullArgs F;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  load_struct(Fg, F);
  load_params(Pg, P);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int D = static_cast<int>(P.D), Dp = static_cast<int>(P.Dp);
  float* Qs = reinterpret_cast<float*>(smem_raw);  // Q^T operator at stride DQ
  float* Xw = Qs + DQ * DQ + warp * 8 * Dp;         // 8 staged columns per warp
  for (int i = threadIdx.x; i < DQ * DQ; i += blockDim.x) Qs[i] = F.QrmQ[i];
  __syncthreads();
  float* xi_e = const_cast<float*>(F.Pe->xi);
  if (blockIdx.x == 0 && warp == 0) {
    const float* x0 = static_cast<const float*>(P.x0);
    for (int i = lane; i < Dp; i += 32) Xw[i] = i < D ? static_cast<float>(x0[i] - P.mean_d[i]) : 0.f;
    __syncwarp();
    float acc[8][4];
    warp_tile8<DQ>(Qs, Xw, Dp, 1, D, acc);
    if (4 * lane < DQ) store4(static_cast<float*>(const_cast<void*>(F.Pe->x0)) + 4 * lane, acc[0]);
    __syncwarp();
  }
  const int64_t ntile = (P.T + 7) / 8;
  for (int64_t tile = static_cast<int64_t>(blockIdx.x) * kWarps + warp; tile < ntile;
       tile += static_cast<int64_t>(gridDim.x) * kWarps) {
    const int64_t t0 = tile * 8;
    const int nc = static_cast<int>(imin64(8, P.T - t0));
    for (int i = lane; i < nc * Dp; i += 32) Xw[i] = P.xi[t0 * Dp + i];
    __syncwarp();
    float acc[8][4];
    warp_tile8<DQ>(Qs, Xw, Dp, nc, D, acc);
    if (4 * lane < DQ)
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (c < nc) store4(xi_e + (t0 + c) * DQ + 4 * lane, acc[c]);
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// eval: per column forward step in the eigenbasis, u', v', r', accept flag
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads)
    full_eval_kernel(const DevParams* __restrict__, const FullArgs* __restrict__ Fg,
                     DevState* __restrict__ st, cudaGraphConditionalHandle, int use_cond) {
  __shared__ DevParams P;  // the eigenbasis view
  __shared__ FullArgs F;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  load_struct(Fg, F);
  __syncthreads();
  load_params(F.Pe, P);
  if (sweep_done(st, use_cond, P.maxiter)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int D = static_cast<int>(P.D), Dp = static_cast<int>(P.Dp);
  Smem<float> sm = carve<float>(smem_raw, P, 1, false);
  const float* Sold = static_cast<const float*>(P.S[st->cur]);
  const float* x0 = static_cast<const float*>(P.x0);
  // the first sweep starts from S = x0 broadcast (DEER.jl:538-542), read in place
  const bool first = st->iter == 0;
  const TapeKey key(P.seed, P.block);
  const float eps = static_cast<float>(P.eps);
  float lam[4] = {0.f, 0.f, 0.f, 0.f};
  if (4 * lane < D) load4(P.prec_f + 4 * lane, lam);
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * kWarps + warp; t < P.T;
       t += static_cast<int64_t>(gridDim.x) * kWarps) {
    const float* xcol = (t == 0 || first) ? x0 : Sold + (t - 1) * Dp;
    Col<float, 1> c;
    column_forward<float, kDiagGauss, 1>(P, sm, key, xcol, static_cast<int>(t), c);
    const double logu = P.logu[t];
    const bool acc = logu < c.la;
    const float gp = sigmoid_slope<float>(c.la - logu);
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
    if (4 * lane < D) load4(first ? x0 + 4 * lane : Sold + t * Dp + 4 * lane, s4);
    float v[4], u[4], r[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const bool in = 4 * lane + e < D;
      const float el = eps * lam[e];
      const float q = c.x[0][e] - c.y[0][e] - eps * c.gy[0][e];
      v[e] = in ? (1.f - el) * c.gy[0][e] - c.gx[0][e] - lam[e] * q * (1.f - 0.5f * el) : 0.f;
      u[e] = in ? gp * (c.y[0][e] - c.x[0][e]) : 0.f;
      r[e] = in ? (acc ? c.y[0][e] : c.x[0][e]) - s4[e] : 0.f;
    }
    if (4 * lane < Dp) {
      store4(F.U + t * Dp + 4 * lane, u);
      store4(F.V + t * Dp + 4 * lane, v);
      store4(F.R + t * Dp + 4 * lane, r);
    }
    if (lane == 0) F.acc[t] = acc ? 1 : 0;
  }
}

// ---------------------------------------------------------------------------
// chunk: the augmented map [Phi' | beta'] of each chunk.  TPC consecutive
// lanes own NCOL columns (column DQ is beta'), lane q of them the row quads
// q, q + TPC, ... in registers (NR = DQ / TPC rows).  Per step: w_j = v'^T
// [Phi'|beta']_{:,j} (log2 TPC shuffles a column), then
// [Phi'|beta'] <- diag(c_t) [Phi'|beta'] + u' w^T + r' e_DQ^T.
// Padded rows and columns stay zero.
// Shared memory returns 128 B a cycle whether lanes share an address or not, so
// the loads of u' and v' bound a step at one column a thread (22 us at D = 64,
// T = 8192; at D = 128, where a lane's rows lay 128 B apart, 150): NCOL = 4 columns
// use each load, and neighbouring lanes read neighbouring quads.
// ---------------------------------------------------------------------------
constexpr int chunk_tpc(int DQ) { return DQ == 16 ? 4 : 8; }
constexpr int chunk_ncol(int DQ) { return DQ <= 32 ? 2 : 4; }
constexpr int chunk_threads(int DQ) {
  return (chunk_tpc(DQ) * (DQ / chunk_ncol(DQ) + 1) + 31) / 32 * 32;
}
template <int DQ>
__global__ void __launch_bounds__(chunk_threads(DQ))
    full_chunk_kernel(const DevParams* __restrict__, const FullArgs* __restrict__ Fg,
                      DevState* __restrict__ st, cudaGraphConditionalHandle, int use_cond) {
  constexpr int TPC = chunk_tpc(DQ), NCOL = chunk_ncol(DQ), NR = DQ / TPC, NQ = NR / 4;
  static_assert(NR % 4 == 0 && (TPC == 4 || TPC == 8) && DQ % NCOL == 0, "chunk tiling");
  __shared__ FullArgs F;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  load_struct(Fg, F);
  __syncthreads();
  if (sweep_done(st, use_cond, F.maxiter)) return;
  const int tid = threadIdx.x;
  const int D = F.D;
  const int L = F.L;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * L;
  const int nt = static_cast<int>(imin64(L, F.T - t0));
  float* Us = reinterpret_cast<float*>(smem_raw);
  float* Vs = Us + L * DQ;
  float* Rs = Vs + L * DQ;
  uint8_t* as = reinterpret_cast<uint8_t*>(Rs + L * DQ);
  {
    const int n4 = nt * DQ / 4;
    const float* gu = F.U + t0 * DQ;
    const float* gv = F.V + t0 * DQ;
    const float* gr = F.R + t0 * DQ;
    for (int i = tid; i < n4; i += blockDim.x) {
      cp_async16(Us + 4 * i, gu + 4 * i);
      cp_async16(Vs + 4 * i, gv + 4 * i);
      cp_async16(Rs + 4 * i, gr + 4 * i);
    }
    cp_async_commit();
    for (int i = tid; i < nt; i += blockDim.x) as[i] = F.acc[t0 + i];
  }
  const int j0 = tid / TPC * NCOL, q = tid % TPC;
  const bool bcol = j0 == DQ;  // the offset's thread: its column is the first
  F2 phi[NCOL][NR / 2], ml[NR / 2];
#pragma unroll
  for (int k = 0; k < NR; k += 2) {
    const int i = 4 * (q + TPC * (k / 4)) + k % 4;
#pragma unroll
    for (int c = 0; c < NCOL; ++c)
      phi[c][k / 2] = pack2(i == j0 + c && i < D ? 1.f : 0.f, i + 1 == j0 + c && i + 1 < D ? 1.f : 0.f);
    ml[k / 2] = pack2(i < D ? 1.f - F.eps * F.lamQ[i] : 0.f,
                      i + 1 < D ? 1.f - F.eps * F.lamQ[i + 1] : 0.f);
  }
  cp_async_wait<0>();
  __syncthreads();
  for (int s = 0; s < nt; ++s) {
    const ulonglong2* v4 = reinterpret_cast<const ulonglong2*>(Vs + s * DQ) + q;
    const ulonglong2* u4 = reinterpret_cast<const ulonglong2*>(Us + s * DQ) + q;
    F2 a01[NCOL], a23[NCOL];
#pragma unroll
    for (int c = 0; c < NCOL; ++c) a01[c] = a23[c] = F2{0ull};
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const ulonglong2 v = v4[k * TPC];
#pragma unroll
      for (int c = 0; c < NCOL; ++c) {
        a01[c] = fma2(F2{v.x}, phi[c][2 * k], a01[c]);
        a23[c] = fma2(F2{v.y}, phi[c][2 * k + 1], a23[c]);
      }
    }
    float w[NCOL];
#pragma unroll
    for (int c = 0; c < NCOL; ++c) {
      float a0, a1, a2, a3;
      unpack2(a01[c], a0, a1);
      unpack2(a23[c], a2, a3);
      w[c] = (a0 + a1) + (a2 + a3);
    }
#pragma unroll
    for (int o = 1; o < TPC; o *= 2)
#pragma unroll
      for (int c = 0; c < NCOL; ++c) w[c] += __shfl_xor_sync(0xffffffffu, w[c], o);
    if (as[s]) {  // uniform across the CTA
#pragma unroll
      for (int c = 0; c < NCOL; ++c)
#pragma unroll
        for (int k = 0; k < NR / 2; ++k) phi[c][k] = mul2(ml[k], phi[c][k]);
    }
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      const ulonglong2 u = u4[k * TPC];
#pragma unroll
      for (int c = 0; c < NCOL; ++c) {
        const F2 ww = pack2(w[c], w[c]);
        phi[c][2 * k] = fma2(F2{u.x}, ww, phi[c][2 * k]);
        phi[c][2 * k + 1] = fma2(F2{u.y}, ww, phi[c][2 * k + 1]);
      }
    }
    if (bcol) {
      const ulonglong2* r4 = reinterpret_cast<const ulonglong2*>(Rs + s * DQ) + q;
#pragma unroll
      for (int k = 0; k < NQ; ++k) {
        const ulonglong2 r = r4[k * TPC];
        phi[0][2 * k] = add2(phi[0][2 * k], F2{r.x});
        phi[0][2 * k + 1] = add2(phi[0][2 * k + 1], F2{r.y});
      }
    }
  }
#pragma unroll
  for (int c = 0; c < NCOL; ++c) {
    const int j = j0 + c;
    if (j > DQ) break;
    float* dst = j == DQ ? F.beta + static_cast<size_t>(blockIdx.x) * DQ
                         : F.Phi + (static_cast<size_t>(blockIdx.x) * DQ + j) * DQ;  // column-major
#pragma unroll
    for (int k = 0; k < NQ; ++k)
      reinterpret_cast<ulonglong2*>(dst)[q + k * TPC] =
          make_ulonglong2(phi[c][2 * k].v, phi[c][2 * k + 1].v);
  }
}

// ---------------------------------------------------------------------------
// group: the maps of a group of G consecutive chunks, [Phi'|beta']_{c+G-1} ... composed
// in order, and before each chunk the composition of those ahead of it in the group.
// A column of the augmented product depends on that column alone, so the DQ + 1 columns
// are split over gridDim.x / ngroups CTAs of NC columns.  A warp forms 4 * RG rows of
// four columns: a lane adds a 4 x 4 tile over every KS-th k, and the KS partial tiles
// are summed by exchanging halves (32 B of shared memory a 16 products; with one row a
// lane it was 20 B a 4, and a step took twice as long).  The maps pass through a ring of three
// slots, copied two steps ahead.  With it the carry runs over the groups and an apply CTA forms its
// entering update by one product with its prefix: the serial chain of a sweep is
// G + nchunks / G steps instead of nchunks (45 of 103 us a sweep at D = 64, T = 8192).
// ---------------------------------------------------------------------------
template <int DQ>
struct GroupTile {
  static constexpr int RG = DQ >= 32 ? 8 : 4, KS = 32 / RG, RB = DQ / (4 * RG), NC = 4 * (8 / RB);
  static constexpr int SX = NC + 4;
  static constexpr size_t smem = sizeof(float) * (3 * (DQ * DQ + DQ) + 2 * DQ * SX);
};
template <int DQ>
__global__ void __launch_bounds__(256)
    full_group_kernel(const DevParams* __restrict__, const FullArgs* __restrict__ Fg,
                      DevState* __restrict__ st, cudaGraphConditionalHandle, int use_cond) {
  using Tile = GroupTile<DQ>;
  constexpr int RG = Tile::RG, KS = Tile::KS, RB = Tile::RB, NC = Tile::NC, SX = Tile::SX;
  __shared__ FullArgs F;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  load_struct(Fg, F);
  __syncthreads();
  if (sweep_done(st, use_cond, F.maxiter)) return;
  float* Ms = reinterpret_cast<float*>(smem_raw);  // three maps, DQ x DQ column-major
  float* bs = Ms + 3 * DQ * DQ;                    // their offsets
  float* xs = bs + 3 * DQ;                         // DQ x SX, the columns, two turns
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row = warp % RB * 4 * RG + lane % RG * 4, cg = 4 * (warp / RB), kq = lane / RG;
  constexpr int slices = (DQ + NC) / NC;
  const int grp = static_cast<int>(blockIdx.x) / slices, slice = static_cast<int>(blockIdx.x) % slices;
  const int ch0 = grp * F.G, n = min(F.G, F.nchunks - ch0);
  auto fetch = [&](int i) {
    if (i < n) {
      const int slot = i % 3;
      const float* src = F.Phi + static_cast<size_t>(ch0 + i) * DQ * DQ;
      float* dst = Ms + slot * DQ * DQ;
      for (int k = tid; k < DQ * DQ / 4; k += 256) cp_async16(dst + 4 * k, src + 4 * k);
      if (tid < DQ / 4)
        cp_async16(bs + slot * DQ + 4 * tid, F.beta + static_cast<size_t>(ch0 + i) * DQ + 4 * tid);
    }
    cp_async_commit();
  };
  fetch(0);
  fetch(1);
  for (int i = tid; i < DQ * NC; i += 256) {
    const int r = i / NC, c = slice * NC + i % NC;
    xs[r * SX + i % NC] = r == c ? 1.f : 0.f;
  }
  // the lane's column once the partial tiles are summed (column DQ is the offset's; past
  // it, unused)
  const int own = cg + 2 * (lane >> 4) + (lane >> 3 & 1), col = slice * NC + own;
  for (int i = 0; i < n; ++i) {
    cp_async_wait<1>();
    __syncthreads();  // map i and the columns are in place, map i - 1's slot is free
    fetch(i + 2);
    const int slot = i % 3;
    const float* M = Ms + slot * DQ * DQ + row;
    const float* x = xs + (i & 1) * DQ * SX + cg;
    F2 a[4][2];
#pragma unroll
    for (int c = 0; c < 4; ++c) a[c][0] = a[c][1] = F2{0ull};
#pragma unroll 4
    for (int k = kq; k < DQ; k += KS) {
      const ulonglong2 m = *reinterpret_cast<const ulonglong2*>(M + k * DQ);
      float v[4];
      load4(x + k * SX, v);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const F2 vv = pack2(v[c], v[c]);
        a[c][0] = fma2(F2{m.x}, vv, a[c][0]);
        a[c][1] = fma2(F2{m.y}, vv, a[c][1]);
      }
    }
    float t[4][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      unpack2(a[c][0], t[c][0], t[c][1]);
      unpack2(a[c][1], t[c][2], t[c][3]);
    }
    const bool hi16 = lane & 16, hi8 = lane & 8;
    float h[2][4], acc[4];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        h[c][e] = (hi16 ? t[c + 2][e] : t[c][e]) +
                  __shfl_xor_sync(0xffffffffu, hi16 ? t[c][e] : t[c + 2][e], 16);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      acc[e] = (hi8 ? h[1][e] : h[0][e]) + __shfl_xor_sync(0xffffffffu, hi8 ? h[0][e] : h[1][e], 8);
    if (KS == 8)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 4);
    if (col == DQ) {
      float b[4];
      load4(bs + slot * DQ + row, b);
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] += b[e];
    }
    float* xn = xs + ((i + 1) & 1) * DQ * SX;
#pragma unroll
    for (int e = 0; e < 4; ++e) xn[(row + e) * SX + own] = acc[e];
    // after chunk i: the prefix of chunk i + 1, or the group's map
    float* phi = i + 1 < n ? F.PPhi + static_cast<size_t>(ch0 + i + 1) * DQ * DQ
                           : F.GPhi + static_cast<size_t>(grp) * DQ * DQ;
    float* beta = i + 1 < n ? F.pbeta + static_cast<size_t>(ch0 + i + 1) * DQ
                            : F.gbeta + static_cast<size_t>(grp) * DQ;
    if (col <= DQ && (KS == 4 || !(lane & 4)))
      store4(col < DQ ? phi + static_cast<size_t>(col) * DQ + row : beta + row, acc);
  }
}

// ---------------------------------------------------------------------------
// carry, over the groups: din_0 = 0, din_{g+1} = Phi'_g din_g + beta'_g (one CTA).  Thread
// (part, row) sums KC terms of row `row` (the map is column-major, so the
// threads of a part read consecutive rows: coalesced), partial sums combined
// through shared memory.  Each thread keeps its KC map entries for the next
// two chunks in registers, loaded from L2 two steps ahead (a three-slot ring),
// so a step waits on no copy.
// ---------------------------------------------------------------------------
template <int DQ>
__global__ void __launch_bounds__(256)
    full_carry_kernel(const DevParams* __restrict__, const FullArgs* __restrict__ Fg,
                      DevState* __restrict__ st, cudaGraphConditionalHandle, int use_cond) {
  constexpr int PARTS = DQ >= 128 ? 2 : 4;
  constexpr int KC = DQ / PARTS;
  static_assert(PARTS * DQ <= 256, "one thread a (part, row)");
  __shared__ FullArgs F;
  __shared__ float vec[2][DQ];
  __shared__ float pbuf[PARTS][DQ];
  load_struct(Fg, F);
  __syncthreads();
  if (sweep_done(st, use_cond, F.maxiter)) return;
  const int tid = threadIdx.x;
  // the groups' maps, or with one chunk a group the chunks'
  const int nch = F.ngroups;
  const float* __restrict__ maps = F.G > 1 ? F.GPhi : F.Phi;
  const float* __restrict__ offs = F.G > 1 ? F.gbeta : F.beta;
  const int row = tid % DQ, part = tid / DQ;
  const bool worker = part < PARTS;
  const int k0 = part * KC;
  for (int i = tid; i < 2 * DQ; i += blockDim.x) (&vec[0][0])[i] = 0.f;
  for (int i = tid; i < DQ; i += blockDim.x) F.din[i] = 0.f;
  float m[3][KC];
  float bt[3] = {0.f, 0.f, 0.f};
  auto fetch = [&](int c, float (&dst)[KC], float& b) {
    if (c < nch - 1) {
      if (worker) {
        const float* Ph = maps + static_cast<size_t>(c) * DQ * DQ + static_cast<size_t>(k0) * DQ + row;
#pragma unroll
        for (int k = 0; k < KC; ++k) dst[k] = __ldcg(Ph + static_cast<size_t>(k) * DQ);
      }
      if (tid < DQ) b = __ldcg(offs + static_cast<size_t>(c) * DQ + tid);
    }
  };
  auto step = [&](int c, const float (&cur)[KC], float b) {
    if (worker) {
      const float* x = vec[c & 1] + k0;
      float a0 = 0.f, a1 = 0.f;
#pragma unroll
      for (int k = 0; k < KC; k += 2) {
        a0 = fmaf(cur[k], x[k], a0);
        a1 = fmaf(cur[k + 1], x[k + 1], a1);
      }
      pbuf[part][row] = a0 + a1;
    }
    __syncthreads();
    if (tid < DQ) {
      float y = b;
#pragma unroll
      for (int p = 0; p < PARTS; ++p) y += pbuf[p][tid];
      vec[(c + 1) & 1][tid] = y;
      F.din[static_cast<size_t>(c + 1) * DQ + tid] = y;
    }
    __syncthreads();
  };
  __syncthreads();
  fetch(0, m[0], bt[0]);
  fetch(1, m[1], bt[1]);
  for (int c = 0; c < nch - 1; c += 3) {
    fetch(c + 2, m[2], bt[2]);
    step(c, m[0], bt[0]);
    if (c + 1 >= nch - 1) break;
    fetch(c + 3, m[0], bt[0]);
    step(c + 1, m[1], bt[1]);
    if (c + 2 >= nch - 1) break;
    fetch(c + 4, m[1], bt[1]);
    step(c + 2, m[2], bt[2]);
  }
}

// ---------------------------------------------------------------------------
// apply: replay each chunk from its entering update (warp 0) while the
// cp.async copies of the old iterates land, rotate back (warp-tiled
// Q delta'), damp both iterates, reduce the convergence metric in the
// original basis and run the convergence test in the last CTA.
// ---------------------------------------------------------------------------
template <int DQ>
__global__ void __launch_bounds__(kThreads)
    full_apply_kernel(const DevParams* __restrict__ Pg, const FullArgs* __restrict__ Fg,
                      DevState* __restrict__ st, cudaGraphConditionalHandle cond, int use_cond) {
  __shared__ DevParams P;   // original basis
  __shared__ FullArgs F;
  __shared__ double r_dm[kWarps], r_sm[kWarps];
  __shared__ int s_bad, s_last;
  __shared__ __align__(16) float s_din[kThreads / DQ][DQ];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int cur = st->cur;
  const bool first = st->iter == 0;
  load_struct(Fg, F);
  load_struct(Pg, P);
  __syncthreads();
  if (sweep_done(st, use_cond, P.maxiter)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int D = static_cast<int>(P.D), Dp = static_cast<int>(P.Dp);
  const int L = F.L;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * L;
  const int nt = static_cast<int>(imin64(L, P.T - t0));
  float* Us = reinterpret_cast<float*>(smem_raw);
  float* Vs = Us + L * DQ;
  float* Rs = Vs + L * DQ;
  float* Qs = Rs + L * DQ;   // DQ x DQ, Q column-major
  float* Eo = Qs + DQ * DQ;  // L x DQ old eigenbasis iterate
  float* So = Eo + L * DQ;   // L x Dp old iterate
  uint8_t* as = reinterpret_cast<uint8_t*>(So + L * Dp);
  {
    const int n4 = nt * DQ / 4;
    const float* gu = F.U + t0 * DQ;
    const float* gv = F.V + t0 * DQ;
    const float* gr = F.R + t0 * DQ;
    for (int i = tid; i < n4; i += blockDim.x) {
      cp_async16(Us + 4 * i, gu + 4 * i);
      cp_async16(Vs + 4 * i, gv + 4 * i);
      cp_async16(Rs + 4 * i, gr + 4 * i);
    }
    for (int i = tid; i < DQ * DQ / 4; i += blockDim.x) cp_async16(Qs + 4 * i, F.QcmQ + 4 * i);
    cp_async_commit();
    if (!first) {
      const float* go = static_cast<const float*>(P.S[cur]) + t0 * Dp;
      const float* ge = F.eS[cur] + t0 * DQ;
      for (int i = tid; i < nt * Dp / 4; i += blockDim.x) cp_async16(So + 4 * i, go + 4 * i);
      for (int i = tid; i < n4; i += blockDim.x) cp_async16(Eo + 4 * i, ge + 4 * i);
    }
    cp_async_commit();
    for (int i = tid; i < nt; i += blockDim.x) as[i] = F.acc[t0 + i];
    if (tid == 0) s_bad = 0;
  }
  // the update entering the chunk: its group's, through the prefix of the group's
  // earlier chunks (the group's first chunk has none)
  const int ch = static_cast<int>(blockIdx.x), grp = ch / F.G;
  {
    constexpr int PARTS = kThreads / DQ, KC = DQ / PARTS;
    const float* gin = F.din + static_cast<size_t>(grp) * DQ;
    const int row = tid % DQ, part = tid / DQ;
    if (ch > grp * F.G) {
      float a = 0.f;
      const float* Ph = F.PPhi + static_cast<size_t>(ch) * DQ * DQ + static_cast<size_t>(part * KC) * DQ + row;
#pragma unroll
      for (int k = 0; k < KC; ++k)
        a = fmaf(__ldcg(Ph + static_cast<size_t>(k) * DQ), __ldcg(gin + part * KC + k), a);
      s_din[part][row] = a;
      if (part == 0) s_din[0][row] += __ldcg(F.pbeta + static_cast<size_t>(ch) * DQ + row);
    } else {
      s_din[part][row] = part == 0 ? __ldcg(gin + row) : 0.f;
    }
  }
  cp_async_wait<1>();
  __syncthreads();
  if (warp == 0) {
    // lanes past DQ carry zeros through the warp reduction
    const bool in = 4 * lane < DQ;
    const float eps = static_cast<float>(P.eps);
    float d[4] = {0.f, 0.f, 0.f, 0.f}, lc[4] = {0.f, 0.f, 0.f, 0.f};
    if (in) {
#pragma unroll
      for (int p = 0; p < kThreads / DQ; ++p) {
        float v[4];
        load4(&s_din[p][4 * lane], v);
#pragma unroll
        for (int e = 0; e < 4; ++e) d[e] += v[e];
      }
      float l4[4];
      load4(F.lamQ + 4 * lane, l4);
#pragma unroll
      for (int e = 0; e < 4; ++e) lc[e] = 4 * lane + e < D ? 1.f - eps * l4[e] : 0.f;
    }
    // step s's u', v', r' and accept flag are loaded during step s - 1
    float u[4] = {0.f, 0.f, 0.f, 0.f}, v[4] = {0.f, 0.f, 0.f, 0.f}, r[4] = {0.f, 0.f, 0.f, 0.f};
    bool a = false;
    if (nt > 0) {
      if (in) {
        load4(Us + 4 * lane, u);
        load4(Vs + 4 * lane, v);
        load4(Rs + 4 * lane, r);
      }
      a = as[0] != 0;
    }
    for (int s = 0; s < nt; ++s) {
      float un[4] = {0.f, 0.f, 0.f, 0.f}, vn[4] = {0.f, 0.f, 0.f, 0.f}, rn[4] = {0.f, 0.f, 0.f, 0.f};
      bool an = false;
      if (s + 1 < nt) {
        if (in) {
          load4(Us + (s + 1) * DQ + 4 * lane, un);
          load4(Vs + (s + 1) * DQ + 4 * lane, vn);
          load4(Rs + (s + 1) * DQ + 4 * lane, rn);
        }
        an = as[s + 1] != 0;
      }
      const float dot = warp_sum((v[0] * d[0] + v[1] * d[1]) + (v[2] * d[2] + v[3] * d[3]));
#pragma unroll
      for (int e = 0; e < 4; ++e) d[e] = fmaf(u[e], dot, (a ? lc[e] : 1.f) * d[e]) + r[e];
      if (in) store4(Rs + s * DQ + 4 * lane, d);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        u[e] = un[e];
        v[e] = vn[e];
        r[e] = rn[e];
      }
      a = an;
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  float* Snew = static_cast<float*>(P.S[cur ^ 1]);
  float* Enew = F.eS[cur ^ 1];
  const float* x0 = static_cast<const float*>(P.x0);
  const float* x0e = F.ex0;
  const float dmp = static_cast<float>(P.damping);
  float dm = 0.f, smx = 0.f;  // maxima are exact in FP32
  bool bad = false;
  for (int tile = warp; 8 * tile < nt; tile += kWarps) {
    const int c0 = 8 * tile;
    const int nc = min(8, nt - c0);
    float acc[8][4];
    warp_tile8<DQ>(Qs, Rs + c0 * DQ, DQ, nc, DQ, acc);
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (c >= nc) break;
      const int64_t t = t0 + c0 + c;
      if (4 * lane < D) {
        float o[4], n[4];
        load4(first ? x0 + 4 * lane : So + (c0 + c) * Dp + 4 * lane, o);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (4 * lane + e < D) {
            n[e] = fmaf(dmp, acc[c][e], o[e]);
            dm = fmaxf(dm, fabsf(n[e] - o[e]));
            smx = fmaxf(smx, fabsf(n[e]));
            bad |= !isfinite(n[e]);
          } else {
            n[e] = 0.f;
          }
        }
        store4(Snew + t * Dp + 4 * lane, n);
      }
      if (4 * lane < DQ) {
        float de[4], eo[4], en[4];
        load4(Rs + (c0 + c) * DQ + 4 * lane, de);
        load4(first ? x0e + 4 * lane : Eo + (c0 + c) * DQ + 4 * lane, eo);
#pragma unroll
        for (int e = 0; e < 4; ++e) en[e] = fmaf(dmp, de[e], eo[e]);
        store4(Enew + t * DQ + 4 * lane, en);
      }
    }
  }
  dm = warp_max(dm);
  smx = warp_max(smx);
  bad = __any_sync(0xffffffffu, bad);
  if (lane == 0) {
    r_dm[warp] = static_cast<double>(dm);
    r_sm[warp] = static_cast<double>(smx);
    if (bad) s_bad = 1;
  }
  __syncthreads();
  if (tid == 0) {
    // this CTA's maxima into its own slot (no contended atomics)
    for (int w = 1; w < kWarps; ++w) {
      r_dm[0] = fmax(r_dm[0], r_dm[w]);
      r_sm[0] = fmax(r_sm[0], r_sm[w]);
    }
    F.part[2 * blockIdx.x] = r_dm[0];
    F.part[2 * blockIdx.x + 1] = r_sm[0];
    if (s_bad) atomicCAS(&st->status, 0, static_cast<int>(kStNonfinite));
    __threadfence();
    const unsigned prev = atomicAdd(&st->done_counter, 1u);
    s_last = prev == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;
  // last CTA: reduce every CTA's slot, the convergence test (DEER.jl:567-578)
  // and loop control
  __threadfence();
  double pd = 0.0, ps = 0.0;
  for (int i = tid; i < static_cast<int>(gridDim.x); i += blockDim.x) {
    pd = fmax(pd, __ldcg(F.part + 2 * i));
    ps = fmax(ps, __ldcg(F.part + 2 * i + 1));
  }
  pd = warp_max(pd);
  ps = warp_max(ps);
  __syncthreads();
  if (lane == 0) {
    r_dm[warp] = pd;
    r_sm[warp] = ps;
  }
  __syncthreads();
  if (tid != 0) return;
  double dmax = 0.0, smax = 0.0;
  for (int w = 0; w < kWarps; ++w) dmax = fmax(dmax, r_dm[w]), smax = fmax(smax, r_sm[w]);
  const double metric = dmax / (P.tol_abs + P.tol_rel * smax);
  const int status = atomicAdd(&st->status, 0);
  const int iter = st->iter;
  const int converged = metric <= 1.0;
  st->metric = metric;
  st->iter = iter + 1;
  st->cur = cur ^ 1;
  st->converged = converged;
  st->done_counter = 0;
  st->dmax_bits = 0;
  st->smax_bits = 0;
  __threadfence();
  const bool more = !converged && (iter + 1 < P.maxiter) && status == 0;
  if (use_cond) cudaGraphSetConditional(cond, more ? 1u : 0u);
}

// ---------------------------------------------------------------------------
// Adjoint kernels
// ---------------------------------------------------------------------------

// Per column t: accept flag of the returned trajectory, the reversed-scan
// multiplier Arev[T - t] = c_t (primed, diagonal) and the objective terms in
// reversed order.  Objective 1: c_t = 2 S_t / T.  Objective 0 (ESJD,
// Rao-Blackwellised): L = (1/T) sum_t alpha_t e_t, e_t = |y_t - x_bar_t|^2,
// alpha_t = min(1, exp(log alpha_t)); term t contributes
//   dL_t/dx_bar_t = (1/T)[alpha' e_t v_t + alpha_t 2 eps H (y_t - x_bar_t)]   to c_{t-1}
//   (1/T)[alpha' e_t dla/deps + alpha_t de_t/deps]                          to the explicit eps term
// with alpha' = d alpha / d log alpha and H = -P.
template <int TK>
__global__ void __launch_bounds__(kThreads)
    adjoint_terms_kernel(const DevParams* __restrict__ Pg, const FullArgs* __restrict__ Fg,
                         int objective, const float* __restrict__ S, float* __restrict__ Brev,
                         float* __restrict__ Arev, double* __restrict__ direct) {
  __shared__ DevParams P;
  __shared__ FullArgs F;
  __shared__ double r_dir[kWarps];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  load_struct(Fg, F);
  load_params(Pg, P);
  constexpr bool dense = TK == kDenseGauss;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int D = static_cast<int>(P.D), Dp = static_cast<int>(P.Dp);
  const int64_t T = P.T;
  Smem<float> sm = carve<float>(smem_raw, P, 1, dense);
  float* Qs = reinterpret_cast<float*>(smem_raw + plan_sweep_smem<float>(Dp, 1, dense).total);
  float* vw = Qs + (dense ? Dp * Dp : 0) + warp * Dp;
  if (dense)
    for (int i = threadIdx.x; i < Dp * Dp; i += blockDim.x) Qs[i] = F.Qrm[i];
  for (int i = lane; i < Dp; i += 32) vw[i] = 0.f;
  __syncthreads();
  const float* x0 = static_cast<const float*>(P.x0);
  const TapeKey key(P.seed, P.block);
  const float eps = static_cast<float>(P.eps);
  const double epsd = P.eps;
  const double invT = 1.0 / static_cast<double>(T);
  float lamq[4] = {0.f, 0.f, 0.f, 0.f};
  if (4 * lane < D) load4(F.lam + 4 * lane, lamq);
  double dir = 0.0;
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * kWarps + warp; t < T;
       t += static_cast<int64_t>(gridDim.x) * kWarps) {
    const float* xcol = t == 0 ? x0 : S + (t - 1) * Dp;
    Col<float, 1> c;
    column_forward<float, TK, 1>(P, sm, key, xcol, static_cast<int>(t), c);
    const double logu = P.logu[t];
    const bool acc = logu < c.la;
    if (lane == 0) F.acc[t] = acc ? 1 : 0;
    if (4 * lane < Dp) {
      float m[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) m[e] = t == 0 ? 1.f : (acc ? 1.f - eps * lamq[e] : 1.f);
      // C_t links lambda_{t-1} (reversed index T - t) to lambda_t; index 0 has no predecessor
      store4(Arev + (t == 0 ? 0 : T - t) * Dp + 4 * lane, m);
    }
    float cvec[4] = {0.f, 0.f, 0.f, 0.f};
    int64_t dst = -1;
    if (objective == 1) {
      if (4 * lane < D) {
        float s4[4];
        load4(S + t * Dp + 4 * lane, s4);
#pragma unroll
        for (int e = 0; e < 4; ++e)
          cvec[e] = 4 * lane + e < D ? static_cast<float>(2.0 * invT * s4[e]) : 0.f;
      }
      dst = T - 1 - t;
    } else {
      const double la = c.la;
      const double alpha = la < 0.0 ? exp(la) : 1.0;
      const double dalpha = la < 0.0 ? alpha : 0.0;
      const float inv_s2e = static_cast<float>(1.0 / P.sqrt2eps);
      float dyx[1][4], dy[1][4], q[1][4], npdy[1][4], npdyx[1][4], v[4];
      double e2 = 0.0, dede = 0.0, qq = 0.0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool in = 4 * lane + e < D;
        dyx[0][e] = in ? c.y[0][e] - c.x[0][e] : 0.f;              // y - x
        dy[0][e] = in ? c.gx[0][e] + c.xi[0][e] * inv_s2e : 0.f;  // dy/deps
        q[0][e] = in ? c.x[0][e] - c.y[0][e] - eps * c.gy[0][e] : 0.f;
        e2 += static_cast<double>(dyx[0][e]) * dyx[0][e];
        dede += 2.0 * static_cast<double>(dyx[0][e]) * dy[0][e];
        qq += static_cast<double>(q[0][e]) * q[0][e];
      }
      if constexpr (dense) {
        float pgy[1][4], pr[1][4], ppr[1][4];
        dense_neg_pv<float, 1>(P, sm, dy, npdy);    // -P dy
        dense_neg_pv<float, 1>(P, sm, dyx, npdyx);  // -P (y - x)
        dense_neg_pv<float, 1>(P, sm, c.gy, pgy);
        dense_neg_pv<float, 1>(P, sm, q, pr);
        dense_neg_pv<float, 1>(P, sm, pr, ppr);
#pragma unroll
        for (int e = 0; e < 4; ++e)
          v[e] = c.gy[0][e] + eps * pgy[0][e] - c.gx[0][e] + pr[0][e] + 0.5f * eps * ppr[0][e];
      } else {
        float lam[4] = {0.f, 0.f, 0.f, 0.f};
        if (4 * lane < D) load4(P.prec_f + 4 * lane, lam);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float el = eps * lam[e];
          npdy[0][e] = -lam[e] * dy[0][e];
          npdyx[0][e] = -lam[e] * dyx[0][e];
          v[e] = (1.f - el) * c.gy[0][e] - c.gx[0][e] - lam[e] * q[0][e] * (1.f - 0.5f * el);
        }
      }
      // dla/deps = g_y.dy - q.dq/(2 eps) + |q|^2/(4 eps^2),  dq = -(dy - eps P dy) - g_y
      double dla = 0.0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (4 * lane + e >= D) continue;
        const double dq = -(static_cast<double>(dy[0][e]) + epsd * npdy[0][e]) - c.gy[0][e];
        dla += static_cast<double>(c.gy[0][e]) * dy[0][e] -
               static_cast<double>(q[0][e]) * dq / (2 * epsd);
      }
      dla = warp_sum(dla) + warp_sum(qq) / (4 * epsd * epsd);
      e2 = warp_sum(e2);
      dede = warp_sum(dede);
      if (lane == 0) dir += invT * (dalpha * dla * e2 + alpha * dede);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        cvec[e] = 4 * lane + e < D ? static_cast<float>(invT * (dalpha * e2 * v[e] +
                                                                alpha * 2.0 * epsd * npdyx[0][e]))
                                   : 0.f;
      dst = t >= 1 ? T - t : -1;  // c_{t-1} sits at reversed index T - 1 - (t - 1)
      if (t == 0 && 4 * lane < Dp) {
        const float z[4] = {0.f, 0.f, 0.f, 0.f};
        store4(Brev + 4 * lane, z);  // c_{T-1} = 0: the last state enters no term
      }
    }
    if (dense) rotate_quad(Qs, vw, D, Dp, cvec);
    if (dst >= 0 && 4 * lane < Dp) store4(Brev + dst * Dp + 4 * lane, cvec);
  }
  if (lane == 0) r_dir[warp] = dir;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < kWarps; ++w) s += r_dir[w];
    if (s != 0.0) atomicAdd(direct, s);
  }
}

// dL/deps and dL/dlog s from the reversed primed adjoint Lrev.
template <int TK>
__global__ void __launch_bounds__(kThreads)
    adjoint_reduce_kernel(const DevParams* __restrict__ Pg, const FullArgs* __restrict__ Fg,
                          int objective, const float* __restrict__ S,
                          const float* __restrict__ Lrev, double* __restrict__ out) {
  __shared__ DevParams P;
  __shared__ FullArgs F;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  load_struct(Fg, F);
  load_params(Pg, P);
  constexpr bool dense = TK == kDenseGauss;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int D = static_cast<int>(P.D), Dp = static_cast<int>(P.Dp);
  const int64_t T = P.T;
  double* red = reinterpret_cast<double*>(smem_raw);  // kWarps x (Dp + 1)
  float* Qs = reinterpret_cast<float*>(red + kWarps * (Dp + 1));
  float* vw = Qs + (dense ? Dp * Dp : 0) + warp * Dp;
  if (dense)
    for (int i = threadIdx.x; i < Dp * Dp; i += blockDim.x) Qs[i] = F.Qrm[i];
  for (int i = lane; i < Dp; i += 32) vw[i] = 0.f;
  __syncthreads();
  const float* x0 = static_cast<const float*>(P.x0);
  const double inv_s2e = 1.0 / P.sqrt2eps;
  float lamq[4] = {0.f, 0.f, 0.f, 0.f};
  if (4 * lane < D) load4(F.lam + 4 * lane, lamq);
  double ge = 0.0, gs[4] = {0.0, 0.0, 0.0, 0.0};
  for (int64_t t = static_cast<int64_t>(blockIdx.x) * kWarps + warp; t < T;
       t += static_cast<int64_t>(gridDim.x) * kWarps) {
    if (!F.acc[t]) continue;  // warp-uniform
    const float* xcol = t == 0 ? x0 : S + (t - 1) * Dp;
    float xm[4] = {0.f, 0.f, 0.f, 0.f}, xi[4] = {0.f, 0.f, 0.f, 0.f};
    if (4 * lane < D) {
      load4(xcol + 4 * lane, xm);
      load4(P.xi + t * Dp + 4 * lane, xi);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        xm[e] = 4 * lane + e < D ? static_cast<float>(xm[e] - P.mean_d[4 * lane + e]) : 0.f;
    }
    if (dense) {
      rotate_quad(Qs, vw, D, Dp, xm);
      rotate_quad(Qs, vw, D, Dp, xi);
    }
    float lm[4] = {0.f, 0.f, 0.f, 0.f};
    if (4 * lane < Dp) load4(Lrev + (T - 1 - t) * Dp + 4 * lane, lm);
    double g = 0.0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (4 * lane + e >= D) continue;
      g += static_cast<double>(lm[e]) *
           (-static_cast<double>(lamq[e]) * xm[e] + static_cast<double>(xi[e]) * inv_s2e);
      if (objective == 1) gs[e] += P.eps * static_cast<double>(lamq[e]) * lm[e] * xm[e];
    }
    ge += warp_sum(g);
  }
  if (4 * lane < Dp)
#pragma unroll
    for (int e = 0; e < 4; ++e) red[warp * (Dp + 1) + 4 * lane + e] = gs[e];
  if (lane == 0) red[warp * (Dp + 1) + Dp] = ge;
  __syncthreads();
  for (int i = threadIdx.x; i <= Dp; i += blockDim.x) {
    double s = 0.0;
    for (int w = 0; w < kWarps; ++w) s += red[w * (Dp + 1) + i];
    if (s != 0.0) {
      if (i == Dp) atomicAdd(out, s);
      else if (i < D) atomicAdd(out + 1 + i, s);
    }
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {

size_t chunk_smem(int Dq, int L) { return sizeof(float) * 3 * static_cast<size_t>(L) * Dq + L + 16; }
size_t apply_smem(int Dq, int64_t Dp, int L) {
  return sizeof(float) * (4 * static_cast<size_t>(L) * Dq + static_cast<size_t>(Dq) * Dq + L * Dp) +
         L + 16;
}

size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

template <int DQ>
void pick_kernels(FullPlan* fp) {
  fp->chunk = reinterpret_cast<const void*>(&full_chunk_kernel<DQ>);
  fp->threads_chunk = chunk_threads(DQ);
  fp->carry = reinterpret_cast<const void*>(&full_carry_kernel<DQ>);
  fp->group = reinterpret_cast<const void*>(&full_group_kernel<DQ>);
  fp->group_slices = (DQ + GroupTile<DQ>::NC) / GroupTile<DQ>::NC;
  fp->smem_group = GroupTile<DQ>::smem;
  fp->apply = reinterpret_cast<const void*>(&full_apply_kernel<DQ>);
  fp->rotate = reinterpret_cast<const void*>(&full_rotate_kernel<DQ>);
}

}  // namespace

int full_stride(int64_t Dp) {
  for (int q = 16; q <= 128; q <<= 1)
    if (Dp <= q) return q;
  return 0;
}

bool full_plan(int64_t Dp, int64_t T, int tkind, int num_sms, int chunks_override, FullPlan* fp) {
  (void)tkind;
  const int Dq = full_stride(Dp);
  if (Dq == 0 || T < 1) return false;
  fp->Dq = Dq;
  switch (Dq) {
    case 16: pick_kernels<16>(fp); break;
    case 32: pick_kernels<32>(fp); break;
    case 64: pick_kernels<64>(fp); break;
    default: pick_kernels<128>(fp); break;
  }
  const size_t budget = 200 * 1024;
  int Lmax = 1;
  while (Lmax < 4096 && chunk_smem(Dq, Lmax + 1) <= budget && apply_smem(Dq, Dp, Lmax + 1) <= budget)
    ++Lmax;
  // The serial chain of a sweep: L steps of the chunk maps and of the replay, G steps of
  // the groups' composition, nchunks / G steps of the carry.  us a step, fitted to sweeps
  // timed over 64 .. 592 chunks: a chunk step takes c_lat, or c_iss for each chunk its SM
  // holds; a group step c_g for each CTA (group_slices a group) its SM holds; a carry step c_c.
  // At D = 64, T = 8192: 56 + 7 + 22 steps or 28 + 14 + 21, 67 to 70 us a sweep, against 64 + 128 steps and
  // 103 us with the carry over the chunks; 64 chunks take 100 us, 592 take 89.  D = 128: 171 us (start 428), 592 chunks 264.
  const int w = Dq == 16 ? 0 : Dq == 32 ? 1 : Dq == 64 ? 2 : 3;
  static constexpr double kStep[4][4] = {{0.30, 0.10, 0.30, 0.30},
                                         {0.30, 0.10, 0.40, 0.30},
                                         {0.35, 0.17, 0.70, 0.30},
                                         {0.60, 0.45, 1.30, 0.60}};
  const double c_lat = kStep[w][0], c_iss = kStep[w][1], c_g = kStep[w][2], c_c = kStep[w][3];
  auto per_sm = [&](int64_t n) { return static_cast<double>((n + num_sms - 1) / num_sms); };
  auto groups = [&](int64_t n, double* cost) {  // chunks a group
    int best = 1;
    *cost = c_c * static_cast<double>(n);
    for (int g = 2; g <= 64 && g <= n; g += 1 + g / 8) {
      const int64_t ng = (n + g - 1) / g;
      const double c = 4.0 + c_g * g * per_sm(ng * fp->group_slices) + c_c * static_cast<double>(ng);
      if (c < *cost) *cost = c, best = g;
    }
    return best;
  };
  int64_t L = 0;
  double best = 0.0, c = 0.0;
  if (chunks_override > 0) {
    L = std::min<int64_t>((T + chunks_override - 1) / chunks_override, Lmax);
  } else {
    const int64_t l0 = std::min<int64_t>(Lmax, (T + 4 * num_sms - 1) / (4 * num_sms));
    for (int64_t l = l0; l <= Lmax && (L == 0 || l <= T); l += 1 + l / 16) {
      const int64_t n = (T + l - 1) / l;
      groups(n, &c);
      c += static_cast<double>(l) * std::max(c_lat, c_iss * per_sm(n));
      if (L == 0 || c < best) best = c, L = l;
    }
  }
  fp->L = static_cast<int>(L);
  fp->nchunks = static_cast<int>((T + L - 1) / L);
  fp->G = groups(fp->nchunks, &c);
  fp->ngroups = (fp->nchunks + fp->G - 1) / fp->G;
  fp->smem_chunk = chunk_smem(Dq, fp->L);
  fp->smem_apply = apply_smem(Dq, Dp, fp->L);
  fp->smem_carry = 0;  // static shared memory only
  fp->smem_eval = plan_sweep_smem<float>(Dq, 1, false).total;
  fp->eval_grid =
      static_cast<int>(std::min<int64_t>((T + kWarps - 1) / kWarps, int64_t(num_sms) * 4));
  fp->eval = reinterpret_cast<const void*>(&full_eval_kernel);
  fp->nnodes = 0;
  auto node = [&](const void* fn, int grid, int threads, size_t smem) {
    fp->nodes[fp->nnodes++] = FullNode{fn, smem, grid, threads};
  };
  node(fp->eval, fp->eval_grid, kThreads, fp->smem_eval);
  node(fp->chunk, fp->nchunks, fp->threads_chunk, fp->smem_chunk);
  if (fp->G > 1) node(fp->group, fp->ngroups * fp->group_slices, 256, fp->smem_group);
  node(fp->carry, 1, 256, fp->smem_carry);
  node(fp->apply, fp->nchunks, kThreads, fp->smem_apply);
  fp->smem_rotate = sizeof(float) * (static_cast<size_t>(Dq) * Dq + kWarps * 8 * Dp);
  fp->rotate_grid = static_cast<int>(
      std::max<int64_t>(1, std::min<int64_t>((T + 8 * kWarps - 1) / (8 * kWarps), num_sms)));
  return true;
}

cudaError_t full_sweep(cudaStream_t s, const FullPlan& fp, const DevParams* Pg, const FullArgs* Fg,
                       DevState* st, cudaGraphConditionalHandle cond, int use_cond) {
  void* args[] = {const_cast<DevParams**>(&Pg), const_cast<FullArgs**>(&Fg), &st, &cond,
                  &use_cond};
  for (int i = 0; i < fp.nnodes; ++i) {
    const FullNode& n = fp.nodes[i];
    const cudaError_t e = cudaLaunchKernel(n.fn, dim3(n.grid), dim3(n.threads), args, n.smem, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// scratch: zero vector | the scan's
size_t full_adjoint_scratch_bytes(int64_t Dp, int64_t T) {
  return al256(4 * Dp) + al256(scan_scratch_bytes(false, Dp, T));
}

cudaError_t full_adjoint(cudaStream_t s, const DevParams* Pg, const FullArgs* Fg,
                         const FullArgs& Fh, int64_t D, int64_t Dp, int64_t T, int tkind,
                         int num_sms, int objective, const float* S, double* out, void* scratch, int* err) {
  const bool dense = tkind == kDenseGauss;
  cudaError_t e = cudaMemsetAsync(out, 0, sizeof(double) * (1 + D), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(Fh.direct, 0, sizeof(double), s);
  if (e != cudaSuccess) return e;
  const int grid =
      static_cast<int>(std::min<int64_t>((T + kWarps - 1) / kWarps, int64_t(num_sms) * 2));
  const size_t st = eval_smem_bytes(Dp, dense);
  const void* tk = dense ? reinterpret_cast<const void*>(&adjoint_terms_kernel<kDenseGauss>)
                         : reinterpret_cast<const void*>(&adjoint_terms_kernel<kDiagGauss>);
  if (st > 0) {
    e = raise_smem_limit(reinterpret_cast<const void*>(tk), st);
    if (e != cudaSuccess) return e;
  }
  float* Brev = Fh.cterm;
  float* Arev = Fh.arev;
  double* dir = Fh.direct;
  void* targs[] = {const_cast<DevParams**>(&Pg), const_cast<FullArgs**>(&Fg), &objective,
                   const_cast<float**>(&S), &Brev, &Arev, &dir};
  e = cudaLaunchKernel(tk, dim3(grid), dim3(kThreads), targs, st, s);
  if (e != cudaSuccess) return e;
  // reverse scan in reversed time: Lrev_tau = Arev_tau * Lrev_{tau-1} + Brev_tau, Lrev_{-1} = 0
  unsigned char* w = static_cast<unsigned char*>(scratch);
  float* zero = reinterpret_cast<float*>(w);
  // the zero vector, and the barrier's word at the start of the scan's scratch
  e = cudaMemsetAsync(zero, 0, al256(4 * Dp) + kScanBarBytes, s);
  if (e != cudaSuccess) return e;
  e = launch_affine_scan(s, false, Dp, T, Arev, Brev, zero, Fh.lam_adj, w + al256(4 * Dp), err);
  if (e != cudaSuccess) return e;
  e = cudaMemcpyAsync(out, Fh.direct, sizeof(double), cudaMemcpyDeviceToDevice, s);
  if (e != cudaSuccess) return e;
  const size_t sr = sizeof(double) * kWarps * (Dp + 1) +
                    sizeof(float) * ((dense ? Dp * Dp : 0) + kWarps * Dp);
  const void* rk = dense ? reinterpret_cast<const void*>(&adjoint_reduce_kernel<kDenseGauss>)
                         : reinterpret_cast<const void*>(&adjoint_reduce_kernel<kDiagGauss>);
  if (sr > 0) {
    e = raise_smem_limit(reinterpret_cast<const void*>(rk), sr);
    if (e != cudaSuccess) return e;
  }
  const float* Lrev = Fh.lam_adj;
  void* rargs[] = {const_cast<DevParams**>(&Pg), const_cast<FullArgs**>(&Fg), &objective,
                   const_cast<float**>(&S), const_cast<float**>(&Lrev), &out};
  return cudaLaunchKernel(rk, dim3(grid), dim3(kThreads), rargs, sr, s);
}

}  // namespace pmcmc
