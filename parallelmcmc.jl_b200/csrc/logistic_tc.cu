// logistic_tc.cu -- one logistic-regression pass on the 5th-generation tensor
// cores (tcgen05 + TMEM + TMA), fused GEMM -> epilogue -> GEMM.
//
// For a tile of trajectory columns (value columns v_t = x_bar_t or y_t, and
// the matching tangent columns z_t or w_t) and all N data rows:
//   GEMM1  L[n, t] = sum_d X[n, d] B[d, t]
//   epilogue (per row n, per column t): p = sigmoid(L), r = y_n - p,
//          s = p (1 - p) L_tangent, loglik = y_n L - softplus(L)  (bayes_logreg.jl:118-154)
//   GEMM2  G[d, t] += sum_n X[n, d] R[n, t],  R = [r | s]
// The N x 2T intermediate never leaves the SM, and the same shared-memory X tile
// serves both GEMMs.  G starts afresh in TMEM after every 128 rows and the epilogue
// threads add the partial sums in registers (round-to-nearest FP32):
// one TMEM accumulation chain over all N rows left the N = 10000 gradient about
// 10x less accurate than an FP32 SGEMM, enough to move the chain by 1.5e-5.
//
// Precision: X, the value columns and r are carried as FP16 hi + lo pairs
// (about 22 significant bits); each value-column product is
// hi*hi + hi*lo + lo*hi with FP32 accumulation.  Tangent columns (only used
// for the Jacobian estimate) and s use a single FP16 term.
//
// Two kernels: logistic_pass_kernel for D <= 256 and logistic_pass_tc_wide_kernel
// above.  Warps 0-15 run the epilogue (warps w, w+4, w+8, w+12 share TMEM lane
// quarter w % 4); one elected lane of warp 16 issues the MMAs.
// Every mbarrier wait is bounded; on timeout the kernel records an error,
// drains its own MMAs and frees TMEM before returning.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "deer_device.cuh"
#include "deer_launch.h"
#include "logistic.h"

namespace pmcmc {
namespace tc {

constexpr int BN = 128;  // data rows per block of the wide variant
constexpr int kThreadsTC = 544;  // 16 epilogue warps + 1 producer warp
constexpr int kEpi = 16;
constexpr int kProd = 16;  // producer / TMEM-owner warp
constexpr int kParts = kEpi / 4;  // epilogue warps per TMEM lane quarter
constexpr uint32_t kTmemCols = 512;
constexpr long long kWaitCycles = 2000000000ll;  // ~1 s at B200 clocks
constexpr uint32_t kBoxX = BN * 128;       // one 64-wide d box of X: 128 rows x 128 B
// R (GEMM2's B operand, N = 96 columns [r hi | s | r lo] by K = BN rows) is
// MN-major with the 128-byte swizzle, like X^T: two 64-column atoms of BN rows
// x 128 B; chunk c (8 columns) of row k sits at chunk c ^ (k & 7).
constexpr uint32_t kRAtom = BN * 128;

__device__ __forceinline__ uint32_t su32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(su32(b))
               : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(
          su32(b)),
      "r"(bytes)
      : "memory");
}
// Bounded wait for the completion of the phase with the given parity: gives up
// after about a second of SM clock (or at once when another CTA of the launch
// has already reported an error).
__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(su32(b)), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity,
                                          const volatile int* err) {
  if (mbar_try(b, parity)) return true;
  const long long start = clock64();
  for (long long i = 0;; ++i) {
    if (mbar_try(b, parity)) return true;
    if ((i & 255) == 255 && (*err || clock64() - start > kWaitCycles)) return false;
  }
}

__device__ __forceinline__ void tma_2d(void* dst, const CUtensorMap* tm, int x, int y,
                                       uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
      "%3}], [%4];" ::"r"(su32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(su32(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(slot)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// One lane of the warp (the same on every call): the issuer of the warp's TMA loads
// and MMAs.  The warp runs the issue loop together and only the instructions
// themselves are predicated, so descriptors and addresses stay in uniform
// registers; a loop inside a lane-0 branch moves every operand there for each
// MMA, 97 cycles an MMA whatever its size, against the 40 - 56 that these
// widths take (M = 128: N = 96 in 56, N = 32 in 40).  The wide pass at N = 5000,
// D = 400, T = 8192 went from 1.26 to 0.91 ms by this alone.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}

// Shared-memory matrix descriptor (tcgen05): start, leading / stride byte
// offsets, version 1, layout (0 = no swizzle, 2 = 128-byte swizzle).
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo,
                                          uint32_t layout) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
  d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(layout & 7u) << 61;
  return d;
}

// Instruction descriptor, kind::f16 with FP16 A/B and FP32 accumulation.
__host__ __device__ constexpr uint32_t idesc_f16(int M, int N, bool a_mn, bool b_mn) {
  return (1u << 4) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

// log(1 + e) for e in [0, 1]: e q(e), q the degree-9 Chebyshev least-squares
// fit of log1p(e) / e on [0, 1] written in powers of e with FP32 coefficients.
// Absolute error below 1.3e-7 on [0, 1] (a correctly rounded FP32 log1p has
// 6e-8; the FP32 rounding of the log-likelihood term it enters is larger than
// either).  FMAs only: no division, no special-function unit.
__device__ __forceinline__ float log1p_unit(float e) {
  float q = -0.0032140363473445177f;
  q = fmaf(q, e, 0.019649166613817215f);
  q = fmaf(q, e, -0.056435029953718185f);
  q = fmaf(q, e, 0.10533228516578674f);
  q = fmaf(q, e, -0.1525145173072815f);
  q = fmaf(q, e, 0.19651491940021515f);
  q = fmaf(q, e, -0.24947808682918549f);
  q = fmaf(q, e, 0.3332909941673279f);
  q = fmaf(q, e, -0.4999985098838806f);
  q = fmaf(q, e, 1.0f);
  return e * q;
}

// Two FP32 values as one FP16x2 word (a in the low half), one conversion.
__device__ __forceinline__ uint32_t half2_bits(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// hi = x with its low 13 mantissa bits cleared: exact in FP16 for
// 2^-14 <= |x| < 65504, and x - hi is exact in FP32 (|x - hi| < 2^-10 |x|).
__device__ __forceinline__ float split_hi(float x) {
  return __uint_as_float(__float_as_uint(x) & 0xffffe000u);
}

// ---------------------------------------------------------------------------
// The pass for D <= 256: one CTA takes 64 trajectory columns and a run of
// 64-row blocks of X.  The columns are the MMAs' A operand, resident for the
// whole run; X streams through shared memory once as the B operand of both GEMMs:
//   GEMM1  L (128 lanes x 64 rows)  = [Bh | Bt] Xl' + Bl Xh' + [Bh | Bt] Xh'
//   GEMM2  G (128 lanes x d)       += [Rh | S] Xl + [Rl | 0] Xh + [Rh | S] Xh
// Lanes: each 32-lane quarter q of TMEM holds value columns 16 q .. 16 q + 15 in
// its lower half and their tangent columns in its upper half (the lanes an M = 64
// MMA writes are the lower halves, so Bl needs no padding).  The small products
// come first, where the accumulator is still small.  TMEM: G in 64 NKB columns,
// two L buffers of 64, [Bh | Bt] in 32 NKB; R overwrites its L in place.
//
// The tensor cores never wait for the epilogue: block b's GEMM1 and block b - 1's
// GEMM2 run while the epilogue turns L(b - 1) and L(b) into R.  Per block 2 x 24
// (NKB = 4) products of 32 and 128 cycles = 3072 cycles at D = 256, and 64 KB of X
// (three stages in flight).  A third of the products' lanes are padding (the lo
// products of the tangent lanes), which the layout pays for keeping X's traffic
// at one read for 64 columns.  The form with X as the A operand (32 columns a CTA,
// one 128 KB block of X, nothing overlapped) took 4.4 us for 128 rows of 32
// columns at first and 3.5 us with its MMAs issued back to back; this takes 2.15 us for
// 64 rows of 64 columns (3650 cycles, of which 3072 on the tensor pipe, at the 1.7 GHz
// the power cap leaves): a pass at N = 10000, D = 256, T = 65536 went from 4.99 and
// 4.12 ms to 2.34 ms, 574 TFLOP/s algorithmic (8 N D T).
//
// A CTA's G is the sum over its rows; `nsplit` CTAs share a tile's rows where the
// tiles alone leave SMs idle, and lg_mid adds their parts.
// ---------------------------------------------------------------------------
constexpr int TB = 64;                        // value columns a CTA
constexpr int RB = 64;                        // rows of X a block
constexpr uint32_t kBox = RB * 128;           // 64 rows (or columns) x 64 values of d, FP16
__host__ __device__ constexpr int stages(int nkb) { return nkb == 4 ? 3 : 4; }
__host__ __device__ constexpr uint32_t pass_smem(int nkb) {
  // Bl | stages x (Xh | Xl) | barriers | alignment slack
  return nkb * kBox + stages(nkb) * 2 * nkb * kBox + 128 + 1024;
}

constexpr int kThreadsPass = 576;             // 16 epilogue warps, the MMA warp, the load warp
constexpr int kLoad = 17;

__device__ __forceinline__ void tma_3d(void* dst, const CUtensorMap* tm, int x, int y, int z,
                                       uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
      "%3, %4}], [%5];" ::"r"(su32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(su32(bar))
      : "memory");
}
// 1 / x for x in [1, 2] (1 ulp).
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// mbar_wait with one answer for the whole warp.
__device__ __forceinline__ bool warp_wait(uint64_t* b, uint32_t parity, const volatile int* err) {
  return __all_sync(0xffffffffu, mbar_wait(b, parity, err));
}

__device__ __forceinline__ void mma_f16_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 8 consecutive TMEM columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// 16 consecutive FP32 TMEM columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// mode 0: value x_bar_t, tangent z_t (probe `probe`); mode 1: value y_t, tangent w_t;
// mode 2: value S_t, no tangent and no G.  G: nsplit parts of 2T x Dp (value block,
// then tangent block), lp: nsplit parts of T.
template <int NKB>
__global__ void __launch_bounds__(kThreadsPass, 1)
    logistic_pass_kernel(const __grid_constant__ CUtensorMap tmXh,
                         const __grid_constant__ CUtensorMap tmXl,
                         const DevParams* __restrict__ Pg, const DevState* __restrict__ st,
                         int mode, int probe, const float* __restrict__ ylab, int64_t N,
                         int64_t T, int64_t Dp, int nsplit, float* __restrict__ G,
                         double* __restrict__ lp, int* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  constexpr int kSt = stages(NKB);
  constexpr uint32_t kHalf = NKB * kBox;  // one of Xh, Xl of a stage
  constexpr int DC = 16 * NKB;            // values of d an epilogue warp owns
  unsigned char* sBl = base;
  unsigned char* sX = base + kHalf;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sX + kSt * 2 * kHalf);
  uint64_t* bar_x = bars;       // [kSt] stage loaded
  uint64_t* bar_f = bars + 4;   // [kSt] the MMAs reading the stage are done
  uint64_t* bar_l = bars + 8;   // [2] L ready
  uint64_t* bar_r = bars + 10;  // [2] R written (and G drained, where it was due)
  uint64_t* bar_g = bars + 12;  // G of two blocks complete
  uint64_t* bar_b = bars + 13;  // column operands written
  uint64_t* bar_z = bars + 14;  // teardown drain
  __shared__ uint32_t s_tmem;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = static_cast<int>(blockIdx.x) / nsplit;
  const int split = static_cast<int>(blockIdx.x) % nsplit;
  const int64_t t0 = static_cast<int64_t>(tile) * TB;
  const int nb_all = static_cast<int>((N + RB - 1) / RB);
  const int b0 = static_cast<int>(static_cast<int64_t>(nb_all) * split / nsplit);
  const int nb = static_cast<int>(static_cast<int64_t>(nb_all) * (split + 1) / nsplit) - b0;
  const bool has_g = mode != 2;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 15; ++i) mbar_init(bars + i, i == 10 || i == 11 || i == 13 ? 32 * kEpi : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kProd) tmem_alloc(&s_tmem, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  const uint32_t tG = tmem, tL = tmem + 256, tB = tmem + 384;

  if (warp == kProd) {
    const bool el = elect_one();
    bool ok = true;
    constexpr uint32_t i1 = idesc_f16(128, RB, false, false), i1h = idesc_f16(64, RB, false, false);
    constexpr uint32_t i2 = idesc_f16(128, 64 * NKB, false, true);
    const uint64_t x1 = sdesc(su32(sX), 16, 1024, 2), x2 = sdesc(su32(sX), kBox, 1024, 2);
    const uint64_t bl = sdesc(su32(sBl), 16, 1024, 2);
    // GEMM2 of block b (in stage s); G starts afresh every second block
    auto gemm2 = [&](int b, int s) {
      if (el) {
        if (has_g) {
          const uint32_t a = tL + 64 * (b & 1);
          const uint64_t xh = x2 + ((s * 2 * kHalf) >> 4), xl = xh + (kHalf >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_f16_ts(tG, a + 16 * k, xl + ((k * 2048) >> 4), i2, ((b & 1) | k) != 0);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_f16_ts(tG, a + 16 * k + 8, xh + ((k * 2048) >> 4), i2, 1);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_f16_ts(tG, a + 16 * k, xh + ((k * 2048) >> 4), i2, 1);
        }
        mma_commit(bar_f + s);
        if (has_g && ((b & 1) || b == nb - 1)) mma_commit(bar_g);
      }
      __syncwarp();
    };
    ok = warp_wait(bar_b, 0, err);
    tc_fence_after();
    int s = 0, sp = 0;  // stage of this block and of the one before
    uint32_t xph = 0;  // phase bit of each stage
    for (int b = 0; b < nb && ok; ++b) {
      if (!(ok = warp_wait(bar_x + s, (xph >> s) & 1u, err))) break;
      xph ^= 1u << s;
      tc_fence_after();
      if (el) {
        const uint32_t d = tL + 64 * (b & 1);
        const uint64_t xh = x1 + ((s * 2 * kHalf) >> 4), xl = xh + (kHalf >> 4);
#pragma unroll
        for (int k = 0; k < 4 * NKB; ++k)
          mma_f16_ts(d, tB + 8 * k, xl + ((k / 4 * kBox + k % 4 * 32) >> 4), i1, k != 0);
#pragma unroll
        for (int k = 0; k < 4 * NKB; ++k)
          mma_f16(d, bl + ((k / 4 * kBox + k % 4 * 32) >> 4),
                  xh + ((k / 4 * kBox + k % 4 * 32) >> 4), i1h, 1);
#pragma unroll
        for (int k = 0; k < 4 * NKB; ++k)
          mma_f16_ts(d, tB + 8 * k, xh + ((k / 4 * kBox + k % 4 * 32) >> 4), i1, 1);
        mma_commit(bar_l + (b & 1));
      }
      __syncwarp();
      if (b > 0) {
        if (!(ok = warp_wait(bar_r + ((b - 1) & 1), ((b - 1) >> 1) & 1, err))) break;
        tc_fence_after();
        gemm2(b - 1, sp);
      }
      sp = s;
      s = s + 1 == kSt ? 0 : s + 1;
    }
    if (ok && nb > 0) {
      ok = warp_wait(bar_r + ((nb - 1) & 1), ((nb - 1) >> 1) & 1, err);
      if (ok) {
        tc_fence_after();
        gemm2(nb - 1, sp);
      }
    }
    if (el) {
      if (!ok) atomicExch(err, 1);
      // drain every MMA this warp issued before TMEM is released
      mma_commit(bar_z);
    }
    __syncwarp();
    if (!warp_wait(bar_z, 0, err) && el) atomicExch(err, 1);
    __syncwarp();
  } else if (warp == kLoad) {
    const bool el = elect_one();
    int s = 0, use = 0;
    for (int b = 0; b < nb; ++b) {
      // the stage's previous block is done with once its GEMM2 has run
      if (use > 0 && !warp_wait(bar_f + s, (use - 1) & 1, err)) break;
      if (el) {
        unsigned char* d = sX + s * 2 * kHalf;
        mbar_expect_tx(bar_x + s, 2 * kHalf);
        tma_3d(d + kHalf, &tmXl, 0, (b0 + b) * RB, 0, bar_x + s);
        tma_3d(d, &tmXh, 0, (b0 + b) * RB, 0, bar_x + s);
      }
      __syncwarp();
      if (++s == kSt) s = 0, ++use;
    }
    // no load is in flight when the CTA ends, not even after a wait that gave up
    for (int i = 0; i < kSt; ++i) {
      const int n = i < s ? use + 1 : use;  // loads into stage i
      if (n > 0) warp_wait(bar_x + i, (n - 1) & 1, err);
    }
  } else {
    // ---- epilogue: lane = (column, value or tangent); warp part = 16 rows, DC values of d ----
    const int quarter = warp & 3, part = warp >> 2;
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const bool tan = lane >= 16;
    const int m = quarter * 16 + (lane & 15);
    const int64_t t = t0 + m;
    const bool in_t = t < T;
    const int d0 = part * DC;
    {  // column operands: [Bh | Bt] to TMEM, Bl to shared memory
      const DevParams& P = *Pg;
      const float* x0 = static_cast<const float*>(P.x0);
      const float* S = static_cast<const float*>(P.S[st->cur]);
      const int iter = st->iter;
      const float* src = nullptr;
      if (in_t) {
        if (mode == 0) src = tan ? nullptr : (iter == 0 || t == 0) ? x0 : S + (t - 1) * Dp;
        else if (mode == 1) src = static_cast<const float*>(P.lg[tan ? 2 : 1]) + t * Dp;
        else src = tan ? nullptr : S + t * Dp;
      }
      const bool probes = mode == 0 && tan && in_t;
      const TapeKey key(P.seed, P.block);
#pragma unroll
      for (int c = 0; c < DC; c += 16) {
        float v[16];
        if (probes) {
          const int d = d0 + c;
          const U4 pb = probe_bits(key, static_cast<uint32_t>(d >> 7),
                                   static_cast<uint32_t>(t + P.t_off), probe, iter);
          const uint32_t w = u4_word(pb, (d >> 5) & 3) >> (d & 31);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = d + i < P.D ? (((w >> i) & 1u) ? 1.f : -1.f) : 0.f;
        } else {
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (src && d0 + c + i < Dp) q = *reinterpret_cast<const float4*>(src + d0 + c + i);
            v[i] = q.x;
            v[i + 1] = q.y;
            v[i + 2] = q.z;
            v[i + 3] = q.w;
          }
        }
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const __half2 h = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
          const float2 f = __half22float2(h);
          hi[i] = *reinterpret_cast<const uint32_t*>(&h);
          lo[i] = half2_bits(v[2 * i] - f.x, v[2 * i + 1] - f.y);
        }
        tmem_st8(tB + lane_off + (d0 + c) / 2, hi);
        if (!tan) {
          const int kb = (d0 + c) >> 6, ch = ((d0 + c) & 63) >> 3;
          unsigned char* row = sBl + kb * kBox + m * 128;
          *reinterpret_cast<uint4*>(row + ((ch ^ (m & 7)) << 4)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          *reinterpret_cast<uint4*>(row + (((ch + 1) ^ (m & 7)) << 4)) = make_uint4(lo[4], lo[5], lo[6], lo[7]);
        }
      }
      tmem_wait_st();
      fence_async_smem();
      tc_fence_before();
      mbar_arrive(bar_b);
    }
    float gacc[DC];  // this lane's G over d0 .. d0 + DC - 1, the blocks' partial sums added here
#pragma unroll
    for (int i = 0; i < DC; ++i) gacc[i] = 0.f;
    // log-likelihood sum, compensated (Kahan) in FP32: ls the sum, lc the running error
    float ls = 0.f, lc = 0.f;
    bool ok = true;
    int drained = 0;
    auto add_g = [&]() {
      if (!(ok = warp_wait(bar_g, drained & 1, err))) return;
      ++drained;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < DC; c += 16) {
        float a[16];
        tmem_ld16(tG + lane_off + d0 + c, a);
#pragma unroll
        for (int i = 0; i < 16; ++i) gacc[c + i] += a[i];
      }
    };
    // labels (0 or 1) of the warp's 16 rows, one block ahead
    const float* yp = ylab + static_cast<int64_t>(b0) * RB + 16 * part + (lane & 15);
    float ynext = nb > 0 ? __ldg(yp) : 0.f;
    for (int b = 0; b < nb; ++b) {
      const uint32_t ybits = __ballot_sync(0xffffffffu, ynext != 0.f) >> (tan ? 8 : 0);
      yp += RB;
      if (b + 1 < nb) ynext = __ldg(yp);
      if (!(ok = warp_wait(bar_l + (b & 1), (b >> 1) & 1, err))) break;
      tc_fence_after();
      const uint32_t la = tL + 64 * (b & 1) + 16 * part + lane_off;
      float v[16];
      tmem_ld16(la, v);
      // rows of this lane: the value lane takes the first 8 of the warp's 16, the tangent
      // lane the last 8; each gets the other's logit or tangent of its rows.
      // Rows past N have X = 0: whatever R holds there adds nothing to G, and only the
      // log-likelihood leaves them out.
      const int nv = static_cast<int>(imin64(
          RB, N - (static_cast<int64_t>(b0 + b) * RB + 16 * part + (tan ? 8 : 0))));
      // With z = l for label 0 and -l for label 1: r = y - p = -+ sigmoid(z), and the
      // log-likelihood term is -softplus(z) = -max(z, 0) - log(1 + e), e = exp(-|l|).  The
      // block's 1 + e are multiplied (at most 2^8, each product rounded once) and take one log.
      float r[8], s[8], prod = 1.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float got = __shfl_xor_sync(0xffffffffu, tan ? v[j] : v[8 + j], 16);
        const float l = tan ? got : v[j], w = tan ? v[8 + j] : got;
        const uint32_t flip = (ybits << (31 - j)) & 0x80000000u;
        const float z = __uint_as_float(__float_as_uint(l) ^ flip);
        const float e = __expf(-fabsf(l));
        const float inv = rcp_approx(1.f + e);
        const float q = e * inv;  // sigmoid(-|l|)
        const float p = z >= 0.f ? inv : q;
        r[j] = __uint_as_float(__float_as_uint(p) ^ flip ^ 0x80000000u);
        s[j] = q * inv * w;
        if (j < nv) {
          prod *= 1.f + e;
          const float y = -fmaxf(z, 0.f) - lc;
          const float sum = ls + y;
          lc = (sum - ls) - y;
          ls = sum;
        }
      }
      {
        const float y = -__logf(prod) - lc;
        const float sum = ls + y;
        lc = (sum - ls) - y;
        ls = sum;
      }
      if (has_g) {
        // R as FP16: r split hi + lo, s one term.  The value lane keeps r of all 16 rows,
        // the tangent lane s; 8 words of hi (or s) and 8 of lo (or zero), in place of L
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float h0 = split_hi(r[2 * i]), h1 = split_hi(r[2 * i + 1]);
          const uint32_t wh = half2_bits(h0, h1);
          const uint32_t wl = half2_bits(r[2 * i] - h0, r[2 * i + 1] - h1);
          const uint32_t ws = half2_bits(s[2 * i], s[2 * i + 1]);
          const uint32_t got = __shfl_xor_sync(0xffffffffu, tan ? wh : ws, 16);
          const uint32_t gotl = __shfl_xor_sync(0xffffffffu, wl, 16);
          hi[i] = tan ? got : wh;
          hi[4 + i] = tan ? ws : got;
          lo[i] = tan ? 0u : wl;
          lo[4 + i] = tan ? 0u : gotl;
        }
        tmem_st8(la, hi);
        tmem_st8(la + 8, lo);
        // the previous two blocks' G, complete while this block's GEMM1 ran; the next
        // GEMM2 starts it afresh after bar_r
        if (b >= 2 && !(b & 1)) add_g();
        tmem_wait_st();
        if (!ok) break;
      }
      tc_fence_before();
      mbar_arrive(bar_r + (b & 1));
    }
    if (ok && has_g && nb > 0) add_g();  // the last blocks
    if (ok && has_g && in_t) {
      float* g = G + (static_cast<int64_t>(split) * 2 * T + (tan ? T : 0) + t) * Dp + d0;
#pragma unroll
      for (int c = 0; c < DC; c += 4)
        if (d0 + c < Dp)
          *reinterpret_cast<float4*>(g + c) = make_float4(gacc[c], gacc[c + 1], gacc[c + 2], gacc[c + 3]);
    }
    if (!ok) atomicExch(err, 1);
    // log-likelihood of a column: 2 lanes x 4 warps, summed in FP64 in a fixed order.  Bl was
    // last read by the last block's GEMM1, complete before its L.
    double* red = reinterpret_cast<double*>(sBl);
    const double sum = static_cast<double>(ls) - static_cast<double>(lc);
    red[(part * 2 + (tan ? 1 : 0)) * TB + m] = sum;
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpi) : "memory");
    if (threadIdx.x < TB && t0 + threadIdx.x < T) {
      double a = 0.0;
      for (int i = 0; i < 8; ++i) a += red[i * TB + threadIdx.x];
      lp[static_cast<int64_t>(split) * T + t0 + threadIdx.x] = a;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == kProd) tmem_dealloc(tmem, kTmemCols);
}

// Builds the FP16 split operands of one pass: Bh/Bl (value columns hi / lo)
// and Bt (tangent columns), each T x Dk (t-major rows, d contiguous).
//   mode 0: value x_bar_t, tangent z_t (probe `probe`); mode 1: value y_t, tangent w_t;
//   mode 2: value S_t, no tangent.
template <typename Real>
__global__ void tc_prep_kernel(const DevParams* __restrict__ Pg, const DevState* __restrict__ st,
                               int mode, int probe, int64_t Dk, __half* __restrict__ Bh,
                               __half* __restrict__ Bl, __half* __restrict__ Bt) {
  const DevParams& P = *Pg;
  const int iter = st->iter;
  const bool from_x0 = iter == 0;
  const Real* S = static_cast<const Real*>(P.S[st->cur]);
  const Real* x0 = static_cast<const Real*>(P.x0);
  const TapeKey key(P.seed, P.block);
  const int64_t n = P.T * Dk;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t t = i / Dk, d = i % Dk;
    float v = 0.f, tv = 0.f;
    if (d < P.D) {
      if (mode == 0) {
        v = static_cast<float>((from_x0 || t == 0) ? x0[d] : S[(t - 1) * P.Dp + d]);
        const U4 pb = probe_bits(key, static_cast<uint32_t>(d >> 7),
                                 static_cast<uint32_t>(t + P.t_off),
                                 probe, iter);
        tv = ((u4_word(pb, static_cast<int>((d >> 5) & 3)) >> (d & 31)) & 1u) ? 1.f : -1.f;
      } else if (mode == 1) {
        v = static_cast<float>(static_cast<const Real*>(P.lg[1])[t * P.Dp + d]);
        tv = static_cast<float>(static_cast<const Real*>(P.lg[2])[t * P.Dp + d]);
      } else {
        v = static_cast<float>(S[t * P.Dp + d]);
      }
    }
    const __half h = __float2half_rn(v);
    Bh[i] = h;
    Bl[i] = __float2half_rn(v - __half2float(h));
    if (mode != 2) Bt[i] = __float2half_rn(tv);
  }
}

// ---------------------------------------------------------------------------
// Wide variant, 256 < D <= 512 (Dk = 512): 16 value columns a CTA (plus 16
// tangent columns) so that B (48 KB) and R fit beside a ring of four X boxes
// (128 KB).  The eight 64-wide d boxes of a row block pass through the ring:
// GEMM1 runs over boxes 0-3, then 4-7 as each slot frees; GEMM2 takes the d
// quarters 2 and 3 from the resident boxes 4-7, then the quarters 0 and 1
// from boxes 0-3 loaded again.  Per 128-row block this is the FLOPs of the
// D <= 256 kernel (half the columns, twice the depth) with 12 box loads
// instead of 8.  Each slot sees three loads and three releases a block, so
// its two mbarriers stay one phase per use.
// ---------------------------------------------------------------------------
constexpr int BTW = 16;          // value columns per CTA (plus BTW tangent columns)
constexpr int kSlots = 4;        // X boxes resident at a time
constexpr int kNkbW = 8;         // 64-wide d boxes of Dk = 512
constexpr uint32_t kBoxBW = 3 * BTW * 128;  // value hi | tangent | value lo rows of a d box

struct LayoutW {
  uint32_t xh, xl, b, r, bars, total;
};

__host__ __device__ inline LayoutW layout_wide() {
  LayoutW L;
  uint32_t off = 0;
  L.xh = off;
  off += kSlots * kBoxX;
  L.xl = off;
  off += kSlots * kBoxX;
  L.b = off;
  off += kNkbW * kBoxBW;
  L.r = off;
  off += kRAtom;  // one 64-column atom: [r hi 16 | s 16 | r lo 16 | unused 16]
  L.bars = off;
  off += 256;
  L.total = off + 1024;
  return L;
}

// 4 consecutive FP32 TMEM columns of this warp's 32 lanes, three times, then
// one wait in the same asm statement.
__device__ __forceinline__ void tmem_ld4x3(uint32_t ta, uint32_t tb, uint32_t tc, float (&a)[4],
                                           float (&b)[4], float (&c)[4]) {
  uint32_t r[12];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%12];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4, %5, %6, %7}, [%13];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8, %9, %10, %11}, [%14];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11])
      : "r"(ta), "r"(tb), "r"(tc)
      : "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    a[i] = __uint_as_float(r[i]);
    b[i] = __uint_as_float(r[4 + i]);
    c[i] = __uint_as_float(r[8 + i]);
  }
}

// 16 consecutive FP32 TMEM columns of this warp's 32 lanes, twice, one wait.
__device__ __forceinline__ void tmem_ld16x2(uint32_t ta, uint32_t tb, float (&a)[16],
                                            float (&b)[16]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, "
      "%26, %27, %28, %29, %30, %31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(ta), "r"(tb)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    a[i] = __uint_as_float(r[i]);
    b[i] = __uint_as_float(r[16 + i]);
  }
}

__global__ void __launch_bounds__(kThreadsTC, 1)
    logistic_pass_tc_wide_kernel(const __grid_constant__ CUtensorMap tmXh,
                                 const __grid_constant__ CUtensorMap tmXl,
                                 const __grid_constant__ CUtensorMap tmBh,
                                 const __grid_constant__ CUtensorMap tmBl,
                                 const __grid_constant__ CUtensorMap tmBt,
                                 const float* __restrict__ ylab, int64_t N, int64_t T,
                                 int64_t Dp, float* __restrict__ G, double* __restrict__ lp,
                                 int has_tangent, int* __restrict__ err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const LayoutW Ly = layout_wide();
  unsigned char* sXh = base + Ly.xh;
  unsigned char* sXl = base + Ly.xl;
  unsigned char* sB = base + Ly.b;
  unsigned char* sR = base + Ly.r;
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + Ly.bars);
  uint64_t* bar_b = bars + 0;   // B loaded
  uint64_t* bar_x = bars + 1;   // [4] slot loaded
  uint64_t* bar_f = bars + 5;   // [4] the MMAs reading the slot are done
  uint64_t* bar_l = bars + 9;   // GEMM1 done (L ready; also GEMM2 of the block before: R free)
  uint64_t* bar_r = bars + 10;  // epilogue wrote R (32 kEpi arrivals)
  uint64_t* bar_g = bars + 11;  // GEMM2 of the block done (G final after the last block)
  uint64_t* bar_z = bars + 12;  // teardown drain
  __shared__ uint32_t s_tmem;
  constexpr int BH = BTW / kParts;  // 4 value columns a thread
  __shared__ double s_red[kEpi][BH];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t0 = static_cast<int64_t>(blockIdx.x) * BTW;
  const int nblocks = static_cast<int>((N + BN - 1) / BN);
  const bool has_g = has_tangent != 0;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 13; ++i) mbar_init(bars + i, i == 10 ? 32 * kEpi : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kProd) tmem_alloc(&s_tmem, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;
  // L: columns [0, 48) = value (hi*hi + lo*hi) | tangent | value hi*lo;
  // G quarter q: columns [64 (q + 1), 64 (q + 1) + 48), the same three parts.
  const uint32_t tL = tmem;
  auto tG = [&](int q) { return tmem + 64u * static_cast<uint32_t>(q + 1); };

  if (warp == kProd) {
    {
      bool ok = true;
      const bool el = elect_one();
      const uint64_t xh1 = sdesc(su32(sXh), 16, 1024, 2), xl1 = sdesc(su32(sXl), 16, 1024, 2);
      const uint64_t b1 = sdesc(su32(sB), 16, 1024, 2), r2 = sdesc(su32(sR), kRAtom, 1024, 2);
      const uint64_t xh2 = sdesc(su32(sXh), kBoxX, 1024, 2),
                     xl2 = sdesc(su32(sXl), kBoxX, 1024, 2);
      uint32_t xph = 0, fph = 0;  // phase bit of each slot's two barriers
      const uint32_t i1_all = idesc_f16(128, 3 * BTW, false, false);
      const uint32_t i1_v = idesc_f16(128, BTW, false, false);
      const uint32_t i2_all = idesc_f16(128, 3 * BTW, true, true);
      const uint32_t i2_v = idesc_f16(128, BTW, true, true);
      auto wait_x = [&](int s) {
        const bool r = mbar_wait(bar_x + s, (xph >> s) & 1u, err);
        xph ^= 1u << s;
        return r;
      };
      auto wait_f = [&](int s) {
        const bool r = mbar_wait(bar_f + s, (fph >> s) & 1u, err);
        fph ^= 1u << s;
        return r;
      };
      auto load_box = [&](int s, int box, int nb) {
        if (el) {
          mbar_expect_tx(bar_x + s, 2 * kBoxX);
          tma_2d(sXh + s * kBoxX, &tmXh, box * 64, nb * BN, bar_x + s);
          tma_2d(sXl + s * kBoxX, &tmXl, box * 64, nb * BN, bar_x + s);
        }
        __syncwarp();
      };
      // GEMM1 over the box in slot s: L += Xh [Bh | Bt | Bl] + Xl Bh
      auto gemm1 = [&](int s, int box) {
        if (el) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            const uint32_t ox = (s * kBoxX + ks * 32) >> 4, ob = (box * kBoxBW + ks * 32) >> 4;
            mma_f16(tL, xh1 + ox, b1 + ob, i1_all, (box | ks) != 0);
            mma_f16(tL, xl1 + ox, b1 + ob, i1_v, 1);
          }
        }
        __syncwarp();
      };
      // GEMM2 for d quarter q from the boxes in slots 2p, 2p + 1
      auto gemm2 = [&](int q, int p, int nb) {
        if (!has_g) return;
        if (el) {
#pragma unroll
          for (int kn = 0; kn < BN / 16; ++kn) {
            const uint32_t ox = (2 * p * kBoxX + kn * 2048) >> 4, orr = (kn * 2048) >> 4;
            // every row block starts G afresh (the epilogue adds the blocks up)
            mma_f16(tG(q), xh2 + ox, r2 + orr, i2_all, kn > 0 ? 1u : 0u);
            mma_f16(tG(q), xl2 + ox, r2 + orr, i2_v, 1);
          }
        }
        __syncwarp();
      };
      auto commit = [&](uint64_t* bar) {
        if (el) mma_commit(bar);
        __syncwarp();
      };
      if (el) {
        mbar_expect_tx(bar_b, kNkbW * kBoxBW);
        for (int kb = 0; kb < kNkbW; ++kb) {
          unsigned char* b = sB + kb * kBoxBW;
          tma_2d(b, &tmBh, kb * 64, static_cast<int>(t0), bar_b);
          tma_2d(b + BTW * 128, has_tangent ? &tmBt : &tmBh, kb * 64, static_cast<int>(t0), bar_b);
          tma_2d(b + 2 * BTW * 128, &tmBl, kb * 64, static_cast<int>(t0), bar_b);
        }
      }
      __syncwarp();
      ok = mbar_wait(bar_b, 0, err);
      if (ok)
        for (int s = 0; s < kSlots; ++s) load_box(s, s, 0);
      for (int nb = 0; nb < nblocks && ok; ++nb) {
        // GEMM1, boxes 0-3
        for (int s = 0; s < kSlots && ok; ++s) {
          if (!(ok = wait_x(s))) break;
          tc_fence_after();
          gemm1(s, s);
          commit(bar_f + s);
        }
        // boxes 4-7 into the slots as they free, then their GEMM1
        for (int s = 0; s < kSlots && ok; ++s) {
          if (!(ok = wait_f(s))) break;
          load_box(s, kSlots + s, nb);
        }
        for (int s = 0; s < kSlots && ok; ++s) {
          if (!(ok = wait_x(s))) break;
          tc_fence_after();
          gemm1(s, kSlots + s);
        }
        if (!ok) break;
        commit(bar_l);
        if (!(ok = mbar_wait(bar_r, nb & 1, err))) break;
        tc_fence_after();
        // GEMM2, quarters 2 and 3 from the resident boxes 4-7
        for (int p = 0; p < 2; ++p) {
          gemm2(2 + p, p, nb);
          commit(bar_f + 2 * p);
          commit(bar_f + 2 * p + 1);
        }
        // boxes 0-3 again, then quarters 0 and 1
        for (int s = 0; s < kSlots && ok; ++s) {
          if (!(ok = wait_f(s))) break;
          load_box(s, s, nb);
        }
        for (int p = 0; p < 2 && ok; ++p) {
          if (!(ok = wait_x(2 * p)) || !(ok = wait_x(2 * p + 1))) break;
          tc_fence_after();
          gemm2(p, p, nb);
          commit(bar_f + 2 * p);
          commit(bar_f + 2 * p + 1);
        }
        if (!ok) break;
        commit(bar_g);
        // the next block's boxes 0-3
        if (nb + 1 < nblocks)
          for (int s = 0; s < kSlots && ok; ++s) {
            if (!(ok = wait_f(s))) break;
            load_box(s, s, nb + 1);
          }
      }
      ok = __all_sync(0xffffffffu, ok);
      if (el) {
        if (!ok) atomicExch(err, 1);
        // drain every MMA this warp issued before TMEM is released
        mma_commit(bar_z);
      }
      __syncwarp();
      if (!mbar_wait(bar_z, 0, err) && el) atomicExch(err, 1);
    }
    __syncwarp();
  } else {
    // ---- epilogue: thread = TMEM lane = data row; warp part = 4 value columns ----
    const int quarter = warp & 3, part = warp >> 2;  // columns [4 part, 4 part + 4)
    const int row = quarter * 32 + lane;
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    float ls[BH], lc[BH];
#pragma unroll
    for (int t = 0; t < BH; ++t) ls[t] = lc[t] = 0.f;
    bool ok = true;
    float y_next = row < N ? __ldg(ylab + row) : 0.f;
    // part q owns d quarter q of G: the row blocks' partial sums of its value
    // (hi*lo added) and tangent columns, added in FP32 with round-to-nearest
    float gv[BTW], gt[BTW];
#pragma unroll
    for (int t = 0; t < BTW; ++t) gv[t] = gt[t] = 0.f;
    auto add_g = [&]() {
      float a[16], b[16], c[16], unused[16];
      tmem_ld16x2(tG(part) + lane_off, tG(part) + lane_off + 2 * BTW, a, b);
      tmem_ld16x2(tG(part) + lane_off + BTW, tG(part) + lane_off + BTW, c, unused);
#pragma unroll
      for (int t = 0; t < BTW; ++t) {
        gv[t] += a[t] + b[t];
        gt[t] += c[t];
      }
    };
    for (int nb = 0; nb < nblocks; ++nb) {
      const int64_t n = static_cast<int64_t>(nb) * BN + row;
      const bool valid = n < N;
      const float yn = y_next;
      if (n + BN < N) y_next = __ldg(ylab + n + BN);
      if (has_g && nb > 0) {
        // the previous block's G partials, final at its GEMM2's commit and kept
        // until this block's R arrives: added while this block's GEMM1 runs
        if (!(ok = mbar_wait(bar_g, (nb - 1) & 1, err))) break;
        tc_fence_after();
        add_g();
      }
      if (!(ok = mbar_wait(bar_l, nb & 1, err))) break;
      tc_fence_after();
      float v[BH], vl[BH], w[BH];
      tmem_ld4x3(tL + lane_off + BH * part, tL + lane_off + 2 * BTW + BH * part,
                 tL + lane_off + BTW + BH * part, v, vl, w);
      float r[BH], sv[BH];
#pragma unroll
      for (int t = 0; t < BH; ++t) {
        const float l = v[t] + vl[t];
        const float e = __expf(-fabsf(l));
        const float inv = __fdividef(1.f, 1.f + e);
        const float p = l >= 0.f ? inv : e * inv;
        r[t] = valid ? yn - p : 0.f;
        sv[t] = (valid && has_tangent) ? p * (1.f - p) * w[t] : 0.f;
        if (valid) {
          const float y = (yn * l - (fmaxf(l, 0.f) + log1p_unit(e))) - lc[t];
          const float sum = ls[t] + y;
          lc[t] = (sum - ls[t]) - y;
          ls[t] = sum;
        }
      }
      if (has_g) {
        uint32_t wh[2], wl[2], ws[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float h0 = split_hi(r[2 * q]), h1 = split_hi(r[2 * q + 1]);
          wh[q] = half2_bits(h0, h1);
          wl[q] = half2_bits(r[2 * q] - h0, r[2 * q + 1] - h1);
          ws[q] = half2_bits(sv[2 * q], sv[2 * q + 1]);
        }
        // 8-column chunks: r hi 0-1, s 2-3, r lo 4-5; this part's half chunk
        unsigned char* rrow = sR + row * 128 + (part & 1) * 8;
        const int sw = row & 7, c = part >> 1;
        *reinterpret_cast<uint2*>(rrow + ((c ^ sw) << 4)) = make_uint2(wh[0], wh[1]);
        *reinterpret_cast<uint2*>(rrow + (((2 + c) ^ sw) << 4)) = make_uint2(ws[0], ws[1]);
        *reinterpret_cast<uint2*>(rrow + (((4 + c) ^ sw) << 4)) = make_uint2(wl[0], wl[1]);
        fence_async_smem();
      }
      tc_fence_before();
      mbar_arrive(bar_r);
    }
    if (ok && has_g && mbar_wait(bar_g, (nblocks - 1) & 1, err)) {
      tc_fence_after();
      add_g();  // the last row block
      const int64_t d = 128 * part + row;
      if (d < Dp) {
#pragma unroll
        for (int t = 0; t < BTW; ++t)
          if (t0 + t < T) {
            G[(t0 + t) * Dp + d] = gv[t];
            G[(T + t0 + t) * Dp + d] = gt[t];
          }
      }
    } else if (!ok) {
      atomicExch(err, 1);
    }
#pragma unroll
    for (int t = 0; t < BH; ++t) {
      const double sum = warp_sum(static_cast<double>(ls[t]) - static_cast<double>(lc[t]));
      if (lane == 0) s_red[warp][t] = sum;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpi) : "memory");
    if (threadIdx.x < BTW && t0 + threadIdx.x < T) {
      const int t = threadIdx.x, hh = t / BH, tt = t % BH;
      double a = 0.0;
      for (int q = 0; q < 4; ++q) a += s_red[4 * hh + q][tt];
      lp[t0 + t] = a;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == kProd) tmem_dealloc(tmem, 512);
}

// lp[t] = the sum of the nsplit partial sums of column t, in order.
__global__ void lp_sum_kernel(const double* __restrict__ parts, int nsplit, int64_t T,
                              double* __restrict__ lp) {
  const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= T) return;
  double a = 0.0;
  for (int p = 0; p < nsplit; ++p) a += parts[static_cast<int64_t>(p) * T + t];
  lp[t] = a;
}

// Bound check of the mbarrier wait used by the tensor-core pass: one thread
// initialises a barrier that expects one arrival, nobody arrives, and the
// bounded wait on phase 0 gives up after kWaitCycles; err[0] = 1 then.
__global__ void mbar_bound_kernel(int* err) {
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_err;
  if (threadIdx.x == 0) {
    s_err = 0;
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) err[0] = mbar_wait(&bar, 0, &s_err) ? 0 : 1;
}

}  // namespace tc


// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 2-D FP16 tensor (rows x cols, row-major) with a 64 x box_rows box, 128-B swizzle.
static bool make_map(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols,
                     uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * 2};
  const cuuint32_t box[2] = {64, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box,
            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

// X (rows x cols FP16, row-major) as 64-column boxes one after another: one load takes
// box_rows rows of every box.
static bool make_map_x(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols,
                       uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[3] = {64, rows, cols / 64};
  const cuuint64_t strides[2] = {cols * 2, 128};
  const cuuint32_t box[3] = {64, box_rows, static_cast<cuuint32_t>(cols / 64)};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(ptr), dims, strides, box,
            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

bool lg_tc_supported(const LogisticDev& X) { return X.Xh != nullptr && encode_fn() != nullptr; }

// CTAs that share a 64-column tile's rows: the split with the fewest steps, counted in
// 64-row blocks a CTA (1.6 us each at D = 256) times waves of 148 CTAs, with about 4
// blocks' time of set-up a CTA and the traffic of the split sums (at 5 TB/s).
int lg_tc_split(const LogisticDev& X, int64_t T) {
  if (X.Dk == 512) return 1;
  const int64_t tiles = (T + tc::TB - 1) / tc::TB, nb = (X.N + tc::RB - 1) / tc::RB;
  int best = 1;
  double cost = 1e300;
  for (int s = 1; s <= 16 && s <= nb; ++s) {
    const double waves = static_cast<double>((tiles * s + 147) / 148);
    const double sums = s > 1 ? s * (T * X.Dp * 16.0 / 5e6) / 1.6 : 0.0;
    const double c = waves * (static_cast<double>((nb + s - 1) / s) + 4.0) + sums;
    if (c < cost) {
      cost = c;
      best = s;
    }
  }
  return best;
}

// error word | the wide variant's FP16 operands, or the split log-likelihood sums
size_t lg_tc_ws_bytes(const LogisticDev& X, int64_t T) {
  if (X.Dk == 512) return 1024 + 3 * static_cast<size_t>(T) * X.Dk * 2;
  return 1024 + 8 * static_cast<size_t>(T) * lg_tc_split(X, T);
}

int* lg_tc_err_word(void* ws) { return static_cast<int*>(ws); }

template <int NKB>
static int launch_pass(cudaStream_t s, const LogisticDev& X, const DevParams* dP,
                       const DevState* dS, double* lp, int mode, int64_t T, int* err, float* G,
                       int probe, int nsplit) {
  CUtensorMap mXh, mXl;
  if (!make_map_x(&mXh, X.Xh, X.Np, X.Dk, tc::RB) ||
      !make_map_x(&mXl, X.Xl, X.Np, X.Dk, tc::RB))
    return 3;
  const uint32_t smem = tc::pass_smem(NKB);
  if (raise_smem_limit(reinterpret_cast<const void*>(tc::logistic_pass_kernel<NKB>), smem) !=
      cudaSuccess)
    return 3;
  const int grid = static_cast<int>((T + tc::TB - 1) / tc::TB) * nsplit;
  tc::logistic_pass_kernel<NKB><<<grid, tc::kThreadsPass, smem, s>>>(
      mXh, mXl, dP, dS, mode, probe, X.y32, X.N, T, X.Dp, nsplit, G, lp, err);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

int lg_tc_pass(cudaStream_t s, const LogisticDev& X, const DevParams* dP, const DevState* dS,
               double* lp, int mode, int64_t T, void* ws, float* G, int probe) {
  const int64_t Dk = X.Dk;
  int* err = lg_tc_err_word(ws);
  unsigned char* buf = static_cast<unsigned char*>(ws) + 1024;
  if (Dk == 512) {  // 256 < D <= 512: the wide variant, 16 value columns a CTA
    __half* Bh = reinterpret_cast<__half*>(buf);
    __half* Bl = Bh + T * Dk;
    __half* Bt = Bl + T * Dk;
    const int g =
        static_cast<int>((T * Dk + 255) / 256 < 148 * 16 ? (T * Dk + 255) / 256 : 148 * 16);
    tc::tc_prep_kernel<float><<<g, 256, 0, s>>>(dP, dS, mode, probe, Dk, Bh, Bl, Bt);
    if (cudaGetLastError() != cudaSuccess) return 3;
    CUtensorMap mXh, mXl, wBh, wBl, wBt;
    if (!make_map(&mXh, X.Xh, X.Np, Dk, tc::BN) || !make_map(&mXl, X.Xl, X.Np, Dk, tc::BN) ||
        !make_map(&wBh, Bh, T, Dk, tc::BTW) || !make_map(&wBl, Bl, T, Dk, tc::BTW) ||
        !make_map(&wBt, Bt, T, Dk, tc::BTW))
      return 3;
    const uint32_t smem = tc::layout_wide().total;
    if (raise_smem_limit(reinterpret_cast<const void*>(tc::logistic_pass_tc_wide_kernel), smem) !=
        cudaSuccess)
      return 3;
    const int grid = static_cast<int>((T + tc::BTW - 1) / tc::BTW);
    tc::logistic_pass_tc_wide_kernel<<<grid, tc::kThreadsTC, smem, s>>>(
        mXh, mXl, wBh, wBl, wBt, X.y32, X.N, T, X.Dp, G, lp, mode != 2 ? 1 : 0, err);
    return cudaGetLastError() == cudaSuccess ? 0 : 3;
  }
  const int ns = lg_tc_split(X, T);
  double* lps = ns > 1 ? reinterpret_cast<double*>(buf) : lp;
  const int rc = Dk == 128
                     ? launch_pass<2>(s, X, dP, dS, lps, mode, T, err, G, probe, ns)
                     : launch_pass<4>(s, X, dP, dS, lps, mode, T, err, G, probe, ns);
  if (rc || ns == 1) return rc;
  const int g = static_cast<int>((T + 255) / 256);
  tc::lp_sum_kernel<<<g, 256, 0, s>>>(lps, ns, T, lp);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

cudaError_t lg_tc_mbar_bound(cudaStream_t s, int* err) {
  tc::mbar_bound_kernel<<<1, 32, 0, s>>>(err);
  return cudaGetLastError();
}

}  // namespace pmcmc
