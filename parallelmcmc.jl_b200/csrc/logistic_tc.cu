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
// Roles: warps 0-15 run the epilogue (warps w, w+4, w+8, w+12 share TMEM lane
// quarter w % 4), warp 16 issues the MMAs and warp 17 the TMA loads (one elected
// lane each).
// Every mbarrier wait is bounded; on timeout the kernel records an error,
// drains its own MMAs and frees TMEM before returning.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "deer_device.cuh"
#include "deer_launch.h"
#include "f32x2.cuh"
#include "logistic.h"

namespace pmcmc {
namespace tc {

constexpr int kEpi = 16;                      // epilogue warps
constexpr int kProd = 16;                     // MMA and TMEM-owner warp
constexpr int kLoad = 17;                     // TMA warp
constexpr int kThreadsPass = 32 * 18;
constexpr uint32_t kTmemCols = 512;
constexpr long long kWaitCycles = 2000000000ll;  // ~1 s at B200 clocks

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
// Bounded wait for the completion of the phase with the given parity: gives up
// after about a second of SM clock (or at once when another CTA of the launch
// has already reported an error).
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity,
                                          const volatile int* err) {
  if (mbar_try(b, parity)) return true;
  const long long start = clock64();
  for (long long i = 0;; ++i) {
    if (mbar_try(b, parity)) return true;
    if ((i & 255) == 255 && (*err || clock64() - start > kWaitCycles)) return false;
  }
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
// widths take (M = 128: N = 96 in 56, N = 32 in 40).
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
// either).  FMAs only: no division, no special-function unit.  One value or, for half
// the instructions, two:
//   float log1p_unit(float e), F2 log1p_unit(F2 e)
template <typename V>
__device__ __forceinline__ V log1p_unit(V e) {
  V q = same<V>(-0.0032140363473445177f);
  q = fma_of(q, e, same<V>(0.019649166613817215f));
  q = fma_of(q, e, same<V>(-0.056435029953718185f));
  q = fma_of(q, e, same<V>(0.10533228516578674f));
  q = fma_of(q, e, same<V>(-0.1525145173072815f));
  q = fma_of(q, e, same<V>(0.19651491940021515f));
  q = fma_of(q, e, same<V>(-0.24947808682918549f));
  q = fma_of(q, e, same<V>(0.3332909941673279f));
  q = fma_of(q, e, same<V>(-0.4999985098838806f));
  q = fma_of(q, e, same<V>(1.0f));
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
// One CTA (D <= 256), or a cluster of two with half of d each (D <= 512), takes 64
// trajectory columns and a run of 64-row blocks of X.  The columns are the MMAs' A
// operand, resident for the whole run; X streams through shared memory once as the B
// operand of both GEMMs:
//   GEMM1  L (128 lanes x 64 rows)  = [Bh | Bt] Xl' + Bl Xh' + [Bh | Bt] Xh'
//   GEMM2  G (128 lanes x d)       += [Rh | S] Xl + [Rl | 0] Xh + [Rh | S] Xh
// Lanes: each 32-lane quarter q of TMEM holds value columns 16 q .. 16 q + 15 in
// its lower half and their tangent columns in its upper half (the lanes an M = 64
// MMA writes are the lower halves, so Bl needs no padding).  The small products
// come first, where the accumulator is still small.  TMEM: G in 64 NKB columns,
// two L buffers of 64, [Bh | Bt] in 32 NKB; R overwrites its L in place.
//
// The tensor cores do not wait for the epilogue: block b's GEMM1 and block b - 1's
// GEMM2 run while the epilogue turns L(b - 1) and L(b) into R.  Per block (NKB = 4)
// 48 products of 32 cycles and 12 of 128 = 3072 cycles, and 64 KB of X.
// A third of the products' lanes are padding (the lo
// products of the tangent lanes), which the layout pays for keeping X's traffic
// at one read for 64 columns.  The form with X as the A operand (32 columns a CTA,
// one 128 KB block of X, nothing overlapped) took 4.4 us for 128 rows of 32
// columns at first and 3.5 us with its MMAs issued back to back; this takes 2.15 us for
// 64 rows of 64 columns (3650 cycles, of which 3072 on the tensor pipe, at the 1.7 GHz
// the power cap leaves): a pass at N = 10000, D = 256, T = 65536 went from 4.99 and
// 4.12 ms to 2.34 ms, 574 TFLOP/s algorithmic (8 N D T); each row's log(1 + e) by itself in
// the epilogue adds 1.3 % to that (3 % with NKB = 2, whose MMAs hide less of it).  The TMEM
// datapath (A operand, accumulators, the epilogue's loads) is active 88 % of the cycles of a
// full wave.
//
// Two CTAs (CL = 2): each forms the logits' sum over its half of d.  Of a warp's 16
// rows each CTA finishes 8: it sends its part of the other 8 to the same warp of the
// peer, and R of its 8 once it has them (st.async into the peer's shared memory, one
// mbarrier a warp and kind).  The exchange makes the epilogue the longer side, about
// 4200 cycles a block.  16 columns a CTA with all of d (three quarters of X loaded
// twice) took 1.26 ms, then 0.91 ms, a pass at N = 5000, D = 400, T = 8192;
// this takes 0.39 ms.
//
// A CTA's G is the sum over its rows; `nsplit` CTAs share a tile's rows where the
// tiles alone leave SMs idle, and lg_mid adds their parts.
// ---------------------------------------------------------------------------
constexpr int TB = 64;                        // value columns a CTA
constexpr int RB = 64;                        // rows of X a block
constexpr uint32_t kBox = RB * 128;           // 64 rows (or columns) x 64 values of d, FP16
constexpr uint32_t kMail = 2 * 32 * 32;       // a warp's two messages, 32 bytes a lane
// Slots of X, half a block (Xl or Xh) each: as many as fit
__host__ __device__ constexpr int slots(int nkb, int cl) { return nkb == 2 ? 8 : cl == 2 ? 5 : 6; }
__host__ __device__ constexpr uint32_t pass_smem(int nkb, int cl) {
  // Bl | slots | mailboxes | barriers | alignment slack
  return (1 + slots(nkb, cl)) * nkb * kBox + (cl == 2 ? kMail * kEpi : 0) + 512 + 1024;
}

__device__ __forceinline__ void tma_3d(void* dst, const CUtensorMap* tm, int x, int y, int z,
                                       uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
      "%3, %4}], [%5];" ::"r"(su32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(su32(bar))
      : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::
                   : "memory");
}
// Messages between the warps of the same index in a cluster's two CTAs, in the
// receiver's shared memory: per block 8 logits (or tangents) a lane, then 4 words of R
// hi (or S) a lane and 4 of R lo a value lane.  A message's buffer is free when the next
// of its kind is sent: a warp sends block b + 1's logits after it has R of block b, which
// the peer sends after reading block b's logits; and the same for R.  Without R (mode 2)
// the blocks' logits take the two messages' places in turn.
struct Mail {
  unsigned char* box;  // [4][32] of 16 bytes
  uint64_t* bar;       // logits, R
  uint32_t to, to_bar;
  __device__ __forceinline__ Mail(unsigned char* b, uint64_t* m, int peer) : box(b), bar(m) {
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(su32(b)), "r"(peer));
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to_bar) : "r"(su32(m)), "r"(peer));
  }
  __device__ __forceinline__ void put(int v, int which, uint32_t a, uint32_t b, uint32_t c,
                                      uint32_t d) const {
    asm volatile(
        "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, "
        "[%5];" ::"r"(to + v * 512 + (threadIdx.x & 31) * 16),
        "r"(a), "r"(b), "r"(c), "r"(d), "r"(to_bar + 8 * which)
        : "memory");
  }
  __device__ __forceinline__ uint4 get(int v) const {
    return *reinterpret_cast<const uint4*>(box + v * 512 + (threadIdx.x & 31) * 16);
  }
  __device__ __forceinline__ bool wait(int which, uint32_t parity, uint32_t bytes,
                                       const volatile int* err) const {
    if ((threadIdx.x & 31) == 0) mbar_expect_tx(bar + which, bytes);
    bool done = false;
    const long long start = clock64();
    for (long long i = 0; !done; ++i) {
      uint32_t d;
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(d)
          : "r"(su32(bar + which)), "r"(parity)
          : "memory");
      done = d != 0;
      if ((i & 255) == 255 && (*err || clock64() - start > kWaitCycles)) break;
    }
    return __all_sync(0xffffffffu, done);
  }
  __device__ __forceinline__ void send_logits(int m, const float (&o)[8]) const {
    put(2 * m, m, __float_as_uint(o[0]), __float_as_uint(o[1]), __float_as_uint(o[2]),
        __float_as_uint(o[3]));
    put(2 * m + 1, m, __float_as_uint(o[4]), __float_as_uint(o[5]), __float_as_uint(o[6]),
        __float_as_uint(o[7]));
  }
  __device__ __forceinline__ bool recv_logits(int m, uint32_t parity, float (&in)[8],
                                              const volatile int* err) const {
    if (!wait(m, parity, 1024, err)) return false;
    const uint4 a = get(2 * m), b = get(2 * m + 1);
    in[0] = __uint_as_float(a.x), in[1] = __uint_as_float(a.y);
    in[2] = __uint_as_float(a.z), in[3] = __uint_as_float(a.w);
    in[4] = __uint_as_float(b.x), in[5] = __uint_as_float(b.y);
    in[6] = __uint_as_float(b.z), in[7] = __uint_as_float(b.w);
    return true;
  }
  __device__ __forceinline__ void send_r(const uint32_t (&hi)[8], const uint32_t (&lo)[8]) const {
    put(2, 1, hi[0], hi[1], hi[2], hi[3]);
    if ((threadIdx.x & 31) < 16) put(3, 1, lo[0], lo[1], lo[2], lo[3]);
  }
  __device__ __forceinline__ bool recv_r(uint32_t parity, uint32_t (&hi)[4], uint32_t (&lo)[4],
                                         const volatile int* err) const {
    if (!wait(1, parity, 768, err)) return false;
    const uint4 a = get(2);
    uint4 b = make_uint4(0, 0, 0, 0);
    if ((threadIdx.x & 31) < 16) b = get(3);
    hi[0] = a.x, hi[1] = a.y, hi[2] = a.z, hi[3] = a.w;
    lo[0] = b.x, lo[1] = b.y, lo[2] = b.z, lo[3] = b.w;
    return true;
  }
};
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
// then tangent block), lp: nsplit CL parts of T.
template <int NKB, int CL>
__global__ void __launch_bounds__(kThreadsPass, 1)
    logistic_pass_kernel(const __grid_constant__ CUtensorMap tmXh,
                         const __grid_constant__ CUtensorMap tmXl,
                         const DevParams* __restrict__ Pg, const DevState* __restrict__ st,
                         int mode, int probe, const float* __restrict__ ylab, int64_t N,
                         int64_t T, int64_t Dp, int nsplit, float* __restrict__ G,
                         double* __restrict__ lp, int guard, int* __restrict__ err) {
  if (guard && solve_ended(st, Pg->maxiter)) return;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  constexpr int kSl = slots(NKB, CL);
  constexpr uint32_t kHalf = NKB * kBox;  // Xh or Xl of a block: one slot
  constexpr int DC = 16 * NKB;            // values of d an epilogue warp owns
  unsigned char* sBl = base;
  unsigned char* sX = base + kHalf;
  unsigned char* sM = sX + kSl * kHalf;  // CL = 2: the warps' mailboxes
  uint64_t* bars = reinterpret_cast<uint64_t*>(sM + (CL == 2 ? kMail * kEpi : 0));
  uint64_t* bar_x = bars;       // [kSl] slot loaded
  uint64_t* bar_f = bars + 8;   // [kSl] the MMAs reading the slot are done
  uint64_t* bar_l = bars + 16;  // [2] L ready
  uint64_t* bar_r = bars + 18;  // [2] R written (and G drained, where it was due)
  uint64_t* bar_g = bars + 20;  // G of two blocks complete
  uint64_t* bar_b = bars + 21;  // column operands written
  uint64_t* bar_z = bars + 22;  // teardown drain
  uint64_t* bar_m = bars + 23;  // CL = 2: [2 kEpi] a warp's message of logits, of R
  __shared__ uint32_t s_tmem;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // a cluster of two CTAs shares tile and rows, each with half of d
  const int rank = CL == 2 ? static_cast<int>(blockIdx.x & 1u) : 0;
  const int unit = static_cast<int>(blockIdx.x) / CL;
  const int tile = unit / nsplit, split = unit % nsplit;
  const int64_t t0 = static_cast<int64_t>(tile) * TB;
  const int nb_all = static_cast<int>((N + RB - 1) / RB);
  const int b0 = static_cast<int>(static_cast<int64_t>(nb_all) * split / nsplit);
  const int nb = static_cast<int>(static_cast<int64_t>(nb_all) * (split + 1) / nsplit) - b0;
  const bool has_g = mode != 2;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 23 + (CL == 2 ? 2 * kEpi : 0); ++i)
      mbar_init(bars + i, i == 18 || i == 19 || i == 21 ? 32 * kEpi : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kProd) tmem_alloc(&s_tmem, kTmemCols);
  tc_fence_before();
  if constexpr (CL == 2) cluster_sync();  // the peer's barriers are set up before any message
  else __syncthreads();
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
    // GEMM2 of block b, its Xl in slot sl and its Xh in slot sh; G starts afresh every
    // second block
    auto gemm2 = [&](int b, int sl, int sh) {
      if (el) {
        const uint32_t a = tL + 64 * (b & 1);
        const uint64_t xl = x2 + ((sl * kHalf) >> 4), xh = x2 + ((sh * kHalf) >> 4);
        if (has_g) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            mma_f16_ts(tG, a + 16 * k, xl + ((k * 2048) >> 4), i2, ((b & 1) | k) != 0);
        }
        if (CL == 2) mma_commit(bar_f + sl);
        if (has_g) {
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_f16_ts(tG, a + 16 * k + 8, xh + ((k * 2048) >> 4), i2, 1);
#pragma unroll
          for (int k = 0; k < 4; ++k) mma_f16_ts(tG, a + 16 * k, xh + ((k * 2048) >> 4), i2, 1);
        }
        mma_commit(bar_f + sh);
        if (has_g && ((b & 1) || b == nb - 1)) mma_commit(bar_g);
      }
      __syncwarp();
    };
    ok = warp_wait(bar_b, 0, err);
    tc_fence_after();
    int sl = 0, sh = 1, pl = 0, ph = 0;  // slots of this block and of the one before
    uint32_t xph = 0;                    // phase bit of each slot
    auto wait_x = [&](int s) {
      const bool r = warp_wait(bar_x + s, (xph >> s) & 1u, err);
      xph ^= 1u << s;
      return r;
    };
    for (int b = 0; b < nb && ok; ++b) {
      const uint32_t d = tL + 64 * (b & 1);
      if (!(ok = wait_x(CL == 1 ? sh : sl))) break;
      tc_fence_after();
      if (el) {
        const uint64_t xl = x1 + ((sl * kHalf) >> 4);
#pragma unroll
        for (int k = 0; k < 4 * NKB; ++k)
          mma_f16_ts(d, tB + 8 * k, xl + ((k / 4 * kBox + k % 4 * 32) >> 4), i1, k != 0);
      }
      if constexpr (CL == 2) {
        __syncwarp();
        if (!(ok = wait_x(sh))) break;
      }
      if (el) {
        const uint64_t xh = x1 + ((sh * kHalf) >> 4);
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
        gemm2(b - 1, pl, ph);
      }
      pl = sl, ph = sh;
      sl = sl + 2 >= kSl ? sl + 2 - kSl : sl + 2;
      sh = sh + 2 >= kSl ? sh + 2 - kSl : sh + 2;
    }
    if (ok && nb > 0) {
      ok = warp_wait(bar_r + ((nb - 1) & 1), ((nb - 1) >> 1) & 1, err);
      if (ok) {
        tc_fence_after();
        gemm2(nb - 1, pl, ph);
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
    // Xl, Xh of block 0, of block 1, ...: one at a time into five slots, or both together
    // into two of an even number, on the barriers of Xh
    constexpr int kStep = CL == 1 ? 2 : 1;
    for (int i = 0; i < 2 * nb; i += kStep) {
      const int sb = s + kStep - 1;
      if (use > 0 && !warp_wait(bar_f + sb, (use - 1) & 1, err)) break;
      if (el) {
        mbar_expect_tx(bar_x + sb, kStep * kHalf);
        tma_3d(sX + s * kHalf, (CL == 2 && (i & 1)) ? &tmXh : &tmXl, 0, (b0 + i / 2) * RB,
               rank * NKB, bar_x + sb);
        if (CL == 1) tma_3d(sX + sb * kHalf, &tmXh, 0, (b0 + i / 2) * RB, 0, bar_x + sb);
      }
      __syncwarp();
      s += kStep;
      if (s == kSl) s = 0, ++use;
    }
    // no load is in flight when the CTA ends, not even after a wait that gave up
    for (int i = kStep - 1; i < kSl; i += kStep) {
      const int n = i < s ? use + 1 : use;  // loads into slot i
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
    const int d0 = part * DC;              // within the CTA's 64 NKB values of d
    const int dg = rank * 64 * NKB + d0;   // of all d
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
          const int d = dg + c;
          const U4 pb = probe_bits(key, static_cast<uint32_t>(d >> 7),
                                   static_cast<uint32_t>(t + P.t_off), probe, iter);
          const uint32_t w = u4_word(pb, (d >> 5) & 3) >> (d & 31);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = d + i < P.D ? (((w >> i) & 1u) ? 1.f : -1.f) : 0.f;
        } else {
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (src && dg + c + i < Dp) q = *reinterpret_cast<const float4*>(src + dg + c + i);
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
    // This lane's rows among the warp's 16: with one CTA the value lane takes the first 8
    // and the tangent lane the last 8; with two, each CTA takes 8 (both CTAs' partial
    // logits summed there) and each lane 4.
    constexpr int NE = CL == 2 ? 4 : 8;
    const int first = (CL == 2 ? 8 * rank : 0) + (tan ? NE : 0);
    [[maybe_unused]] Mail mail(sM + warp * kMail, bar_m + 2 * warp, rank ^ 1);
    // labels (0 or 1) of the warp's 16 rows, one block ahead
    const float* yp = ylab + static_cast<int64_t>(b0) * RB + 16 * part + (lane & 15);
    float ynext = nb > 0 ? __ldg(yp) : 0.f;
    for (int b = 0; b < nb; ++b) {
      const uint32_t ybits = __ballot_sync(0xffffffffu, ynext != 0.f) >> first;
      yp += RB;
      if (b + 1 < nb) ynext = __ldg(yp);
      if (!(ok = warp_wait(bar_l + (b & 1), (b >> 1) & 1, err))) break;
      tc_fence_after();
      const uint32_t la = tL + 64 * (b & 1) + 16 * part + lane_off;
      float v[16];
      tmem_ld16(la, v);
      if constexpr (CL == 2) {
        // the peer's rows go there, and its part of this CTA's rows comes here
        float o[8], in[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rank ? v[j] : v[8 + j];
        const int m = has_g ? 0 : b & 1;
        mail.send_logits(m, o);
        if (!(ok = mail.recv_logits(m, (has_g ? b : b >> 1) & 1, in, err))) break;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (rank ? v[8 + j] : v[j]) + in[j];
      }
      // each lane gets the other's logit or tangent of its rows
      // Rows past N have X = 0: whatever R holds there adds nothing to G, and only the
      // log-likelihood leaves them out.
      const int nv = static_cast<int>(imin64(
          RB, N - (static_cast<int64_t>(b0 + b) * RB + 16 * part + first)));
      // With z = l for label 0 and -l for label 1: r = y - p = -+ sigmoid(z), and the
      // log-likelihood term is -softplus(z) = -max(z, 0) - log(1 + e), e = exp(-|l|): each
      // row's log(1 + e) by itself, accurate relative to e.  (One log of the rows' product of
      // 1 + e, 4 instructions a row fewer, loses up to 6e-8 a row, more than all of log(1 + e)
      // where the rows are well separated.)
      float r[NE], s[NE];
#pragma unroll
      for (int j = 0; j < NE; j += 2) {
        float z[2], w[2], e[2], inv[2], q[2], lg[2];
        uint32_t flip[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float got = __shfl_xor_sync(0xffffffffu, tan ? v[j + i] : v[NE + j + i], 16);
          const float l = tan ? got : v[j + i];
          w[i] = tan ? v[NE + j + i] : got;
          flip[i] = (ybits << (31 - j - i)) & 0x80000000u;
          z[i] = __uint_as_float(__float_as_uint(l) ^ flip[i]);
          e[i] = __expf(-fabsf(l));
          inv[i] = rcp_approx(1.f + e[i]);
        }
        const F2 e2 = pack2(e[0], e[1]), inv2 = pack2(inv[0], inv[1]), q2 = e2 * inv2;
        unpack2(q2, q[0], q[1]);  // sigmoid(-|l|)
        unpack2(q2 * inv2 * pack2(w[0], w[1]), s[j], s[j + 1]);
        unpack2(log1p_unit(e2), lg[0], lg[1]);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float p = z[i] >= 0.f ? inv[i] : q[i];
          r[j + i] = __uint_as_float(__float_as_uint(p) ^ flip[i] ^ 0x80000000u);
          if (j + i < nv) {
            const float y = -(fmaxf(z[i], 0.f) + lg[i]) - lc;
            const float sum = ls + y;
            lc = (sum - ls) - y;
            ls = sum;
          }
        }
      }
      if (has_g) {
        // R as FP16: r split hi + lo, s one term.  The value lane keeps r of all 16 rows,
        // the tangent lane s; 8 words of hi (or s) and 8 of lo (or zero), in place of L
        constexpr int NW = NE / 2;
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < NW; ++i) {
          const float h0 = split_hi(r[2 * i]), h1 = split_hi(r[2 * i + 1]);
          const uint32_t wh = half2_bits(h0, h1);
          const uint32_t wl = half2_bits(r[2 * i] - h0, r[2 * i + 1] - h1);
          const uint32_t ws = half2_bits(s[2 * i], s[2 * i + 1]);
          const uint32_t got = __shfl_xor_sync(0xffffffffu, tan ? wh : ws, 16);
          const uint32_t gotl = __shfl_xor_sync(0xffffffffu, wl, 16);
          hi[i] = tan ? got : wh;
          hi[NW + i] = tan ? ws : got;
          lo[i] = tan ? 0u : wl;
          lo[NW + i] = tan ? 0u : gotl;
        }
        if constexpr (CL == 2) {  // 4 words of each here; the other 4 from the peer
          uint32_t ph[4], pl[4];
          mail.send_r(hi, lo);
          if (!(ok = mail.recv_r(b & 1, ph, pl, err))) break;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t h = hi[i], l = lo[i];
            hi[i] = rank ? ph[i] : h;
            hi[4 + i] = rank ? h : ph[i];
            lo[i] = rank ? pl[i] : l;
            lo[4 + i] = rank ? l : pl[i];
          }
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
      float* g = G + (static_cast<int64_t>(split) * 2 * T + (tan ? T : 0) + t) * Dp + dg;
#pragma unroll
      for (int c = 0; c < DC; c += 4)
        if (dg + c < Dp)
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
      lp[static_cast<int64_t>(split * CL + rank) * T + t0 + threadIdx.x] = a;
    }
  }
  tc_fence_before();
  if constexpr (CL == 2) cluster_sync();  // the peer's messages to this CTA have arrived
  else __syncthreads();
  tc_fence_after();
  if (warp == kProd) tmem_dealloc(tmem, kTmemCols);
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

// The same for Mail::wait: a warp waits for a message that its peer never sends.
__global__ void mail_bound_kernel(int* err) {
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ __align__(16) unsigned char box[kMail];
  __shared__ int s_err;
  if (threadIdx.x == 0) {
    s_err = 0;
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const Mail mail(box, bar, 0);
  const bool got = mail.wait(0, 0, 1024, &s_err);
  if (threadIdx.x == 0) err[0] = got ? 0 : 1;
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

// X (rows x cols FP16, row-major) as 64-column boxes one after another: one load takes
// box_rows rows of `boxes` of them.
static bool make_map_x(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols,
                       uint32_t box_rows, uint32_t boxes) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[3] = {64, rows, cols / 64};
  const cuuint64_t strides[2] = {cols * 2, 128};
  const cuuint32_t box[3] = {64, box_rows, boxes};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(ptr), dims, strides, box,
            estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
         CUDA_SUCCESS;
}

bool lg_tc_supported(const LogisticDev& X) { return X.Xh != nullptr && encode_fn() != nullptr; }

// CTAs (pairs of CTAs for D > 256) that share a 64-column tile's rows: the split with
// the fewest steps, counted in 64-row blocks a CTA (1.6 us each at D = 256) times waves
// of a CTA an SM (a pair two), with about 4 blocks' time of set-up a CTA and the traffic of
// the split sums (at 5 TB/s).
int lg_tc_split(const LogisticDev& X, int64_t T) {
  const int64_t tiles = (T + tc::TB - 1) / tc::TB, nb = (X.N + tc::RB - 1) / tc::RB;
  const int64_t slots = X.Dk == 512 ? X.num_sms / 2 : X.num_sms;
  int best = 1;
  double cost = 1e300;
  for (int s = 1; s <= 16 && s <= nb; ++s) {
    const double waves = static_cast<double>((tiles * s + slots - 1) / slots);
    const double sums = s > 1 ? s * (T * X.Dp * 16.0 / 5e6) / 1.6 : 0.0;
    const double c = waves * (static_cast<double>((nb + s - 1) / s) + 4.0) + sums;
    if (c < cost) {
      cost = c;
      best = s;
    }
  }
  return best;
}

// error word | the log-likelihood sums of the parts
size_t lg_tc_ws_bytes(const LogisticDev& X, int64_t T) {
  return 1024 + 16 * static_cast<size_t>(T) * lg_tc_split(X, T);
}

int* lg_tc_err_word(void* ws) { return static_cast<int*>(ws); }

template <int NKB, int CL>
static int launch_pass(cudaStream_t s, const LogisticDev& X, const DevParams* dP,
                       const DevState* dS, double* lp, int mode, int64_t T, int* err, float* G,
                       int probe, int nsplit, bool guard) {
  CUtensorMap mXh, mXl;
  if (!make_map_x(&mXh, X.Xh, X.Np, X.Dk, tc::RB, NKB) ||
      !make_map_x(&mXl, X.Xl, X.Np, X.Dk, tc::RB, NKB))
    return 3;
  const auto fn = tc::logistic_pass_kernel<NKB, CL>;
  const uint32_t smem = tc::pass_smem(NKB, CL);
  if (raise_smem_limit(reinterpret_cast<const void*>(fn), smem) != cudaSuccess) return 3;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>((T + tc::TB - 1) / tc::TB) * nsplit * CL);
  cfg.blockDim = dim3(tc::kThreadsPass);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = CL;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, mXh, mXl, dP, dS, mode, probe,
                            static_cast<const float*>(X.y32), X.N, T, X.Dp, nsplit, G, lp,
                            guard ? 1 : 0, err) == cudaSuccess
             ? 0
             : 3;
}

int lg_tc_lp_count(const LogisticDev& X, int64_t T) {
  return lg_tc_split(X, T) * (X.Dk == 512 ? 2 : 1);
}
static double* lp_parts(void* ws) {
  return reinterpret_cast<double*>(static_cast<unsigned char*>(ws) + 1024);
}
const double* lg_tc_lp_parts(void* ws) { return lp_parts(ws); }

int lg_tc_pass(cudaStream_t s, const LogisticDev& X, const DevParams* dP, const DevState* dS,
               double* lp, int mode, int64_t T, void* ws, float* G, int probe, bool guard) {
  int* err = lg_tc_err_word(ws);
  const int ns = lg_tc_split(X, T), np = lg_tc_lp_count(X, T);
  double* lps = lp && np == 1 ? lp : lp_parts(ws);
  const int rc =
      X.Dk == 128   ? launch_pass<2, 1>(s, X, dP, dS, lps, mode, T, err, G, probe, ns, guard)
      : X.Dk == 256 ? launch_pass<4, 1>(s, X, dP, dS, lps, mode, T, err, G, probe, ns, guard)
                    : launch_pass<4, 2>(s, X, dP, dS, lps, mode, T, err, G, probe, ns, guard);
  if (rc || !lp || np == 1) return rc;
  const int g = static_cast<int>((T + 255) / 256);
  tc::lp_sum_kernel<<<g, 256, 0, s>>>(lps, np, T, lp);
  return cudaGetLastError() == cudaSuccess ? 0 : 3;
}

cudaError_t lg_tc_mbar_bound(cudaStream_t s, int* err) {
  tc::mbar_bound_kernel<<<1, 32, 0, s>>>(err);
  return cudaGetLastError();
}

cudaError_t lg_tc_mail_bound(cudaStream_t s, int* err) {
  tc::mail_bound_kernel<<<1, 32, 0, s>>>(err);
  return cudaGetLastError();
}

}  // namespace pmcmc
