// scan_noalloc.cu -- the diagonal affine scan for callers that cannot allocate
// device memory.
//
// Some callers may not call cudaMalloc once they are running: a process that
// reserved its whole device memory budget up front in its own pool (a Julia
// session whose CUDA.jl pool owns the device, a serving process with a fixed
// memory budget), or a latency-critical loop that cannot afford the implicit
// device synchronisation of an allocation.  pmcmc_affine_scan_diag_noalloc
// serves them: the caller passes device inputs and outputs, and the scan's
// scratch (the barrier's word, the chunks' maps and states) lives in the
// file-scope array below instead of a handle's workspace.  No cudaMalloc,
// cudaFree or allocating library routine is called.
//
// The array is kPmcmcNoallocScratchBytes (4 MiB) on every GPU that loads the
// library, held until the process exits.  It is shared by all calls on a
// device; each call clears the barrier's word and writes what else it reads
// there.  Calls that overlap on the GPU (different streams, or several host
// threads) race on the array and must be serialised by the caller.  The array's memory
// is taken when the module is loaded on a device, which under lazy loading is
// the first call there: callers that give every free byte to their own pool
// make one small call first.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "../../include/pmcmc_deer.h"
#include "deer_launch.h"

namespace {

constexpr size_t kPmcmcNoallocScratchBytes = size_t(4) << 20;
static_assert(kPmcmcNoallocScratchBytes == PMCMC_NOALLOC_SCRATCH_BYTES, "keep in step");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kPmcmcNoallocScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_setup_mu;
void* g_scratch_addr[kMaxDevices] = {};

// Device address of the scratch array for the current device, looked up once
// per device (the host-side symbol is not a device address).
int scratch_for_current_device(void** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    return PMCMC_ERR_CUDA;
  }
  std::lock_guard<std::mutex> lk(g_setup_mu);
  if (!g_scratch_addr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
      cudaGetLastError();
      return PMCMC_ERR_CUDA;
    }
    g_scratch_addr[dev] = p;
  }
  *out = g_scratch_addr[dev];
  return PMCMC_OK;
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

}  // namespace

extern "C" int pmcmc_affine_scan_diag_noalloc(int32_t dtype, int64_t D, int64_t T, const void* A,
                                              const void* B, const void* s0, void* S,
                                              void* stream) {
  if (dtype != PMCMC_F32 && dtype != PMCMC_F64) return PMCMC_ERR_ARGUMENT;
  if (D < 0 || T < 0) return PMCMC_ERR_DIMENSION;
  if (T == 0 || D == 0) return PMCMC_OK;
  if (!A || !B || !s0 || !S || S == A || S == B) return PMCMC_ERR_ARGUMENT;
  const bool f64 = dtype == PMCMC_F64;
  const size_t es = f64 ? 8 : 4;
  if (3 * es * static_cast<size_t>(D) > 200 * 1024) return PMCMC_ERR_UNSUPPORTED;
  const int TT = pmcmc::scan_tile_cols(D, T);
  const int64_t nt = (T + TT - 1) / TT;
  // the largest size served: three arrays of nt maps and 4 bytes a chunk
  const size_t need = align256(64 + 4 * static_cast<size_t>(nt)) + 3 * align256(es * nt * D);
  if (need > kPmcmcNoallocScratchBytes) return PMCMC_ERR_NOMEM;  // beyond the fixed maximum

  void* base = nullptr;
  const int rc = scratch_for_current_device(&base);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the barrier's word is the array's first, the error flag follows it; both are cleared, so
  // that a wait that gave up, or calls that overlapped, leave nothing to the next call
  int* err = static_cast<int*>(base) + 1;
  int flag = 0;
  if (cudaMemsetAsync(base, 0, pmcmc::kScanBarBytes, s) != cudaSuccess ||
      pmcmc::launch_affine_scan(s, f64, D, T, A, B, s0, S, base, err) != cudaSuccess ||
      cudaMemcpyAsync(&flag, err, sizeof flag, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess) {
    cudaGetLastError();
    return PMCMC_ERR_CUDA;
  }
  return flag ? PMCMC_ERR_TIMEOUT : PMCMC_OK;
}
