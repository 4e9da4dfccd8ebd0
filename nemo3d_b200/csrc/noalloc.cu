// tbgpu_hx_dot_noalloc: H*x with the fused dot product, allocating nothing.
//
// The regular entry points reduce the dot product through scratch that the
// context allocates with cudaMalloc the first time it is needed.  Some
// callers cannot have the library allocate at that point: applications that
// have handed the whole device memory to their own pool allocator (the
// Hamiltonian of a dot of tens of millions of atoms fills most of the HBM),
// and eigensolver loops that call H*x thousands of times and cannot accept
// the implicit device-wide synchronisation of cudaMalloc/cudaFree inside the
// loop.  This entry point
// takes the reduction scratch from a fixed array in this file instead.
//
// The scratch: kMaxBlocks (2048) block partials plus a completion counter,
// 16,640 bytes held on every device that loads the library, until the
// process exits.  The product needs one block per SM at most.  Sizes that were
// refused when it took one block per 24 atoms (10 orbitals with a Bloch vector
// set) or 48 (5 orbitals) and so more than 2048 of them, above 49,152 and
// 98,304 atoms, are refused still (TBGPU_E_ARG): the interface says so.
//
// The array is shared by every call and keeps the last call's contents; the
// counter is cleared before each launch.  Calls that overlap on the GPU (from
// different streams or host threads) race on it and must be serialised by
// the caller.  The first call on a device looks up the array's device address
// (cudaGetSymbolAddress, with that device current); that first call should
// come before any stream capture.
#include <mutex>

#include "launch.cuh"
#include "tbgpu_internal.cuh"

namespace tbgpu {
namespace {

constexpr int kMaxBlocks = 2048;
constexpr int kMaxDevices = 64;

// [0, kMaxBlocks): block partials; the next 8 bytes: the completion counter
static __device__ __align__(256) double g_noalloc_scratch[kMaxBlocks + 32];

// The counter is cleared by a kernel and not by a memset: the product behind it
// and the product before it then overlap it as they overlap each other
// (launch.cuh), where a memset waits and is waited for in full.  216 atoms,
// back to back: sp3s* with spin 8.7 against 12.0 us, sp3d5s* with spin 7.8
// against 10.3 (10.3 and 12.3 by the lane-gather and warp-staged kernels).
__global__ void k_clear(unsigned int *counter) {
  wait_for_previous();
  *counter = 0u;
}

std::mutex g_setup_mutex;
double *g_scratch_dev[kMaxDevices] = {nullptr};

// Device address of g_noalloc_scratch on the current device (looked up once).
int scratch_address(int device, double **out) {
  if (device < 0 || device >= kMaxDevices) return set_error(TBGPU_E_ARG);
  std::lock_guard<std::mutex> lock(g_setup_mutex);
  if (!g_scratch_dev[device]) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p)
      return set_error(TBGPU_E_CUDA);
    g_scratch_dev[device] = static_cast<double *>(p);
  }
  *out = g_scratch_dev[device];
  return TBGPU_OK;
}

}  // namespace
}  // namespace tbgpu

using namespace tbgpu;

extern "C" int tbgpu_hx_dot_noalloc(tbgpu_ctx *ctx, double shift, const double *x_dev,
                                    double *y_dev, double *dot_dev) {
  if (!ctx || !x_dev || !y_dev || !dot_dev || misaligned16(x_dev) || misaligned16(y_dev))
    return set_error(TBGPU_E_ARG);
  Ctx &c = *reinterpret_cast<Ctx *>(ctx);
  if (!c.built) return set_error(TBGPU_E_STATE);
  int cur = -1;
  if (cudaGetDevice(&cur) != cudaSuccess) return set_error(TBGPU_E_CUDA);
  if (cur != c.device) return set_error(TBGPU_E_ARG);  // the context's device must be current
  double *scratch = nullptr;
  int rc = scratch_address(c.device, &scratch);
  if (rc) return rc;
  unsigned int *counter = reinterpret_cast<unsigned int *>(scratch + kMaxBlocks);
  launch_overlapped(k_clear, 1, 1, 0, c.stream, counter);
  TB_CUDA(cudaGetLastError());
  return launch_spmv_scratch(c, x_dev, y_dev, shift, scratch, counter, kMaxBlocks, dot_dev,
                             c.stream);
}
