// Allocation-free Laplacian inverse (ib_op_laplacian_inv_noalloc, include/ibgb300_ops.h).
//
// Some callers cannot call cudaMalloc in the loop that solves: programs whose device memory is
// owned by another allocator or memory pool (a Julia or Python host that hands this library
// only the arrays it already owns), and time-critical loops that must not pay for an
// allocation's implicit synchronisation of the whole device.  ib_op_laplacian_inv allocates a
// work buffer on its first and on its largest calls; this variant has it in a fixed array compiled into
// the library instead, and runs the same transform kernels as ib_op_laplacian_inv on the same
// handle.
//
// The array is a file-scope __device__ variable of kNoAllocMaxValues FP64 values (32 MiB).
// Every GPU that loads the library holds it until the process exits.  In host code its name
// only stands in for the symbol and is not a device address; every call looks up the device
// address (cudaGetSymbolAddress, with the handle's device current; the lookup does not
// synchronise) and passes that address to the kernels, so a re-created context cannot leave a
// stale address behind.  The first call on a device also loads the module there, so it should
// come before any stream capture.
//
// All calls share the one array and it keeps the last call's contents.  The solve overwrites
// every value it reads before reading it, so nothing needs clearing; but calls that overlap on
// the GPU (other streams, other threads, other handles on the same device) race on it.
#include "ib_common.cuh"
#include "ibgb300_ops.h"

#include <mutex>

namespace {

constexpr size_t kNoAllocMaxValues = (size_t)1 << 22;  // 4,194,304 doubles = 32 MiB

static __device__ __align__(256) double g_noalloc_work[kNoAllocMaxValues];

}  // namespace

extern "C" int ib_op_laplacian_inv_noalloc(ib_handle* h, int32_t batch, const double* b, double* x) {
  ib::LapView v;
  if (!ib_handle_lap_view(h, &v) || batch < 1 || !b || !x) return IB_ERR_INVALID;
  if ((size_t)batch * (size_t)v.g.nG > kNoAllocMaxValues)
    return ib_handle_fail(h, IB_ERR_INVALID,
                          "ib_op_laplacian_inv_noalloc: batch * (nx-1)*(ny-1) exceeds the 4194304-value work array");
  ib::DeviceGuard guard(v.device);
  cudaError_t e = guard.err;
  void* wp = nullptr;
  if (e == cudaSuccess) e = cudaGetSymbolAddress(&wp, g_noalloc_work);
  if (e != cudaSuccess) return ib_handle_fail(h, IB_ERR_CUDA, cudaGetErrorString(e));
  double* w = static_cast<double*>(wp);
  // x = F2D(mlap .* F2D(b)): x pass into the fixed work array, y pass out of it, x pass in place
  e = ib::fx_fwd<double>(v.g, v.ax, b, w, batch, nullptr, v.stream);
  if (e == cudaSuccess) e = ib::fx_ypass(v.g, v.ay, w, x, batch, v.mlap, 0, 0, v.stream);
  if (e == cudaSuccess) e = ib::fx_inv<double>(v.g, v.ax, x, x, batch, nullptr, v.stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(v.stream);
  if (e != cudaSuccess) return ib_handle_fail(h, IB_ERR_CUDA, cudaGetErrorString(e));
  return IB_OK;
}
