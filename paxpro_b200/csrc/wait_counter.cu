// wait_counter.cu -- the per-device count of kernel waits that ran out.
//
// The propagation kernels give up a bounded wait for their asynchronous
// copies instead of hanging, and count it.  The count is a word of mapped host
// memory: the kernels reach it through the pointer in their parameters (they
// write it only when a wait runs out), and the host reads it after any
// synchronisation without a copy of its own.  (Three counters in device memory
// cost three copies, each with its own synchronisation, at every result read:
// some 55 of the 70 us of a 2048-point pxp_get_saved.)
#include <cuda_runtime.h>

#include <mutex>

#include "pxp_kernels.h"

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_mutex;
unsigned *g_host[kMaxDevices] = {}, *g_dev[kMaxDevices] = {};
}  // namespace

// Allocated the first time a device is asked for and kept until the process
// exits; null when that failed.
unsigned *pxp::wait_counter(int device, unsigned **dev) {
  std::lock_guard<std::mutex> lk(g_mutex);
  if (device < 0 || device >= kMaxDevices) return nullptr;
  if (g_host[device] == nullptr) {
    void *h = nullptr, *d = nullptr;
    if (cudaHostAlloc(&h, sizeof(unsigned), cudaHostAllocMapped | cudaHostAllocPortable) !=
            cudaSuccess ||
        cudaHostGetDevicePointer(&d, h, 0) != cudaSuccess) {
      cudaGetLastError();
      if (h) cudaFreeHost(h);
      return nullptr;
    }
    *(unsigned *)h = 0;
    g_host[device] = (unsigned *)h;
    g_dev[device] = (unsigned *)d;
  }
  if (dev) *dev = g_dev[device];
  return g_host[device];
}
