// hw_noalloc.cu -- one RHS evaluation that allocates no device memory.
//
// Its scratch (the stage input, the RHS output and the intermediate
// fields of the RHS) lives in the file-scope array g_rhs_scratch below instead
// of per-context cudaMalloc'd buffers.  Every GPU that loads this library holds
// the array (1 MiB) until the process exits.  Host code cannot pass the array's
// name to a kernel: the name is a host-side stand-in, not a device address.  The
// device address is fetched once per device with cudaGetSymbolAddress (with that
// device current) on the first call and reused.
//
// Everything else the RHS reads or writes stays in the context: the tables, the
// member's breaking state (crest records, B, the breaking.dat log), which a
// breaking deck's RHS advances exactly as hw_rhs does, and the member's RHS
// counter.
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "hw_kernels.h"

namespace {

using namespace hwdev;

constexpr int kNoAllocMaxNx = 4096;   // largest grid the static scratch covers
constexpr int kSlots = 4 + kScratch;  // 2N stage input + 2N output + the fields, in N double2 units
static __device__ __align__(256) double2 g_rhs_scratch[size_t(kSlots) * kNoAllocMaxNx];

constexpr int kMaxDevices = 128;

// per-device set-up done by the first call on that device (the scratch array's
// device address), under a lock so that two host threads making their first call on
// one device at once do it once
struct DeviceScratch {
  bool ready = false;
  double2* ptr = nullptr;
};
DeviceScratch g_scratch_addr[kMaxDevices];
std::mutex g_setup_lock;

}  // namespace

int hw_noalloc_max_nx() { return kNoAllocMaxNx; }

// Launch the no-allocation RHS for member mi (grid N, slice M, cluster C) on stream s,
// with the member's device (dev) current.  The first call on a device looks up the
// scratch array's device address, once, under a lock.
bool hw_noalloc_rhs_launch(DevMember* mems, int mi, int N, int M, int C, double t, const double* y,
                           double* dy, cudaStream_t s, int dev, std::string& err) {
  if (N > kNoAllocMaxNx) {
    err = "hw_rhs_noalloc: Nx=" + std::to_string(N) + " exceeds the " + std::to_string(kNoAllocMaxNx) +
          "-point limit of its static scratch";
    return false;
  }
  if (dev < 0 || dev >= kMaxDevices) {
    err = "hw_rhs_noalloc: device ordinal " + std::to_string(dev) + " out of range";
    return false;
  }
  cudaError_t e = cudaSuccess;
  DeviceScratch& ds = g_scratch_addr[dev];
  {
    std::lock_guard<std::mutex> lk(g_setup_lock);
    if (!ds.ready) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_rhs_scratch);
      if (e != cudaSuccess) {
        err = std::string("hw_rhs_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e);
        return false;
      }
      ds.ptr = static_cast<double2*>(p);
      ds.ready = true;
    }
  }
  switch (M) {
    case 256: e = hw_rhs_256(mems, mi, C, t, y, dy, ds.ptr, s); break;
    case 512: e = hw_rhs_512(mems, mi, C, t, y, dy, ds.ptr, s); break;
    case 1024: e = hw_rhs_1024(mems, mi, C, t, y, dy, ds.ptr, s); break;
    case 2048: e = hw_rhs_2048(mems, mi, C, t, y, dy, ds.ptr, s); break;
    default: e = cudaErrorInvalidValue;
  }
  if (e != cudaSuccess) {
    err = std::string("hw_rhs_noalloc: launch: ") + cudaGetErrorString(e);
    return false;
  }
  return true;
}
