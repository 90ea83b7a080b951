// hw_pinned.hpp -- the mapped pinned buffers of the host calls, kept past their contexts.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <vector>

namespace hw {

// A new pinned buffer costs 0.15 to 2.6 ms, a context of 512 points without it 0.9, so
// contexts hand theirs on.  At most kKept buffers wait here, each of at most 4 x 32768 + 3
// doubles and the rest of a page; of more, the larger ones.
//
// The pages are this process's own, pinned by registration: a device reset ends the
// registration and leaves the memory, so a buffer that waited through one is registered
// again, and nobody else's memory can stand at its address meanwhile.
class PinnedBuffers {
 public:
  struct Block {
    double* p = nullptr;     // host address
    double* dev = nullptr;   // the device's address of it
    size_t n = 0;
  };
  cudaError_t take(size_t n, Block& out) {
    Block b;
    {
      std::lock_guard<std::mutex> lk(m_);
      size_t best = kept_.size();   // the smallest that is large enough
      for (size_t i = 0; i < kept_.size(); ++i)
        if (kept_[i].n >= n && (best == kept_.size() || kept_[i].n < kept_[best].n)) best = i;
      if (best < kept_.size()) {
        b = kept_[best];
        kept_.erase(kept_.begin() + long(best));
      }
    }
    const bool fresh = !b.p;
    if (fresh) {
      b.n = (std::max<size_t>(n, 4096) * sizeof(double) + kPage - 1) / kPage * kPage / sizeof(double);
      b.p = static_cast<double*>(std::aligned_alloc(kPage, b.n * sizeof(double)));
      if (!b.p) return cudaErrorMemoryAllocation;
    }
    unsigned flags = 0;
    cudaError_t e = fresh ? cudaErrorInvalidValue : cudaHostGetFlags(&flags, b.p);
    if (e != cudaSuccess) {
      if (!fresh) cudaGetLastError();
      e = cudaHostRegister(b.p, b.n * sizeof(double), cudaHostRegisterMapped | cudaHostRegisterPortable);
    }
    if (e == cudaSuccess) e = cudaHostGetDevicePointer(reinterpret_cast<void**>(&b.dev), b.p, 0);
    if (e != cudaSuccess) {
      cudaGetLastError();
      release(b);
      return e;
    }
    out = b;
    return cudaSuccess;
  }
  void give(Block b) {
    if (!b.p) return;
    {
      std::lock_guard<std::mutex> lk(m_);
      if (kept_.size() < kKept) {
        kept_.push_back(b);
        return;
      }
      auto least = std::min_element(kept_.begin(), kept_.end(), [](const Block& x, const Block& y) { return x.n < y.n; });
      if (least->n < b.n) std::swap(*least, b);
    }
    release(b);
  }

 private:
  static void release(const Block& b) {
    if (cudaHostUnregister(b.p) != cudaSuccess) cudaGetLastError();   // (a reset unregistered it)
    std::free(b.p);
  }
  static constexpr size_t kKept = 4, kPage = 4096;
  std::mutex m_;
  std::vector<Block> kept_;
};

}  // namespace hw
