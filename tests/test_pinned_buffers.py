"""The pool of mapped pinned buffers (csrc/hw_pinned.hpp) against a stand-in for the
runtime's pinning calls, on the CPU: a buffer that waited through a device reset is pinned
again and is never memory that someone else pinned meanwhile, small buffers do not keep a
larger one out, a failing registration leaves nothing behind, and threads never share one."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#pragma once
#include <cstdlib>
#include <map>
#include <mutex>
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2,
                   cudaErrorHostMemoryAlreadyRegistered = 712, cudaErrorHostMemoryNotRegistered = 713 };
enum { cudaHostRegisterPortable = 1, cudaHostRegisterMapped = 2, cudaHostAllocPortable = 1, cudaHostAllocMapped = 2 };
struct Fake {
  std::mutex m;
  std::map<void*, int> pinned;   // 1: registered by the pool, 2: allocated, 3: another owner's
  void* hole = nullptr;          // address of an allocation that a reset freed
  int registered = 0, fail = 0;
};
inline Fake& fake() { static Fake f; return f; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaHostGetFlags(unsigned* f, void* p) {
  std::lock_guard<std::mutex> lk(fake().m);
  *f = 0;
  return fake().pinned.count(p) ? cudaSuccess : cudaErrorInvalidValue;
}
inline cudaError_t cudaHostRegister(void* p, size_t, unsigned) {
  std::lock_guard<std::mutex> lk(fake().m);
  if (fake().fail) return cudaErrorMemoryAllocation;
  if (fake().pinned.count(p)) return cudaErrorHostMemoryAlreadyRegistered;
  fake().pinned[p] = 1;
  ++fake().registered;
  return cudaSuccess;
}
inline cudaError_t cudaHostUnregister(void* p) {
  std::lock_guard<std::mutex> lk(fake().m);
  return fake().pinned.erase(p) ? cudaSuccess : cudaErrorHostMemoryNotRegistered;
}
inline cudaError_t cudaHostGetDevicePointer(void** d, void* p, unsigned) {
  std::lock_guard<std::mutex> lk(fake().m);
  *d = p;
  return fake().pinned.count(p) ? cudaSuccess : cudaErrorInvalidValue;
}
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::aligned_alloc(4096, (n + 4095) / 4096 * 4096);
  std::lock_guard<std::mutex> lk(fake().m);
  fake().pinned[*p] = 2;
  return cudaSuccess;
}
template <class T> cudaError_t cudaHostAlloc(T** p, size_t n, unsigned f) { return cudaHostAlloc((void**)p, n, f); }
inline cudaError_t cudaFreeHost(void* p) {
  std::lock_guard<std::mutex> lk(fake().m);
  if (!fake().pinned.erase(p)) return cudaErrorInvalidValue;
  std::free(p);
  return cudaSuccess;
}
// a device reset ends registrations and frees allocations; another owner then pins what
// stands at a freed address
inline void reset_and_repin() {
  std::lock_guard<std::mutex> lk(fake().m);
  std::map<void*, int> after;
  for (auto& e : fake().pinned) if (e.second != 1) after[e.first] = 3;
  fake().pinned = after;
}
"""

PROGRAM = r"""
#include "hw_pinned.hpp"
#include <cstdio>
#include <set>
#include <thread>
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
using Pool = hw::PinnedBuffers;

int main() {
  {   // handed on, at least as large as asked for, mapped
    Pool p;
    Pool::Block a, b;
    CHECK(p.take(2051, a) == cudaSuccess && a.n >= 2051 && a.dev == a.p);
    a.p[a.n - 1] = 1.0;
    p.give(a);
    CHECK(p.take(100, b) == cudaSuccess && b.p == a.p && fake().registered == 1);
    // through a reset: pinned again, and the pool's own
    p.give(b);
    reset_and_repin();
    Pool::Block c;
    CHECK(p.take(100, c) == cudaSuccess && fake().pinned.count(c.p) && fake().pinned[c.p] == 1);
    c.p[c.n - 1] = 2.0;
    // a reset while it is out
    reset_and_repin();
    p.give(c);
    CHECK(p.take(100, a) == cudaSuccess && fake().pinned[a.p] == 1);
    p.give(a);
  }
  {   // four small ones do not keep a large one out; the smallest that fits is taken
    Pool p;
    Pool::Block s[5], big, again;
    for (auto& b : s) CHECK(p.take(4096, b) == cudaSuccess);
    CHECK(p.take(4 * 32768 + 3, big) == cudaSuccess);
    for (auto& b : s) p.give(b);
    CHECK(!fake().pinned.count(s[4].p));   // the fifth small one was let go
    p.give(big);
    CHECK(p.take(4096, again) == cudaSuccess && again.n < big.n);
    CHECK(p.take(4 * 32768 + 3, again) == cudaSuccess && again.p == big.p);
  }
  {   // a registration that fails: the error, no block, and the next one works
    Pool p;
    Pool::Block a;
    fake().fail = 1;
    CHECK(p.take(100, a) == cudaErrorMemoryAllocation && !a.p);
    fake().fail = 0;
    CHECK(p.take(100, a) == cudaSuccess && a.p);
  }
  {   // threads
    Pool p;
    std::mutex m;
    std::set<double*> out;
    int shared = 0;
    std::vector<std::thread> ts;
    for (int t = 0; t < 8; ++t)
      ts.emplace_back([&, t] {
        for (int i = 0; i < 2000; ++i) {
          Pool::Block b;
          if (p.take(size_t(1000 * (1 + (t + i) % 7)), b) != cudaSuccess) { ++shared; return; }
          { std::lock_guard<std::mutex> lk(m); if (!out.insert(b.p).second) ++shared; }
          b.p[b.n - 1] = t;
          { std::lock_guard<std::mutex> lk(m); out.erase(b.p); }
          p.give(b);
        }
      });
    for (auto& t : ts) t.join();
    CHECK(shared == 0);
  }
  return 0;
}
"""


def test_pool(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(FAKE)
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(tmp_path), "-I",
                    os.path.join(ROOT, "hawassi_c_b200", "csrc"), "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")],
                   check=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
