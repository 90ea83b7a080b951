// hw2d_engine.cu -- C ABI of the 2D engine: tables upload, the
// RHS entry points and the device-resident rkf45 loop.
//
// One step attempt is a fixed launch sequence captured once as a CUDA graph:
//   [RHS k1, if needed] [RHS stages 2..6] combine control [RHS k_out, if accepted] finalize
// Every kernel reads the device control block (t, h, h0, done, buffer indices)
// and does nothing once the target time is reached, so the host replays the
// graph in batches and reads the control block back between batches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/hawassi_b200.h"
#include "hw2d.cuh"
#include "hw2d_brk.cuh"
#include "hw2d_out.cuh"
#include "hw2d_var.cuh"
#include "hw2d_wall.cuh"
#include "hw_setup.hpp"

using hw2d::Ctl2;
using hw2d::RK2;
using hw2d::Tab2;
using hw2d::Work2;

namespace {

std::string g_err2d;

constexpr int kMinM = 64, kMaxM = 1024;
constexpr int kMaxRef2 = 16;   // reference depths
constexpr long long kMaxAttemptsPerRun = 2000000;

template <int M>
size_t smem_bytes(int slices) { return (size_t)slices * hwdev::padded(M) * sizeof(double2); }

// the slices of each pass
template <int M>
void set_attrs() {
  cudaFuncSetAttribute(hw2d::k2_rowA<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2_colB<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(6));
  cudaFuncSetAttribute(hw2d::k2_rowC<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(6));
  cudaFuncSetAttribute(hw2d::k2_colD<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2_rowE<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2_colH3<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2_rowI3<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(6));
  cudaFuncSetAttribute(hw2d::k2_colH1<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(4));
  cudaFuncSetAttribute(hw2d::k2_rowH1<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(4));
  cudaFuncSetAttribute(hw2d::k2v_row1<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2v_col2<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(6));
  cudaFuncSetAttribute(hw2d::k2v_row3<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(6));
  cudaFuncSetAttribute(hw2d::k2v_col4<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(6));
  cudaFuncSetAttribute(hw2d::k2v_row5<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(6));
  cudaFuncSetAttribute(hw2d::k2v_col6<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(6));
  cudaFuncSetAttribute(hw2d::k2v_row7<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(6));
  cudaFuncSetAttribute(hw2d::k2b_rowI<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2b_colI<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2b_sbcol<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2b_sbrow<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2w_row1<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2w_col2<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2w_row3<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2w_rowV1<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(4));
  cudaFuncSetAttribute(hw2d::k2w_colV2<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(4));
  cudaFuncSetAttribute(hw2d::k2w_rowV3<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(2));
  cudaFuncSetAttribute(hw2d::k2o_row<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(4));
  cudaFuncSetAttribute(hw2d::k2o_col<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes<M>(4));
}

// the output stage's two passes (row M = nx, column M = ny)
template <int M>
void launch_out(int which, int nblocks, cudaStream_t s, const Tab2& tb, const double2* z, double2* P, double* phys,
                float* f32) {
  const int blk = hw2d::kThr2;
  if (which == 0) hw2d::k2o_row<M><<<nblocks, blk, smem_bytes<M>(4), s>>>(tb, z, P);
  else hw2d::k2o_col<M><<<nblocks, blk, smem_bytes<M>(4), s>>>(tb, P, phys, f32);
}
void out_pass(int M, int which, int nb, cudaStream_t s, const Tab2& tb, const double2* z, double2* P, double* phys,
              float* f32) {
  switch (M) {
    case 64: launch_out<64>(which, nb, s, tb, z, P, phys, f32); break;
    case 128: launch_out<128>(which, nb, s, tb, z, P, phys, f32); break;
    case 256: launch_out<256>(which, nb, s, tb, z, P, phys, f32); break;
    case 512: launch_out<512>(which, nb, s, tb, z, P, phys, f32); break;
    default: launch_out<1024>(which, nb, s, tb, z, P, phys, f32); break;
  }
}

// the flat bottom's wall round trip (row M = nx, column M = ny)
template <int M>
void launch_wall(int which, int nblocks, cudaStream_t s, const Tab2& tb, const Work2& w, const Ctl2* ctl, int cond) {
  const int blk = hw2d::kThr2;
  if (which == 0) hw2d::k2w_row1<M><<<nblocks, blk, smem_bytes<M>(2), s>>>(tb, w, ctl, cond);
  else if (which == 1) hw2d::k2w_col2<M><<<nblocks, blk, smem_bytes<M>(2), s>>>(tb, w, ctl, cond);
  else if (which == 2) hw2d::k2w_row3<M><<<nblocks, blk, smem_bytes<M>(2), s>>>(tb, w, ctl, cond);
  else if (which == 3) hw2d::k2w_rowV1<M><<<nblocks, blk, smem_bytes<M>(4), s>>>(tb, w, ctl, cond);
  else if (which == 4) hw2d::k2w_colV2<M><<<nblocks, blk, smem_bytes<M>(4), s>>>(tb, w, ctl, cond);
  else hw2d::k2w_rowV3<M><<<nblocks, blk, smem_bytes<M>(2), s>>>(tb, w, ctl, cond);
}
void wall_pass(int M, int which, int nb, cudaStream_t s, const Tab2& tb, const Work2& w, const Ctl2* ctl, int cond) {
  switch (M) {
    case 64: launch_wall<64>(which, nb, s, tb, w, ctl, cond); break;
    case 128: launch_wall<128>(which, nb, s, tb, w, ctl, cond); break;
    case 256: launch_wall<256>(which, nb, s, tb, w, ctl, cond); break;
    case 512: launch_wall<512>(which, nb, s, tb, w, ctl, cond); break;
    default: launch_wall<1024>(which, nb, s, tb, w, ctl, cond); break;
  }
}

// the breaking kernels of one RHS (row passes: row length M = nx; column passes: M = ny)
template <int M>
void launch_brk_row(int which, int nblocks, cudaStream_t s, const Tab2& tb, const Work2& w, const hw2d::Brk2& b,
                    const RK2& rk, const Ctl2* ctl, int mode, int cond, double2* out) {
  const int blk = hw2d::kThr2;
  if (which == 0) hw2d::k2b_rowI<M><<<nblocks, blk, smem_bytes<M>(2), s>>>(tb, w, b, rk, ctl, mode, cond, out);
  else hw2d::k2b_sbrow<M><<<nblocks, blk, smem_bytes<M>(2), s>>>(tb, b, rk, ctl, mode, cond, out);
}
template <int M>
void launch_brk_col(int which, int nblocks, cudaStream_t s, const Tab2& tb, const Work2& w, const hw2d::Brk2& b,
                    const Ctl2* ctl, int mode, int cond) {
  const int blk = hw2d::kThr2;
  if (which == 0) hw2d::k2b_colI<M><<<nblocks, blk, smem_bytes<M>(2), s>>>(tb, b, ctl, mode, cond);
  else hw2d::k2b_sbcol<M><<<nblocks, blk, smem_bytes<M>(2), s>>>(tb, w, b, ctl, mode, cond);
}
void brk_row(int M, int which, int nb, cudaStream_t s, const Tab2& tb, const Work2& w, const hw2d::Brk2& b,
             const RK2& rk, const Ctl2* ctl, int mode, int cond, double2* out) {
  switch (M) {
    case 64: launch_brk_row<64>(which, nb, s, tb, w, b, rk, ctl, mode, cond, out); break;
    case 128: launch_brk_row<128>(which, nb, s, tb, w, b, rk, ctl, mode, cond, out); break;
    case 256: launch_brk_row<256>(which, nb, s, tb, w, b, rk, ctl, mode, cond, out); break;
    case 512: launch_brk_row<512>(which, nb, s, tb, w, b, rk, ctl, mode, cond, out); break;
    default: launch_brk_row<1024>(which, nb, s, tb, w, b, rk, ctl, mode, cond, out); break;
  }
}
void brk_col(int M, int which, int nb, cudaStream_t s, const Tab2& tb, const Work2& w, const hw2d::Brk2& b,
             const Ctl2* ctl, int mode, int cond) {
  switch (M) {
    case 64: launch_brk_col<64>(which, nb, s, tb, w, b, ctl, mode, cond); break;
    case 128: launch_brk_col<128>(which, nb, s, tb, w, b, ctl, mode, cond); break;
    case 256: launch_brk_col<256>(which, nb, s, tb, w, b, ctl, mode, cond); break;
    case 512: launch_brk_col<512>(which, nb, s, tb, w, b, ctl, mode, cond); break;
    default: launch_brk_col<1024>(which, nb, s, tb, w, b, ctl, mode, cond); break;
  }
}

// the passes of one RHS: rows (row length M = nx) and columns (M = ny)
enum RowPass { kRowA, kRowC, kRowE, kRowI3, kRowH1, kRowV1, kRowV3, kRowV5, kRowV7 };
enum ColPass { kColB, kColD, kColH3, kColH1, kColV2, kColV4, kColV6 };

struct PassArgs {
  cudaStream_t s;
  const Tab2& tb;
  const Work2& w;
  const RK2& rk;
  Ctl2* ctl;
  int mode, cond;
  double2* out;
};

template <int M>
void launch_row(RowPass which, int cubic, const PassArgs& a) {
  const Tab2& tb = a.tb;
  const int nb = tb.ny / 2;
  const int t2 = hw2d::kThr2, t4 = hw2d::kThr4;
  switch (which) {
    case kRowA:
      hw2d::k2_rowA<M><<<dim3(nb, tb.model == 3 ? 3 : 2), t2, smem_bytes<M>(2), a.s>>>(tb, a.w, a.ctl, a.ctl, a.mode, a.cond);
      break;
    case kRowC: hw2d::k2_rowC<M><<<nb, t4, smem_bytes<M>(6), a.s>>>(tb, a.w, a.ctl, a.cond); break;
    case kRowE: hw2d::k2_rowE<M><<<dim3(nb, 3), t2, smem_bytes<M>(2), a.s>>>(tb, a.w, a.rk, a.ctl, a.mode, a.cond, a.out); break;
    case kRowI3: hw2d::k2_rowI3<M><<<nb, t4, smem_bytes<M>(6), a.s>>>(tb, a.w, a.ctl, a.cond); break;
    case kRowH1: hw2d::k2_rowH1<M><<<nb, t4, smem_bytes<M>(4), a.s>>>(tb, a.w, a.rk, a.ctl, a.mode, a.cond, a.out); break;
    case kRowV1:
      hw2d::k2v_row1<M><<<dim3(nb, 2 + tb.nk), t2, smem_bytes<M>(2), a.s>>>(tb, a.w, a.ctl, a.ctl, a.mode, a.cond);
      break;
    case kRowV3: hw2d::k2v_row3<M><<<nb, t4, smem_bytes<M>(6), a.s>>>(tb, a.w, a.ctl, a.cond); break;
    case kRowV5: hw2d::k2v_row5<M><<<nb, t4, smem_bytes<M>(6), a.s>>>(tb, a.w, a.ctl, a.cond, cubic); break;
    case kRowV7: hw2d::k2v_row7<M><<<nb, t4, smem_bytes<M>(6), a.s>>>(tb, a.w, a.ctl, a.cond, cubic); break;
  }
}
template <int M>
void launch_col(ColPass which, int cubic, const PassArgs& a) {
  const Tab2& tb = a.tb;
  const int nb = tb.nx / 2;
  const int t2 = hw2d::kThr2, t4 = hw2d::kThr4;
  switch (which) {
    case kColB: hw2d::k2_colB<M><<<nb, t4, smem_bytes<M>(6), a.s>>>(tb, a.w, a.ctl, a.cond); break;
    case kColD: hw2d::k2_colD<M><<<dim3(nb, 3), t2, smem_bytes<M>(2), a.s>>>(tb, a.w, a.ctl, a.cond); break;
    case kColH3: hw2d::k2_colH3<M><<<nb, t2, smem_bytes<M>(2), a.s>>>(tb, a.w, a.ctl, a.cond); break;
    case kColH1: hw2d::k2_colH1<M><<<nb, t4, smem_bytes<M>(4), a.s>>>(tb, a.w, a.ctl, a.cond); break;
    case kColV2: hw2d::k2v_col2<M><<<nb, t4, smem_bytes<M>(6), a.s>>>(tb, a.w, a.ctl, a.cond); break;
    case kColV4: hw2d::k2v_col4<M><<<nb, t4, smem_bytes<M>(6), a.s>>>(tb, a.w, a.ctl, a.cond, cubic); break;
    case kColV6: hw2d::k2v_col6<M><<<nb, t4, smem_bytes<M>(6), a.s>>>(tb, a.w, a.ctl, a.cond); break;
  }
}
void row_pass(RowPass which, const PassArgs& a, int cubic = 0) {
  switch (a.tb.nx) {
    case 64: launch_row<64>(which, cubic, a); break;
    case 128: launch_row<128>(which, cubic, a); break;
    case 256: launch_row<256>(which, cubic, a); break;
    case 512: launch_row<512>(which, cubic, a); break;
    default: launch_row<1024>(which, cubic, a); break;
  }
}
void col_pass(ColPass which, const PassArgs& a, int cubic = 0) {
  switch (a.tb.ny) {
    case 64: launch_col<64>(which, cubic, a); break;
    case 128: launch_col<128>(which, cubic, a); break;
    case 256: launch_col<256>(which, cubic, a); break;
    case 512: launch_col<512>(which, cubic, a); break;
    default: launch_col<1024>(which, cubic, a); break;
  }
}

void set_all_attrs() {
  static bool done[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || done[dev]) return;
  set_attrs<64>(); set_attrs<128>(); set_attrs<256>(); set_attrs<512>(); set_attrs<1024>();
  cudaFuncSetAttribute(hw2d::k2b_sort, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)(hw2d::kBrkPeakCap * sizeof(int)));
  done[dev] = true;
}

std::vector<double2> twiddles(int n) {
  std::vector<double2> t(n);
  for (int q = 0; q < n; ++q) {
    const double a = 2.0 * M_PI * double(q) / double(n);
    t[q] = make_double2(std::cos(a), -std::sin(a));
  }
  return t;
}

bool pow2_in_range(int v) { return v >= kMinM && v <= kMaxM && (v & (v - 1)) == 0; }

}  // namespace

struct hw2d_ctx {
  int device = 0;
  int nx = 0, ny = 0;
  size_t n = 0;
  cudaStream_t own_stream = nullptr, stream = nullptr;
  Tab2 tb{};
  Work2 w{};
  RK2 rk{};
  Ctl2* ctl = nullptr;     // device
  Ctl2* hctl = nullptr;    // pinned host copy
  hw2d::Brk2 brk{};        // kinematic breaking (brk.on = 0: off)
  double* dref = nullptr;  // 6n staging for reference-layout transfers
  double* href = nullptr;  // the same on small grids, mapped and pinned, for hw2d_rhs (behind hctl)
  double2* dout = nullptr; // 3n direct RHS output
  std::vector<void*> allocs;
  cudaGraphExec_t attempt = nullptr;
  cudaStream_t graph_stream = nullptr;
  double h_first = 0.0;
  // output stage (allocated at first use)
  double2* oP = nullptr;    // 2n packed transforms
  double* ophys = nullptr;  // 3n eta, u, v
  float* of32 = nullptr;    // 3n float copies
  float* hf32 = nullptr;    // pinned host copy of of32
  int* ogpt = nullptr;      // gauge grid points
  double* ogval = nullptr;  // 3 values per gauge
  double* hgval = nullptr;  // pinned host copy of ogval
  int ogcap = 0;
  long long launches = 0;   // kernels issued (graph nodes counted one by one)
  int per_rhs = 5;
  std::string err;

  // Grids whose right-hand side moves through a mapped buffer: one call in copies and so,
  // 64x64 97 and 78 us, 128x64 121 and 97, 128x128 175 and 172, 256x128 270 and 312 (the
  // host's own copy into the buffer costs more than the driver's staging)
  static constexpr size_t kMappedPoints = 128 * 64;
  template <class T>
  T* dalloc(size_t count) {
    void* p = nullptr;
    if (cudaMalloc(&p, count * sizeof(T)) != cudaSuccess) return nullptr;
    allocs.push_back(p);
    return static_cast<T*>(p);
  }
  template <class T>
  T* upload(const std::vector<T>& v) {
    T* p = dalloc<T>(v.size());
    if (p && cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) return nullptr;
    return p;
  }
  // a failed runtime call: record it (with the call's own error) and return 1
  int fail(const char* what, cudaError_t e) {
    err = std::string(what) + ": " + cudaGetErrorString(e);
    cudaGetLastError();
    return 1;
  }
  bool check(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      err = std::string(what) + ": " + cudaGetErrorString(e);
      return false;
    }
    return true;
  }
  void rhs_launch(int mode, int cond, cudaStream_t s, double2* out) {
    const int rows = ny / 2, cols = nx / 2;
    if (mode != 0) hw2d::k2_stage<<<hw2d::kCombBlocks, 256, 0, s>>>(tb.aal, rk, w, ctl, mode, cond, n);
    per_rhs = 1;
    const PassArgs a{s, tb, w, rk, ctl, mode, cond, out};
    auto row = [&](RowPass p, int cubic = 0) { row_pass(p, a, cubic); ++per_rhs; };
    auto col = [&](ColPass p, int cubic = 0) { col_pass(p, a, cubic); ++per_rhs; };
    if (tb.var) {
      row(kRowV1);
      col(kColV2);
      row(kRowV3);
    } else {
      if (tb.wallchar) {
        const int base = tb.refl_one ? 3 : 0;
        wall_pass(nx, base + 0, rows, s, tb, w, ctl, cond);
        wall_pass(ny, base + 1, cols, s, tb, w, ctl, cond);
        wall_pass(nx, base + 2, rows, s, tb, w, ctl, cond);
        per_rhs += 3;
      }
      row(kRowA);
    }
    if (tb.model == 1) {
      col(kColH1);
      row(kRowH1);
      return;
    }
    if (tb.var) {
      for (int cubic = 0; cubic <= (tb.model == 3 ? 1 : 0); ++cubic) {
        col(kColV4, cubic);
        row(kRowV5, cubic);
        col(kColV6, cubic);
        row(kRowV7, cubic);
      }
    } else {
      col(kColB);
      row(kRowC);
      if (tb.model == 3) {
        col(kColH3);
        row(kRowI3);
      }
    }
    if (!tb.chi_one) col(kColD);
    row(kRowE);
    if (brk.on) brk_launch(mode, cond, s, out);
  }
  // the breaking kernels after the assembly pass (both bottoms)
  void brk_launch(int mode, int cond, cudaStream_t s, double2* out) {
    const int rows = ny / 2, cols = nx / 2;
    const int gb = (int)std::min<size_t>((n + 255) / 256, 4 * 148);
    brk_row(nx, 0, rows, s, tb, w, brk, rk, ctl, mode, cond, out);
    brk_col(ny, 0, cols, s, tb, w, brk, ctl, mode, cond);
    hw2d::k2b_peaks<<<gb, 256, 0, s>>>(tb, w, brk, ctl, mode, cond);
    hw2d::k2b_sort<<<1, hw2d::kBrkSortThreads, hw2d::kBrkPeakCap * sizeof(int), s>>>(brk, ctl, mode, cond);
    hw2d::k2b_machine<<<1, 32, 0, s>>>(tb, w, brk, ctl, mode, cond);
    hw2d::k2b_flux<<<gb, 256, 0, s>>>(tb, w, brk, ctl, mode, cond);
    brk_col(ny, 1, cols, s, tb, w, brk, ctl, mode, cond);
    brk_row(nx, 1, rows, s, tb, w, brk, rk, ctl, mode, cond, out);
    per_rhs += 8;
  }
  long long kernels_per_attempt() const { return (brk.on ? 7LL : 6LL) * per_rhs + 3; }
  // One attempt of a step.  Without breaking only a run's first attempt forms its own k1
  // (an accepted one leaves the next one's), so that right-hand side is launched ahead of the
  // attempts: as a conditional part of each it was six to thirteen empty kernels of 1.3 us.
  void attempt_launch(cudaStream_t s) {
    if (brk.on) rhs_launch(1, hw2d::kIfK1, s, nullptr);
    for (int st = 2; st <= 6; ++st) rhs_launch(st, hw2d::kIfStage, s, nullptr);
    if (brk.on) {
      // gsl_odeiv2's order: dydt_out of the candidate state before the step control
      hw2d::k2_combine<<<hw2d::kCombBlocks, hw2d::kCombThreads, 0, s>>>(tb.aal, rk, w, ctl, n);
      rhs_launch(8, hw2d::kIfStage, s, nullptr);
      hw2d::k2_control<<<1, 256, 0, s>>>(ctl, w, hw2d::kCombBlocks);
      hw2d::k2_finalize<<<1, 1, 0, s>>>(ctl);
      return;
    }
    hw2d::k2_combine<<<hw2d::kCombBlocks, hw2d::kCombThreads, 0, s>>>(tb.aal, rk, w, ctl, n);
    hw2d::k2_control<<<1, 256, 0, s>>>(ctl, w, hw2d::kCombBlocks);
    rhs_launch(7, hw2d::kIfKout, s, nullptr);
    hw2d::k2_finalize<<<1, 1, 0, s>>>(ctl);
  }
  bool build_graph() {
    if (attempt) return true;
    if (cudaStreamCreateWithFlags(&graph_stream, cudaStreamNonBlocking) != cudaSuccess) {
      err = "stream create failed";
      return false;
    }
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(graph_stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
      err = "graph capture failed to start";
      return false;
    }
    attempt_launch(graph_stream);
    if (cudaStreamEndCapture(graph_stream, &g) != cudaSuccess || !g) {
      err = "graph capture failed";
      cudaGetLastError();
      return false;
    }
    const cudaError_t e = cudaGraphInstantiate(&attempt, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
      err = std::string("graph instantiate: ") + cudaGetErrorString(e);
      return false;
    }
    return true;
  }
  bool read_ctl() {
    if (cudaMemcpyAsync(hctl, ctl, sizeof(Ctl2), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
        cudaStreamSynchronize(stream) != cudaSuccess)
      return check("control read-back");
    return true;
  }
  // evolve on the device until t1 (or one accepted step when one_step)
  int run(double t1, bool one_step) {
    if (!build_graph()) return 1;
    hw2d::k2_begin<<<1, 1, 0, stream>>>(ctl, t1);
    hw2d::k2_spread<<<hw2d::kCombBlocks, 256, 0, stream>>>(tb.aal, rk, w, ctl, n);
    launches += 2;
    if (!check("begin")) return 1;
    if (!read_ctl()) return 1;
    const long long acc0 = hctl->acc;
    long long launched = 0;
    if (!brk.on && !hctl->done && hctl->need_k1) {
      rhs_launch(1, hw2d::kIfK1, stream, nullptr);
      launches += per_rhs;
      if (!check("first right-hand side")) return 1;
    }
    for (;;) {
      if (hctl->done) break;
      if (launched > kMaxAttemptsPerRun) {
        err = "time integration stopped: attempt budget of one run exceeded (step size collapsed)";
        return 1;
      }
      // as many attempts as the present step asks for, sixteen at most: one past the end is
      // some forty empty kernels (50 us), one short another read of the control block (15 us)
      const int batch = one_step ? 1 : (int)std::min(16.0, std::max(1.0, std::ceil((t1 - hctl->t) / hctl->h - 0.01)));
      launched += batch;
      for (int b = 0; b < batch; ++b)
        if (const cudaError_t e = cudaGraphLaunch(attempt, stream); e != cudaSuccess) return fail("graph launch", e);
      launches += batch * kernels_per_attempt();
      if (!read_ctl()) return 1;
      if (hctl->status != hw2d::kOk) break;
      if (one_step && hctl->acc > acc0) {
        // stop here: the next call recomputes its dydt_in like GSL's evolve_apply
        break;
      }
    }
    if (hctl->status == hw2d::kNonFinite) { err = "non-finite state (the step size collapsed)"; return 1; }
    if (hctl->status == hw2d::kStepFailed) { err = "time integration failed (too many rejected steps)"; return 1; }
    if (hctl->status == hw2d::kBreakCapacity) { err = "breaking: a capacity (peaks, crests or nodes) was exceeded"; return 1; }
    return 0;
  }
  bool ensure_out(int ngauge) {
    if (!oP) {
      oP = dalloc<double2>(2 * n);
      ophys = dalloc<double>(3 * n);
      of32 = dalloc<float>(3 * n);
      if (!oP || !ophys || !of32 || cudaMallocHost(&hf32, 3 * n * sizeof(float)) != cudaSuccess) {
        err = "output buffers: out of memory";
        return false;
      }
    }
    if (ngauge > ogcap) {
      if (hgval) cudaFreeHost(hgval);
      hgval = nullptr;
      ogpt = dalloc<int>(ngauge);
      ogval = dalloc<double>(3 * (size_t)ngauge);
      if (!ogpt || !ogval || cudaMallocHost(&hgval, 3 * (size_t)ngauge * sizeof(double)) != cudaSuccess) {
        err = "gauge buffers: out of memory";
        return false;
      }
      ogcap = ngauge;
    }
    return true;
  }
  // eta, u, v of the current state (hctl must be current) into ophys (and of32)
  void fields_launch(cudaStream_t s, bool keep_f32) {
    out_pass(nx, 0, ny / 2, s, tb, rk.y[hctl->cur], oP, ophys, nullptr);
    out_pass(ny, 1, nx / 2, s, tb, rk.y[hctl->cur], oP, ophys, keep_f32 ? of32 : nullptr);
    launches += 2;
  }
  ~hw2d_ctx() {
    if (hf32) cudaFreeHost(hf32);
    if (hgval) cudaFreeHost(hgval);
    if (attempt) cudaGraphExecDestroy(attempt);
    if (graph_stream) cudaStreamDestroy(graph_stream);
    for (void* p : allocs) cudaFree(p);
    if (hctl) cudaFreeHost(hctl);
    if (own_stream) cudaStreamDestroy(own_stream);
  }
};

extern "C" {

hw2d_ctx* hw2d_create(const hw2d_tables* t, const hw_opts* o) {
  if (!t || !t->kx || !t->ky || !t->c2d || !t->l2d || !t->aal || !t->charac || !t->chiadj) {
    g_err2d = "hw2d_create: missing table";
    return nullptr;
  }
  if (!pow2_in_range(t->nx) || !pow2_in_range(t->ny)) {
    g_err2d = "hw2d_create: nx and ny must be powers of two in [64, 1024]";
    return nullptr;
  }
  if (t->model < 1 || t->model > 3) {
    g_err2d = "hw2d_create: model must be 1 (HS1), 2 (HS2) or 3 (HS3)";
    return nullptr;
  }
  const bool var_tables = t->gam_min && t->gam_plus && t->csq_min && t->csq_plus && t->om2_min && t->om2_plus;
  const bool mid_tables = t->gam_mid && t->csq_mid && t->om2_mid;
  if ((t->gam_mid || t->csq_mid || t->om2_mid) && !(mid_tables && var_tables)) {
    g_err2d = "hw2d_create: three reference depths need all of gam, csq, om2 for the min, mid and plus depths";
    return nullptr;
  }
  const bool kref = t->nrefk != 0;
  if (kref && (t->nrefk < 2 || t->nrefk > kMaxRef2 || !t->gam_k || !t->csq_k || !t->om2_k)) {
    g_err2d = "hw2d_create: K reference depths need 2 <= nrefk <= 16 and gam_k, csq_k, om2_k";
    return nullptr;
  }
  if (kref && (var_tables || t->gam_mid)) {
    g_err2d = "hw2d_create: give either the min/plus(/mid) tables or the K-reference tables, not both";
    return nullptr;
  }
  if (t->model == 1 && t->breaking) {
    // rhs_AB1_2DF_uv / rhs_AB1_2DB_uv never call breaking_process: under HS1 a breaking
    // deck is the plain HS1 run, so the tables must say breaking = 0
    g_err2d = "hw2d_create: HS1 runs no breaking process (rhs_AB1_2DF_uv, rhs_AB1_2DB_uv); pass breaking = 0";
    return nullptr;
  }
  if (t->propagation < 0 || t->propagation > 2) {
    g_err2d = "hw2d_create: propagation must be 0 (Uni+), 1 (Uni-) or 2 (Bi)";
    return nullptr;
  }
  auto* c = new hw2d_ctx();
  c->device = o ? o->device : 0;
  if (cudaSetDevice(c->device) != cudaSuccess) {
    g_err2d = "hw2d_create: cannot select the CUDA device";
    delete c;
    return nullptr;
  }
  set_all_attrs();
  const int nx = t->nx, ny = t->ny;
  const size_t n = (size_t)nx * ny;
  c->nx = nx; c->ny = ny; c->n = n;
  const bool has_src = t->nt >= 2 && t->sig && t->tsig && t->newgam;

  // host tables (reference formulas: C2d^2/grav as pow(C2d, 2)/grav, 7*Cpeak*charac)
  std::vector<double> c2g(n), damp(n);
  bool chi_one = true;
  for (size_t q = 0; q < n; ++q) {
    c2g[q] = std::pow(t->c2d[q], 2) / hw2d::kGrav;
    damp[q] = 7 * t->cpeak * t->charac[q];
    if (t->chiadj[q] != 1.0) chi_one = false;
  }
  Tab2& tb = c->tb;
  tb.nx = nx; tb.ny = ny; tb.n = (int)n; tb.model = t->model; tb.chi_one = chi_one ? 1 : 0;
  tb.has_src = has_src ? 1 : 0;
  tb.fac_src = t->propagation == 2 ? 2.0 : 1.0;
  tb.kx = c->upload(std::vector<double>(t->kx, t->kx + nx));
  tb.ky = c->upload(std::vector<double>(t->ky, t->ky + ny));
  tb.c2g = c->upload(c2g);
  tb.l2d = c->upload(std::vector<double>(t->l2d, t->l2d + n));
  tb.aal = c->upload(std::vector<double>(t->aal, t->aal + n));
  tb.damp = c->upload(damp);
  tb.chi = c->upload(std::vector<double>(t->chiadj, t->chiadj + n));
  tb.twx = c->upload(twiddles(nx));
  tb.twy = c->upload(twiddles(ny));
  if (has_src) {
    const double sk = t->propagation == 0 ? -1.0 : (t->propagation == 1 ? 1.0 : 0.0);
    std::vector<double> ss(n, 0.0);
    if (t->skewgam)
      for (size_t q = 0; q < n; ++q) ss[q] = sk * t->skewgam[q];
    tb.gsrc = c->upload(std::vector<double>(t->newgam, t->newgam + n));
    tb.ssrc = c->upload(ss);
    const int nt = t->nt;
    tb.nt = nt;
    std::vector<double> ts(t->tsig, t->tsig + nt);
    tb.t0 = ts[0];
    tb.tl = ts[size_t(nt - 1)];
    tb.dts = ts[1] - ts[0];
    std::vector<double> sig((size_t)ny * nt), sigc((size_t)ny * nt), sigs((size_t)ny * nt, 0.0),
        sigsc((size_t)ny * nt, 0.0);
    for (int i = 0; i < ny; ++i) {
      std::vector<double> a(t->sig + (size_t)i * nt, t->sig + (size_t)(i + 1) * nt);
      std::vector<double> ca = hw::natural_spline_c(ts, a);
      std::copy(a.begin(), a.end(), sig.begin() + (size_t)i * nt);
      std::copy(ca.begin(), ca.end(), sigc.begin() + (size_t)i * nt);
      if (t->sigskew) {
        std::vector<double> b(t->sigskew + (size_t)i * nt, t->sigskew + (size_t)(i + 1) * nt);
        std::vector<double> cb = hw::natural_spline_c(ts, b);
        std::copy(b.begin(), b.end(), sigs.begin() + (size_t)i * nt);
        std::copy(cb.begin(), cb.end(), sigsc.begin() + (size_t)i * nt);
      }
    }
    tb.tsig = c->upload(ts);
    tb.sig = c->upload(sig);
    tb.sigc = c->upload(sigc);
    tb.sigs = c->upload(sigs);
    tb.sigsc = c->upload(sigsc);
    c->h_first = (ts[nt - 1] - ts[0]) / (nt - 1) / 5.0;   // h = dt/5 (2d/fun_odesolver.c:2580)
  } else {
    c->h_first = 1e-3;
  }
  if (o && o->h0 > 0) c->h_first = o->h0;
  const bool var = kref || (t->gam_min && t->gam_plus && t->csq_min && t->csq_plus && t->om2_min && t->om2_plus);
  tb.var = var ? 1 : 0;
  if (var) {
    // rows of the reference depths: K given ones, or min, (mid,) plus in HSSgen's order
    auto rows = [&](const double* all, const double* lo, const double* mid, const double* hi) {
      std::vector<double> v;
      if (kref) v.assign(all, all + (size_t)t->nrefk * n);
      else
        for (const double* r : {lo, mid, hi})
          if (r) v.insert(v.end(), r, r + n);
      return v;
    };
    tb.nk = kref ? t->nrefk : (t->gam_mid ? 3 : 2);
    tb.gk = c->upload(rows(t->gam_k, t->gam_min, t->gam_mid, t->gam_plus));
    tb.ck = c->upload(rows(t->csq_k, t->csq_min, t->csq_mid, t->csq_plus));
    tb.ok = c->upload(rows(t->om2_k, t->om2_min, t->om2_mid, t->om2_plus));
  }
  if (t->wallchar) {
    tb.wallchar = c->upload(std::vector<double>(t->wallchar, t->wallchar + n));
    if (!var) tb.c2d = c->upload(std::vector<double>(t->c2d, t->c2d + n));
    if (!var && t->refl_coef == 1) {
      // fun_delphiH1hat's refl_coef == 1 branch needs fun_gradient(wallchar)
      // (2d/functions.c:392-460, called at :741): periodic forward and backward
      // differences, the forward ones clipped to <= 0, the backward ones to >= 0
      if (!(t->dx > 0) || !(t->dy > 0)) {
        g_err2d = "hw2d_create: walls with refl_coef 1 need dx and dy";
        delete c;
        return nullptr;
      }
      std::vector<double> gx(n), gy(n);
      const double* f = t->wallchar;
      for (int i = 0; i < ny; ++i)
        for (int j = 0; j < nx; ++j) {
          const size_t q = (size_t)i * nx + j;
          double Fx = (j < nx - 1) ? (f[q + 1] - f[q]) / t->dx : (f[(size_t)i * nx] - f[q]) / t->dx;
          double Fy = (i < ny - 1) ? (f[q + nx] - f[q]) / t->dy : (f[j] - f[q]) / t->dy;
          double Bx = (j > 0) ? (f[q] - f[q - 1]) / t->dx : (f[q] - f[(size_t)i * nx + nx - 1]) / t->dx;
          double By = (i > 0) ? (f[q] - f[q - nx]) / t->dy : (f[q] - f[(size_t)(ny - 1) * nx + j]) / t->dy;
          if (Fx > 0) Fx = 0;
          if (Fy > 0) Fy = 0;
          if (Bx < 0) Bx = 0;
          if (By < 0) By = 0;
          gx[q] = Fx + Bx;
          gy[q] = Fy + By;
        }
      tb.refl_one = 1;
      tb.gwx = c->upload(gx);
      tb.gwy = c->upload(gy);
    }
  }

  hw2d::Brk2& bk = c->brk;
  if (t->breaking) {
    if (!t->bathy || !t->brchar || !t->x || !t->y || !(t->dx > 0) || !(t->dy > 0) || !(t->dt_out > 0) ||
        !(t->rsearch > 0)) {
      g_err2d = "hw2d_create: breaking tables missing or invalid";
      delete c;
      return nullptr;
    }
    bk.on = 1;
    bk.bathy = c->upload(std::vector<double>(t->bathy, t->bathy + n));
    bk.pbchar = c->upload(std::vector<double>(t->brchar, t->brchar + n));
    bk.x = c->upload(std::vector<double>(t->x, t->x + nx));
    bk.y = c->upload(std::vector<double>(t->y, t->y + ny));
    bk.dx = t->dx; bk.dy = t->dy; bk.thr = t->max_eta_init; bk.tstar = t->tstar; bk.rsearch = t->rsearch;
    bk.kbc = t->kbc; bk.tc = t->tc; bk.delb = t->delb; bk.cur_u = t->cur_u; bk.t0 = t->t0; bk.dt_out = t->dt_out;
    bk.B = c->dalloc<double>(n);
    bk.flux = c->dalloc<double>(n);
    bk.P = c->dalloc<double2>(n);
    bk.dh = c->dalloc<double2>(n);
    bk.sb = c->dalloc<double2>(2 * n);
    bk.peaks = c->dalloc<int>(hw2d::kBrkPeakCap);
    bk.CB = c->dalloc<hw2d::Crest2>(hw2d::kBrkCrestCap);
    bk.CBNew = c->dalloc<hw2d::Crest2>(hw2d::kBrkCrestCap);
    bk.CBPrev = c->dalloc<hw2d::Crest2>(hw2d::kBrkCrestCap);
    bk.cap_nodes = (int)std::max<size_t>(4096, n / 4);
    bk.bn[0] = c->dalloc<int2>(bk.cap_nodes);
    bk.bn[1] = c->dalloc<int2>(bk.cap_nodes);
    bk.bnp = c->dalloc<int2>(bk.cap_nodes);
    bk.cap_rec = 1 << 18;
    bk.cap_log = (long long)std::max<size_t>(1 << 16, 4 * n);
    bk.log_t = c->dalloc<double>(bk.cap_rec);
    bk.log_cnt = c->dalloc<int>(bk.cap_rec);
    bk.log_nodes = c->dalloc<int2>((size_t)bk.cap_log);
    bk.st = c->dalloc<hw2d::BrkSt>(1);
    const bool bok = bk.bathy && bk.pbchar && bk.x && bk.y && bk.B && bk.flux && bk.P && bk.dh && bk.sb && bk.peaks &&
                     bk.CB && bk.CBNew && bk.CBPrev && bk.bn[0] && bk.bn[1] && bk.bnp && bk.log_t && bk.log_cnt &&
                     bk.log_nodes && bk.st;
    if (!bok) {
      g_err2d = "hw2d_create: device allocation failed (breaking)";
      delete c;
      return nullptr;
    }
    hw2d::BrkSt s0{};
    s0.sb_zero = 1;   // Sb_xhat, Sb_yhat start at zero
    cudaMemcpy(bk.st, &s0, sizeof s0, cudaMemcpyHostToDevice);
    cudaMemset(bk.B, 0, n * sizeof(double));
    cudaMemset(bk.sb, 0, 2 * n * sizeof(double2));
  }

  Work2& w = c->w;
  w.dph = bk.on ? c->dalloc<double2>(n) : nullptr;
  const int K = tb.nk, nd = chi_one ? 2 : (bk.on ? 1 : 0);
  w.z = c->dalloc<double2>(3 * n);
  w.R = c->dalloc<double2>((size_t)(var ? 2 + K : 3) * n);
  w.Q = c->dalloc<double2>((size_t)std::max(1 + K, 3 + nd + (K + 1) / 2) * n);
  w.T = c->dalloc<double2>(3 * n);
  w.D = c->dalloc<double2>(3 * n);
  w.W = chi_one ? nullptr : c->dalloc<double2>(3 * n);
  w.V = c->dalloc<double2>(3 * n);
  w.phys = c->dalloc<double>(3 * n);
  w.op = c->dalloc<double>(2 * n);
  if (var || t->wallchar) w.H1 = c->dalloc<double2>(n);
  if (!var && t->wallchar) w.WP = c->dalloc<double2>((tb.refl_one ? 2 : 1) * n);   // the wall's round trip
  w.insig = c->dalloc<double>(ny);
  w.insigs = c->dalloc<double>(ny);
  w.part = c->dalloc<double>(hw2d::kCombBlocks);
  RK2& rk = c->rk;
  for (int i = 0; i < 2; ++i) rk.y[i] = c->dalloc<double2>(3 * n);
  for (int i = 0; i < 2; ++i) rk.kk[i] = c->dalloc<double2>(3 * n);
  for (int i = 0; i < 5; ++i) rk.ks[i] = c->dalloc<double2>(3 * n);
  c->dref = c->dalloc<double>(6 * n);
  c->dout = c->dalloc<double2>(3 * n);
  c->ctl = c->dalloc<Ctl2>(1);
  bool ok = tb.kx && tb.ky && tb.c2g && tb.l2d && tb.aal && tb.damp && tb.chi && tb.twx && tb.twy && w.z && w.R &&
            w.Q && w.T && w.D && w.V && w.phys && w.op && w.insig && w.insigs && w.part && c->dref && c->dout && c->ctl &&
            (chi_one || w.W) && (!has_src || (tb.gsrc && tb.ssrc && tb.sig && tb.sigc && tb.sigs && tb.sigsc)) &&
            (!bk.on || w.dph) && (!var || (tb.gk && tb.ck && tb.ok && w.H1)) &&
            (!t->wallchar || (tb.wallchar && w.H1 &&
                              (var || (w.WP && tb.c2d && (!tb.refl_one || (tb.gwx && tb.gwy))))));
  for (int i = 0; i < 2; ++i) ok = ok && rk.y[i] && rk.kk[i];
  for (int i = 0; i < 5; ++i) ok = ok && rk.ks[i];
  // the pinned control block, with the mapped buffer behind it where there is one
  const size_t mapped = n <= hw2d_ctx::kMappedPoints ? 6 * n : 0;
  static_assert(sizeof(Ctl2) % sizeof(double) == 0, "the buffer follows aligned");
  if (ok && cudaHostAlloc(&c->hctl, sizeof(Ctl2) + mapped * sizeof(double), cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();
    ok = false;
  }
  if (ok && mapped) c->href = reinterpret_cast<double*>(c->hctl + 1);
  if (!ok) {
    g_err2d = "hw2d_create: device allocation failed";
    delete c;
    return nullptr;
  }
  cudaStreamCreateWithFlags(&c->own_stream, cudaStreamNonBlocking);
  c->stream = c->own_stream;
  Ctl2 h{};
  h.eps_abs = (o && o->eps_abs > 0) ? o->eps_abs : 1e-3;
  h.eps_rel = (o && o->eps_rel > 0) ? o->eps_rel : 1e-2;
  h.h = c->h_first;
  h.need_k1 = 1;
  h.done = 1;
  h.brk = bk.on;
  cudaMemcpy(c->ctl, &h, sizeof h, cudaMemcpyHostToDevice);
  cudaMemset(rk.y[0], 0, 3 * n * sizeof(double2));
  if (!c->check("hw2d_create")) {
    g_err2d = c->err;
    delete c;
    return nullptr;
  }
  return c;
}

void hw2d_destroy(hw2d_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  cudaStreamSynchronize(c->stream);
  delete c;
}

const char* hw2d_last_error(const hw2d_ctx* c) { return c ? c->err.c_str() : g_err2d.c_str(); }
int hw2d_nx(const hw2d_ctx* c) { return c ? c->nx : 0; }
int hw2d_ny(const hw2d_ctx* c) { return c ? c->ny : 0; }

int hw2d_rhs(hw2d_ctx* c, double t, const double* y, double* dydt) {
  if (!c || !y || !dydt) return 1;
  cudaSetDevice(c->device);
  const size_t n = c->n;
  // the mapped buffer where there is one: the layout kernels read and write it over PCIe
  double* ref = c->href ? c->href : c->dref;
  if (c->href) std::memcpy(ref, y, 6 * n * sizeof(double));
  else cudaMemcpyAsync(ref, y, 6 * n * sizeof(double), cudaMemcpyHostToDevice, c->stream);
  hw2d::k2_to_internal<<<592, 256, 0, c->stream>>>(ref, c->w.z, n, c->ctl, t);
  c->rhs_launch(0, hw2d::kAlways, c->stream, c->dout);
  hw2d::k2_to_reference<<<592, 256, 0, c->stream>>>(c->dout, ref, n);
  c->launches += c->per_rhs + 2;
  if (!c->href) cudaMemcpyAsync(dydt, ref, 6 * n * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
  if (const cudaError_t e = cudaStreamSynchronize(c->stream); e != cudaSuccess) return c->fail("hw2d_rhs", e);
  if (!c->check("hw2d_rhs")) return 1;
  if (c->href) std::memcpy(dydt, ref, 6 * n * sizeof(double));
  if (c->brk.on) {
    hw2d::BrkSt st{};
    if (const cudaError_t e = cudaMemcpy(&st, c->brk.st, sizeof st, cudaMemcpyDeviceToHost); e != cudaSuccess)
      return c->fail("hw2d_rhs", e);
    if (st.err & (hw2d::kBrkErrPeaks | hw2d::kBrkErrCrests | hw2d::kBrkErrNodes)) {
      c->err = "breaking: a capacity (peaks, crests or nodes) was exceeded";
      return 1;
    }
  }
  return 0;
}

int hw2d_gsl_rhs(double t, const double* y, double* dydt, void* params) {
  return hw2d_rhs(static_cast<hw2d_ctx*>(params), t, y, dydt);
}

int hw2d_set_state(hw2d_ctx* c, double t, double h, const double* y) {
  if (!c || !y) return 1;
  cudaSetDevice(c->device);
  if (!c->read_ctl()) return 1;
  Ctl2 s = *c->hctl;
  s.t = t;
  s.h = h > 0 ? h : c->h_first;
  s.cur = 0;
  s.need_k1 = 1;
  s.need_kout = 0;
  s.done = 1;
  s.status = hw2d::kOk;
  *c->hctl = s;
  cudaMemcpyAsync(c->dref, y, 6 * c->n * sizeof(double), cudaMemcpyHostToDevice, c->stream);
  hw2d::k2_to_internal<<<592, 256, 0, c->stream>>>(c->dref, c->rk.y[0], c->n, nullptr, 0.0);
  c->launches += 1;
  cudaMemcpyAsync(c->ctl, c->hctl, sizeof(Ctl2), cudaMemcpyHostToDevice, c->stream);
  if (const cudaError_t e = cudaStreamSynchronize(c->stream); e != cudaSuccess) return c->fail("hw2d_set_state", e);
  return c->check("hw2d_set_state") ? 0 : 1;
}

int hw2d_get_state(hw2d_ctx* c, double* t, double* h, double* y) {
  if (!c) return 1;
  cudaSetDevice(c->device);
  if (!c->read_ctl()) return 1;
  if (t) *t = c->hctl->t;
  if (h) *h = c->hctl->h;
  if (y) {
    hw2d::k2_to_reference<<<592, 256, 0, c->stream>>>(c->rk.y[c->hctl->cur], c->dref, c->n);
    c->launches += 1;
    cudaMemcpyAsync(y, c->dref, 6 * c->n * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    if (const cudaError_t e = cudaStreamSynchronize(c->stream); e != cudaSuccess) return c->fail("hw2d_get_state", e);
  }
  return c->check("hw2d_get_state") ? 0 : 1;
}

int hw2d_run_to_time(hw2d_ctx* c, double t1) {
  if (!c) return 1;
  cudaSetDevice(c->device);
  return c->run(t1, false);
}

int hw2d_evolve_apply(hw2d_ctx* c, double* t, double t1, double* h, double* y) {
  if (!c || !t || !h || !y) return 1;
  if (hw2d_set_state(c, *t, *h, y)) return 1;
  // gsl_odeiv2_evolve_apply rejects a step whose direction disagrees with t1 - t
  const double dt = t1 - *t;
  if ((dt < 0.0 && *h > 0.0) || (dt > 0.0 && *h < 0.0)) {
    c->err = "step direction does not match t1 - t";
    return 1;
  }
  if (c->run(t1, true)) return 1;
  return hw2d_get_state(c, t, h, y);
}

int hw2d_stats(const hw2d_ctx* cc, long long* r, long long* a, long long* j) {
  auto* c = const_cast<hw2d_ctx*>(cc);
  if (!c || !c->read_ctl()) return 1;
  if (r) *r = c->hctl->rhs;
  if (a) *a = c->hctl->acc;
  if (j) *j = c->hctl->rej;
  return 0;
}

long long hw2d_launches(const hw2d_ctx* c) { return c ? c->launches : 0; }

int hw2d_breaking_fields(hw2d_ctx* c, double* B, double* sbx, double* sby, int* flagbr, int* ncrest) {
  if (!c || !c->brk.on) return -1;
  cudaSetDevice(c->device);
  if (const cudaError_t e = cudaStreamSynchronize(c->stream); e != cudaSuccess)
    return c->fail("hw2d_breaking_fields", e);
  const size_t n = c->n;
  struct Copy { void* dst; const void* src; size_t bytes; };
  hw2d::BrkSt st{};
  const Copy copies[4] = {{B, c->brk.B, n * sizeof(double)}, {sbx, c->brk.sb, n * sizeof(double2)},
                          {sby, c->brk.sb + n, n * sizeof(double2)}, {&st, c->brk.st, sizeof st}};
  for (const Copy& k : copies)
    if (k.dst)
      if (const cudaError_t e = cudaMemcpy(k.dst, k.src, k.bytes, cudaMemcpyDeviceToHost); e != cudaSuccess)
        return c->fail("hw2d_breaking_fields", e);
  if (flagbr) *flagbr = st.flagbr;
  if (ncrest) *ncrest = st.flagbr == 2 ? st.ncbprev : 0;
  return 0;
}

long long hw2d_breaking_log_nodes(hw2d_ctx* c) {
  if (!c || !c->brk.on) return -1;
  cudaSetDevice(c->device);
  hw2d::BrkSt st{};
  if (cudaStreamSynchronize(c->stream) != cudaSuccess ||
      cudaMemcpy(&st, c->brk.st, sizeof st, cudaMemcpyDeviceToHost) != cudaSuccess)
    return -1;
  return st.nlog;
}

int hw2d_breaking_log(hw2d_ctx* c, double* times, int* counts, int* nodes, int cap_rec, long long cap_nodes) {
  if (!c || !c->brk.on) return -1;
  cudaSetDevice(c->device);
  hw2d::BrkSt st{};
  if (cudaStreamSynchronize(c->stream) != cudaSuccess ||
      cudaMemcpy(&st, c->brk.st, sizeof st, cudaMemcpyDeviceToHost) != cudaSuccess)
    return -1;
  const int nr = std::min(st.nrec, std::max(cap_rec, 0));
  const long long nn = std::min(st.nlog, std::max(cap_nodes, 0LL));
  if (times && nr > 0 && cudaMemcpy(times, c->brk.log_t, nr * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess)
    return -1;
  if (counts && nr > 0 && cudaMemcpy(counts, c->brk.log_cnt, nr * sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
    return -1;
  if (nodes && nn > 0 && cudaMemcpy(nodes, c->brk.log_nodes, nn * sizeof(int2), cudaMemcpyDeviceToHost) != cudaSuccess)
    return -1;
  if (st.err & hw2d::kBrkErrLog) return -2;
  return st.nrec;
}

int hw2d_fields(hw2d_ctx* c, double* eta, double* u, double* v) {
  if (!c) return 1;
  cudaSetDevice(c->device);
  if (!c->ensure_out(0) || !c->read_ctl()) return 1;
  c->fields_launch(c->stream, false);
  if (!c->check("hw2d_fields")) return 1;
  double* dst[3] = {eta, u, v};
  for (int f = 0; f < 3; ++f)
    if (dst[f])
      if (const cudaError_t e = cudaMemcpyAsync(dst[f], c->ophys + f * c->n, c->n * sizeof(double),
                                                cudaMemcpyDeviceToHost, c->stream);
          e != cudaSuccess)
        return c->fail("hw2d_fields", e);
  if (const cudaError_t e = cudaStreamSynchronize(c->stream); e != cudaSuccess) return c->fail("hw2d_fields", e);
  return 0;
}

namespace {

// the file set of ode_solver_uv's output loop; every file is closed on the way out
struct OutFiles {
  FILE* part[3] = {nullptr, nullptr, nullptr};   // Hawassi_eta/u/v_NN.dat
  FILE* gauge[3] = {nullptr, nullptr, nullptr};  // Hawassi_eta/u/v_gauge.dat
  void close_part() {
    for (FILE*& f : part)
      if (f) { fclose(f); f = nullptr; }
  }
  ~OutFiles() {
    close_part();
    for (FILE*& f : gauge)
      if (f) { fclose(f); f = nullptr; }
  }
};

// print_xt (2d/fun_odesolver.c:2532-2563)
bool write_constant(const std::string& path, const hw2d_outputs* o, int nx, int ny, int ntpart) {
  FILE* f = fopen(path.c_str(), "wb");
  if (!f) return false;
  std::vector<double> th(ntpart);
  for (int j = 0; j < ntpart; ++j) th[j] = (0 + j) * o->dt;
  const double NX = nx, NT = ntpart, NY = ny;
  const size_t n = (size_t)nx * ny;
  bool ok = fwrite(&NX, sizeof(double), 1, f) == 1 && fwrite(o->x, sizeof(double), nx, f) == (size_t)nx &&
            fwrite(&NY, sizeof(double), 1, f) == 1 && fwrite(o->y, sizeof(double), ny, f) == (size_t)ny &&
            fwrite(&NT, sizeof(double), 1, f) == 1 &&
            fwrite(th.data(), sizeof(double), ntpart, f) == (size_t)ntpart &&
            fwrite(&o->hs, sizeof(double), 1, f) == 1 && fwrite(&o->kp, sizeof(double), 1, f) == 1 &&
            fwrite(&o->wp, sizeof(double), 1, f) == 1 && fwrite(o->kx, sizeof(double), nx, f) == (size_t)nx &&
            fwrite(o->ky, sizeof(double), ny, f) == (size_t)ny && fwrite(o->bathy, sizeof(double), n, f) == n &&
            fwrite(o->cfsa, sizeof(double), n, f) == n;
  if (ok && o->chiadjphi) ok = fwrite(o->chiadjphi, sizeof(double), n, f) == n;
  return fclose(f) == 0 && ok;
}

}  // namespace

int hw2d_run_outputs(hw2d_ctx* c, const hw2d_outputs* o) {
  if (!c || !o) return -1;
  cudaSetDevice(c->device);
  auto fail = [&](const std::string& m) {
    c->err = m;
    return -1;
  };
  if (!o->outdir || o->nt < 1 || !o->tout) return fail("outputs: outdir, nt and tout are required");
  if (o->npartition < 1 || o->nt / o->npartition < 1) return fail("outputs: npartition must be in [1, nt]");
  if (!o->x || !o->y || !o->kx || !o->ky || !o->bathy || !o->cfsa)
    return fail("outputs: x, y, kx, ky, bathy and cfsa are required (Constant_01.dat)");
  if (o->ngauge < 0 || (o->ngauge > 0 && (!o->xgauge || !o->ygauge || !(o->dx > 0) || !(o->dy > 0))))
    return fail("outputs: gauges need xgauge, ygauge, dx and dy");
  const int nx = c->nx, ny = c->ny, ng = o->ngauge;
  const size_t n = c->n;
  const int ntpart = o->nt / o->npartition;
  // index_gauge (2d/functions.c:774-781): the nearest grid point
  std::vector<int> gx(ng), gy(ng), gpt(ng);
  for (int j = 0; j < ng; ++j) {
    const double fx = std::round((o->xgauge[j] - o->x[0]) / o->dx), fy = std::round((o->ygauge[j] - o->y[0]) / o->dy);
    if (!(fx >= 0 && fx < nx && fy >= 0 && fy < ny)) return fail("Gauges are outside of the domain!");
    gx[j] = (int)fx;
    gy[j] = (int)fy;
    gpt[j] = gy[j] * nx + gx[j];
  }
  if (!c->ensure_out(ng)) return -1;
  if (ng > 0)
    if (const cudaError_t e = cudaMemcpy(c->ogpt, gpt.data(), ng * sizeof(int), cudaMemcpyHostToDevice);
        e != cudaSuccess)
      return -c->fail("gauge upload", e);
  const std::string pre(o->outdir);
  OutFiles files;
  static const char* kField[3] = {"eta", "u", "v"};
  if (ng > 0)
    for (int f = 0; f < 3; ++f) {
      files.gauge[f] = fopen((pre + "Hawassi_" + kField[f] + "_gauge.dat").c_str(), "wb");
      if (!files.gauge[f]) return fail("cannot open " + pre + "Hawassi_" + kField[f] + "_gauge.dat");
    }
  int ipart = 1;
  char name[64];
  for (int i = 0; i < o->nt; ++i) {
    if (c->run(o->tout[i], false)) return -1;
    const double t = c->hctl->t;
    const bool first = (i % ntpart) == 0;
    const bool uv = o->uv_every_sample || first;
    c->fields_launch(c->stream, true);
    if (ng > 0) {
      hw2d::k2o_gauge<<<(ng + 127) / 128, 128, 0, c->stream>>>(c->ophys, c->ogpt, ng, n, c->ogval);
      c->launches += 1;
      cudaMemcpyAsync(c->hgval, c->ogval, 3 * (size_t)ng * sizeof(double), cudaMemcpyDeviceToHost, c->stream);
    }
    cudaMemcpyAsync(c->hf32, c->of32, (uv ? 3 : 1) * n * sizeof(float), cudaMemcpyDeviceToHost, c->stream);
    if (const cudaError_t e = cudaStreamSynchronize(c->stream); e != cudaSuccess) return -c->fail("output stage", e);
    if (!c->check("output stage")) return -1;
    if (first) {
      // the reference opens the next partition's files without closing the last ones
      files.close_part();
      for (int f = 0; f < 3; ++f) {
        snprintf(name, sizeof name, "Hawassi_%s_%02d.dat", kField[f], ipart);
        files.part[f] = fopen((pre + name).c_str(), "wb");
        if (!files.part[f]) return fail("cannot open " + pre + name);
      }
      if (i == 0) {
        snprintf(name, sizeof name, "Constant_%02d.dat", ipart);
        if (!write_constant(pre + name, o, nx, ny, ntpart)) return fail("cannot write " + pre + name);
      }
      ++ipart;
    }
    bool ok = fwrite(c->hf32, sizeof(float), n, files.part[0]) == n;
    if (uv)
      ok = ok && fwrite(c->hf32 + n, sizeof(float), n, files.part[1]) == n &&
           fwrite(c->hf32 + 2 * n, sizeof(float), n, files.part[2]) == n;
    for (FILE* f : files.part) ok = ok && fflush(f) == 0;
    if (ng > 0) {
      // print_data_gauges_uv (2d/fun_odesolver.c:427-476)
      for (int f = 0; f < 3; ++f) {
        FILE* g = files.gauge[f];
        if (i == 0) {
          fprintf(g, "0 ");
          for (int j = 0; j < ng; ++j) fprintf(g, "%f ", o->x[gx[j]]);
          fprintf(g, "\n");
          fprintf(g, "0 ");
          for (int j = 0; j < ng; ++j) fprintf(g, "%f ", o->y[gy[j]]);
          fprintf(g, "\n");
        }
        fprintf(g, "%f ", t);
        for (int j = 0; j < ng; ++j) fprintf(g, "%f ", c->hgval[3 * j + f]);
        fprintf(g, "\n");
        ok = ok && fflush(g) == 0;
      }
    }
    if (!ok) return fail("output files: write failed");
    if (std::isnan(c->hf32[n - 1])) {
      snprintf(name, sizeof name, "Time stepping failed at t=%fs.", t);
      return fail(name);
    }
  }
  if (c->brk.on) {
    // breaking.dat (2d/breaking.c:707-718): "t" then " x y " per break node, one line a record
    const int nrec = hw2d_breaking_log(c, nullptr, nullptr, nullptr, 0, 0);
    if (nrec < 0) return fail(nrec == -2 ? "breaking log overflowed" : "breaking log read failed");
    const long long nn = hw2d_breaking_log_nodes(c);
    std::vector<double> tr(nrec);
    std::vector<int> cnt(nrec), nodes(2 * (size_t)std::max(nn, 0LL));
    if (hw2d_breaking_log(c, tr.data(), cnt.data(), nodes.data(), nrec, nn) != nrec)
      return fail("breaking log read failed");
    FILE* f = fopen((pre + "breaking.dat").c_str(), "w");
    if (!f) return fail("cannot open " + pre + "breaking.dat");
    size_t k = 0;
    for (int r = 0; r < nrec; ++r) {
      fprintf(f, "%lf ", tr[r]);
      for (int j = 0; j < cnt[r] && k < (size_t)nn; ++j, ++k) fprintf(f, " %d %d ", nodes[2 * k], nodes[2 * k + 1]);
      fprintf(f, "\n");
    }
    if (fclose(f) != 0) return fail("cannot write " + pre + "breaking.dat");
  }
  return o->nt;
}

int hw2d_set_stream(hw2d_ctx* c, void* s) {
  if (!c) return 1;
  c->stream = s ? static_cast<cudaStream_t>(s) : c->own_stream;
  return 0;
}

int hw2d_synchronize(hw2d_ctx* c) {
  if (!c) return 1;
  return cudaStreamSynchronize(c->stream) == cudaSuccess ? 0 : 1;
}

}  // extern "C"
