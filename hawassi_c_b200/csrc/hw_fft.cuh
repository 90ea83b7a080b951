// hw_fft.cuh -- FP64 complex FFT of one member's grid, distributed over the C
// CTAs of a thread-block cluster.  Each CTA owns a slice of M = N / C points in
// shared memory (T = M / 8 threads, 8 points per thread).
//
// Layouts (index i within the CTA of cluster rank c):
//   physical ("block"):  global grid index n = c*M + i
//   spectral ("cyclic"): global wavenumber index kk = c + C*i
// Forward transform (block -> cyclic) is a decimation-in-frequency four-step:
// a C-point DFT across the cluster (read from the peers' shared memory through
// DSMEM) times the twiddle W_N^(i*c), then a local M-point Stockham FFT.  The
// inverse (cyclic -> block) is the transpose: local M-point inverse FFT, then
// the twiddle and the C-point DFT across the cluster.  With C == 1 the cross
// step vanishes.  Sign convention and scaling follow FFTW (unnormalised,
// forward exponent -1).
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

namespace hwdev {

namespace cg = cooperative_groups;

constexpr int kPts = 8;  // points per thread

// bank swizzle: position i of a slice is stored at i with its low three bits XORed
// by bits 3-5 (a permutation inside each group of 8 double2 = 128 bytes = all 32
// banks), which keeps the stride-8 stores of the first Stockham pass conflict-free
// while unit-stride accesses stay conflict-free; unlike a pad slot per 8 points it
// costs no shared memory, which the SM gives to L1 instead
__device__ __forceinline__ int pidx(int i) { return i ^ ((i >> 3) & 7); }
__host__ __device__ constexpr int padded(int m) { return m; }

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

// twiddle exp(sign * 2 pi i q / N) from the table tw[q] = exp(-2 pi i q / N)
__device__ __forceinline__ double2 twd(const double2* __restrict__ tw, int q, int sign) {
  double2 w = __ldg(tw + q);
  return sign > 0 ? make_double2(w.x, -w.y) : w;
}

// multiply by exp(sign * i pi / 2) = sign * i
__device__ __forceinline__ double2 mul_pm_i(double2 a, int sign) {
  return sign > 0 ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

template <int R>
__device__ __forceinline__ void dft_small(double2* v, int sign);

template <>
__device__ __forceinline__ void dft_small<2>(double2* v, int) {
  double2 a = v[0], b = v[1];
  v[0] = cadd(a, b);
  v[1] = csub(a, b);
}

template <>
__device__ __forceinline__ void dft_small<4>(double2* v, int sign) {
  double2 d0 = cadd(v[0], v[2]), d2 = csub(v[0], v[2]);
  double2 d1 = cadd(v[1], v[3]), d3 = mul_pm_i(csub(v[1], v[3]), sign);
  v[0] = cadd(d0, d1);
  v[2] = csub(d0, d1);
  v[1] = cadd(d2, d3);
  v[3] = csub(d2, d3);
}

template <>
__device__ __forceinline__ void dft_small<8>(double2* v, int sign) {
  const double r = 0.70710678118654752440084436210485;  // sqrt(1/2)
  double2 b[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    b[i] = cadd(v[i], v[i + 4]);
    b[i + 4] = csub(v[i], v[i + 4]);
  }
  // b5 *= w^1, b6 *= w^2, b7 *= w^3 with w = exp(sign * 2 pi i / 8)
  {
    double2 a = b[5];
    b[5] = make_double2(r * (a.x - sign * a.y), r * (a.y + sign * a.x));
    b[6] = mul_pm_i(b[6], sign);
    a = b[7];
    b[7] = make_double2(r * (-a.x - sign * a.y), r * (-a.y + sign * a.x));
  }
  double2 e[4] = {b[0], b[1], b[2], b[3]}, o[4] = {b[4], b[5], b[6], b[7]};
  dft_small<4>(e, sign);
  dft_small<4>(o, sign);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    v[2 * m] = e[m];
    v[2 * m + 1] = o[m];
  }
}


// w^1..w^(R-1) from w^1: one table load per butterfly, powers by short products
// (w^2 = w w, w^3 = w^2 w, w^4 = w^2 w^2, w^5 = w^4 w, w^6 = w^4 w^2, w^7 = w^4 w^3)
template <int R>
__device__ __forceinline__ void twiddle_powers(double2 w1, double2* w) {
  w[1] = w1;
  if constexpr (R > 2) {
    w[2] = cmul(w1, w1);
    w[3] = cmul(w[2], w1);
  }
  if constexpr (R > 4) {
    w[4] = cmul(w[2], w[2]);
    w[5] = cmul(w[4], w1);
    w[6] = cmul(w[4], w[2]);
    w[7] = cmul(w[4], w[3]);
  }
}

// 16-point DFT as 4 x 4
template <>
__device__ __forceinline__ void dft_small<16>(double2* v, int sign) {
  constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173, r = 0.70710678118654752440;
#pragma unroll
  for (int n = 0; n < 4; ++n) {
    double2 t[4] = {v[n], v[n + 4], v[n + 8], v[n + 12]};
    dft_small<4>(t, sign);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[n + 4 * k] = t[k];
  }
  // x W16^(n k), n the column, k the row of the 4 x 4 block
  const double sg = double(sign);
  auto rot = [&](double2 a, double c, double s) { return make_double2(c * a.x - sg * s * a.y, c * a.y + sg * s * a.x); };
  v[5] = rot(v[5], c1, s1);
  v[6] = rot(v[6], r, r);
  v[7] = rot(v[7], s1, c1);
  v[9] = rot(v[9], r, r);
  v[10] = mul_pm_i(v[10], sign);
  v[11] = rot(v[11], -r, r);
  v[13] = rot(v[13], s1, c1);
  v[14] = rot(v[14], -r, r);
  v[15] = rot(v[15], -c1, -s1);
#pragma unroll
  for (int k = 0; k < 4; ++k) dft_small<4>(v + 4 * k, sign);
  // v[4 k2 + k1] holds X[4 k1 + k2]
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = a + 1; b < 4; ++b) {
      const double2 t = v[4 * a + b];
      v[4 * a + b] = v[4 * b + a];
      v[4 * b + a] = t;
    }
}

// the TP threads of one slice: within a warp, or the warps of group g by their own barrier
template <int TP>
__device__ __forceinline__ void slice_sync(int g) {
  if constexpr (TP > 32) asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(TP) : "memory");
  else __syncwarp();
}

// One in-place Stockham radix-R pass of an M-point slice by M/16 threads (rank tid of group
// g), 16 points each.  xo turns the slice's swizzle (pidx(i) ^ xo); tw_stride converts an
// index in units of 1/M of a turn to the table's.  Lanes with act = false only keep step.
template <int M, int R>
__device__ __forceinline__ void slice_pass(double2* buf, int xo, int Ns, const double2* __restrict__ tw, int tw_stride,
                                           int sign, int tid, int g, bool act) {
  constexpr int TP = M / 16, NB = M / R, BPT = 16 / R;
  double2 v[BPT][R];
  if (act) {
#pragma unroll
    for (int u = 0; u < BPT; ++u)
#pragma unroll
      for (int r = 0; r < R; ++r) v[u][r] = buf[pidx(tid + u * TP + r * NB) ^ xo];
  }
  slice_sync<TP>(g);
  if (act) {
#pragma unroll
    for (int u = 0; u < BPT; ++u) {
      const int j = tid + u * TP, jm = j & (Ns - 1);
      if (Ns > 1) {
        const int qb = jm * (M / (Ns * R)) * tw_stride;
        if constexpr (R == 16) {
          // powers from w, w^2, w^4, w^8: at most three factors each
          const double2 w1 = twd(tw, qb, sign), w2 = twd(tw, 2 * qb, sign), w4 = twd(tw, 4 * qb, sign),
                        w8 = twd(tw, 8 * qb, sign), w3 = cmul(w2, w1);
          const double2 lo[4] = {make_double2(1.0, 0.0), w1, w2, w3};
#pragma unroll
          for (int r = 1; r < 4; ++r) v[u][r] = cmul(v[u][r], lo[r]);
#pragma unroll
          for (int h = 1; h < 4; ++h) {
            const double2 wh = h == 1 ? w4 : (h == 2 ? w8 : cmul(w8, w4));
            v[u][4 * h] = cmul(v[u][4 * h], wh);
#pragma unroll
            for (int r = 1; r < 4; ++r) v[u][4 * h + r] = cmul(v[u][4 * h + r], cmul(wh, lo[r]));
          }
        } else {
          double2 w[R];
          twiddle_powers<R>(twd(tw, qb, sign), w);
#pragma unroll
          for (int r = 1; r < R; ++r) v[u][r] = cmul(v[u][r], w[r]);
        }
      }
      dft_small<R>(v[u], sign);
      const int d = (j - jm) * R + jm;
#pragma unroll
      for (int r = 0; r < R; ++r) buf[pidx(d + r * Ns) ^ xo] = v[u][r];
    }
  }
  slice_sync<TP>(g);
}

// M-point transform of a slice, natural order in and out; radix 16 where it saves a pass.
// 1024 points take one pass of 16 and two of 8, in any order at the same cost (a run of 4096
// points in four CTAs 16.9 ms, with 8, 8, 16 or 8, 16, 8 16.5 and 17.7) and to the same error
// (one right-hand side within 7e-17 of the oracle).  16, 8, 8 is the order whose roundings
// leave a 1024-point run to t = 6 s the oracle's step sequence, 776 accepted steps and eta
// 1.2e-10 apart; with the others step control passes a threshold on the other side after
// a clipped step: 787 steps, 1.35e-9, which is the truncation error at rtol 1e-6.
template <int M>
__device__ __forceinline__ void slice_fft(double2* buf, int xo, const double2* __restrict__ tw, int tw_stride, int sign,
                                          int tid, int g, bool act) {
  if constexpr (M == 2048) {
    slice_pass<M, 8>(buf, xo, 1, tw, tw_stride, sign, tid, g, act);
    slice_pass<M, 16>(buf, xo, 8, tw, tw_stride, sign, tid, g, act);
    slice_pass<M, 16>(buf, xo, 128, tw, tw_stride, sign, tid, g, act);
  } else if constexpr (M == 1024) {
    slice_pass<M, 16>(buf, xo, 1, tw, tw_stride, sign, tid, g, act);
    slice_pass<M, 8>(buf, xo, 16, tw, tw_stride, sign, tid, g, act);
    slice_pass<M, 8>(buf, xo, 128, tw, tw_stride, sign, tid, g, act);
  } else if constexpr (M == 512) {
    slice_pass<M, 8>(buf, xo, 1, tw, tw_stride, sign, tid, g, act);
    slice_pass<M, 8>(buf, xo, 8, tw, tw_stride, sign, tid, g, act);
    slice_pass<M, 8>(buf, xo, 64, tw, tw_stride, sign, tid, g, act);
  } else if constexpr (M == 256) {
    slice_pass<M, 16>(buf, xo, 1, tw, tw_stride, sign, tid, g, act);
    slice_pass<M, 16>(buf, xo, 16, tw, tw_stride, sign, tid, g, act);
  } else if constexpr (M == 128) {
    slice_pass<M, 8>(buf, xo, 1, tw, tw_stride, sign, tid, g, act);
    slice_pass<M, 16>(buf, xo, 8, tw, tw_stride, sign, tid, g, act);
  } else {
    static_assert(M == 64, "slices of 64 to 2048 points");
    slice_pass<M, 8>(buf, xo, 1, tw, tw_stride, sign, tid, g, act);
    slice_pass<M, 8>(buf, xo, 8, tw, tw_stride, sign, tid, g, act);
  }
}

// A member's two slices, M/16 of the CTA's M/8 threads each.  Sixteen points a thread:
// three passes for 2048 points where eight points took four, and a barrier of one
// slice's warps only; a slice of up to 512 points is one warp's.
template <int M>
__device__ __forceinline__ void local_fft2(double2* A, double2* B, const double2* __restrict__ tw, int tw_stride, int sign) {
  constexpr int TP = M / 16;
  const int g = threadIdx.x / TP;
  slice_fft<M>(g ? B : A, 0, tw, tw_stride, sign, threadIdx.x % TP, g, true);
  __syncthreads();
}

// One in-place Stockham radix-R pass of a single slice by all M/8 threads, eight points
// each (half the threads, as in the pair, would leave the CTA's other warps idle).
template <int M, int R>
__device__ __forceinline__ void stockham_pass(double2* buf, int Ns, const double2* __restrict__ tw,
                                              int tw_stride, int sign) {
  constexpr int T = M / kPts;
  constexpr int NB = M / R;
  constexpr int BPT = kPts / R;
  double2 v[BPT][R];
  const int tid = threadIdx.x;
#pragma unroll
  for (int u = 0; u < BPT; ++u) {
    const int j = tid + u * T;
#pragma unroll
    for (int r = 0; r < R; ++r) v[u][r] = buf[pidx(j + r * NB)];
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < BPT; ++u) {
    const int j = tid + u * T;
    const int jm = j & (Ns - 1);
    if (Ns > 1) {
      const int qb = jm * (M / (Ns * R));
      double2 w[R];
      twiddle_powers<R>(twd(tw, qb * tw_stride, sign), w);
#pragma unroll
      for (int r = 1; r < R; ++r) v[u][r] = cmul(v[u][r], w[r]);
    }
    dft_small<R>(v[u], sign);
    const int idxD = (j - jm) * R + jm;
#pragma unroll
    for (int r = 0; r < R; ++r) buf[pidx(idxD + r * Ns)] = v[u][r];
  }
  __syncthreads();
}

// Local M-point transform of a single slice, natural order in and out: radix-8 passes
// while they divide, then one radix-4 or radix-2 pass
template <int M>
__device__ __forceinline__ void local_fft(double2* buf, const double2* __restrict__ tw, int tw_stride, int sign) {
  int Ns = 1;
  constexpr int L8 = (M >= 512) ? 3 : (M >= 64 ? 2 : 1);
  constexpr int rem = M / (1 << (3 * L8));
#pragma unroll
  for (int p = 0; p < L8; ++p) {
    stockham_pass<M, 8>(buf, Ns, tw, tw_stride, sign);
    Ns *= 8;
  }
  if constexpr (rem == 4) stockham_pass<M, 4>(buf, Ns, tw, tw_stride, sign);
  else if constexpr (rem == 2) stockham_pass<M, 2>(buf, Ns, tw, tw_stride, sign);
}

// Cross-CTA step of the distributed transform, as gather / C-point DFT / scatter:
// the M positions of the slice are shared out over the C*T threads of the cluster;
// the thread owning position i gathers the C values at i from every CTA's slice,
// applies the C-point DFT (forward: then the twiddles W_N^(i k1); inverse: the
// twiddles W_N^-(i k1) first) and stores output j into CTA j's slice at i.
// Every position is owned by exactly one thread of the cluster -- with sixteen CTAs by two
// neighbouring lanes, which have eight of its sixteen values each -- so the values are
// rewritten without a barrier after they were read: one cluster barrier before (the slices
// are complete) and one after.
// (A sum over sixteen peers for each point instead, with two barriers more and the products
// in shared memory, left sixteen CTAs slower than eight; now 16384 points on a slope take
// 359 us an RHS in sixteen and 430 in eight.)
template <int C>
struct Cross {
  static constexpr int H = C > kPts ? C / kPts : 1;   // threads to a position
  static constexpr int R = C / H;                     // values to a thread
  static constexpr int PER = kPts / R;                // positions to a thread
  static_assert(H == 1 || H == 2, "clusters of up to 16 CTAs");
  static __device__ __forceinline__ int half() { return H > 1 ? int(threadIdx.x) & (H - 1) : 0; }
  // the q-th position of this thread in CTA c; value e's CTA on the spectral and the physical side
  template <int T>
  static __device__ __forceinline__ int at(int c, int q) {
    return c * (T / H) + int(threadIdx.x) / H + q * (C * T / H);
  }
  static __device__ __forceinline__ int spectral(int e) { return e * H + half(); }
  static __device__ __forceinline__ int physical(int e) { return e + R * half(); }
};

// values v of one position from the spectral to the physical side, and back.  The twiddles
// are formed anew on each side: kept across the pointwise work they took the registers that
// its loads need.  With two threads to a position the 16-point DFT is two 8-point ones
// (even and odd CTAs) and a butterfly between the lanes; each lane stores only after the
// exchange, and so after its partner's loads.
__device__ __forceinline__ double2 lane_swap(double2 v) {
  return make_double2(__shfl_xor_sync(0xffffffffu, v.x, 1), __shfl_xor_sync(0xffffffffu, v.y, 1));
}
// x exp(sign 2 pi i n / 16), n = 0..7
template <int N16>
__device__ __forceinline__ double2 rot16(double2 a, int sign) {
  constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173, r = 0.70710678118654752440;
  constexpr double co[8] = {1.0, c1, r, s1, 0.0, -s1, -r, -c1}, si[8] = {0.0, s1, r, c1, 1.0, c1, r, s1};
  if constexpr (N16 == 0) return a;
  if constexpr (N16 == 4) return mul_pm_i(a, sign);
  const double sg = double(sign), c = co[N16], t = si[N16];
  return make_double2(c * a.x - sg * t * a.y, c * a.y + sg * t * a.x);
}
template <int N16 = 0>
__device__ __forceinline__ void lanes_in(double2* v, int h) {
  if constexpr (N16 < 8) {
    if (h) v[N16] = rot16<N16>(v[N16], +1);
    const double2 p = lane_swap(v[N16]);
    v[N16] = h ? csub(p, v[N16]) : cadd(v[N16], p);
    lanes_in<N16 + 1>(v, h);
  }
}
template <int N16 = 0>
__device__ __forceinline__ void lanes_out(double2* v, int h) {
  if constexpr (N16 < 8) {
    const double2 p = lane_swap(v[N16]);
    v[N16] = h ? rot16<N16>(csub(p, v[N16]), -1) : cadd(v[N16], p);
    lanes_out<N16 + 1>(v, h);
  }
}
// the position's twiddles: value e times W_N^(sign i spectral(e))
template <int C>
__device__ __forceinline__ void cross_twiddle(double2* v, const double2* __restrict__ tw, int i, int sign) {
  using X = Cross<C>;
  double2 w[X::R > 1 ? X::R : 2];
  twiddle_powers<X::R>(twd(tw, X::H * i, sign), w);
#pragma unroll
  for (int e = 1; e < X::R; ++e) v[e] = cmul(v[e], w[e]);
  if constexpr (X::H > 1) {
    if (X::half()) {
      const double2 w1 = twd(tw, i, sign);
#pragma unroll
      for (int e = 0; e < X::R; ++e) v[e] = cmul(v[e], w1);
    }
  }
}
template <int C>
__device__ __forceinline__ void cross_in(double2* v, const double2* __restrict__ tw, int i) {
  cross_twiddle<C>(v, tw, i, +1);
  dft_small<Cross<C>::R>(v, +1);
  if constexpr (Cross<C>::H > 1) lanes_in(v, Cross<C>::half());
}
template <int C>
__device__ __forceinline__ void cross_out(double2* v, const double2* __restrict__ tw, int i) {
  if constexpr (Cross<C>::H > 1) lanes_out(v, Cross<C>::half());
  dft_small<Cross<C>::R>(v, -1);
  cross_twiddle<C>(v, tw, i, -1);
}

template <int M, int C, int NBUF>
__device__ __forceinline__ void cross_gs(double2* A, double2* B, const double2* __restrict__ tw, int c, int sign) {
  using X = Cross<C>;
  constexpr int T = M / kPts;
  cg::cluster_group cl = cg::this_cluster();
  double2 va[X::PER][X::R], vb[X::PER][X::R];
  cl.sync();
#pragma unroll
  for (int q = 0; q < X::PER; ++q) {
    const int i = X::template at<T>(c, q);
#pragma unroll
    for (int e = 0; e < X::R; ++e) {
      const int r = sign > 0 ? X::spectral(e) : X::physical(e);
      va[q][e] = cl.map_shared_rank(A, r)[pidx(i)];
      if constexpr (NBUF == 2) vb[q][e] = cl.map_shared_rank(B, r)[pidx(i)];
    }
  }
#pragma unroll
  for (int q = 0; q < X::PER; ++q) {
    const int i = X::template at<T>(c, q);
    if (sign > 0) {
      cross_in<C>(va[q], tw, i);
      if constexpr (NBUF == 2) cross_in<C>(vb[q], tw, i);
    } else {
      cross_out<C>(va[q], tw, i);
      if constexpr (NBUF == 2) cross_out<C>(vb[q], tw, i);
    }
#pragma unroll
    for (int e = 0; e < X::R; ++e) {
      const int r = sign > 0 ? X::physical(e) : X::spectral(e);
      cl.map_shared_rank(A, r)[pidx(i)] = va[q][e];
      if constexpr (NBUF == 2) cl.map_shared_rank(B, r)[pidx(i)] = vb[q][e];
    }
  }
  cl.sync();
}

// dispatch on the cluster size
template <int M, int NBUF>
__device__ __forceinline__ void cross_step(double2* A, double2* B, const double2* __restrict__ tw, int C, int c, int sign) {
  if (C == 2) cross_gs<M, 2, NBUF>(A, B, tw, c, sign);
  else if (C == 4) cross_gs<M, 4, NBUF>(A, B, tw, c, sign);
  else if (C == 8) cross_gs<M, 8, NBUF>(A, B, tw, c, sign);
  else cross_gs<M, 16, NBUF>(A, B, tw, c, sign);
}

// cluster-wide barrier (block barrier when the member is a single CTA)
__device__ __forceinline__ void member_sync(int C) {
  if (C > 1) cg::this_cluster().sync();
  else __syncthreads();
}

// Forward FFT: physical block slice in buf -> spectral cyclic slice in buf.
template <int M>
__device__ __noinline__ void fft_forward(double2* buf, const double2* __restrict__ tw, int C, int c) {
  if (C > 1) cross_step<M, 1>(buf, buf, tw, C, c, -1);
  else __syncthreads();
  local_fft<M>(buf, tw, C, -1);
}

// Inverse FFT (unnormalised): spectral cyclic slice in buf -> physical block slice in buf.
template <int M>
__device__ __noinline__ void fft_inverse(double2* buf, const double2* __restrict__ tw, int C, int c) {
  __syncthreads();
  local_fft<M>(buf, tw, C, +1);
  if (C > 1) cross_step<M, 1>(buf, buf, tw, C, c, +1);
}

// Dual transforms: two M-point slices (A and B) in one sweep -- twice the
// independent work per thread, one set of twiddle loads and barriers for both.
template <int M>
__device__ __noinline__ void fft_forward2(double2* A, double2* B, const double2* __restrict__ tw, int C, int c) {
  if (C > 1) cross_step<M, 2>(A, B, tw, C, c, -1);
  else __syncthreads();
  local_fft2<M>(A, B, tw, C, -1);
}

template <int M>
__device__ __noinline__ void fft_inverse2(double2* A, double2* B, const double2* __restrict__ tw, int C, int c) {
  __syncthreads();
  local_fft2<M>(A, B, tw, C, +1);
  if (C > 1) cross_step<M, 2>(A, B, tw, C, c, +1);
}

// The local (in-CTA) part of a distributed transform alone, for callers that do the
// cross-CTA step themselves: sign +1 is the inverse's first half, -1 the forward's
// second half.  Barrier on entry (the caller wrote the slices) and on exit.
template <int M>
__device__ __noinline__ void fft_local(double2* A, const double2* __restrict__ tw, int C, int sign) {
  __syncthreads();
  local_fft<M>(A, tw, C, sign);
}
template <int M>
__device__ __noinline__ void fft_local2(double2* A, double2* B, const double2* __restrict__ tw, int C, int sign) {
  __syncthreads();
  local_fft2<M>(A, B, tw, C, sign);
}

}  // namespace hwdev
