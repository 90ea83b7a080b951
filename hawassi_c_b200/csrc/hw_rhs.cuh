// hw_rhs.cuh -- what the pseudo-spectral Hamiltonian right-hand sides of one member
// share, executed by the CTAs of one thread-block cluster (or one CTA): stage values,
// the ownership of Hermitian pairs, packing and splitting of two real signals in one
// complex transform, the influx signal.  hw_rhs_fast.cuh holds HS2 on a flat bottom,
// hw_rhs_gen.cuh the rest.
#pragma once

#include "hw_device.cuh"

namespace hwdev {

// Fehlberg coefficients (GSL rkf45)
__device__ constexpr double RK_ah[5] = {1.0 / 4.0, 3.0 / 8.0, 12.0 / 13.0, 1.0, 1.0 / 2.0};
__device__ constexpr double RK_b3[2] = {3.0 / 32.0, 9.0 / 32.0};
__device__ constexpr double RK_b4[3] = {1932.0 / 2197.0, -7200.0 / 2197.0, 7296.0 / 2197.0};
__device__ constexpr double RK_b5[4] = {8341.0 / 4104.0, -32832.0 / 4104.0, 29440.0 / 4104.0, -845.0 / 4104.0};
__device__ constexpr double RK_b6[5] = {-6080.0 / 20520.0, 41040.0 / 20520.0, -28352.0 / 20520.0, 9295.0 / 20520.0,
                                        -5643.0 / 20520.0};
__device__ constexpr double RK_c1 = 902880.0 / 7618050.0;
__device__ constexpr double RK_c3 = 3953664.0 / 7618050.0;
__device__ constexpr double RK_c4 = 3855735.0 / 7618050.0;
__device__ constexpr double RK_c5 = -1371249.0 / 7618050.0;
__device__ constexpr double RK_c6 = 277020.0 / 7618050.0;
__device__ constexpr double RK_ec1 = 1.0 / 360.0;
__device__ constexpr double RK_ec3 = -128.0 / 4275.0;
__device__ constexpr double RK_ec4 = -2197.0 / 75240.0;
__device__ constexpr double RK_ec5 = 1.0 / 50.0;
__device__ constexpr double RK_ec6 = 2.0 / 55.0;

// the stage input of an RK stage: zs = y + h sum_j b_sj k_j (s = 2..6), or zs = y
// itself (s = 1: the state a first or last derivative is evaluated at; s = 0: zs holds it)
struct StageSrc {
  const double2* y;
  const double2* k[5];
  int s;
  int sig;      // entry of the step's influx signals at this stage's time (-1: not formed)
  double h;
};

// IEEE products and sums without fused multiply-add: the stepper's arithmetic
// rounds like GSL's (compiled without contraction)
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }

// one element of the stage input of stage S (1: the state itself), in GSL rkf45's
// expression forms, from values already loaded: k[j] is k_(j+1)
template <int S>
__device__ __forceinline__ double stage_comb(double y, double h, const double* k) {
  if constexpr (S == 1) return y;
  else if constexpr (S == 2) return radd(y, rmul(rmul(RK_ah[0], h), k[0]));
  else if constexpr (S == 3) return radd(y, rmul(h, radd(rmul(RK_b3[0], k[0]), rmul(RK_b3[1], k[1]))));
  else {
    auto b = [](int j) { return S == 4 ? RK_b4[j] : (S == 5 ? RK_b5[j] : RK_b6[j]); };
    double v = radd(rmul(b(0), k[0]), rmul(b(1), k[1]));
#pragma unroll
    for (int j = 2; j < S - 1; ++j) v = radd(v, rmul(b(j), k[j]));
    return radd(y, rmul(h, v));
  }
}

// the operands of stage value q: loaded apart from their use, so that a thread has
// those of several values in flight
template <int S>
struct StageOps {
  double2 y, k[S > 1 ? S - 1 : 1];
  __device__ __forceinline__ void load(const double2* __restrict__ ys, const double2* const* ks, int q) {
    y = ys[q];
#pragma unroll
    for (int j = 0; j < S - 1; ++j) k[j] = ks[j][q];
  }
  __device__ __forceinline__ double2 value(double h) const {
    double kx[S > 1 ? S - 1 : 1], ky[S > 1 ? S - 1 : 1];
#pragma unroll
    for (int j = 0; j < S - 1; ++j) {
      kx[j] = k[j].x;
      ky[j] = k[j].y;
    }
    return make_double2(stage_comb<S>(y.x, h, kx), stage_comb<S>(y.y, h, ky));
  }
};

// the stepper's buffers: y, ynew, k1..k6, kout (accepted steps swap pointers)
struct Bufs {
  double2* y;
  double2* yn;
  double2* k[7];
};

// Scratch of one CTA in static shared memory, beside the transform slices.  What every
// thread needs alike (the stage description, the buffers) stands here once, and not in
// each thread's local memory: with 256 threads and kilobyte frames that overflows the L1
// cache, and every access to it waited for L2.
constexpr int kRed = 48;
constexpr int kRedPv = 40, kRedPs = 41;   // influx signals at the stage time
template <int M>
struct Scratch {
  double red[kRed];
  StageSrc stg;         // stage input of the coming RHS (stg.s = 0: zs holds it)
  Bufs bufs;
  int full;             // dz is written outside the alias band too (as zeros)
  double2 sig[7];       // influx signal and its integral at the step's times: k1, stages 2..6, kout
  // breaking (CTA 0's counters serve the member; live in every CTA)
  int npk, above;       // crests that passed the test, eta above the threshold somewhere
  int live;             // some node breaks: the force is not zero
  int idle, iter;       // no crest is tracked and every record clear (-1: not known); ITERbdt
  int ncand;
  unsigned short cand[M];   // grid points of this CTA's threads above the breaking threshold
};

// what a device function of the member is given, by value (a few registers)
template <int M>
struct Ctx {
  static constexpr int T = M / kPts;
  const DevMember& d;
  double2* buf;   // M-point transform slice in shared memory; the second one follows it
  Scratch<M>* sc;
  int c;          // rank of this CTA in the member's cluster
  __device__ __forceinline__ double2* buf2() const { return buf + padded(M); }
};

// The Hermitian pairs {k, N-k} of the member, each owned by one thread wherever spectral
// values are formed: CTA c takes the first half of its slice, i < M / 2, with the
// partners, which lie in the second half of CTA (C - c) mod C.  Positions 0 and M / 2
// of CTA 0 are their own partners; they go as one "pair" of two such points (self).
// The owner is the same in every phase, so the RK vectors need no barrier between the
// phase that writes them and the ones that read them.
struct PairAt {
  int i, j, p, pp;   // slice indices and positions of the two points
  bool self;
};
template <int M>
__device__ __forceinline__ PairAt pair_at(int c, int cq, int i) {
  PairAt r;
  r.i = i;
  r.self = c == 0 && i == 0;
  r.j = r.self ? M / 2 : (c == 0 ? M - i : M - 1 - i);
  r.p = c * M + r.i;
  r.pp = cq * M + r.j;
  return r;
}

// dynamic shared memory of the 1D kernels of slice M: two padded FFT slices (no more:
// what the SM does not give to shared memory serves as L1 cache)
__host__ __device__ constexpr size_t slice_smem_bytes(int m) { return 2 * size_t(padded(m)) * sizeof(double2); }

template <int M>
__device__ __forceinline__ Ctx<M> make_ctx(const DevMember& d, double2* smem, Scratch<M>& sc, int rank) {
  return Ctx<M>{d, smem, &sc, rank};
}

#define HW_FOREACH(X)                            \
  _Pragma("unroll") for (int u = 0; u < kPts; ++u)  \
    if (const int idx = int(threadIdx.x) + u * Ctx<M>::T, p = (X).c * M + idx; true)

// permuted position of the wavenumber N - kk, for the spectral entry at slice index idx
template <int M>
__device__ __forceinline__ int partner_pos(Ctx<M> X, int idx) {
  const DevMember& d = X.d;
  const int kk = X.c + (idx << d.logC);
  const int kp = (d.N - kk) & (d.N - 1);
  return (kp & (d.C - 1)) * M + (kp >> d.logC);
}

// Hermitian part (A[k] + conj A[N-k]) / 2: the spectrum whose inverse transform is
// the real part of the inverse transform of A (the reference keeps only the real part).
__device__ __forceinline__ double2 herm(double2 a, double2 ap) {
  return make_double2(0.5 * (a.x + ap.x), 0.5 * (a.y - ap.y));
}
// (A + i B) * s
__device__ __forceinline__ double2 pack(double2 a, double2 b, double s) {
  return make_double2((a.x - b.y) * s, (a.y + b.x) * s);
}
// spectra of the real and imaginary input parts from Z = FFT(a + i b)
__device__ __forceinline__ double2 split_re(double2 z, double2 zp) {
  return make_double2(0.5 * (z.x + zp.x), 0.5 * (z.y - zp.y));
}
__device__ __forceinline__ double2 split_im(double2 z, double2 zp) {
  return make_double2(0.5 * (z.y + zp.y), -0.5 * (z.x - zp.x));
}
// prod_1ik (1d/functions.c:297): (i a) * B
__device__ __forceinline__ double2 mul_ik(double a, double2 b) {
  return make_double2((0.0 * b.x) - (a * b.y), (0.0 * b.y) + (a * b.x));
}

// forward FFT of the physical slice in buf, then f(u, idx, p, Z, Zpartner) for each
// of this thread's spectral points (Zpartner read from the owning CTA by DSMEM)
template <int M, class F>
__device__ __forceinline__ void fft_forward_split(Ctx<M> X, F&& f) {
  const DevMember& d = X.d;
  fft_forward<M>(X.buf, d.tw, d.C, X.c);
  const double2* pb = X.buf;
  if (d.C > 1) {
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    pb = cl.map_shared_rank(X.buf, (d.C - X.c) & (d.C - 1));
  }
  double2 Z[kPts], Zp[kPts];
  HW_FOREACH(X) {
    (void)p;
    Z[u] = X.buf[pidx(idx)];
    const int jp = X.c == 0 ? ((M - idx) & (M - 1)) : (M - 1 - idx);
    Zp[u] = pb[pidx(jp)];
  }
  member_sync(d.C);
  HW_FOREACH(X) { f(u, idx, p, Z[u], Zp[u]); }
}

// inverse FFT of the spectral slice in buf; g(u, idx, p, v) for each physical point
template <int M, class G>
__device__ __forceinline__ void fft_inverse_then(Ctx<M> X, G&& g) {
  const DevMember& d = X.d;
  fft_inverse<M>(X.buf, d.tw, d.C, X.c);
  HW_FOREACH(X) { g(u, idx, p, X.buf[pidx(idx)]); }
}

// natural cubic spline evaluation (GSL cspline + bsearch index rule) of the influx
// signal and its running integral at t.  Both need the same interval: every value of a
// guessed one is loaded at once, and the guess moves on if the samples' times ask for it.
__device__ __forceinline__ double2 influx_at(const DevMember& d, double t) {
  const double nan = __longlong_as_double(0x7ff8000000000000ULL);
  if (!(t >= d.tt0 && t <= d.ttl)) return make_double2(nan, nan);
  const int n = d.n_in;
  int lo = int((t - d.tt0) / d.tth);
  lo = lo < 0 ? 0 : (lo > n - 2 ? n - 2 : lo);
  double xl, xh, y0, y1, c0, c1, s0, s1, e0, e1;
  for (;;) {
    xl = d.tt[lo]; xh = d.tt[lo + 1];
    y0 = d.ins[lo]; y1 = d.ins[lo + 1]; c0 = d.insc[lo]; c1 = d.insc[lo + 1];
    s0 = d.skw[lo]; s1 = d.skw[lo + 1]; e0 = d.skwc[lo]; e1 = d.skwc[lo + 1];
    if (lo > 0 && xl > t) --lo;
    else if (lo < n - 2 && xh <= t) ++lo;
    else break;
  }
  const double h = xh - xl, delx = t - xl;
  auto cubic = [&](double a, double b, double ci, double cp) {
    const double dy = b - a;
    const double bb = dy / h - h * (cp + 2.0 * ci) / 3.0;
    const double dd = (cp - ci) / (3.0 * h);
    return a + delx * (bb + delx * (ci + delx * dd));
  };
  return make_double2(cubic(y0, y1, c0, c1), cubic(s0, s1, e0, e1));
}

// breaking hooks (implemented in hw_breaking.cuh)
template <int M>
__device__ __forceinline__ void breaking_reset(Ctx<M> X);
template <int M>
__device__ __forceinline__ void breaking_scan(Ctx<M> X, const double2* PE, const double* Heta, int hs);
template <int M>
__device__ __forceinline__ void breaking_lead(Ctx<M> X, double t, const double2* PE, const double* Heta, int hs);
template <int M>
__device__ __noinline__ void breaking_force(Ctx<M> X, const double2* PE, const double2* AEadj, double2* Rb);
// HS2 on a flat bottom (hw_rhs_fast.cuh) and every other right-hand side (hw_rhs_gen.cuh)
template <int M>
__device__ __noinline__ void rhs_hs2_flat(Ctx<M> X, double t, double2* __restrict__ dz);
template <int M>
__device__ __noinline__ void rhs_gen(Ctx<M> X, double t, double2* __restrict__ dz);

// One RHS evaluation dz = f(t, zs), zs = [eta^ | u^] (permuted spectral, 2N).
template <int M>
__device__ __forceinline__ void rhs_eval(Ctx<M> X, double t, double2* __restrict__ dz) {
  if (X.d.model == 2 && X.d.flat) rhs_hs2_flat<M>(X, t, dz);
  else rhs_gen<M>(X, t, dz);
}

}  // namespace hwdev
