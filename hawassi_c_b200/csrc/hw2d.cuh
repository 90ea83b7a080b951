// hw2d.cuh -- HAWASSI 2D right-hand sides: what every bottom and order shares, the
// passes of a flat bottom (rhs_AB1/AB2/AB3_2DF_uv, 2d/fun_odesolver.c:4404-4734), and
// the rkf45 attempt's stepper kernels.
//
// A 2D transform is a row pass and a column pass.  Row passes run one CTA per row
// pair {r, Ny-r} (with {0, Ny/2} sharing a CTA): that pair holds every point's
// conjugate mirror (-ky, -kx), so the Hermitian operations the reference
// performs on whole arrays (fftwcomplex_2d_sym before an inverse transform, real
// parts after it, the split of two real fields packed into one complex transform)
// are CTA-local.  Column passes run one CTA per column pair {2c, 2c+1}.  A CTA holds
// slices (rows or columns) of M points in shared memory, each transformed by M/16
// threads.
//
// What an RHS cannot do without is fewer transforms than its terms name, because
// they are linear: delu H2^ and delv H2^ (and the cubic ones) enter only as their sum,
// whose operator part is L (eta L phi)^ of one real field; L phi is the sum of M0u
// and M0v in physical space; the damping of u, v, and of eta less the source, are added
// where the adjusted terms are in physical space.  HS2 on a flat bottom:
//   A row   (eta, u), (v, L phi)                                      -> inverse rows
//   B col   inverse -> eta u, eta v, eta L phi, deletaH2, two to a field -> forward
//   C row   forward, split -> S(i kx deletaH2^), S(i ky deletaH2^), S(delu + delv) -> inverse
//   D col   inverse, x ChiAdj, with the damping and the source        -> forward
//   E row   forward -> dt Z (x aal)
// is 13 field passes (a field: two slices in one direction) where one of the terms each
// takes 24.  HS3 adds one round trip between C and D, HS1 leaves C and D out.
// Passes whose fields are independent (A, D, E) run a CTA per field, so that several
// share an SM.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

#include "hw_fft.cuh"

namespace hw2d {

using hwdev::cadd;
using hwdev::cconj;
using hwdev::cmul;
using hwdev::cscale;
using hwdev::csub;
using hwdev::padded;
using hwdev::pidx;

constexpr double kGrav = 9.80665;

struct Tab2 {
  int nx, ny, n, model, nt, chi_one, has_src;
  double fac_src;               // 1 (Uni+/-) or 2 (Bi)
  const double* kx;             // [nx]
  const double* ky;             // [ny]
  const double* c2g;            // C2d^2 / g
  const double* l2d;
  const double* aal;
  const double* damp;           // 7 Cpeak fbdy.charac
  const double* chi;            // ChiAdj
  const double* gsrc;           // newGam
  const double* ssrc;           // +-SkewGam (sign of the propagation)
  double t0, tl, dts;           // first, last line-signal time, second minus first
  const double* tsig;           // [nt]
  const double* sig;            // [ny][nt] line signals and their spline coefficients
  const double* sigc;
  const double* sigs;
  const double* sigsc;
  const double2* twx;           // exp(-2 pi i q / nx)
  const double2* twy;           // exp(-2 pi i q / ny)
  int var;
  const double* wallchar;       // dominfo.wallchar (harbour walls), nullptr: none
  const double* c2d;            // Oprt.C2d (flat bottom with walls only)
  int refl_one;                 // flat bottom, refl_coef == 1: fun_delphiH1hat's flux branch
  const double* gwx;            // fun_gradient(wallchar) (refl_one only)
  const double* gwy;
  // varying bottom: K reference depths (HSSgen_2depth, HSSgen_3depth, and the same sum over
  // K depths of the plain K-reference and the learned operators), rows [K][N] of the
  // weights (physical), C^2 and Omega^2 (spectral); var = nk = 0 on a flat bottom
  int nk;
  const double* gk;
  const double* ck;
  const double* ok;
};

struct Work2 {
  double2* z;                   // stage input, 3 fields
  double2* R;                   // row pass -> column pass
  double2* Q;                   // column pass -> row pass
  double2* D;                   // spectrum of damping of eta less the source (breaking, ChiAdj = 1);
                                // of damping of u and v (ChiAdj = 1)
  double2* W;                   // C -> D, 3 fields
  double2* V;                   // -> E, 3 fields
  double2* T;                   // left half of every row: delu + delv (0), deletaH (1), L of the
                                // operand's kept part (2)
  double* insig;                // [ny] line signal at the stage time
  double* insigs;
  double* part;                 // per-block maxima of the error ratio
  double* phys;                 // eta, u, v in physical space (3 real fields)
  double* op;                   // operand of an HSS, L phi in physical space (2 real fields)
  double2* H1;                  // delphiH1^ (varying bottom; flat bottom with walls)
  double2* WP;                  // flat bottom with walls: the round trip of (C u^, C v^)
  double2* dph;                 // breaking: delphiH^ as the assembly forms it (nullptr: off)
};

// device control block of the stepper (one per engine)
struct Ctl2 {
  double t, h, h0, t1, t_direct, eps_abs, eps_rel;
  int final_step, done, status, cur, k1i, need_k1, need_kout, attempts;
  long long rhs, acc, rej;
  // kinematic breaking on: every evolve_apply evaluates its own dydt_in and every
  // attempt its dydt_out (mode 8) before the step control, as gsl_odeiv2 does,
  // since each RHS past tprev advances the breaking state
  int brk;
};

enum { kOk = 0, kNonFinite = 1, kStepFailed = 2, kBreakCapacity = 3 };
// RHS launch conditions
enum { kAlways = 0, kIfK1 = 1, kIfStage = 2, kIfKout = 3 };

struct RK2 {
  double2* y[2];                // state, 3 fields each
  double2* kk[2];               // k1 / kout pair
  double2* ks[5];               // k2..k6
};

__device__ constexpr double A2_ah[5] = {1.0 / 4.0, 3.0 / 8.0, 12.0 / 13.0, 1.0, 1.0 / 2.0};
__device__ constexpr double A2_b3[2] = {3.0 / 32.0, 9.0 / 32.0};
__device__ constexpr double A2_b4[3] = {1932.0 / 2197.0, -7200.0 / 2197.0, 7296.0 / 2197.0};
__device__ constexpr double A2_b5[4] = {8341.0 / 4104.0, -32832.0 / 4104.0, 29440.0 / 4104.0, -845.0 / 4104.0};
__device__ constexpr double A2_b6[5] = {-6080.0 / 20520.0, 41040.0 / 20520.0, -28352.0 / 20520.0, 9295.0 / 20520.0,
                                        -5643.0 / 20520.0};
__device__ constexpr double A2_c[5] = {902880.0 / 7618050.0, 3953664.0 / 7618050.0, 3855735.0 / 7618050.0,
                                       -1371249.0 / 7618050.0, 277020.0 / 7618050.0};
__device__ constexpr double A2_ec[5] = {1.0 / 360.0, -128.0 / 4275.0, -2197.0 / 75240.0, 1.0 / 50.0, 2.0 / 55.0};

__device__ __forceinline__ bool rhs_active(const Ctl2* c, int cond) {
  if (cond == kAlways) return true;
  if (cond == kIfKout) return c->need_kout != 0;
  if (c->done) return false;
  if (cond == kIfK1) return c->need_k1 != 0;
  return true;
}

// ---------------------------------------------------------------------------
// M-point transforms of slices in shared memory
// ---------------------------------------------------------------------------
// Position i of slice s: the swizzle of the 1D slices, odd slices turned by half a
// 128-byte group, so that the two columns of a pair, which lie side by side in memory
// and go to neighbouring slices, meet no bank conflict.
__device__ __forceinline__ int sidx(int M, int s, int i) { return s * M + (pidx(i) ^ ((s & 1) << 2)); }
__device__ __forceinline__ double2 slot(const double2* sm, int M, int s, int i) { return sm[sidx(M, s, i)]; }
__device__ __forceinline__ void put(double2* sm, int M, int s, int i, double2 v) { sm[sidx(M, s, i)] = v; }

// threads of a CTA that transforms two slices at a time, or four (1024 points; on
// shorter slices the threads that no transform needs share the pointwise work: at
// 256 x 128, M/16 threads a slice and no more took 65 us an RHS against 39), and the
// CTAs that an SM's registers hold at 128 a thread (16 points and their twiddles).
// 256 and 512 threads at 1024 points, one CTA less an SM, took 764 us an RHS against 665.
__host__ __device__ constexpr int ctas(int threads) { return 512 / threads; }
constexpr int kThr2 = 128, kThr4 = 256;

// slices [s0, s0 + ns) by a CTA of NT threads, NT / (M/16) at a time; CTA-wide
// barriers on entry and exit (the phases around read and write every slice).  Sixteen
// points a thread: two passes of radix 16 for 256 points, three for 512 and 1024 where
// eight points a thread took three and four, and no barrier wider than two warps.
template <int M, int NT>
__device__ __forceinline__ void fft_slices(double2* sm, int s0, int ns, const double2* __restrict__ tw, int sign) {
  constexpr int TP = M / 16, G = NT / TP;
  const int g = threadIdx.x / TP, tid = threadIdx.x % TP;
  __syncthreads();
  for (int base = 0; base < ns; base += G) {
    const int s = s0 + base + g;
    const bool act = base + g < ns;
    if (TP > 32 && !act) break;
    hwdev::slice_fft<M>(sm + s * M, (s & 1) << 2, tw, 1, sign, tid, g, act);
  }
  __syncthreads();
}

// global -> shared copies without registers: every copy of a phase is in flight at once
__device__ __forceinline__ void copy16(double2* dst, const double2* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---------------------------------------------------------------------------
// row-pair geometry and the Hermitian operators
// ---------------------------------------------------------------------------
struct Pair {
  int r[2];      // rows held (slice 2f + k holds row r[k] of field f)
  int flip;      // the mirror of row r[k] is r[k ^ flip]
  __device__ __forceinline__ int row(int k) const { return k ? r[1] : r[0]; }
};

__device__ __forceinline__ Pair row_pair(int b, int Ny) {
  Pair p;
  p.flip = b != 0;
  p.r[0] = b;
  p.r[1] = b == 0 ? Ny / 2 : Ny - b;
  return p;
}

// columns j and Nx - j of both rows: four points, each other's mirrors.  The
// reference's symmetrisation takes the right half of a row from the left one, so what
// is formed spectrally is formed at s = 0 alone and conjugated; columns 0 and Nx / 2,
// their own mirrors, go as one quad (self) of which both are formed.
struct Quad {
  int r[2], cc[2], flip;
  bool self;
  __device__ __forceinline__ Quad(const Pair& P, int j, int Nx) {
    r[0] = P.r[0];
    r[1] = P.r[1];
    flip = P.flip;
    self = j == 0;
    cc[0] = j;
    cc[1] = self ? Nx / 2 : Nx - j;
  }
  __device__ __forceinline__ bool has(int s) const { return s == 0 || self; }
  __device__ __forceinline__ size_t at(int k, int s, int Nx) const { return (size_t)r[k] * Nx + cc[s]; }
};

// spectra of the two real fields packed in slices s0, s0 + 1, at point (k, s)
__device__ __forceinline__ void split_at(const double2* sm, int M, int s0, const Quad& Q, int k, int s, double2& A,
                                         double2& B) {
  const double2 z = slot(sm, M, s0 + k, Q.cc[s]);
  const double2 m = slot(sm, M, s0 + (k ^ Q.flip), Q.cc[Q.self ? s : s ^ 1]);
  A = make_double2(0.5 * (z.x + m.x), 0.5 * (z.y - m.y));
  B = make_double2(0.5 * (z.y + m.y), -0.5 * (z.x - m.x));
}

// the reference's fftwcomplex_2d_sym (S) at a point of column 0 (s = 0) or Nx / 2, or
// (herm) the Hermitian part of it, which the real part of the inverse transform sees
__device__ __forceinline__ double2 self_sym(double2 a, double2 m, int r, int s, int Ny, bool herm) {
  if (r == 0 || r == Ny / 2) return make_double2(a.x, 0.0);
  if (s == 0) return r < Ny / 2 ? a : cconj(m);
  return herm ? make_double2(0.5 * (a.x + m.x), 0.5 * (a.y - m.y)) : a;
}

// E(S(x)) + i E(S(y)) into slices s0, s0 + 1 at the quad's points; x[k][s] for s = 0
// (and 1 in a self quad)
__device__ __forceinline__ void emit_pack(double2* sm, int M, int s0, const Quad& Q, int Ny, const double2 x[2][2],
                                          const double2 y[2][2]) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (!Q.self) {
      const double2 a = x[k][0], b = y[k][0], c = Q.flip ? x[k ^ 1][0] : x[k][0], d = Q.flip ? y[k ^ 1][0] : y[k][0];
      put(sm, M, s0 + k, Q.cc[0], make_double2(a.x - b.y, a.y + b.x));
      put(sm, M, s0 + k, Q.cc[1], make_double2(c.x + d.y, d.x - c.y));
    } else {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const double2 a = self_sym(x[k][s], Q.flip ? x[k ^ 1][s] : x[k][s], Q.r[k], s, Ny, true);
        const double2 b = self_sym(y[k][s], Q.flip ? y[k ^ 1][s] : y[k][s], Q.r[k], s, Ny, true);
        put(sm, M, s0 + k, Q.cc[s], make_double2(a.x - b.y, a.y + b.x));
      }
    }
  }
}
// S(x) (not its Hermitian part) into slices s0, s0 + 1
__device__ __forceinline__ void emit_sym(double2* sm, int M, int s0, const Quad& Q, int Ny, const double2 x[2][2]) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (!Q.self) {
      put(sm, M, s0 + k, Q.cc[0], x[k][0]);
      put(sm, M, s0 + k, Q.cc[1], cconj(Q.flip ? x[k ^ 1][0] : x[k][0]));
    } else {
#pragma unroll
      for (int s = 0; s < 2; ++s)
        put(sm, M, s0 + k, Q.cc[s], self_sym(x[k][s], Q.flip ? x[k ^ 1][s] : x[k][s], Q.r[k], s, Ny, false));
    }
  }
}

// split Z = FFT(a + i b) at a point given Z there (z) and at its mirror (zm)
__device__ __forceinline__ void split2(double2 z, double2 zm, double2& A, double2& B) {
  A = make_double2(0.5 * (z.x + zm.x), 0.5 * (z.y - zm.y));
  B = make_double2(0.5 * (z.y + zm.y), -0.5 * (z.x - zm.x));
}

__device__ __forceinline__ double2 zero2() { return make_double2(0.0, 0.0); }
// mul by -i s: (x, y) -> (s y, -s x)
__device__ __forceinline__ double2 mul_mi(double2 a, double s) { return make_double2(s * a.y, -s * a.x); }
// mul by +i s
__device__ __forceinline__ double2 mul_pi(double2 a, double s) { return make_double2(-s * a.y, s * a.x); }

// GSL natural cubic spline evaluation of a row's line signal and its quadrature at x
// (the bsearch's interval: a guess from the even spacing of the samples, moved on where
// their times ask for it)
__device__ __forceinline__ double2 line_signal(const Tab2& tb, int r, double x) {
  const double nan = __longlong_as_double(0x7ff8000000000000ULL);
  if (x < tb.t0 || x > tb.tl || x != x) return make_double2(nan, nan);
  const int n = tb.nt;
  const size_t o = (size_t)r * n;
  int lo = (int)((x - tb.t0) / tb.dts);
  lo = lo < 0 ? 0 : (lo > n - 2 ? n - 2 : lo);
  double xl, xh, y0, y1, c0, c1, s0, s1, e0, e1;
  for (;;) {
    xl = tb.tsig[lo]; xh = tb.tsig[lo + 1];
    y0 = tb.sig[o + lo]; y1 = tb.sig[o + lo + 1]; c0 = tb.sigc[o + lo]; c1 = tb.sigc[o + lo + 1];
    s0 = tb.sigs[o + lo]; s1 = tb.sigs[o + lo + 1]; e0 = tb.sigsc[o + lo]; e1 = tb.sigsc[o + lo + 1];
    if (lo > 0 && xl > x) --lo;
    else if (lo < n - 2 && xh <= x) ++lo;
    else break;
  }
  const double h = xh - xl, dx = x - xl;
  auto cubic = [&](double a, double b, double ci, double cip) {
    const double dy = b - a;
    const double bi = dy / h - h * (cip + 2.0 * ci) / 3.0;
    const double di = (cip - ci) / (3.0 * h);
    return a + dx * (bi + dx * (ci + dx * di));
  };
  return make_double2(cubic(y0, y1, c0, c1), cubic(s0, s1, e0, e1));
}

// modes: 0 direct RHS, 1 k1 (dydt_in), 2..6 the rkf45 stages, 7 k_out after an
// accepted step (reused as the next k1), 8 dydt_out of the attempt's candidate
// state at t + h before the step control (breaking runs)
__device__ __forceinline__ double stage_time(const Ctl2* c, int mode) {
  if (mode == 0) return c->t_direct;
  if (mode == 1 || mode == 7) return c->t;
  if (mode == 8) return c->t + c->h0;
  return c->t + A2_ah[mode - 2] * c->h0;
}

// IEEE products and sums without fused multiply-add (GSL's rounding)
__device__ __forceinline__ double rm2(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ra2(double a, double b) { return __dadd_rn(a, b); }

// stage input at element q (3n double2 per state): GSL rkf45's expression forms
__device__ __forceinline__ double2 stage_value(const RK2& B, const Ctl2* c, int mode, size_t q) {
  if (mode == 8) return B.y[c->cur ^ 1][q];
  const double2 y = B.y[c->cur][q];
  if (mode <= 1 || mode == 7) return y;
  const double h = c->h0;
  const double2 a = B.kk[c->k1i][q];
  if (mode == 2) {
    const double f = rm2(A2_ah[0], h);
    return make_double2(ra2(y.x, rm2(f, a.x)), ra2(y.y, rm2(f, a.y)));
  }
  const double2 b = B.ks[0][q];
  if (mode == 3)
    return make_double2(ra2(y.x, rm2(h, ra2(rm2(A2_b3[0], a.x), rm2(A2_b3[1], b.x)))),
                        ra2(y.y, rm2(h, ra2(rm2(A2_b3[0], a.y), rm2(A2_b3[1], b.y)))));
  const double2 c3 = B.ks[1][q];
  if (mode == 4)
    return make_double2(
        ra2(y.x, rm2(h, ra2(ra2(rm2(A2_b4[0], a.x), rm2(A2_b4[1], b.x)), rm2(A2_b4[2], c3.x)))),
        ra2(y.y, rm2(h, ra2(ra2(rm2(A2_b4[0], a.y), rm2(A2_b4[1], b.y)), rm2(A2_b4[2], c3.y)))));
  const double2 c4 = B.ks[2][q];
  if (mode == 5)
    return make_double2(
        ra2(y.x, rm2(h, ra2(ra2(ra2(rm2(A2_b5[0], a.x), rm2(A2_b5[1], b.x)), rm2(A2_b5[2], c3.x)),
                            rm2(A2_b5[3], c4.x)))),
        ra2(y.y, rm2(h, ra2(ra2(ra2(rm2(A2_b5[0], a.y), rm2(A2_b5[1], b.y)), rm2(A2_b5[2], c3.y)),
                            rm2(A2_b5[3], c4.y)))));
  const double2 c5 = B.ks[3][q];
  return make_double2(
      ra2(y.x, rm2(h, ra2(ra2(ra2(ra2(rm2(A2_b6[0], a.x), rm2(A2_b6[1], b.x)), rm2(A2_b6[2], c3.x)),
                              rm2(A2_b6[3], c4.x)),
                          rm2(A2_b6[4], c5.x)))),
      ra2(y.y, rm2(h, ra2(ra2(ra2(ra2(rm2(A2_b6[0], a.y), rm2(A2_b6[1], b.y)), rm2(A2_b6[2], c3.y)),
                              rm2(A2_b6[3], c4.y)),
                          rm2(A2_b6[4], c5.y)))));
}

// the buffer an RHS of the given mode writes
__device__ __forceinline__ double2* rhs_out(const RK2& rk, const Ctl2* ctl, int mode, double2* direct_out) {
  if (mode == 0) return direct_out;
  if (mode == 1) return rk.kk[ctl->k1i];
  if (mode == 7 || mode == 8) return rk.kk[ctl->k1i ^ 1];
  return rk.ks[mode - 2];
}

// ---------------------------------------------------------------------------
// Stage input z = y + h sum_j b_sj k_j, a streaming pass ahead of the first row pass (mode 1
// and 7: z = y).  It and the combination move the points inside the alias mask alone:
// outside it every k_j is zero, so z and both states are what they were when the run
// began, which is when k2_spread writes them.  Bound by memory: at 1024^2 points, 39 in a
// hundred of them inside, a right-hand side with its stage took 670 us, 650 so.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
k2_stage(const double* __restrict__ aal, RK2 rk, Work2 w, const Ctl2* __restrict__ ctl, int mode, int cond, size_t n) {
  if (!rhs_active(ctl, cond)) return;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
    if (aal[q] == 0.0) continue;
#pragma unroll
    for (int f = 0; f < 3; ++f) w.z[f * n + q] = stage_value(rk, ctl, mode, f * n + q);
  }
}

// the points outside the alias mask, in the stage input and the other state
__global__ void __launch_bounds__(256)
k2_spread(const double* __restrict__ aal, RK2 rk, Work2 w, const Ctl2* __restrict__ ctl, size_t n) {
  if (ctl->done) return;
  const double2* __restrict__ y = rk.y[ctl->cur];
  double2* __restrict__ yn = rk.y[ctl->cur ^ 1];
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
    if (aal[q] != 0.0) continue;
#pragma unroll
    for (int f = 0; f < 3; ++f) w.z[f * n + q] = yn[f * n + q] = y[f * n + q];
  }
}

// ---------------------------------------------------------------------------
// what the passes share
// ---------------------------------------------------------------------------
// nf fields (two rows each) into / out of slices s0...
template <int M, int NT>
__device__ __forceinline__ void row_load(double2* sm, int s0, int nf, const double2* __restrict__ F, const Pair& P, size_t n) {
  for (int s = 0; s < 2 * nf; ++s) {
    const double2* src = F + (s >> 1) * n + (size_t)P.row(s & 1) * M;
    for (int j = threadIdx.x; j < M; j += NT) copy16(sm + sidx(M, s0 + s, j), src + j);
  }
  copies_done();
}
template <int M, int NT>
__device__ __forceinline__ void row_store(const double2* sm, int s0, int nf, double2* __restrict__ F, const Pair& P, size_t n) {
  for (int s = 0; s < 2 * nf; ++s) {
    double2* dst = F + (s >> 1) * n + (size_t)P.row(s & 1) * M;
#pragma unroll 4
    for (int j = threadIdx.x; j < M; j += NT) dst[j] = slot(sm, M, s0 + s, j);
  }
}
// the same for column pairs (slice 2f + k = field f, column 2c + k): neighbouring lanes
// take the two columns, 32 contiguous bytes of a row
template <int M, int NT>
__device__ __forceinline__ void col_load(double2* sm, int s0, int nf, const double2* __restrict__ F, int Nx, int c, size_t n) {
  for (int f = 0; f < nf; ++f) {
    const double2* src = F + f * n + 2 * c;
    for (int t = threadIdx.x; t < 2 * M; t += NT)
      copy16(sm + sidx(M, s0 + 2 * f + (t & 1), t >> 1), src + (size_t)(t >> 1) * Nx + (t & 1));
  }
  copies_done();
}
template <int M, int NT>
__device__ __forceinline__ void col_store(const double2* sm, int s0, int nf, double2* __restrict__ F, int Nx, int c, size_t n) {
  for (int f = 0; f < nf; ++f) {
    double2* dst = F + f * n + 2 * c;
#pragma unroll 4
    for (int t = threadIdx.x; t < 2 * M; t += NT)
      dst[(size_t)(t >> 1) * Nx + (t & 1)] = slot(sm, M, s0 + 2 * f + (t & 1), t >> 1);
  }
}
// physical point t of a column pair
struct ColPt {
  int y, k;
  size_t q;
  __device__ __forceinline__ ColPt(int t, int c, int Nx) : y(t >> 1), k(t & 1), q((size_t)(t >> 1) * Nx + 2 * c + (t & 1)) {}
};

// damping of eta less the source in physical space; D0's field
__device__ __forceinline__ double eta_loss(const Tab2& tb, const Work2& w, size_t q, int y, double damp, double eta) {
  double d = damp * eta;
  if (tb.has_src) d -= tb.fac_src * w.insig[y] * tb.gsrc[q] + w.insigs[y] * tb.ssrc[q];
  return d;
}

// how the damping travels: 0 in pass D's physical space; with breaking, whose update
// rewrites dt eta^, that of eta by itself as a spectrum (1); with ChiAdj = 1, where no
// pass D runs, all three as spectra (2)
__device__ __forceinline__ int damp_fields(const Tab2& tb, const Work2& w) { return tb.chi_one ? 2 : (w.dph ? 1 : 0); }

// Column pass: the loss fields from physical space to w.Q's fields f0..., once the slices'
// own fields are stored (a batch of their own keeps every pass at six slices, two CTAs to
// an SM at 1024 points)
template <int M, int NT>
__device__ __forceinline__ void send_loss(double2* sm, int f0, int nd, const Tab2& tb, const Work2& w, int c, size_t n) {
  if (nd == 0) return;
  __syncthreads();
#pragma unroll 2
  for (int t = threadIdx.x; t < 2 * M; t += NT) {
    const ColPt p(t, c, tb.nx);
    const double dm = tb.damp[p.q];
    put(sm, M, p.k, p.y, make_double2(eta_loss(tb, w, p.q, p.y, dm, w.phys[p.q]), nd == 2 ? dm * w.phys[n + p.q] : 0.0));
    if (nd == 2) put(sm, M, 2 + p.k, p.y, make_double2(dm * w.phys[2 * n + p.q], 0.0));
  }
  fft_slices<M, NT>(sm, 0, 2 * nd, tb.twy, -1);
  col_store<M, NT>(sm, 0, nd, w.Q + f0 * n, tb.nx, c, n);
}
// Row pass: their spectra into w.D, ahead of the pass's own fields
template <int M, int NT>
__device__ __forceinline__ void store_loss(double2* sm, int f0, int nd, const Tab2& tb, const Work2& w, const Pair& P, size_t n) {
  if (nd == 0) return;
  row_load<M, NT>(sm, 0, nd, w.Q + f0 * n, P, n);
  fft_slices<M, NT>(sm, 0, 2 * nd, tb.twx, -1);
#pragma unroll 1
  for (int j = threadIdx.x; j < M / 2; j += NT) {
    const Quad Q(P, j, M);
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const size_t q = Q.at(k, s, M);
        double2 a, b;
        split_at(sm, M, 0, Q, k, s, a, b);
        w.D[q] = a;
        if (nd == 2) {
          w.D[n + q] = b;
          split_at(sm, M, 2, Q, k, s, a, b);
          w.D[2 * n + q] = a;
        }
      }
  }
  __syncthreads();
}

// the adjustment's input at a quad: S(i kx dH), S(i ky dH), S(a) into slices 0..5
__device__ __forceinline__ void emit_adjust(double2* sm, int M, const Quad& Q, const Tab2& tb, const double2 dH[2][2],
                                            const double2 a[2][2]) {
  double2 x[2][2];
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int s = 0; s < 2; ++s)
      if (Q.has(s)) x[k][s] = mul_pi(dH[k][s], tb.kx[Q.cc[s]]);
  emit_sym(sm, M, 0, Q, tb.ny, x);
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int s = 0; s < 2; ++s)
      if (Q.has(s)) x[k][s] = mul_pi(dH[k][s], tb.ky[Q.r[k]]);
  emit_sym(sm, M, 2, Q, tb.ny, x);
  emit_sym(sm, M, 4, Q, tb.ny, a);
}
// and on its way: inverse rows into w.W, or with ChiAdj = 1, which leaves S(A) as it is,
// the terms with the damping of u and v straight into w.V
template <int M, int NT>
__device__ __forceinline__ void send_adjust(double2* sm, const Pair& P, const Tab2& tb, const Work2& w, size_t n) {
  if (!tb.chi_one) {
    fft_slices<M, NT>(sm, 0, 6, tb.twx, +1);
    row_store<M, NT>(sm, 0, 3, w.W, P, n);
    return;
  }
  __syncthreads();
  for (int s = 0; s < 6; ++s) {
    const size_t row = (size_t)P.row(s & 1) * M;
    for (int j = threadIdx.x; j < M; j += NT) {
      double2 v = slot(sm, M, s, j);
      if (s < 4) v = cadd(v, w.D[(1 + (s >> 1)) * n + row + j]);
      w.V[(s >> 1) * n + row + j] = v;
    }
  }
}

// the first row pass's extras: the RHS counter and the two rows' line signals at the
// stage time, by the last warp's lanes
__device__ __forceinline__ void stage_extras(const Tab2& tb, const Work2& w, const Pair& P, const Ctl2* ctl, Ctl2* ctlw, int mode,
                                             int NT) {
  if (blockIdx.y != 0) return;
  if (blockIdx.x == 0 && threadIdx.x == 0 && ctlw) ctlw->rhs += 1;
  const int l = NT - 1 - (int)threadIdx.x;
  if (tb.has_src && l < 2) {
    const double2 s = line_signal(tb, P.r[l], stage_time(ctl, mode));
    w.insig[P.r[l]] = s.x;
    w.insigs[P.r[l]] = s.y;
  }
}

// ---------------------------------------------------------------------------
// A: row pass of the flat bottom, one CTA per row pair and field:
//    0 (eta, u); 1 (v, L phi) under HS2, (v, M0u) under HS3, (v, -) under HS1; 2 (M0v, -)
// ---------------------------------------------------------------------------
template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2_rowA(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, Ctl2* ctlw, int mode, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = M, Ny = tb.ny, f = blockIdx.y;
  const size_t n = (size_t)tb.n;
  const Pair P = row_pair(blockIdx.x, Ny);
  stage_extras(tb, w, P, ctl, ctlw, mode, NT);
#pragma unroll 2
  for (int j = threadIdx.x; j < Nx / 2; j += NT) {
    const Quad Q(P, j, Nx);
    double2 x[2][2], y[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (!Q.has(s)) continue;
        const size_t q = Q.at(k, s, Nx);
        if (f == 0) {
          x[k][s] = w.z[q];
          y[k][s] = w.z[n + q];
        } else {
          const double2 zu = w.z[n + q], zv = w.z[2 * n + q];
          // M0 u^ = -i (C^2/g) kx u^, M0 v^ = -i (C^2/g) ky v^
          const double cg = tb.c2g[q];
          const double2 mu = mul_mi(zu, cg * tb.kx[Q.cc[s]]), mv = mul_mi(zv, cg * tb.ky[Q.r[k]]);
          x[k][s] = f == 1 ? zv : mv;
          y[k][s] = f == 2 || tb.model == 1 ? zero2() : (tb.model == 3 ? mu : cadd(mu, mv));
        }
      }
    emit_pack(sm, M, 0, Q, Ny, x, y);
  }
  fft_slices<M, NT>(sm, 0, 2, tb.twx, +1);
  row_store<M, NT>(sm, 0, 1, w.R + f * n, P, n);
}

// ---------------------------------------------------------------------------
// B: column pass of the flat bottom, inverse -> products (each x wallchar,
//    2d/fun_odesolver.c:3239-3249) -> forward.  Fields: 0 (eta L phi, eta u),
//    1 (eta v, deletaH2), under HS3 2 (eta^2 M0u, eta^2 M0v), then the loss fields.
// ---------------------------------------------------------------------------
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2_colB(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = tb.nx, c = blockIdx.x, nd = damp_fields(tb, w);
  const size_t n = (size_t)tb.n;
  const bool hs3 = tb.model == 3;
  const int nin = hs3 ? 3 : 2, np = hs3 ? 3 : 2;
  col_load<M, NT>(sm, 0, nin, w.R, Nx, c, n);
  fft_slices<M, NT>(sm, 0, 2 * nin, tb.twy, +1);
  const double invN = 1.0 / ((double)tb.n);
#pragma unroll 2
  for (int t = threadIdx.x; t < 2 * M; t += NT) {
    const ColPt p(t, c, Nx);
    const double wc = tb.wallchar ? tb.wallchar[p.q] : 1.0;
    const double2 P1 = slot(sm, M, p.k, p.y), P2 = slot(sm, M, 2 + p.k, p.y);
    const double eta = P1.x * invN, u = P1.y * invN, v = P2.x * invN;
    double lphi = P2.y * invN;
    if (hs3) {
      const double m0u = lphi, m0v = slot(sm, M, 4 + p.k, p.y).x * invN;
      lphi = m0u + m0v;
      put(sm, M, 4 + p.k, p.y, make_double2(eta * eta * m0u * wc, eta * eta * m0v * wc));
      w.op[n + p.q] = lphi;
    }
    w.phys[p.q] = eta;
    w.phys[n + p.q] = u;
    w.phys[2 * n + p.q] = v;
    put(sm, M, p.k, p.y, make_double2(eta * lphi * wc, eta * u * wc));
    put(sm, M, 2 + p.k, p.y, make_double2(eta * v * wc, 0.5 * ((u * u + v * v) - lphi * lphi) * wc));
  }
  fft_slices<M, NT>(sm, 0, 2 * np, tb.twy, -1);
  col_store<M, NT>(sm, 0, np, w.Q, Nx, c, n);
  send_loss<M, NT>(sm, np, nd, tb, w, c, n);
}

// ---------------------------------------------------------------------------
// C: row pass of the flat bottom, forward, split.  HS2: the adjustment's input -> inverse
//    rows.  HS3 (fun_termshat_AB3_2DF_uv, :3512-3897): the second-order terms less
//    (kx^2 (eta^2 M0u)^ + ky^2 (eta^2 M0v)^) / 2 are kept, and (L (eta L phi), div(grad phi))
//    goes to physical space.
// ---------------------------------------------------------------------------
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2_rowC(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = M, Ny = tb.ny, nd = damp_fields(tb, w);
  const size_t n = (size_t)tb.n;
  const bool hs3 = tb.model == 3;
  const int np = hs3 ? 3 : 2;
  const Pair P = row_pair(blockIdx.x, Ny);
  store_loss<M, NT>(sm, np, nd, tb, w, P, n);
  row_load<M, NT>(sm, 0, np, w.Q, P, n);
  fft_slices<M, NT>(sm, 0, 2 * np, tb.twx, -1);
#pragma unroll 1
  for (int j = threadIdx.x; j < Nx / 2; j += NT) {
    const Quad Q(P, j, Nx);
    double2 dH[2][2], a[2][2], lq[2][2], dv[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (!Q.has(s)) continue;
        const size_t q = Q.at(k, s, Nx);
        const double L = tb.l2d[q], kx = tb.kx[Q.cc[s]], ky = tb.ky[Q.r[k]];
        double2 qh, eu, ev;
        split_at(sm, M, 0, Q, k, s, qh, eu);
        split_at(sm, M, 2, Q, k, s, ev, dH[k][s]);
        // delu H2^ + delv H2^ = -L (eta L phi)^ - i kx (eta u)^ - i ky (eta v)^
        lq[k][s] = cscale(qh, L);
        a[k][s] = csub(cadd(mul_mi(eu, kx), mul_mi(ev, ky)), lq[k][s]);
        if (hs3) {
          double2 cu, cv;
          split_at(sm, M, 4, Q, k, s, cu, cv);
          a[k][s] = csub(a[k][s], cadd(cscale(cu, 0.5 * (kx * kx)), cscale(cv, 0.5 * (ky * ky))));
          dv[k][s] = cadd(mul_pi(w.z[n + q], kx), mul_pi(w.z[2 * n + q], ky));
          w.T[q] = a[k][s];
          w.T[n + q] = dH[k][s];
        }
      }
    if (hs3) emit_pack(sm, M, 0, Q, Ny, lq, dv);
    else emit_adjust(sm, M, Q, tb, dH, a);
  }
  if (hs3) {
    fft_slices<M, NT>(sm, 0, 2, tb.twx, +1);
    row_store<M, NT>(sm, 0, 1, w.R, P, n);
  } else {
    send_adjust<M, NT>(sm, P, tb, w, n);
  }
}

// ---------------------------------------------------------------------------
// HS3: the cubic products from L (eta L phi), div(grad phi) in physical space:
//   p  = eta L(eta L phi) + eta^2 div(grad phi) / 2, whose L^ adds to delu + delv,
//   h3 = L phi (eta div(grad phi) + L(eta L phi)) = deletaH3
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 cubic_products(const Tab2& tb, const Work2& w, size_t q, size_t n, double lel, double divg) {
  const double eta = w.phys[q], lphi = w.op[n + q];
  const double wc = tb.wallchar ? tb.wallchar[q] : 1.0;
  return make_double2(eta * lel + 0.5 * (eta * eta * divg * wc), lphi * eta * divg + lphi * lel);
}
template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2_colH3(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = tb.nx, c = blockIdx.x;
  const size_t n = (size_t)tb.n;
  col_load<M, NT>(sm, 0, 1, w.R, Nx, c, n);
  fft_slices<M, NT>(sm, 0, 2, tb.twy, +1);
  const double invN = 1.0 / ((double)tb.n);
#pragma unroll 4
  for (int t = threadIdx.x; t < 2 * M; t += NT) {
    const ColPt p(t, c, Nx);
    const double2 a = slot(sm, M, p.k, p.y);
    put(sm, M, p.k, p.y, cubic_products(tb, w, p.q, n, a.x * invN, a.y * invN));
  }
  fft_slices<M, NT>(sm, 0, 2, tb.twy, -1);
  col_store<M, NT>(sm, 0, 1, w.Q, Nx, c, n);
}
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2_rowI3(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = M;
  const size_t n = (size_t)tb.n;
  const Pair P = row_pair(blockIdx.x, tb.ny);
  row_load<M, NT>(sm, 0, 1, w.Q, P, n);
  fft_slices<M, NT>(sm, 0, 2, tb.twx, -1);
#pragma unroll 1
  for (int j = threadIdx.x; j < Nx / 2; j += NT) {
    const Quad Q(P, j, Nx);
    double2 dH[2][2], a[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (!Q.has(s)) continue;
        const size_t q = Q.at(k, s, Nx);
        double2 ph, h3;
        split_at(sm, M, 0, Q, k, s, ph, h3);
        a[k][s] = cadd(w.T[q], cscale(ph, tb.l2d[q]));
        dH[k][s] = cadd(w.T[n + q], h3);
      }
    emit_adjust(sm, M, Q, tb, dH, a);
  }
  send_adjust<M, NT>(sm, P, tb, w, n);
}

// ---------------------------------------------------------------------------
// D: column pass, one CTA per column pair and field f: inverse -> x ChiAdj / N, with the
//    damping (and source) that no spectrum carries -> forward.  The adjustment's complex
//    intermediate is kept (the Nyquist column of S(A) is not Hermitian).
// ---------------------------------------------------------------------------
template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2_colD(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = tb.nx, c = blockIdx.x, f = blockIdx.y;
  const size_t n = (size_t)tb.n;
  const bool loss = f < 2 || !w.dph;
  const double* __restrict__ src = w.phys + (f == 2 ? 0 : f + 1) * n;
  col_load<M, NT>(sm, 0, 1, w.W + f * n, Nx, c, n);
  fft_slices<M, NT>(sm, 0, 2, tb.twy, +1);
  const double invN = 1.0 / ((double)tb.n);
#pragma unroll 4
  for (int t = threadIdx.x; t < 2 * M; t += NT) {
    const ColPt p(t, c, Nx);
    const double ch = tb.chi[p.q] * invN;
    double d = 0.0;
    if (loss) {
      const double dm = tb.damp[p.q], v = src[p.q];
      d = f == 2 ? -eta_loss(tb, w, p.q, p.y, dm, v) : dm * v;
    }
    const double2 a = slot(sm, M, p.k, p.y);
    put(sm, M, p.k, p.y, make_double2(a.x * ch + d, a.y * ch));
  }
  fft_slices<M, NT>(sm, 0, 2, tb.twy, -1);
  col_store<M, NT>(sm, 0, 1, w.V + f * n, Nx, c, n);
}

// ---------------------------------------------------------------------------
// E: row pass, one CTA per row pair and component (0 u, 1 v, 2 eta): forward -> dt Z
// ---------------------------------------------------------------------------
// delphiH1^ at a point: the operator's on a varying bottom, the wall branch's on a flat
// one with walls, else -i (kx C^2/g u^ + ky C^2/g v^)
__device__ __forceinline__ double2 delphi_h1(const Tab2& tb, const Work2& w, size_t q, size_t n, double kx, double ky) {
  if (tb.var || tb.wallchar) return w.H1[q];
  const double cg = tb.c2g[q];
  return cadd(mul_mi(w.z[n + q], cg * kx), mul_mi(w.z[2 * n + q], cg * ky));
}
template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2_rowE(Tab2 tb, Work2 w, RK2 rk, const Ctl2* __restrict__ ctl, int mode, int cond, double2* __restrict__ direct_out) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = M, f = blockIdx.y;
  const size_t n = (size_t)tb.n;
  const Pair P = row_pair(blockIdx.x, tb.ny);
  const bool dspec = tb.chi_one || w.dph;   // the damping of eta comes as a spectrum
  row_load<M, NT>(sm, 0, 1, w.V + f * n, P, n);
  if (tb.chi_one) __syncthreads();
  else fft_slices<M, NT>(sm, 0, 2, tb.twx, -1);
  double2* out = rhs_out(rk, ctl, mode, direct_out) + (f == 2 ? 0 : f + 1) * n;
  for (int k = 0; k < 2; ++k) {
    const int r = P.row(k);
    const double ky = tb.ky[r];
#pragma unroll 4
    for (int j = threadIdx.x; j < Nx; j += NT) {
      const size_t q = (size_t)r * Nx + j;
      const double kx = tb.kx[j], a = tb.aal[q];
      const double2 v = slot(sm, M, k, j);
      if (f == 2) {
        const double2 dphi = cadd(delphi_h1(tb, w, q, n, kx, ky), v);
        const double2 d = dspec ? w.D[q] : zero2();
        if (w.dph) w.dph[q] = dphi;
        out[q] = make_double2((dphi.x - d.x) * a, (dphi.y - d.y) * a);
      } else {
        const double2 h = mul_mi(w.z[q], kGrav * (f == 0 ? kx : ky));
        out[q] = make_double2((h.x - v.x) * a, (h.y - v.y) * a);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// HS1 (rhs_AB1_2DF_uv / rhs_AB1_2DB_uv, 2d/fun_odesolver.c:4350-4456): no H2 terms.  Column
// pass: eta, u, v (inverse transforms of pass A's fields; on a varying bottom already in
// physical space) -> their damping; row pass: dt Z.
// ---------------------------------------------------------------------------
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2_colH1(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = tb.nx, c = blockIdx.x;
  const size_t n = (size_t)tb.n;
  if (!tb.var) {
    col_load<M, NT>(sm, 0, 2, w.R, Nx, c, n);
    fft_slices<M, NT>(sm, 0, 4, tb.twy, +1);
  }
  const double invN = 1.0 / ((double)tb.n);
#pragma unroll 2
  for (int t = threadIdx.x; t < 2 * M; t += NT) {
    const ColPt p(t, c, Nx);
    double eta, u, v;
    if (tb.var) {
      eta = w.phys[p.q];
      u = w.phys[n + p.q];
      v = w.phys[2 * n + p.q];
    } else {
      const double2 a = slot(sm, M, p.k, p.y), b = slot(sm, M, 2 + p.k, p.y);
      eta = a.x * invN;
      u = a.y * invN;
      v = b.x * invN;
    }
    const double dm = tb.damp[p.q];
    put(sm, M, p.k, p.y, make_double2(eta_loss(tb, w, p.q, p.y, dm, eta), dm * u));
    put(sm, M, 2 + p.k, p.y, make_double2(dm * v, 0.0));
  }
  fft_slices<M, NT>(sm, 0, 4, tb.twy, -1);
  col_store<M, NT>(sm, 0, 2, w.Q, Nx, c, n);
}
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2_rowH1(Tab2 tb, Work2 w, RK2 rk, const Ctl2* __restrict__ ctl, int mode, int cond, double2* __restrict__ direct_out) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = M;
  const size_t n = (size_t)tb.n;
  const Pair P = row_pair(blockIdx.x, tb.ny);
  row_load<M, NT>(sm, 0, 2, w.Q, P, n);
  fft_slices<M, NT>(sm, 0, 4, tb.twx, -1);
  double2* out = rhs_out(rk, ctl, mode, direct_out);
  for (int k = 0; k < 2; ++k) {
    const int r = P.row(k);
    const double ky = tb.ky[r];
#pragma unroll 2
    for (int j = threadIdx.x; j < Nx; j += NT) {
      const size_t q = (size_t)r * Nx + j;
      const double kx = tb.kx[j], a = tb.aal[q];
      const int jm = (Nx - j) & (Nx - 1), km = k ^ P.flip;
      double2 de, du, dv, none;
      split2(slot(sm, M, k, j), slot(sm, M, km, jm), de, du);
      split2(slot(sm, M, 2 + k, j), slot(sm, M, 2 + km, jm), dv, none);
      const double2 ze = w.z[q], dphi = delphi_h1(tb, w, q, n, kx, ky);
      const double2 hu = mul_mi(ze, kGrav * kx), hv = mul_mi(ze, kGrav * ky);
      out[q] = make_double2((dphi.x - de.x) * a, (dphi.y - de.y) * a);
      out[n + q] = make_double2((hu.x - du.x) * a, (hu.y - du.y) * a);
      out[2 * n + q] = make_double2((hv.x - dv.x) * a, (hv.y - dv.y) * a);
    }
  }
}

// ---------------------------------------------------------------------------
// stepper kernels
// ---------------------------------------------------------------------------
constexpr int kCombBlocks = 592;   // 4 x 148 SMs
constexpr int kCombThreads = 256;

// y_new = y + h0 sum c_i k_i into y[cur ^ 1]; per-block max of |yerr| / D0
__global__ void __launch_bounds__(kCombThreads)
k2_combine(const double* __restrict__ aal, RK2 rk, Work2 w, const Ctl2* __restrict__ ctl, size_t n) {
  __shared__ double red[kCombThreads / 32];
  __shared__ int badw[kCombThreads / 32];
  if (ctl->done) return;
  const double h = ctl->h0, er = ctl->eps_rel, ea = ctl->eps_abs;
  const double2* __restrict__ y = rk.y[ctl->cur];
  double2* __restrict__ yn = rk.y[ctl->cur ^ 1];
  const double2* __restrict__ k1 = rk.kk[ctl->k1i];
  double rm = 2.2250738585072014e-308;
  int bad = 0;
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < n; p += (size_t)gridDim.x * blockDim.x) {
    if (aal[p] == 0.0) continue;
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const size_t q = s * n + p;
      const double2 a = k1[q], c = rk.ks[1][q], e = rk.ks[2][q], f = rk.ks[3][q], g = rk.ks[4][q], yy = y[q];
      const double dix = ra2(ra2(ra2(ra2(rm2(A2_c[0], a.x), rm2(A2_c[1], c.x)), rm2(A2_c[2], e.x)), rm2(A2_c[3], f.x)),
                             rm2(A2_c[4], g.x));
      const double diy = ra2(ra2(ra2(ra2(rm2(A2_c[0], a.y), rm2(A2_c[1], c.y)), rm2(A2_c[2], e.y)), rm2(A2_c[3], f.y)),
                             rm2(A2_c[4], g.y));
      const double2 nv = make_double2(ra2(yy.x, rm2(h, dix)), ra2(yy.y, rm2(h, diy)));
      yn[q] = nv;
      const double ex = rm2(h, ra2(ra2(ra2(ra2(rm2(A2_ec[0], a.x), rm2(A2_ec[1], c.x)), rm2(A2_ec[2], e.x)),
                                       rm2(A2_ec[3], f.x)), rm2(A2_ec[4], g.x)));
      const double ey = rm2(h, ra2(ra2(ra2(ra2(rm2(A2_ec[0], a.y), rm2(A2_ec[1], c.y)), rm2(A2_ec[2], e.y)),
                                       rm2(A2_ec[3], f.y)), rm2(A2_ec[4], g.y)));
      const double rx = fabs(ex) / fabs(ra2(rm2(er, fabs(nv.x)), ea));
      const double ry = fabs(ey) / fabs(ra2(rm2(er, fabs(nv.y)), ea));
      bad |= (!(rx == rx) || !(ry == ry) || isinf(nv.x) || isinf(nv.y)) ? 1 : 0;
      rm = fmax(rm, fmax(rx, ry));
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    rm = fmax(rm, __shfl_xor_sync(0xffffffffu, rm, o));
    bad |= __shfl_xor_sync(0xffffffffu, bad, o);
  }
  if ((threadIdx.x & 31) == 0) { red[threadIdx.x >> 5] = rm; badw[threadIdx.x >> 5] = bad; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double m = red[0];
    int b = badw[0];
    for (int i = 1; i < kCombThreads / 32; ++i) { m = fmax(m, red[i]); b |= badw[i]; }
    w.part[blockIdx.x] = b ? __longlong_as_double(0x7ff0000000000000ULL) : m;
  }
}

__device__ __forceinline__ void set_prologue(Ctl2* c) {
  const double dt = c->t1 - c->t;
  double h0 = c->h;
  c->final_step = 0;
  if ((dt >= 0.0 && h0 > dt) || (dt < 0.0 && h0 < dt)) { h0 = dt; c->final_step = 1; }
  c->h0 = h0;
}

// std_control_hadjust + gsl_odeiv2_evolve_apply's accept / retry decision
__global__ void k2_control(Ctl2* c, const Work2 w, int nparts) {
  __shared__ double red[32];
  if (c->done) return;
  double m = 2.2250738585072014e-308;
  bool nonfin = false;
  for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
    const double v = w.part[i];
    if (!(v <= 1.7976931348623157e308)) nonfin = true;
    m = fmax(m, v);
  }
  const int anynf = __syncthreads_or(nonfin ? 1 : 0);
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x != 0) return;
  double rmax = red[0];
  for (int i = 1; i < (int)(blockDim.x / 32); ++i) rmax = fmax(rmax, red[i]);
  c->need_k1 = 0;   // the attempt's k1 is in place
  if (anynf) { c->status = kNonFinite; c->done = 1; return; }
  const double t0 = c->t, h_old = c->h0;
  const double tn = c->final_step ? c->t1 : t0 + h_old;
  int adj = 0;
  double hn = h_old;
  if (rmax > 1.1) {
    double r = 0.9 / pow(rmax, 1.0 / 5.0);
    if (r < 0.2) r = 0.2;
    hn = r * h_old;
    adj = -1;
  } else if (rmax < 0.5) {
    double r = 0.9 / pow(rmax, 1.0 / 6.0);
    if (r > 5.0) r = 5.0;
    if (r < 1.0) r = 1.0;
    hn = r * h_old;
    adj = 1;
  }
  if (adj == -1) {
    const double t_next = tn + hn;
    if (fabs(hn) < fabs(h_old) && t_next != tn) {
      c->rej += 1;
      if (++c->attempts > 1000) { c->status = kStepFailed; c->done = 1; return; }
      c->h = hn;
      set_prologue(c);
      return;
    }
    hn = h_old;
  }
  c->acc += 1;
  c->attempts = 0;
  c->cur ^= 1;
  const double tk = t0 + h_old;
  c->t = tn;
  c->h = hn;
  if (tk == tn && !c->brk) c->need_kout = 1;
  else c->need_k1 = 1;
  if (!(c->t < c->t1)) c->done = 1;
  else set_prologue(c);
}

__global__ void k2_finalize(Ctl2* c) {
  if (c->need_kout) {
    c->k1i ^= 1;
    c->need_kout = 0;
  }
}

__global__ void k2_begin(Ctl2* c, double t1) {
  c->t1 = t1;
  c->status = kOk;
  c->attempts = 0;
  c->done = (c->t < t1) ? 0 : 1;
  if (!c->done) set_prologue(c);
}

// reference layout [Re eta | Im eta | Re u | Im u | Re v | Im v] <-> 3 double2 fields; with a
// control block, the time of a direct right-hand side as well
__global__ void k2_to_internal(const double* __restrict__ yr, double2* __restrict__ yi, size_t n, Ctl2* ctl, double t) {
  if (ctl && blockIdx.x == 0 && threadIdx.x == 0) ctl->t_direct = t;
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < 3 * n; q += (size_t)gridDim.x * blockDim.x) {
    const size_t f = q / n, p = q - f * n;
    yi[q] = make_double2(yr[2 * f * n + p], yr[(2 * f + 1) * n + p]);
  }
}
__global__ void k2_to_reference(const double2* __restrict__ yi, double* __restrict__ yr, size_t n) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < 3 * n; q += (size_t)gridDim.x * blockDim.x) {
    const size_t f = q / n, p = q - f * n;
    const double2 v = yi[q];
    yr[2 * f * n + p] = v.x;
    yr[(2 * f + 1) * n + p] = v.y;
  }
}

}  // namespace hw2d
