// hw_stepper.cuh -- the RKF45 stage / error-norm / step-control loop of one
// member, entirely on the device.  It restates GSL's rkf45 stepper (Fehlberg
// tableau, 5th-order solution propagated), the standard control built by
// gsl_odeiv_control_y_new (a_y = 1, a_dydt = 0, safety 0.9, order 5, decrease
// above 1.1, increase below 0.5, factors clamped to [0.2, 5]) and the legacy
// gsl_odeiv_evolve_apply (dydt_in at every call, final-step clipping, retry on
// decrease).  The reference calls these at 1d/functions.c:532-553.
#pragma once

#include "hw_rhs.cuh"

namespace hwdev {

// max over the member (all CTAs of the cluster); identical result in every thread
template <int M>
__device__ __forceinline__ double member_max(Ctx<M> X, double v) {
  const DevMember& d = X.d;
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int w = int(threadIdx.x) >> 5;
  constexpr int NW = Ctx<M>::T / 32;
  __syncthreads();
  if ((int(threadIdx.x) & 31) == 0) X.sc->red[w] = v;
  __syncthreads();
  double m = X.sc->red[0];
  for (int i = 1; i < NW; ++i) m = fmax(m, X.sc->red[i]);
  if (d.C > 1) {
    cg::cluster_group cl = cg::this_cluster();
    if (int(threadIdx.x) == 0) X.sc->red[NW] = m;
    cl.sync();
    m = *cl.map_shared_rank(X.sc->red + NW, 0);
    for (int r = 1; r < d.C; ++r) m = fmax(m, *cl.map_shared_rank(X.sc->red + NW, r));
    cl.sync();
  }
  return m;
}

// ynew = y + h sum c_i k_i ; yerr = h sum ec_i k_i ; returns max |yerr| / D0, with D0 =
// eps_rel |ynew| + eps_abs.  Pairs outside the alias band are left out: their k_i are
// zero, so ynew = y there (both buffers hold it since the launch began) and yerr = 0.
// A thread keeps the numerator and denominator of its largest ratio and divides once.
template <int M>
__device__ __noinline__ double final_combine(Ctx<M> X, double h) {
  const DevMember& d = X.d;
  const Bufs& B = X.sc->bufs;
  constexpr int T = Ctx<M>::T;
  const double2* __restrict__ ys = B.y;
  const double2* __restrict__ k1 = B.k[0];
  const double2* __restrict__ k3 = B.k[2];
  const double2* __restrict__ k4 = B.k[3];
  const double2* __restrict__ k5 = B.k[4];
  const double2* __restrict__ k6 = B.k[5];
  double2* __restrict__ yn = B.yn;
  const double er = d.eps_rel, ea = d.eps_abs;
  const int N = d.N, act = d.act, cq = (d.C - X.c) & (d.C - 1);
  double num = 0.0, den = 1.0;
  bool bad = false;
  auto one = [&](double y, double a, double c, double e, double f, double g) {
    const double di = radd(radd(radd(radd(rmul(RK_c1, a), rmul(RK_c3, c)), rmul(RK_c4, e)), rmul(RK_c5, f)),
                           rmul(RK_c6, g));
    const double v = radd(y, rmul(h, di));
    const double ex = fabs(rmul(h, radd(radd(radd(radd(rmul(RK_ec1, a), rmul(RK_ec3, c)), rmul(RK_ec4, e)),
                                             rmul(RK_ec5, f)), rmul(RK_ec6, g))));
    const double D = fabs(radd(rmul(er, fabs(v)), ea));
    bad = bad || !(ex <= 1.7976931348623157e308) || !(fabs(v) <= 1.7976931348623157e308);
    if (ex * den > num * D) {
      num = ex;
      den = D;
    }
    return v;
  };
#pragma unroll 1
  for (int u = 0; u < kPts / 2; ++u) {
    const PairAt r = pair_at<M>(X.c, cq, int(threadIdx.x) + u * T);
    if (r.i >= act) continue;
#pragma unroll 1
    for (int off = 0; off <= N; off += N) {
      const int q0 = r.p + off, q1 = r.pp + off;
      const double2 y0 = ys[q0], a0 = k1[q0], c0 = k3[q0], e0 = k4[q0], f0 = k5[q0], g0 = k6[q0];
      const double2 y1 = ys[q1], a1 = k1[q1], c1 = k3[q1], e1 = k4[q1], f1 = k5[q1], g1 = k6[q1];
      yn[q0] = make_double2(one(y0.x, a0.x, c0.x, e0.x, f0.x, g0.x), one(y0.y, a0.y, c0.y, e0.y, f0.y, g0.y));
      yn[q1] = make_double2(one(y1.x, a1.x, c1.x, e1.x, f1.x, g1.x), one(y1.y, a1.y, c1.y, e1.y, f1.y, g1.y));
    }
  }
  double rm = fmax(num / den, 2.2250738585072014e-308);   // DBL_MIN
  if (bad) rm = __longlong_as_double(0x7ff0000000000000ULL);   // +inf: forces a failure path
  return member_max(X, rm);
}

// Outside the alias band every k_i is zero and the state stays what it is: the second
// state buffer and the stage input take those points once, when a launch begins.
template <int M>
__device__ __forceinline__ void spread_unmoved(Ctx<M> X) {
  const DevMember& d = X.d;
  const int cq = (d.C - X.c) & (d.C - 1);
  for (int u = 0; u < kPts / 2; ++u) {
    const PairAt r = pair_at<M>(X.c, cq, int(threadIdx.x) + u * Ctx<M>::T);
    if (r.i < d.act) continue;
    for (int off = 0; off <= d.N; off += d.N) {
      d.ynew[r.p + off] = d.zs[r.p + off] = d.y[r.p + off];
      d.ynew[r.pp + off] = d.zs[r.pp + off] = d.y[r.pp + off];
    }
  }
}

struct StepState {
  double t, h;
  int status, k1_valid;
  long long rhs, acc, rej;
};

// stage s of a step of size h as the coming RHS's input: y + h sum_j b_sj k_j, or (s = 1)
// the state y itself, and entry sig of the step's influx signals; the RHS's first barrier
// makes it known
template <int M>
__device__ __forceinline__ void set_stage(Ctx<M> X, const double2* y, int s, int sig, double h) {
  if (threadIdx.x == 0) {
    const Bufs& B = X.sc->bufs;
    X.sc->stg = StageSrc{y, {B.k[0], B.k[1], B.k[2], B.k[3], B.k[4]}, s, X.d.has_influx ? sig : -1, h};
  }
}

// one RHS evaluation at the state src itself (the RHS copies it into zs)
template <int M>
__device__ __forceinline__ void rhs_at(Ctx<M> X, StepState& S, double t, const double2* src, double2* out, int sig) {
  set_stage(X, src, 1, sig, 0.0);
  rhs_eval<M>(X, t, out);
  ++S.rhs;
}

// gsl_odeiv_evolve_apply with rkf45 and control_y, one member
template <int M>
__device__ __noinline__ void evolve_apply(Ctx<M> X, StepState& S, double t1) {
  const DevMember& d = X.d;
  Bufs& B = X.sc->bufs;
  const double t0 = S.t;
  double h0 = S.h;
  const double dt = t1 - t0;
  if ((dt < 0.0 && h0 > 0.0) || (dt > 0.0 && h0 < 0.0)) { S.status = kStepFailed; return; }
  bool need_k1 = d.exact || !S.k1_valid;
  int attempts = 0;
  for (;;) {
    bool final_step = false;
    if ((dt >= 0.0 && h0 > dt) || (dt < 0.0 && h0 < dt)) { h0 = dt; final_step = true; }
    // The influx signals at the attempt's seven times, each by a thread of its own: one
    // wait for the samples and divisions an attempt instead of one an RHS (4 thousand
    // cycles of an RHS's 40 in a single tank)
    if (d.has_influx && threadIdx.x < 7) {
      const int j = threadIdx.x;
      X.sc->sig[j] = influx_at(d, j == 0 ? t0 : (j == 6 ? t0 + h0 : t0 + RK_ah[j - 1] * h0));
    }
    if (need_k1) rhs_at(X, S, t0, B.y, B.k[0], 0);
    need_k1 = false;
    for (int s = 2; s <= 6; ++s) {
      // the RHS forms its own stage input from y and the k's (into zs as well)
      set_stage(X, B.y, s, s - 1, h0);
      rhs_eval<M>(X, t0 + RK_ah[s - 2] * h0, B.k[s - 1]);
      ++S.rhs;
    }
    member_sync(d.C);
    const double rmax = final_combine(X, h0);
    if (d.exact) rhs_at(X, S, t0 + h0, B.yn, B.k[6], 6);
    const double tn = final_step ? t1 : t0 + h0;
    // std_control_hadjust (order 5)
    const double h_old = h0;
    int adj = 0;
    double hn = h0;
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
    if (!(rmax <= 1.7976931348623157e308)) { S.status = kNonFinite; return; }   // NaN/inf state: freeze
    if (adj == -1) {
      const double t_next = tn + hn;
      if (fabs(hn) < fabs(h_old) && t_next != tn) {
        ++S.rej;
        h0 = hn;
        if (++attempts > 200) { S.status = kStepFailed; return; }
        continue;
      }
      hn = h_old;
    }
    // accepted
    if (!d.exact) {
      // pure RHS: derivative at the new point serves as the next dydt_in when the
      // next call starts exactly at t0 + h0
      const double tk = t0 + h0;
      if (tk == tn) {
        rhs_at(X, S, tk, B.yn, B.k[6], 6);
        S.k1_valid = 1;
      } else {
        S.k1_valid = 0;
      }
    } else {
      S.k1_valid = 0;
    }
    __syncthreads();   // every thread has read the buffers' addresses
    if (threadIdx.x == 0) {
      double2* ty = B.y; B.y = B.yn; B.yn = ty;
      if (S.k1_valid) { double2* tk = B.k[0]; B.k[0] = B.k[6]; B.k[6] = tk; }
    }
    __syncthreads();
    S.t = tn;
    S.h = hn;
    ++S.acc;
    return;
  }
}

}  // namespace hwdev
