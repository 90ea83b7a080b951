// hw_rhs_gen.cuh -- the right-hand sides other than HS2 on a flat bottom: HS1
// (rhs_HsF1, 1d/rhs.c:1-94), HS3 on a flat bottom and HS2 / HS3 on a varying bottom
// with K reference depths (rhs_HsF2, rhs_HsF3, 1d/rhs.c:96-398; HSS,
// 1d/functions.c:2861-2977; Op_M0 / Op_M1, :2979-3015).
//
// The varying-bottom operator of a real field a with spectrum a^ is
//   HSS(a) = 1/2 [ F( sum_j gam_j Re F^-1(C_j a^) ) + sum_j C_j F(gam_j a) ].
// The first sum is taken in physical space, so K reference depths ask for K real inverse
// transforms, K real forward ones and one more (the transform is linear; K forward
// transforms of each gam_j s_j gave the same sum).  Real fields go four to a sweep, two
// to a complex transform and two transforms to a pass over the slices: an iteration
// takes up to four fields to physical space, does there what the points need and takes
// up to four back.  Where a sweep's last iteration ends, the pair's owner forms the next
// sweep's input in place.  A sweep starts with the fields that its operand is formed
// from (eta, u; M0 u; L(eta M0 u)) and carries the model's own products beside the
// gam_j images: 15 complex transforms for HS2 with three reference depths (17 with an
// HSS by itself), 40 with sixteen (55).
//
// What bounds it: the barriers and load latencies between the transforms.  Fields that
// outlive an iteration (physical and spectral sums, eta, u, M0 u) lie in the member's
// global scratch, each read and written by the one thread that owns the point or pair.
#pragma once

#include "hw_rhs_fast.cuh"

namespace hwdev {

// One iteration of a sweep: nin packed spectra (slices A, B) to physical space, op at
// every point, nout packed fields back.  op.load(n) reads what point n needs, op(n, L, a, b)
// turns the transformed values into the next ones; two points' loads are in flight
// together.  The meeting of cross-CTA steps is cross_products'.
template <int M, int C, class Op>
__device__ __forceinline__ void meet_cross(Ctx<M> X, int nin, int nout, const Op& op) {
  using P = Cross<C>;
  constexpr int T = M / kPts, R = P::R;
  const DevMember& d = X.d;
  double2 *A = X.buf, *B = X.buf2();
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
#pragma unroll 1
  for (int q = 0; q < P::PER; ++q) {
    const int i = P::template at<T>(X.c, q);
    double2 va[R], vb[R];
#pragma unroll
    for (int e = 0; e < R; ++e) {
      va[e] = cl.map_shared_rank(A, P::spectral(e))[pidx(i)];
      vb[e] = nin == 2 ? cl.map_shared_rank(B, P::spectral(e))[pidx(i)] : czero();
    }
    cross_in<C>(va, d.tw, i);
    if (nin == 2) cross_in<C>(vb, d.tw, i);
#pragma unroll
    for (int e = 0; e < R; e += 2) {
      const int n0 = P::physical(e) * M + i, n1 = P::physical(e + 1) * M + i;
      const typename Op::L l0 = op.load(n0), l1 = op.load(n1);
      op(n0, l0, va[e], vb[e]);
      op(n1, l1, va[e + 1], vb[e + 1]);
    }
    cross_out<C>(va, d.tw, i);
    if (nout == 2) cross_out<C>(vb, d.tw, i);
#pragma unroll
    for (int e = 0; e < R; ++e) {
      cl.map_shared_rank(A, P::spectral(e))[pidx(i)] = va[e];
      if (nout == 2) cl.map_shared_rank(B, P::spectral(e))[pidx(i)] = vb[e];
    }
  }
  cl.sync();
}

// (op is made here, between the transforms' calls, from the member's description and the
// iteration: its fields stay in registers)
template <int M, class Op>
__device__ __noinline__ void meet(Ctx<M> X, int nin, int nout, int it) {
  const DevMember& d = X.d;
  const int C = d.C;
  if (C > 1) {
    if (nin == 2) fft_local2<M>(X.buf, X.buf2(), d.tw, C, +1);
    else fft_local<M>(X.buf, d.tw, C, +1);
    if (C == 2) meet_cross<M, 2>(X, nin, nout, Op(X, it));
    else if (C == 4) meet_cross<M, 4>(X, nin, nout, Op(X, it));
    else if (C == 8) meet_cross<M, 8>(X, nin, nout, Op(X, it));
    else meet_cross<M, 16>(X, nin, nout, Op(X, it));
    if (nout == 2) fft_local2<M>(X.buf, X.buf2(), d.tw, C, -1);
    else fft_local<M>(X.buf, d.tw, C, -1);
    return;
  }
  if (nin == 2) fft_inverse2<M>(X.buf, X.buf2(), d.tw, C, X.c);
  else fft_inverse<M>(X.buf, d.tw, C, X.c);
  {
    const Op op(X, it);
    double2 *A = X.buf, *B = X.buf2();
#pragma unroll 1
    for (int u = 0; u < kPts; u += 2) {
      const int i0 = int(threadIdx.x) + u * Ctx<M>::T, i1 = i0 + Ctx<M>::T, n0 = X.c * M + i0, n1 = X.c * M + i1;
      const typename Op::L l0 = op.load(n0), l1 = op.load(n1);
      double2 a0 = A[pidx(i0)], a1 = A[pidx(i1)];
      double2 b0 = nin == 2 ? B[pidx(i0)] : czero(), b1 = nin == 2 ? B[pidx(i1)] : czero();
      op(n0, l0, a0, b0);
      op(n1, l1, a1, b1);
      A[pidx(i0)] = a0;
      A[pidx(i1)] = a1;
      if (nout == 2) {
        B[pidx(i0)] = b0;
        B[pidx(i1)] = b1;
      }
    }
  }
  if (nout == 2) fft_forward2<M>(X.buf, X.buf2(), d.tw, C, X.c);
  else fft_forward<M>(X.buf, d.tw, C, X.c);
}

// How K reference depths fill a sweep's iterations.  First sweep: fields in 0 eta, 1 u, then
// the images; out gam_j u, and at index `at`, once the last image is in, the sum.  The others:
// in one pair, then four images to an iteration; out three products, gam_j q, the sum.
struct Plan {
  int at, nit;
};
__device__ __forceinline__ Plan first_plan(int K) {
  const int at = K % 4 == 3 ? K + 1 : K;
  return Plan{at, at / 4 + 1};
}
__device__ __forceinline__ Plan rest_plan(int K) {
  const int nimg = (K + 3) / 4, at = K > 0 ? (3 + K > 4 * nimg ? 3 + K : 4 * nimg) : 3;
  return Plan{at, at / 4 + 1};
}
template <int M>
__device__ __forceinline__ int refs(const Ctx<M>& X) { return X.d.flat ? 0 : X.d.nref; }

// point n above the breaking threshold inside the window: listed for the criterion
template <int M>
struct Listing {
  int w0, w1;
  double thr;
  unsigned short* cand;
  int* ncand;
  __device__ __forceinline__ explicit Listing(const Ctx<M>& X)
      : w0(X.d.xbstart), w1(X.d.brk ? X.d.xbstart + X.d.lenIF : X.d.xbstart), thr(X.d.MaxEtaInit), cand(X.sc->cand),
        ncand(&X.sc->ncand) {}
  __device__ __forceinline__ void operator()(int n, double e) const {
    if (n >= w0 && n < w1 && !(e < thr)) cand[atomicAdd(ncand, 1)] = (unsigned short)n;
  }
};

// HS1: eta, u -> their damping
template <int M>
struct OpLinear {
  const double* __restrict__ damp;
  __device__ __forceinline__ OpLinear(Ctx<M> X, int) : damp(X.d.damp) {}
  struct L { double dm; };
  __device__ __forceinline__ L load(int n) const { return L{__ldg(damp + n)}; }
  __device__ __forceinline__ void operator()(int, const L& l, double2& a, double2&) const {
    a = make_double2(l.dm * a.x, l.dm * a.y);
  }
};

// First sweep, HSS(u^).  Fields to physical space: 0 eta, 1 u, 2 + j the image of u^ under
// C_j; fields back: j < K gam_j u, and at index at (past the last image's iteration) the sum
// of gam_j times the images.
template <int M>
struct OpFirst {
  const double* __restrict__ gam;
  double2* PE;
  double* S;
  int N, K, it, at, more;
  Listing<M> list;
  __device__ __forceinline__ OpFirst(Ctx<M> X, int it_)
      : gam(X.d.gam), PE(X.d.sc[0]), S(reinterpret_cast<double*>(X.d.sc[5])), N(X.d.N), K(X.d.nref), it(it_),
        at(first_plan(X.d.nref).at), more(it_ + 1 < first_plan(X.d.nref).nit), list(X) {}
  struct L { double u, s, g[6]; };   // g[m]: gam of reference 4 it - 2 + m
  __device__ __forceinline__ L load(int n) const {
    L l;
    l.u = l.s = 0.0;
    if (it > 0) {
      l.u = PE[n].y;
      l.s = S[n];
    }
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const int j = 4 * it - 2 + m;
      l.g[m] = j >= 0 && j < K ? __ldg(gam + size_t(j) * N + n) : 0.0;
    }
    return l;
  }
  __device__ __forceinline__ void operator()(int n, const L& l, double2& a, double2& b) const {
    double u = l.u, s = l.s;
    if (it == 0) {
      PE[n] = a;
      u = a.y;
      list(n, a.x);
      s = l.g[2] * b.x + l.g[3] * b.y;
    } else {
      s += l.g[0] * a.x + l.g[1] * a.y + l.g[2] * b.x + l.g[3] * b.y;
    }
    if (more) S[n] = s;
    double o[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) o[r] = 4 * it + r == at ? s : l.g[r + 2] * u;
    a = make_double2(o[0], o[1]);
    b = make_double2(o[2], o[3]);
  }
};

// Second sweep, the second-order products and HSS((eta M0 u)^); third sweep (CUBIC), the
// third-order ones and HSS((A3 + B3 / 2)^).  Fields to physical space in iteration 0:
// (M0 u, H(eta) or d_x u), or (L eta M0 u, H(eta)); then the images of the operand q under
// C_j, 4 (it - 1) + r.  Fields back: 0, 1, 2 the products, 3 + j gam_j q, at index at the sum.
// HS3 on a flat bottom has no references and enters the second sweep with eta, u in
// slice A, M0 u, d_x u in slice B (START).
template <int M, bool CUBIC>
struct OpRest {
  const double* __restrict__ gam;
  double2 *PE, *PM, *PA;
  double* S;
  int N, K, it, at, more, start;
  Listing<M> list;
  __device__ __forceinline__ OpRest(Ctx<M> X, int it_)
      : gam(X.d.gam), PE(X.d.sc[0]), PM(X.d.sc[1]), PA(X.d.sc[7]), S(reinterpret_cast<double*>(X.d.sc[5])), N(X.d.N),
        K(refs(X)), it(it_), at(rest_plan(refs(X)).at), more(it_ + 1 < rest_plan(refs(X)).nit),
        start(!CUBIC && refs(X) == 0 && it_ == 0), list(X) {}
  struct L { double2 e, m; double lm, s, g[5]; };   // g[m]: gam of reference 4 it - 4 + m
  __device__ __forceinline__ L load(int n) const {
    L l;
    l.e = l.m = czero();
    l.lm = l.s = 0.0;
    if (!start) l.e = PE[n];
    if (it > 0 || CUBIC) l.m = PM[n];
    if (CUBIC && it > 0) l.lm = PA[n].x;
    if (it > 1) l.s = S[n];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const int j = 4 * it - 4 + m;
      l.g[m] = j >= 0 && j < K ? __ldg(gam + size_t(j) * N + n) : 0.0;
    }
    return l;
  }
  __device__ __forceinline__ void operator()(int n, const L& l, double2& a, double2& b) const {
    double2 e = l.e, m = l.m;
    double lm = l.lm;
    if (it == 0) {
      if (CUBIC) {
        PA[n] = a;
        lm = a.x;
      } else {
        if (start) {
          e = a;
          PE[n] = e;
          list(n, e.x);
        }
        m = start ? b : a;
        PM[n] = m;
      }
    }
    // (1d/functions.c:1486-1498, 1590-1625, 3515-3540)
    const double q = CUBIC ? e.x * lm + 0.5 * (e.x * e.x * m.y) : e.x * m.x;
    if (it == 0) {
      a = CUBIC ? make_double2(e.x * e.x * m.x, m.x * (e.x * m.y + lm)) : make_double2(e.x * e.y, q);
      b = make_double2(CUBIC ? q : e.y * e.y - m.x * m.x, l.g[4] * q);
      return;
    }
    const double s = l.s + (l.g[0] * a.x + l.g[1] * a.y + l.g[2] * b.x + l.g[3] * b.y);
    if (more) S[n] = s;
    double o[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) o[r] = 4 * it + r == at ? s : l.g[r + 1] * q;
    a = make_double2(o[0], o[1]);
    b = make_double2(o[2], o[3]);
  }
};

// the four real fields' spectra at a pair: f at the first point, g at its partner
struct Four {
  double2 f[4], g[4];
  __device__ __forceinline__ Four(const PairAt& r, double2 z, double2 zp, double2 y, double2 yp) {
    f[0] = split_re(z, r.self ? z : zp);
    f[1] = split_im(z, r.self ? z : zp);
    f[2] = split_re(y, r.self ? y : yp);
    f[3] = split_im(y, r.self ? y : yp);
    if (r.self) {
      g[0] = split_re(zp, zp);
      g[1] = split_im(zp, zp);
      g[2] = split_re(yp, yp);
      g[3] = split_im(yp, yp);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] = cconj(f[i]);
    }
  }
};

// Spectral side of one iteration: field r of the four is the image of reference j0 + r
// (0 <= j0 + r < K), the sum (index at - 4 it) or something else.  Returns the pair's
// parts of sum_j C_j F(gam_j q) + F(sum) added to acc.
struct RefRows {
  double c[4], cq[4];
  __device__ __forceinline__ void load(const double* __restrict__ Csq, int N, int K, int j0, const PairAt& r) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = j0 + i;
      const bool in = j >= 0 && j < K;
      c[i] = in ? __ldg(Csq + size_t(j) * N + r.p) : 0.0;
      cq[i] = in ? __ldg(Csq + size_t(j) * N + r.pp) : 0.0;
    }
  }
  __device__ __forceinline__ void add_sum(int s) {   // field s carries the summed images
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i == s) c[i] = cq[i] = 1.0;
  }
};

// the images of a^ under references j0 .. j0 + 3 into the slices
__device__ __forceinline__ void emit_refs(double2* A, double2* Aq, double2* B, double2* Bq, const PairAt& r,
                                          const RefRows& t, int n, double2 a, double2 ap, double invN) {
  emit_pair(A, Aq, r, cscale(a, t.c[0]), cscale(ap, t.cq[0]), cscale(a, t.c[1]), cscale(ap, t.cq[1]), invN);
  if (n == 2) emit_pair(B, Bq, r, cscale(a, t.c[2]), cscale(ap, t.cq[2]), cscale(a, t.c[3]), cscale(ap, t.cq[3]), invN);
}

// Spectral side of the first sweep's iteration `it`: the pair's owner adds its part of the
// sum and forms the next input in place, at the end M0 u^ with H(eta) or d_x u.
template <int M>
__device__ __noinline__ void first_spectral(Ctx<M> X, int it, int nout) {
  const DevMember& d = X.d;
  constexpr int T = Ctx<M>::T;
  const int N = d.N, K = d.nref, at = first_plan(K).at, last = it + 1 == first_plan(K).nit;
  const bool hs3 = d.model == 3, brk = d.brk != 0;
  const double invN = d.invN;
  double2 *acc = d.sc[4], *M0h = d.sc[6];
  const double2 *ZE = d.zs, *ZU = d.zs + N;
  const double* __restrict__ kt = d.k;
  const PairBufs<M> pb(X);
  double2 *A = X.buf, *B = X.buf2();
  const int nnext = K + 2 - 4 * (it + 1) > 2 ? 2 : 1;
#pragma unroll 1
  for (int u = 0; u < kPts / 2; ++u) {
    const PairAt r = pair_at<M>(X.c, pb.cq, int(threadIdx.x) + u * T);
    RefRows back, next;
    back.load(d.Csq, N, K, 4 * it, r);
    back.add_sum(at - 4 * it);
    double2 s = czero(), sq = czero();
    if (it > 0) {
      s = acc[r.p];
      sq = acc[r.pp];
    }
    // the next input's operands: u^ again, or (last) eta^ and u^ with k
    const double2 w = ZU[r.p], wp = ZU[r.pp], e = ZE[r.p], ep = ZE[r.pp];
    const double k = kt[r.p], kq = kt[r.pp];
    if (!last) next.load(d.Csq, N, K, 4 * it + 2, r);
    const double2 y = nout == 2 ? B[pidx(r.i)] : czero(), yp = nout == 2 ? pb.Bq[pidx(r.j)] : czero();
    const Four F(r, A[pidx(r.i)], pb.Aq[pidx(r.j)], y, yp);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s = cadd(s, cscale(F.f[i], back.c[i]));
      sq = cadd(sq, cscale(F.g[i], back.cq[i]));
    }
    if (!last) {
      acc[r.p] = s;
      acc[r.pp] = sq;
      emit_refs(A, pb.Aq, B, pb.Bq, r, next, nnext, w, wp, invN);
    } else {
      // M0 u^ = -i k HSS / g
      const double2 m = cmi(0.5 / kG * k, s), mq = cmi(0.5 / kG * kq, sq);
      M0h[r.p] = m;
      M0h[r.pp] = mq;
      double2 h = czero(), hq = czero();
      if (hs3) {
        h = cmi(-k, w);
        hq = cmi(-kq, wp);
      } else if (brk) {
        h = hilbert_hat(k, e);
        hq = hilbert_hat(kq, ep);
      }
      emit_pair(A, pb.Aq, r, m, mq, h, hq, invN);
    }
  }
}

// Spectral side of a later sweep's iteration (see OpRest): the model's terms in iteration 0,
// the sum, and at the end L q^ into the terms and the next input (the nonlinear adjustment's,
// or, under HS3 after the second-order sweep, L (eta M0 u)^ with H(eta)).
template <int M, bool CUBIC>
__device__ __noinline__ void rest_spectral(Ctx<M> X, int it, int nout) {
  const DevMember& d = X.d;
  constexpr int T = Ctx<M>::T;
  const int N = d.N, K = refs(X), at = rest_plan(K).at, last = it + 1 == rest_plan(K).nit;
  const bool hs3 = d.model == 3, brk = d.brk != 0, final_sweep = CUBIC || !hs3;
  const double invN = d.invN;
  double2 *AE = d.sc[2], *AU = d.sc[3], *acc = d.sc[4], *Q = d.sc[10];
  const double2* ZE = d.zs;
  const double* __restrict__ kt = d.k;
  const double* __restrict__ c1t = d.c1;
  const PairBufs<M> pb(X);
  double2 *A = X.buf, *B = X.buf2();
  const int nnext = K - 4 * it > 2 ? 2 : 1;
#pragma unroll 1
  for (int u = 0; u < kPts / 2; ++u) {
    const PairAt r = pair_at<M>(X.c, pb.cq, int(threadIdx.x) + u * T);
    RefRows back, next;
    back.load(d.Csq, N, K, 4 * it - 3, r);
    if (K > 0) back.add_sum(at - 4 * it);
    double2 s = czero(), sq = czero(), q = czero(), qq = czero(), ae = czero(), aeq = czero(), au = czero(),
            auq = czero(), e = czero(), ep = czero();
    if (it > 0) {
      s = acc[r.p];
      sq = acc[r.pp];
      q = Q[r.p];
      qq = Q[r.pp];
    }
    const double k = kt[r.p], kq = kt[r.pp];
    const double L = K > 0 ? 0.5 / kG * (k * k) : k * c1t[r.p], Lq = K > 0 ? 0.5 / kG * (kq * kq) : kq * c1t[r.pp];
    if (CUBIC || it > 0) {
      ae = AE[r.p];
      aeq = AE[r.pp];
      au = AU[r.p];
      auq = AU[r.pp];
    }
    if (!CUBIC && hs3 && brk && last) {
      e = ZE[r.p];
      ep = ZE[r.pp];
    }
    if (!last) next.load(d.Csq, N, K, 4 * it, r);
    const double2 y = nout == 2 ? B[pidx(r.i)] : czero(), yp = nout == 2 ? pb.Bq[pidx(r.j)] : czero();
    const Four F(r, A[pidx(r.i)], pb.Aq[pidx(r.j)], y, yp);
    if (it == 0) {
      if (CUBIC) {
        // D3, F3: -k^2 D3^ / 2 and -i k F3^
        ae = make_double2(ae.x - 0.5 * (k * k) * F.f[0].x, ae.y - 0.5 * (k * k) * F.f[0].y);
        aeq = make_double2(aeq.x - 0.5 * (kq * kq) * F.g[0].x, aeq.y - 0.5 * (kq * kq) * F.g[0].y);
        au = cadd(au, cmi(k, F.f[1]));
        auq = cadd(auq, cmi(kq, F.g[1]));
      } else {
        // -i k (eta u)^ and -i k (u^2 - (M0 u)^2)^ / 2
        ae = cmi(k, F.f[0]);
        aeq = cmi(kq, F.g[0]);
        au = cmi(0.5 * k, F.f[2]);
        auq = cmi(0.5 * kq, F.g[2]);
      }
      q = CUBIC ? F.f[2] : F.f[1];
      qq = CUBIC ? F.g[2] : F.g[1];
      if (!last) {
        Q[r.p] = q;
        Q[r.pp] = qq;
      }
      if (K > 0) {
        s = cscale(F.f[3], back.c[3]);
        sq = cscale(F.g[3], back.cq[3]);
      } else {   // flat: the operator's multiplier is the table's
        s = q;
        sq = qq;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        s = cadd(s, cscale(F.f[i], back.c[i]));
        sq = cadd(sq, cscale(F.g[i], back.cq[i]));
      }
    }
    if (last) {
      // L q^ = k^2 HSS / g: minus L (eta M0 u)^, or plus L (A3 + B3 / 2)^
      const double2 l = cscale(s, L), lq = cscale(sq, Lq);
      ae = CUBIC ? cadd(ae, l) : csub(ae, l);
      aeq = CUBIC ? cadd(aeq, lq) : csub(aeq, lq);
      if (final_sweep) {
        emit_pair(A, pb.Aq, r, ae, aeq, au, auq, invN);   // into the nonlinear adjustment
      } else {
        emit_pair(A, pb.Aq, r, l, lq, brk ? hilbert_hat(k, e) : czero(), brk ? hilbert_hat(kq, ep) : czero(), invN);
      }
    } else {
      acc[r.p] = s;
      acc[r.pp] = sq;
      emit_refs(A, pb.Aq, B, pb.Bq, r, next, nnext, q, qq, invN);
    }
    if (it == 0 || (last && !final_sweep)) {
      AE[r.p] = ae;
      AE[r.pp] = aeq;
      AU[r.p] = au;
      AU[r.pp] = auq;
    }
  }
}

template <int M, bool CUBIC>
__device__ __forceinline__ void rest_sweep(Ctx<M> X, double t) {
  const int nit = rest_plan(refs(X)).nit;
  const bool final_sweep = CUBIC || X.d.model != 3;
  for (int it = 0; it < nit; ++it) {
    const int K = refs(X), nout = rest_plan(K).at + 1 - 4 * it > 2 ? 2 : 1;
    const int nin = it == 0 ? (!CUBIC && K == 0 ? 2 : 1) : (K - 4 * (it - 1) > 2 ? 2 : 1);
    meet<M, OpRest<M, CUBIC>>(X, nin, nout, it);
    // breaking criterion on eta, u, H(eta), complete member-wide by now
    const bool done = final_sweep && it + 1 == nit;
    const double* Heta = X.d.model == 3 ? &X.d.sc[7][0].y : &X.d.sc[1][0].y;
    if (X.d.brk && done) breaking_scan(X, X.d.sc[0], Heta, 2);
    member_sync(X.d.C);
    rest_spectral<M, CUBIC>(X, it, nout);
    if (done) lead_and_influx(X, t, X.d.sc[0], Heta);
    if (X.d.C > 1) cg::this_cluster().sync();
  }
}

// Scratch fields: sc[0] eta, u in physical space; sc[1] M0 u with H(eta) or d_x u; sc[2], sc[3]
// spectral terms; sc[4] spectral and sc[5] physical sum of an HSS; sc[6] M0 u^; sc[7] L (eta M0 u)
// with H(eta); sc[8] the breaking flux; sc[10] the operand's spectrum; sc[11] the breaking force.
template <int M>
__device__ __noinline__ void rhs_gen(Ctx<M> X, double t, double2* __restrict__ dz) {
  const int C = X.d.C;
  breaking_reset(X);
  if (X.d.model == 1) {
    stage_phase<M, kWithNone>(X);
    meet<M, OpLinear<M>>(X, 1, 1, 0);
    lead_and_influx(X, t, nullptr, nullptr);
    member_sync(C);
    assemble<M, kAsmLinear, false>(X, dz, nullptr, nullptr, nullptr, nullptr);
    member_sync(C);
    return;
  }
  if (X.d.flat) {
    stage_phase<M, kWithM0Dx>(X);
  } else {
    stage_phase<M, kWithRefs>(X);
    const int nit = first_plan(X.d.nref).nit;
    for (int it = 0; it < nit; ++it) {
      const int K = X.d.nref, nin = K + 2 - 4 * it > 2 ? 2 : 1, nout = first_plan(K).at + 1 - 4 * it > 2 ? 2 : 1;
      meet<M, OpFirst<M>>(X, nin, nout, it);
      member_sync(C);
      first_spectral(X, it, nout);
      if (C > 1) cg::this_cluster().sync();
    }
  }
  rest_sweep<M, false>(X, t);
  if (X.d.model == 3) rest_sweep<M, true>(X, t);
  finish_rhs(X, dz, X.d.flat ? nullptr : X.d.sc[6]);
}

}  // namespace hwdev
