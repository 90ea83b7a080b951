// hw_rhs_fast.cuh -- HS2 on a flat bottom (rhs_HsF2 with ifft_fft_Hsf2,
// 1d/rhs.c:96-241, 1d/functions.c:1458-1526), the hot path of the plain and the
// batched runs, with the fields kept in two shared-memory slices:
//   * stage input -> Hermitian packing, pair by pair;
//   * eta, u and M0 u, Hilbert(eta) from one dual inverse transform;
//   * the three real products from one dual forward transform;
//   * the nonlinear adjustment: one inverse transform, ChiAdj, and a dual forward
//     transform that also carries the damping of eta and u.
// What bounds it: the latency of the loads between the transforms.  Each phase names
// its loads before its stores, the pair's owner forms both of its points (half the
// table loads), and outside the alias band, where aal = 0 and every k_j is zero (half
// the pairs under HS2), nothing but y is read.  Against loads taken point by point
// (B200, 256 ragged members, thousand cycles a CTA and RHS): stage input 57 -> 16,
// assembly 32 -> 10, H2 terms 14 -> 5, criterion 21 -> 7, the transforms 38 as before;
// three output samples of the ensemble 111 -> 69 ms, ten of one 4096-point tank (512-point
// slices) 27.6 -> 17.1 ms.
#pragma once

#include "hw_rhs.cuh"

namespace hwdev {

// (A + i B) s of a pair's first point, and of its partner, from the Hermitian parts
// A, B at the first (the partner's are their conjugates)
__device__ __forceinline__ double2 pack_conj(double2 a, double2 b, double s) {
  return make_double2((a.x + b.y) * s, (b.x - a.y) * s);
}

// shared-memory slices of the CTA that holds the partners
template <int M>
struct PairBufs {
  double2 *Aq, *Bq;
  int cq;
  __device__ __forceinline__ explicit PairBufs(Ctx<M> X) {
    cq = (X.d.C - X.c) & (X.d.C - 1);
    Aq = X.buf;
    Bq = X.buf2();
    if (cq != X.c) {
      cg::cluster_group cl = cg::this_cluster();
      Aq = cl.map_shared_rank(X.buf, cq);
      Bq = cl.map_shared_rank(X.buf2(), cq);
    }
  }
};

// one complex transform's input at a pair from two spectra x, y (given at both points,
// not necessarily Hermitian): (herm x + i herm y) / N, real parts only as the reference
__device__ __forceinline__ void emit_pair(double2* A, double2* Aq, const PairAt& r, double2 x, double2 xp, double2 y,
                                          double2 yp, double invN) {
  if (r.self) {   // (one thread of a member)
    A[pidx(r.i)] = pack(herm(x, x), herm(y, y), invN);
    A[pidx(r.j)] = pack(herm(xp, xp), herm(yp, yp), invN);
  } else {
    const double2 E = herm(x, xp), F = herm(y, yp);
    A[pidx(r.i)] = pack(E, F, invN);
    Aq[pidx(r.j)] = pack_conj(E, F, invN);
  }
}
__device__ __forceinline__ double2 cmi(double s, double2 a) { return make_double2(s * a.y, -s * a.x); }   // -i s a
__device__ __forceinline__ double2 czero() { return make_double2(0.0, 0.0); }
// Hilbert transform's multiplier (1d/breaking.c:133-143): -i sign(k)
__device__ __forceinline__ double2 hilbert_hat(double k, double2 e) {
  return k == 0 ? czero() : cmi(copysign(1.0, k), e);
}

// what the first inverse transform carries beside eta and u
enum : int { kWithM0Hilbert = 0, kWithM0Dx = 1, kWithRefs = 2, kWithNone = 3 };

// Stage input of stage S (y + h sum_j b_sj k_j, kept in zs for the assembly) and its
// Hermitian packing for the first inverse transform: A <- eta^ + i u^ and, by `with`,
// B <- M0 u^ + i H(eta)^ (flat HS2), M0 u^ + i (d_x u)^ (flat HS3), the images of u^
// under the first two reference depths (varying bottom) or nothing (HS1).  On a flat
// bottom M0 u^ = -i c1 u^, and the Hilbert multiplier takes the sign of c1 = (C^2/g) k.
// The stage is a template argument so that a pair's loads (up to 24) are independent
// of any branch and in flight together.
template <int M, int S, int WITH>
__device__ __noinline__ void stage_pack(Ctx<M> X) {
  const DevMember& d = X.d;
  constexpr int T = Ctx<M>::T;
  const double2* y = X.sc->stg.y;
  const double2* ks[S > 1 ? S - 1 : 1];
#pragma unroll
  for (int j = 0; j < S - 1; ++j) ks[j] = X.sc->stg.k[j];
  const double h = X.sc->stg.h, invN = d.invN;
  const int N = d.N, c = X.c, act = d.act;
  const double* __restrict__ t1 = WITH == kWithRefs ? d.Csq : d.c1;
  const double* __restrict__ t2 = WITH == kWithRefs ? d.Csq + N : d.k;
  double2* zw = d.zs;
  const bool brk = d.brk != 0;
  const PairBufs<M> pb(X);
  double2 *A = X.buf, *B = X.buf2(), *Aq = pb.Aq, *Bq = pb.Bq;
  auto emit = [&](const PairAt& r, double a, double aq, double b, double bq, double2 e, double2 ep, double2 w, double2 wp) {
    emit_pair(A, Aq, r, e, ep, w, wp, invN);
    if constexpr (WITH == kWithM0Hilbert) {
      double2 s = czero(), sp = czero();
      if (brk) {
        s = hilbert_hat(a, e);
        sp = hilbert_hat(aq, ep);
      }
      emit_pair(B, Bq, r, cmi(a, w), cmi(aq, wp), s, sp, invN);
    } else if constexpr (WITH == kWithM0Dx) {
      emit_pair(B, Bq, r, cmi(a, w), cmi(aq, wp), cmi(-b, w), cmi(-bq, wp), invN);
    } else if constexpr (WITH == kWithRefs) {
      emit_pair(B, Bq, r, cscale(w, a), cscale(wp, aq), cscale(w, b), cscale(wp, bq), invN);
    }
  };
#pragma unroll 1
  for (int u = 0; u < kPts / 2; ++u) {
    const PairAt r = pair_at<M>(c, pb.cq, int(threadIdx.x) + u * T);
    double a = 0.0, aq = 0.0, b = 0.0, bq = 0.0;
    if constexpr (WITH != kWithNone) {
      a = t1[r.p];
      aq = t1[r.pp];
    }
    if constexpr (WITH == kWithM0Dx || WITH == kWithRefs) {
      b = t2[r.p];
      bq = t2[r.pp];
    }
    if (r.i < act) {
      StageOps<S> oe, oep, ow, owp;
      oe.load(y, ks, r.p);
      oep.load(y, ks, r.pp);
      ow.load(y, ks, N + r.p);
      owp.load(y, ks, N + r.pp);
      const double2 e = oe.value(h), ep = oep.value(h), w = ow.value(h), wp = owp.value(h);
      if (S > 1 || zw != y) {   // (a direct RHS's state is zs itself)
        zw[r.p] = e;
        zw[r.pp] = ep;
        zw[N + r.p] = w;
        zw[N + r.pp] = wp;
      }
      emit(r, a, aq, b, bq, e, ep, w, wp);
    } else {
      emit(r, a, aq, b, bq, y[r.p], y[r.pp], y[N + r.p], y[N + r.pp]);
    }
  }
}

// the stage phase with its barriers.  Every RHS leaves the slices unread by the other
// CTAs (a barrier follows its last partner reads), so they can be written at once; with
// zs written by the caller (stage 0), other threads' writes of it and the start of the
// partner CTA come first.
template <int M, int WITH>
__device__ __forceinline__ void stage_phase(Ctx<M> X) {
  __syncthreads();   // the stage description
  const int stage = X.sc->stg.s;
  if (stage == 0) {
    member_sync(X.d.C);
    if (threadIdx.x == 0) X.sc->stg.y = X.d.zs;
    __syncthreads();
  }
  switch (stage) {
    case 2: stage_pack<M, 2, WITH>(X); break;
    case 3: stage_pack<M, 3, WITH>(X); break;
    case 4: stage_pack<M, 4, WITH>(X); break;
    case 5: stage_pack<M, 5, WITH>(X); break;
    case 6: stage_pack<M, 6, WITH>(X); break;
    default: stage_pack<M, 1, WITH>(X); break;
  }
  if (X.d.C > 1) cg::this_cluster().sync();   // the partners' slices are written
}

// the influx source term of the assembly (1d/rhs.c:659-693) from the loaded kernels
__device__ __forceinline__ double2 source_term(int mode, double2 gx, double2 gs, double pv, double ps) {
  if (mode == 0) return make_double2(0.5 * (pv * gx.x - ps * gs.x), 0.5 * (pv * gx.y - ps * gs.y));
  if (mode == 1) return make_double2(0.5 * (pv * gx.x + ps * gs.x), 0.5 * (pv * gx.y + ps * gs.y));
  if (mode == 2) return make_double2(pv * gx.x, pv * gx.y);
  return make_double2(0.0, 0.0);
}

// Cluster members: the inverse transform's cross-CTA step, the pointwise work in
// physical space and the next forward transform's cross-CTA step meet at the same
// index set -- position i of every CTA's slice, i.e. the physical points r M + i
// (r = 0..C-1) -- so the thread owning position i (the ownership of cross_gs) does
// all three in registers: gather, twiddle, inverse C-point DFT, pointwise step,
// forward C-point DFT, twiddle, scatter.  Two cluster barriers replace four and the
// physical fields never pass through shared memory.

// What the first meeting does at physical point n (1d/functions.c:1486-1498), given
// e = (eta, u), m = (M0 u, H(eta)): a <- (eta u) + i (eta M0 u), b <- u^2 - (M0 u)^2.
// (eta, u) goes to global memory where the damping zones read it back, and with
// breaking everywhere, beside H(eta) and a list of the points above the threshold.
template <int M>
__device__ __forceinline__ void product_point(Ctx<M> X, int n, double2 e, double2 m, double damp, double2* PE,
                                              double2* PM, double2& a, double2& b) {
  const DevMember& d = X.d;
  if (d.brk) {
    PE[n] = e;
    PM[n].y = m.y;
    if (n >= d.xbstart && n < d.xbstart + d.lenIF && !(e.x < d.MaxEtaInit))
      X.sc->cand[atomicAdd(&X.sc->ncand, 1)] = (unsigned short)n;
  } else if (damp != 0.0) {
    PE[n] = e;
  }
  a = make_double2(e.x * e.y, e.x * m.x);
  b = make_double2(e.y * e.y - m.x * m.x, 0.0);
}

// What the second meeting does (1d/rhs.c:695-715): the nonlinear terms times ChiAdj,
// paired with the damping of eta and u
__device__ __forceinline__ void adjust_point(const double2* PE, int n, double chi, double damp, double2& a, double2& b) {
  a = make_double2(a.x * chi, a.y * chi);
  b = make_double2(0.0, 0.0);
  if (damp != 0.0) {
    const double2 e = PE[n];
    b = make_double2(damp * e.x, damp * e.y);
  }
}

template <int M, int C>
__device__ __forceinline__ void cross_products(Ctx<M> X, double2* A, double2* B, double2* PE, double2* PM) {
  using P = Cross<C>;
  constexpr int T = M / kPts, R = P::R;
  const DevMember& d = X.d;
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
#pragma unroll
  for (int q = 0; q < P::PER; ++q) {
    const int i = P::template at<T>(X.c, q);
    double2 va[R], vb[R];
    double dm[R];
#pragma unroll
    for (int e = 0; e < R; ++e) {
      va[e] = cl.map_shared_rank(A, P::spectral(e))[pidx(i)];
      vb[e] = cl.map_shared_rank(B, P::spectral(e))[pidx(i)];
      dm[e] = __ldg(d.damp + P::physical(e) * M + i);
    }
    cross_in<C>(va, d.tw, i);
    cross_in<C>(vb, d.tw, i);
#pragma unroll
    for (int e = 0; e < R; ++e)
      product_point<M>(X, P::physical(e) * M + i, va[e], vb[e], dm[e], PE, PM, va[e], vb[e]);
    cross_out<C>(va, d.tw, i);
    cross_out<C>(vb, d.tw, i);
#pragma unroll
    for (int e = 0; e < R; ++e) {
      cl.map_shared_rank(A, P::spectral(e))[pidx(i)] = va[e];
      cl.map_shared_rank(B, P::spectral(e))[pidx(i)] = vb[e];
    }
  }
  cl.sync();
}

template <int M, int C>
__device__ __forceinline__ void cross_adjust(Ctx<M> X, double2* A, double2* B, const double2* PE) {
  using P = Cross<C>;
  constexpr int T = M / kPts, R = P::R;
  const DevMember& d = X.d;
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
#pragma unroll
  for (int q = 0; q < P::PER; ++q) {
    const int i = P::template at<T>(X.c, q);
    double2 va[R], vb[R];
    double dm[R], ch[R];
#pragma unroll
    for (int e = 0; e < R; ++e) {
      va[e] = cl.map_shared_rank(A, P::spectral(e))[pidx(i)];
      dm[e] = __ldg(d.damp + P::physical(e) * M + i);
      ch[e] = __ldg(d.chi + P::physical(e) * M + i);
    }
    cross_in<C>(va, d.tw, i);
#pragma unroll
    for (int e = 0; e < R; ++e) adjust_point(PE, P::physical(e) * M + i, ch[e], dm[e], va[e], vb[e]);
    cross_out<C>(va, d.tw, i);
    cross_out<C>(vb, d.tw, i);
#pragma unroll
    for (int e = 0; e < R; ++e) {
      cl.map_shared_rank(A, P::spectral(e))[pidx(i)] = va[e];
      cl.map_shared_rank(B, P::spectral(e))[pidx(i)] = vb[e];
    }
  }
  cl.sync();
}

template <int M>
__device__ __forceinline__ void cross_products_any(Ctx<M> X, double2* A, double2* B, double2* PE, double2* PM) {
  if (X.d.C == 2) cross_products<M, 2>(X, A, B, PE, PM);
  else if (X.d.C == 4) cross_products<M, 4>(X, A, B, PE, PM);
  else if (X.d.C == 8) cross_products<M, 8>(X, A, B, PE, PM);
  else cross_products<M, 16>(X, A, B, PE, PM);
}
template <int M>
__device__ __forceinline__ void cross_adjust_any(Ctx<M> X, double2* A, double2* B, const double2* PE) {
  if (X.d.C == 2) cross_adjust<M, 2>(X, A, B, PE);
  else if (X.d.C == 4) cross_adjust<M, 4>(X, A, B, PE);
  else if (X.d.C == 8) cross_adjust<M, 8>(X, A, B, PE);
  else cross_adjust<M, 16>(X, A, B, PE);
}

// Assembly of dz (1d/rhs.c:217-228, 373-385, 73-83): delta H1 + adjusted nonlinear terms
// + breaking force + 2 force - damping, times aal, for the pairs inside the alias band;
// outside it dz is zero, and was when the buffer was made.  delta H1 of eta is M0h on a varying
// bottom (VAR), else -i c1 u^.  MODE: the adjusted terms come from slice A
// (damping from B), from scratch with the force (some node breaks; damping from B), or
// there are none (HS1; damping from A).
enum : int { kAsmSlices = 0, kAsmLive = 1, kAsmLinear = 2 };
template <int M, int MODE, bool VAR>
__device__ __noinline__ void assemble(Ctx<M> X, double2* __restrict__ dz, const double2* M0h, const double2* AE,
                                      const double2* AU, const double2* RB) {
  const DevMember& d = X.d;
  constexpr int T = Ctx<M>::T;
  const int N = d.N, c = X.c, act = d.act, mode = d.has_influx ? d.prop_mode : 3;
  const PairBufs<M> pb(X);
  const double2 *A = X.buf, *Aq = pb.Aq;
  const double2 *B = MODE == kAsmLinear ? X.buf : X.buf2(), *Bq = MODE == kAsmLinear ? pb.Aq : pb.Bq;
  const double2* zs = d.zs;
  const double* __restrict__ kt = d.k;
  const double* __restrict__ c1t = d.c1;
  const double* __restrict__ aalt = d.aal;
  const double2* __restrict__ gxt = d.gamX;
  const double2* __restrict__ gst = d.gamXs;
  const int sig = X.sc->stg.sig;
  const double pv = sig < 0 ? X.sc->red[kRedPv] : X.sc->sig[sig].x, ps = sig < 0 ? X.sc->red[kRedPs] : X.sc->sig[sig].y;
#pragma unroll 1
  for (int u = 0; u < kPts / 2; ++u) {
    const PairAt r = pair_at<M>(c, pb.cq, int(threadIdx.x) + u * T);
    if (r.i >= act) {
      if (X.sc->full) dz[r.p] = dz[r.pp] = dz[N + r.p] = dz[N + r.pp] = czero();
      continue;
    }
    const int pos[2] = {r.p, r.pp};
    double2 ze[2], h1[2], gx[2], gs[2], ae[2], au[2];
    double kk[2], c1[2], al[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      ze[s] = zs[pos[s]];
      h1[s] = VAR ? M0h[pos[s]] : zs[N + pos[s]];
      c1[s] = VAR ? 0.0 : c1t[pos[s]];
      kk[s] = kt[pos[s]];
      al[s] = aalt[pos[s]];
      gx[s] = gs[s] = ae[s] = au[s] = czero();
      if (mode != 3) {
        gx[s] = gxt[pos[s]];
        gs[s] = gst[pos[s]];
      }
      if constexpr (MODE == kAsmLive) {
        const double2 f = RB[pos[s]];
        ae[s] = AE[pos[s]];
        au[s] = cadd(AU[pos[s]], f);
      }
    }
    const double2 z = A[pidx(r.i)], zp = Aq[pidx(r.j)], zb = B[pidx(r.i)], zbp = Bq[pidx(r.j)];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const double2 a = s ? zp : z, b = s ? zbp : zb;
      const double2 aq = r.self ? a : (s ? z : zp), bq = r.self ? b : (s ? zb : zbp);
      if constexpr (MODE == kAsmSlices) {
        ae[s] = split_re(a, aq);
        au[s] = split_im(a, aq);
      }
      const double2 de = split_re(b, bq), du = split_im(b, bq);
      const double gk = kG * kk[s];
      const double2 f = source_term(mode, gx[s], gs[s], pv, ps);
      const double2 te = cadd(VAR ? h1[s] : cmi(c1[s], h1[s]), ae[s]);
      const double2 tu = make_double2(gk * ze[s].y + au[s].x, -gk * ze[s].x + au[s].y);
      dz[pos[s]] = make_double2((te.x + 2 * f.x - de.x) * al[s], (te.y + 2 * f.y - de.y) * al[s]);
      dz[N + pos[s]] = make_double2((tu.x - du.x) * al[s], (tu.y - du.y) * al[s]);
    }
  }
}

// beside the last spectral phase: the breaking machine's leader and, where the step has not
// formed them, by another thread the influx signals at the stage time (read after the
// phase's barrier)
template <int M>
__device__ __forceinline__ void lead_and_influx(Ctx<M> X, double t, const double2* PE, const double* Heta) {
  if (X.d.brk) breaking_lead(X, t, PE, Heta, 2);
  if (X.d.has_influx && X.sc->stg.sig < 0 && int(threadIdx.x) == Ctx<M>::T - 1) {
    const double2 s = influx_at(X.d, t);
    X.sc->red[kRedPv] = s.x;
    X.sc->red[kRedPs] = s.y;
  }
}

// From the packed nonlinear terms in slice A to dz: the nonlinear adjustment with the
// damping, the breaking force where some node breaks, the assembly.
template <int M>
__device__ __noinline__ void finish_rhs(Ctx<M> X, double2* __restrict__ dz, const double2* M0h) {
  const DevMember& d = X.d;
  constexpr int T = Ctx<M>::T;
  const int C = d.C;
  double2* A = X.buf;
  double2* Bf = X.buf2();
  const double2* PE = d.sc[0];
  if (C > 1) {
    fft_local<M>(A, d.tw, C, +1);
    cross_adjust_any<M>(X, A, Bf, PE);
    fft_local2<M>(A, Bf, d.tw, C, -1);
  } else {
    double dm[kPts], ch[kPts];
    HW_FOREACH(X) {
      (void)idx;
      dm[u] = __ldg(d.damp + p);
      ch[u] = __ldg(d.chi + p);
    }
    fft_inverse<M>(A, d.tw, C, X.c);
    HW_FOREACH(X) {
      double2 a = A[pidx(idx)], b;
      adjust_point(PE, p, ch[u], dm[u], a, b);
      A[pidx(idx)] = a;
      Bf[pidx(idx)] = b;
    }
    fft_forward2<M>(A, Bf, d.tw, C, X.c);
  }
  member_sync(C);
  // (the leader's word is in every CTA since the transforms' barriers)
  const bool rb_live = d.brk != 0 && X.sc->live;
  if (!rb_live) {
    if (M0h) assemble<M, kAsmSlices, true>(X, dz, M0h, nullptr, nullptr, nullptr);
    else assemble<M, kAsmSlices, false>(X, dz, nullptr, nullptr, nullptr, nullptr);
    member_sync(C);   // the partner reads of the slices are done
    return;
  }
  // kinematic breaking: the eddy-viscosity force on the u-equation takes slice A, so
  // the adjusted terms move to global memory; the damping stays in slice B
  double2 *AE = d.sc[2], *AU = d.sc[3], *RB = d.sc[11];
  const PairBufs<M> pb(X);
#pragma unroll 1
  for (int u = 0; u < kPts / 2; ++u) {
    const PairAt r = pair_at<M>(X.c, pb.cq, int(threadIdx.x) + u * T);
    const double2 z = A[pidx(r.i)], zp = pb.Aq[pidx(r.j)];
    AE[r.p] = split_re(z, r.self ? z : zp);
    AU[r.p] = split_im(z, r.self ? z : zp);
    AE[r.pp] = split_re(zp, r.self ? zp : z);
    AU[r.pp] = split_im(zp, r.self ? zp : z);
  }
  member_sync(C);
  breaking_force<M>(X, PE, AE, RB);
  member_sync(C);
  if (M0h) assemble<M, kAsmLive, true>(X, dz, M0h, AE, AU, RB);
  else assemble<M, kAsmLive, false>(X, dz, nullptr, AE, AU, RB);
  member_sync(C);
}

template <int M>
__device__ __noinline__ void rhs_hs2_flat(Ctx<M> X, double t, double2* __restrict__ dz) {
  const DevMember& d = X.d;
  constexpr int T = Ctx<M>::T;
  const int C = d.C;
  double2* A = X.buf;
  double2* Bf = X.buf2();
  double2* PE = d.sc[0];   // physical (eta, u)           [breaking, and in the damping zones]
  double2* PM = d.sc[1];   // physical (., Hilbert eta)   [breaking only]
  const bool brk = d.brk != 0;
  const PairBufs<M> pb(X);

  // (0)-(1) stage input and its packing
  breaking_reset(X);
  stage_phase<M, kWithM0Hilbert>(X);
  // (2) products in physical space (1d/functions.c:1486-1498)
  const bool fused = C > 1;
  if (fused) {
    fft_local2<M>(A, Bf, d.tw, C, +1);
    cross_products_any<M>(X, A, Bf, PE, PM);
    fft_local2<M>(A, Bf, d.tw, C, -1);
  } else {
    double dm[kPts];
    HW_FOREACH(X) {
      (void)idx;
      dm[u] = __ldg(d.damp + p);
    }
    fft_inverse2<M>(A, Bf, d.tw, C, X.c);
    HW_FOREACH(X) {
      double2 a, b;
      product_point<M>(X, p, A[pidx(idx)], Bf[pidx(idx)], dm[u], PE, PM, a, b);
      A[pidx(idx)] = a;
      Bf[pidx(idx)] = b;
    }
    fft_forward2<M>(A, Bf, d.tw, C, X.c);
  }
  // breaking criterion (1d/breaking.c:36-95) on eta, u, H(eta): the transform's
  // barriers made PE / PM complete member-wide
  if (brk) breaking_scan(X, PE, &PM[0].y, 2);
  // (3) spectra of the products, H2 terms (1d/rhs.c:141-147) and, in the same
  // pass, the Hermitian packing of the nonlinear adjustment (1d/rhs.c:695-715): the
  // pair's owner reads both transformed values and rewrites them in place
  member_sync(C);
  {
    const double* __restrict__ kt = d.k;
    const double* __restrict__ c1t = d.c1;
    const double invN = d.invN;
    double kk[kPts], cc[kPts];
#pragma unroll
    for (int u = 0; u < kPts / 2; ++u) {
      const PairAt r = pair_at<M>(X.c, pb.cq, int(threadIdx.x) + u * T);
      kk[2 * u] = kt[r.p];
      kk[2 * u + 1] = kt[r.pp];
      cc[2 * u] = c1t[r.p];
      cc[2 * u + 1] = c1t[r.pp];
    }
    // -L (eta M0u)^ - i k (eta u)^ and -i k (u^2 - (M0u)^2)^ / 2 at one point
    auto terms = [&](double k, double c1, double2 a, double2 ap, double2 b, double2 bp, double2& te, double2& tu) {
      const double2 ah = split_re(a, ap), bh = split_im(a, ap), ch = split_re(b, bp);
      const double L = k * c1;
      te = make_double2(-L * bh.x + k * ah.y, -L * bh.y - k * ah.x);
      tu = make_double2(0.5 * k * ch.y, -0.5 * k * ch.x);
    };
#pragma unroll
    for (int u = 0; u < kPts / 2; ++u) {
      const PairAt r = pair_at<M>(X.c, pb.cq, int(threadIdx.x) + u * T);
      const double2 z1 = A[pidx(r.i)], z1p = pb.Aq[pidx(r.j)], z2 = Bf[pidx(r.i)], z2p = pb.Bq[pidx(r.j)];
      double2 te, tu, teq, tuq;
      if (u == 0 && r.self) {
        terms(kk[0], cc[0], z1, z1, z2, z2, te, tu);
        terms(kk[1], cc[1], z1p, z1p, z2p, z2p, teq, tuq);
        A[pidx(r.i)] = pack(herm(te, te), herm(tu, tu), invN);
        A[pidx(r.j)] = pack(herm(teq, teq), herm(tuq, tuq), invN);
        continue;
      }
      terms(kk[2 * u], cc[2 * u], z1, z1p, z2, z2p, te, tu);
      terms(kk[2 * u + 1], cc[2 * u + 1], z1p, z1, z2p, z2, teq, tuq);
      const double2 E = herm(te, teq), U = herm(tu, tuq);
      A[pidx(r.i)] = pack(E, U, invN);
      pb.Aq[pidx(r.j)] = pack_conj(E, U, invN);
    }
  }
  lead_and_influx(X, t, PE, &PM[0].y);
  member_sync(C);
  // (4) nonlinear adjustment, damping, breaking force, assembly
  finish_rhs(X, dz, nullptr);
}

}  // namespace hwdev
