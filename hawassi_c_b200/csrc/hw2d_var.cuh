// hw2d_var.cuh -- HAWASSI 2D right-hand sides on a varying bottom with K reference
// depths (rhs_AB1/AB2/AB3_2DB_uv, 2d/fun_odesolver.c:4350-4402, 4542-4626, 4735-4844;
// fun_termshat_AB1/AB2/AB3_2DB_uv :2874-2960, 3327-3510, 4104-4296; HSSgen_2depth /
// HSSgen_3depth :500-697; K = 2 and 3 in the reference, up to 16 for the plain
// K-reference operator and the learned blend).  The operator of a real field a,
//   HSS(a; O) = 1/2 [ F( sum_j gam_j Re F^-1 S(O_j a^) ) + sum_j O_j F(gam_j a) ],
// takes K real inverse transforms, K real forward ones and one more: the weighted images
// are summed in physical space and go back once.  It is linear, so
//   C^2 u, C^2 v are needed only as kx C^2 u^ + ky C^2 v^ (delphiH1^, and L phi = its
//     image), the second-order operator term only as L (eta L phi)^ of one real field,
//     the third-order ones as L p^ of one (hw2d.cuh, cubic_products).
// Passes:
//   V1 row   (eta, u), (v, -), (C_j u, C_j v) for every j               -> inverse rows
//   V2 col   inverse -> eta, u, v; sum gam_j (C_j u, C_j v), (gam_j u, gam_j v) -> forward
//   V3 row   forward -> delphiH1^ (kept), L phi (HS3: M0u, M0v)         -> inverse rows
//   V4 col   inverse -> the products and gam_j (eta L phi), two to a field -> forward
//   V5 row   forward -> the terms kept, Omega_j (eta L phi)^            -> inverse rows
//   V6 col   inverse -> sum gam_j Omega_j (.)                           -> forward
//   V7 row   forward -> the adjustment's input                          -> inverse rows
// and D, E as on a flat bottom.  HS3: V7 sends (L (eta L phi), div(grad phi)) instead, and
// V4, V5, V6, V7 run once more on the cubic products.  HS1 ends after V3.
// Fields beyond the first few go through the column and row passes two or four slices
// at a time, so a CTA's shared memory does not grow with K and two CTAs share an SM.
#pragma once

#include "hw2d.cuh"

namespace hw2d {

// V1: one CTA per row pair and field (blockIdx.y): 0 (eta, u), 1 (v, -), 2 + j
template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2v_row1(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, Ctl2* ctlw, int mode, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = M, f = blockIdx.y;
  const size_t n = (size_t)tb.n;
  const Pair P = row_pair(blockIdx.x, tb.ny);
  stage_extras(tb, w, P, ctl, ctlw, mode, NT);
  const double* __restrict__ O = tb.ck + (f > 1 ? f - 2 : 0) * n;
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
        } else if (f == 1) {
          x[k][s] = w.z[2 * n + q];
          y[k][s] = zero2();
        } else {
          const double o = O[q];
          x[k][s] = cscale(w.z[n + q], o);
          y[k][s] = cscale(w.z[2 * n + q], o);
        }
      }
    emit_pack(sm, M, 0, Q, tb.ny, x, y);
  }
  fft_slices<M, NT>(sm, 0, 2, tb.twx, +1);
  row_store<M, NT>(sm, 0, 1, w.R + f * n, P, n);
}

// V2: slices 0, 1 the sum, 2..5 two references at a time.  Fields out: 0 the sum
// (u in the real, v in the imaginary part), 1 + j (gam_j u, gam_j v).
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2v_col2(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = tb.nx, c = blockIdx.x, K = tb.nk;
  const size_t n = (size_t)tb.n;
  const double invN = 1.0 / ((double)tb.n);
  col_load<M, NT>(sm, 2, 2, w.R, Nx, c, n);
  fft_slices<M, NT>(sm, 2, 4, tb.twy, +1);
#pragma unroll 4
  for (int t = threadIdx.x; t < 2 * M; t += NT) {
    const ColPt p(t, c, Nx);
    const double2 a = slot(sm, M, 2 + p.k, p.y), b = slot(sm, M, 4 + p.k, p.y);
    w.phys[p.q] = a.x * invN;
    w.phys[n + p.q] = a.y * invN;
    w.phys[2 * n + p.q] = b.x * invN;
    put(sm, M, p.k, p.y, zero2());
  }
  for (int j = 0; j < K; j += 2) {
    const int nj = K - j > 1 ? 2 : 1;
    __syncthreads();   // the slices' last readers are done
    col_load<M, NT>(sm, 2, nj, w.R + (2 + j) * n, Nx, c, n);
    fft_slices<M, NT>(sm, 2, 2 * nj, tb.twy, +1);
#pragma unroll 2
    for (int t = threadIdx.x; t < 2 * M; t += NT) {
      const ColPt p(t, c, Nx);
      const double u = w.phys[n + p.q], v = w.phys[2 * n + p.q];
      double2 s = slot(sm, M, p.k, p.y);
      for (int i = 0; i < nj; ++i) {
        const double g = tb.gk[(j + i) * n + p.q], gn = g * invN;
        const double2 a = slot(sm, M, 2 + 2 * i + p.k, p.y);
        s = cadd(s, cscale(a, gn));
        put(sm, M, 2 + 2 * i + p.k, p.y, make_double2(g * u, g * v));
      }
      put(sm, M, p.k, p.y, s);
    }
    fft_slices<M, NT>(sm, 2, 2 * nj, tb.twy, -1);
    col_store<M, NT>(sm, 2, nj, w.Q + (1 + j) * n, Nx, c, n);
  }
  fft_slices<M, NT>(sm, 0, 2, tb.twy, -1);
  col_store<M, NT>(sm, 0, 1, w.Q, Nx, c, n);
}

// V3: slices 0..3 two fields at a time, 4, 5 the sum kx (.) + ky (.); under HS3 0, 1 one field
// at a time, 2, 3 the sum's kx part at the points that the symmetrisation keeps (columns up
// to Nx / 2)
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2v_row3(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = M, K = tb.nk;
  const size_t n = (size_t)tb.n;
  const bool hs3 = tb.model == 3;
  const Pair P = row_pair(blockIdx.x, tb.ny);
  const int step = hs3 ? 1 : 2;
  for (int f = 0; f <= K; f += step) {
    const int nf = K + 1 - f < step ? 1 : step;
    __syncthreads();
    row_load<M, NT>(sm, 0, nf, w.Q + f * n, P, n);
    fft_slices<M, NT>(sm, 0, 2 * nf, tb.twx, -1);
#pragma unroll 1
    for (int j = threadIdx.x; j < Nx / 2; j += NT) {
      const Quad Q(P, j, Nx);
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const size_t q = Q.at(k, s, Nx);
          const double kx = tb.kx[Q.cc[s]], ky = tb.ky[Q.r[k]];
          // field 0 is the summed images (coefficient 1), field 1 + j reference j's
          const double o0 = f == 0 ? 1.0 : tb.ck[(f - 1) * n + q], o1 = nf == 2 ? tb.ck[f * n + q] : 0.0;
          double2 a, b;
          split_at(sm, M, 0, Q, k, s, a, b);
          double2 pu = cscale(a, o0), pv = cscale(b, o0);
          if (nf == 2) {
            split_at(sm, M, 2, Q, k, s, a, b);
            pu = cadd(pu, cscale(a, o1));
            pv = cadd(pv, cscale(b, o1));
          }
          double2 t = cadd(cscale(pu, kx), cscale(pv, ky));
          if (f > 0) t = cadd(t, slot(sm, M, 4 + k, Q.cc[s]));
          put(sm, M, 4 + k, Q.cc[s], t);
          if (hs3 && Q.has(s)) {
            double2 tu = cscale(pu, kx);
            if (f > 0) tu = cadd(tu, slot(sm, M, 2 + k, Q.cc[s]));
            put(sm, M, 2 + k, Q.cc[s], tu);
          }
        }
    }
  }
  // delphiH1^ = -i (kx C^2 u^ + ky C^2 v^) / g (2d/fun_odesolver.c:2943-2946, 4560-4563)
  const double h = 0.5 / kGrav;
#pragma unroll 1
  for (int j = threadIdx.x; j < Nx / 2; j += NT) {
    const Quad Q(P, j, Nx);
    double2 x[2][2], y[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const double2 t = mul_mi(slot(sm, M, 4 + k, Q.cc[s]), h);
        w.H1[Q.at(k, s, Nx)] = t;
        if (!Q.has(s)) continue;
        x[k][s] = t;
        y[k][s] = zero2();
        if (hs3) {
          x[k][s] = mul_mi(slot(sm, M, 2 + k, Q.cc[s]), h);
          y[k][s] = csub(t, x[k][s]);
        }
      }
    if (tb.model != 1) emit_pack(sm, M, 4, Q, tb.ny, x, y);
  }
  if (tb.model == 1) return;
  fft_slices<M, NT>(sm, 4, 2, tb.twx, +1);
  row_store<M, NT>(sm, 4, 1, w.R, P, n);
}

// the products' fields of pass V4 in w.Q; the loss fields and the gam_j pairs follow
__device__ __forceinline__ int products(const Tab2& tb, int cubic) { return cubic ? 1 : (tb.model == 3 ? 3 : 2); }

// V4: column pass, inverse -> products -> forward; then gam_j q, four references at a time.
// cubic = 0: L phi (HS3: M0u, M0v) in; fields 0 (q, eta u), 1 (eta v, deletaH2), under HS3
// 2 (eta^2 M0u, eta^2 M0v), the loss fields; q = eta L phi.  cubic = 1: L q, div(grad phi) in;
// field 0 (p, h3); q = p.
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2v_col4(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond, int cubic) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = tb.nx, c = blockIdx.x, K = tb.nk, nd = cubic ? 0 : damp_fields(tb, w);
  const size_t n = (size_t)tb.n;
  const bool hs3 = tb.model == 3;
  const int np = products(tb, cubic), f0 = np + nd;
  const double invN = 1.0 / ((double)tb.n);
  col_load<M, NT>(sm, 0, 1, w.R, Nx, c, n);
  fft_slices<M, NT>(sm, 0, 2, tb.twy, +1);
#pragma unroll 2
  for (int t = threadIdx.x; t < 2 * M; t += NT) {
    const ColPt p(t, c, Nx);
    const double2 a = cscale(slot(sm, M, p.k, p.y), invN);
    if (cubic) {
      const double2 r = cubic_products(tb, w, p.q, n, a.x, a.y);
      put(sm, M, p.k, p.y, r);
      w.op[p.q] = r.x;
    } else {
      const double wc = tb.wallchar ? tb.wallchar[p.q] : 1.0;
      const double eta = w.phys[p.q], u = w.phys[n + p.q], v = w.phys[2 * n + p.q];
      const double lphi = hs3 ? a.x + a.y : a.x, q = eta * lphi * wc;
      put(sm, M, p.k, p.y, make_double2(q, eta * u * wc));
      put(sm, M, 2 + p.k, p.y, make_double2(eta * v * wc, 0.5 * ((u * u + v * v) - lphi * lphi) * wc));
      w.op[p.q] = q;
      if (hs3) {
        put(sm, M, 4 + p.k, p.y, make_double2(eta * eta * a.x * wc, eta * eta * a.y * wc));
        w.op[n + p.q] = lphi;
      }
    }
  }
  fft_slices<M, NT>(sm, 0, 2 * np, tb.twy, -1);
  col_store<M, NT>(sm, 0, np, w.Q, Nx, c, n);
  send_loss<M, NT>(sm, np, nd, tb, w, c, n);
  for (int j = 0; j < K; j += 4) {
    const int nf = K - j > 2 ? 2 : 1;
    __syncthreads();
#pragma unroll 2
    for (int t = threadIdx.x; t < 2 * M; t += NT) {
      const ColPt p(t, c, Nx);
      const double q = w.op[p.q];
      double g[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] = j + i < K ? tb.gk[(j + i) * n + p.q] : 0.0;
      put(sm, M, p.k, p.y, make_double2(g[0] * q, g[1] * q));
      if (nf == 2) put(sm, M, 2 + p.k, p.y, make_double2(g[2] * q, g[3] * q));
    }
    fft_slices<M, NT>(sm, 0, 2 * nf, tb.twy, -1);
    col_store<M, NT>(sm, 0, nf, w.Q + (f0 + j / 2) * n, Nx, c, n);
  }
}

// V5: row pass, forward, split; what the images still to come do not change is kept in w.T
// (delu + delv, deletaH, and 1/2 sum_j Omega_j F(gam_j q) / g), and Omega_j q^ goes to
// physical space, two references to a field
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2v_row5(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond, int cubic) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = M, K = tb.nk, nd = cubic ? 0 : damp_fields(tb, w);
  const size_t n = (size_t)tb.n;
  const bool hs3 = tb.model == 3;
  const int np = products(tb, cubic), f0 = np + nd;
  const Pair P = row_pair(blockIdx.x, tb.ny);
  store_loss<M, NT>(sm, np, nd, tb, w, P, n);
  row_load<M, NT>(sm, 0, np, w.Q, P, n);
  fft_slices<M, NT>(sm, 0, 2 * np, tb.twx, -1);
#pragma unroll 1
  for (int j = threadIdx.x; j < Nx / 2; j += NT) {
    const Quad Q(P, j, Nx);
    double2 keep[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (!Q.has(s)) continue;
        const size_t q = Q.at(k, s, Nx);
        double2 qh, b;
        split_at(sm, M, 0, Q, k, s, qh, b);
        keep[k][s] = qh;
        if (cubic) {
          w.T[n + q] = cadd(w.T[n + q], b);   // deletaH3
        } else {
          const double kx = tb.kx[Q.cc[s]], ky = tb.ky[Q.r[k]];
          double2 ev, dH;
          split_at(sm, M, 2, Q, k, s, ev, dH);
          double2 a = cadd(mul_mi(b, kx), mul_mi(ev, ky));   // -i kx (eta u)^ - i ky (eta v)^
          if (hs3) {
            double2 cu, cv;
            split_at(sm, M, 4, Q, k, s, cu, cv);
            a = csub(a, cadd(cscale(cu, 0.5 * (kx * kx)), cscale(cv, 0.5 * (ky * ky))));
          }
          w.T[q] = a;
          w.T[n + q] = dH;
        }
      }
    // q^ stays in slices 0, 1 at the points that the symmetrisation keeps
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s)
        if (Q.has(s)) put(sm, M, k, Q.cc[s], keep[k][s]);
  }
  const double h = 0.5 / kGrav;
  for (int j0 = 0; j0 < K; j0 += 4) {
    const int nf = K - j0 > 2 ? 2 : 1;
    __syncthreads();
    row_load<M, NT>(sm, 2, nf, w.Q + (f0 + j0 / 2) * n, P, n);
    fft_slices<M, NT>(sm, 2, 2 * nf, tb.twx, -1);
#pragma unroll 1
    for (int j = threadIdx.x; j < Nx / 2; j += NT) {
      const Quad Q(P, j, Nx);
      double2 x[4][2][2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          if (!Q.has(s)) continue;
          const size_t q = Q.at(k, s, Nx);
          double o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] = j0 + i < K ? tb.ok[(j0 + i) * n + q] : 0.0;
          double2 acc = j0 > 0 ? w.T[2 * n + q] : zero2();
          double2 a, b;
          split_at(sm, M, 2, Q, k, s, a, b);
          acc = cadd(acc, cadd(cscale(a, h * o[0]), cscale(b, h * o[1])));
          if (nf == 2) {
            split_at(sm, M, 4, Q, k, s, a, b);
            acc = cadd(acc, cadd(cscale(a, h * o[2]), cscale(b, h * o[3])));
          }
          w.T[2 * n + q] = acc;
          const double2 qh = slot(sm, M, k, Q.cc[s]);
#pragma unroll
          for (int i = 0; i < 4; ++i) x[i][k][s] = cscale(qh, o[i]);
        }
      emit_pack(sm, M, 2, Q, tb.ny, x[0], x[1]);
      if (nf == 2) emit_pack(sm, M, 4, Q, tb.ny, x[2], x[3]);
    }
    fft_slices<M, NT>(sm, 2, 2 * nf, tb.twx, +1);
    row_store<M, NT>(sm, 2, nf, w.R + (j0 / 2) * n, P, n);
  }
}

// V6: slices 0, 1 the sum of the weighted images (real), 2..5 four references at a time
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2v_col6(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = tb.nx, c = blockIdx.x, K = tb.nk;
  const size_t n = (size_t)tb.n;
  const double invN = 1.0 / ((double)tb.n);
  for (int j = 0; j < K; j += 4) {
    const int nf = K - j > 2 ? 2 : 1;
    __syncthreads();
    col_load<M, NT>(sm, 2, nf, w.R + (j / 2) * n, Nx, c, n);
    fft_slices<M, NT>(sm, 2, 2 * nf, tb.twy, +1);
#pragma unroll 2
    for (int t = threadIdx.x; t < 2 * M; t += NT) {
      const ColPt p(t, c, Nx);
      double g[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) g[i] = j + i < K ? tb.gk[(j + i) * n + p.q] : 0.0;
      const double2 a = slot(sm, M, 2 + p.k, p.y), b = nf == 2 ? slot(sm, M, 4 + p.k, p.y) : zero2();
      double s = (g[0] * a.x + g[1] * a.y + (g[2] * b.x + g[3] * b.y)) * invN;
      if (j > 0) s += slot(sm, M, p.k, p.y).x;
      put(sm, M, p.k, p.y, make_double2(s, 0.0));
    }
  }
  fft_slices<M, NT>(sm, 0, 2, tb.twy, -1);
  col_store<M, NT>(sm, 0, 1, w.Q, Nx, c, n);
}

// V7: row pass, forward: L q^ = (sum_j Omega_j F(gam_j q) + F(sum)) / (2 g).  The second-order
// operand's enters delu + delv with a minus, the cubic one's with a plus; under HS3 the
// former, with div(grad phi), goes to physical space for the cubic products.
template <int M>
__global__ void __launch_bounds__(kThr4, ctas(kThr4))
k2v_row7(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond, int cubic) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr4;
  const int Nx = M;
  const size_t n = (size_t)tb.n;
  const bool more = tb.model == 3 && !cubic;
  const double h = 0.5 / kGrav;
  const Pair P = row_pair(blockIdx.x, tb.ny);
  row_load<M, NT>(sm, 0, 1, w.Q, P, n);
  fft_slices<M, NT>(sm, 0, 2, tb.twx, -1);
#pragma unroll 1
  for (int j = threadIdx.x; j < Nx / 2; j += NT) {
    const Quad Q(P, j, Nx);
    double2 dH[2][2], a[2][2], lq[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (!Q.has(s)) continue;
        const size_t q = Q.at(k, s, Nx);
        double2 x, none;
        split_at(sm, M, 0, Q, k, s, x, none);
        lq[k][s] = cadd(w.T[2 * n + q], cscale(x, h));
        a[k][s] = cubic ? cadd(w.T[q], lq[k][s]) : csub(w.T[q], lq[k][s]);
        if (more) {
          w.T[q] = a[k][s];
          dH[k][s] = cadd(mul_pi(w.z[n + q], tb.kx[Q.cc[s]]), mul_pi(w.z[2 * n + q], tb.ky[Q.r[k]]));
        } else {
          dH[k][s] = w.T[n + q];
        }
      }
    if (more) emit_pack(sm, M, 0, Q, tb.ny, lq, dH);
    else emit_adjust(sm, M, Q, tb, dH, a);
  }
  if (more) {
    fft_slices<M, NT>(sm, 0, 2, tb.twx, +1);
    row_store<M, NT>(sm, 0, 1, w.R, P, n);
  } else {
    send_adjust<M, NT>(sm, P, tb, w, n);
  }
}

}  // namespace hw2d
