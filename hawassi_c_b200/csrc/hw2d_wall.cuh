// hw2d_wall.cuh -- harbour walls on the flat bottom: fun_delphiH1hat's branch for
// refl_coef < 1 (2d/fun_odesolver.c:2172-2219).  With walls the flat RHS takes
// delphiH1^ = -i (kx (C/g) F(wallchar Re F^-1 S(C u^)) + ky (C/g) F(wallchar Re F^-1 S(C v^)))
// instead of -i (kx C^2/g u^ + ky C^2/g v^): one round trip of the pair (C u^, C v^)
// through physical space, packed as one complex transform each way.
//   W1 (row pass)  E(S(C u^)) + i E(S(C v^)) -> inverse row FFT
//   W2 (col pass)  inverse column FFT, x wallchar / N (both real fields), forward column FFT
//   W3 (row pass)  forward row FFT, split, x C/g, -i (kx . + ky .) -> delphiH1^ (w.H1)
// The H2 products of the column pass carry wallchar as well (:3239-3249).
//
// With refl_coef == 1 the branch at :2105-2170 runs instead: Flux = Re F^-1 S(C^2/g u^)
// (both components), divC2u from the symmetrised spectra, and
// delphiH1^ = F(divC2u wallchar) - F(Flux . grad wallchar):
//   V1 (row pass)  E(S(C^2/g u^)) + i E(S(C^2/g v^)), E(S(D)) with D = -i(kx S(.) + ky S(.))
//                  -> inverse row FFT (four slices)
//   V2 (col pass)  inverse column FFT -> Flux, divC2u -> divC2u wallchar + i Flux . grad
//                  wallchar -> forward column FFT
//   V3 (row pass)  forward row FFT, split, difference -> delphiH1^ (w.H1)
#pragma once

#include "hw2d.cuh"

namespace hw2d {

template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2w_row1(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = tb.nx, Ny = tb.ny;
  const size_t n = (size_t)tb.n;
  const Pair P = row_pair(blockIdx.x, Ny);
#pragma unroll 2
  for (int j = threadIdx.x; j < Nx / 2; j += NT) {
    const Quad Q(P, j, Nx);
    double2 A[2][2], B[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (!Q.has(s)) continue;
        const size_t q = Q.at(k, s, Nx);
        const double C = tb.c2d[q];
        const double2 zu = w.z[n + q], zv = w.z[2 * n + q];
        A[k][s] = make_double2(C * zu.x, C * zu.y);
        B[k][s] = make_double2(C * zv.x, C * zv.y);
      }
    emit_pack(sm, M, 0, Q, Ny, A, B);
  }
  fft_slices<M, NT>(sm, 0, 2, tb.twx, +1);
  row_store<M, NT>(sm, 0, 1, w.WP, P, n);
}

template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2w_col2(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = tb.nx;
  const int c = blockIdx.x;
  const size_t n = (size_t)tb.n;
  col_load<M, NT>(sm, 0, 1, w.WP, Nx, c, n);
  fft_slices<M, NT>(sm, 0, 2, tb.twy, +1);
  const double invN = 1.0 / ((double)tb.n);
#pragma unroll 4
  for (int t = threadIdx.x; t < 2 * M; t += NT) {
      const ColPt p(t, c, Nx);
      const size_t q = p.q;
      const double2 v = slot(sm, M, p.k, p.y);
      const double wc = tb.wallchar[q];
      put(sm, M, p.k, p.y, make_double2(v.x * invN * wc, v.y * invN * wc));
    }
  fft_slices<M, NT>(sm, 0, 2, tb.twy, -1);
  col_store<M, NT>(sm, 0, 1, w.WP, Nx, c, n);
}

template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2w_row3(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = tb.nx, Ny = tb.ny;
  const Pair P = row_pair(blockIdx.x, Ny);
  row_load<M, NT>(sm, 0, 1, w.WP, P, (size_t)tb.n);
  fft_slices<M, NT>(sm, 0, 2, tb.twx, -1);
  for (int k = 0; k < 2; ++k) {
    const int r = P.row(k);
    const double kyv = tb.ky[r];
    for (int j = threadIdx.x; j < Nx; j += NT) {
      const size_t q = (size_t)r * Nx + j;
      double2 X, Y;   // F(wallchar C u), F(wallchar C v)
      split2(slot(sm, M, k, j), slot(sm, M, k ^ P.flip, (Nx - j) % Nx), X, Y);
      const double cg = tb.c2d[q] / kGrav;
      const double2 du = make_double2(cg * X.x, cg * X.y), dv = make_double2(cg * Y.x, cg * Y.y);
      const double kxv = tb.kx[j];
      w.H1[q] = make_double2(kxv * du.y + kyv * dv.y, -kxv * du.x - kyv * dv.x);
    }
  }
}

template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2w_rowV1(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = tb.nx, Ny = tb.ny;
  const size_t n = (size_t)tb.n;
  const Pair P = row_pair(blockIdx.x, Ny);
#pragma unroll 2
  for (int j = threadIdx.x; j < Nx / 2; j += NT) {
    const Quad Q(P, j, Nx);
    double2 A[2][2], B[2][2], D[2][2], Z[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (!Q.has(s)) continue;
        const size_t q = Q.at(k, s, Nx);
        const double cg = tb.c2g[q];
        const double2 zu = w.z[n + q], zv = w.z[2 * n + q];
        A[k][s] = make_double2(cg * zu.x, cg * zu.y);
        B[k][s] = make_double2(cg * zv.x, cg * zv.y);
      }
    // divC2u^ = -i (kx S(.) + ky S(.)) from the symmetrised spectra
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (!Q.has(s)) continue;
        double2 sa = A[k][s], sb = B[k][s];
        if (Q.self) {
          sa = self_sym(sa, Q.flip ? A[k ^ 1][s] : sa, Q.r[k], s, Ny, false);
          sb = self_sym(sb, Q.flip ? B[k ^ 1][s] : sb, Q.r[k], s, Ny, false);
        }
        D[k][s] = cadd(mul_mi(sa, tb.kx[Q.cc[s]]), mul_mi(sb, tb.ky[Q.r[k]]));
        Z[k][s] = zero2();
      }
    emit_pack(sm, M, 0, Q, Ny, A, B);
    emit_pack(sm, M, 2, Q, Ny, D, Z);
  }
  fft_slices<M, NT>(sm, 0, 4, tb.twx, +1);
  row_store<M, NT>(sm, 0, 2, w.WP, P, n);
}

template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2w_colV2(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = tb.nx;
  const size_t n = (size_t)tb.n;
  const int c = blockIdx.x;
  col_load<M, NT>(sm, 0, 2, w.WP, Nx, c, n);
  fft_slices<M, NT>(sm, 0, 4, tb.twy, +1);
  const double invN = 1.0 / ((double)tb.n);
#pragma unroll 4
  for (int t = threadIdx.x; t < 2 * M; t += NT) {
      const ColPt p(t, c, Nx);
      const size_t q = p.q;
      const double2 fl = slot(sm, M, p.k, p.y), dv = slot(sm, M, 2 + p.k, p.y);
      const double fx = fl.x * invN, fy = fl.y * invN, div = dv.x * invN;
      put(sm, M, p.k, p.y, make_double2(div * tb.wallchar[q], fx * tb.gwx[q] + fy * tb.gwy[q]));
    }
  fft_slices<M, NT>(sm, 0, 2, tb.twy, -1);
  col_store<M, NT>(sm, 0, 1, w.WP, Nx, c, n);
}

template <int M>
__global__ void __launch_bounds__(kThr2, ctas(kThr2))
k2w_rowV3(Tab2 tb, Work2 w, const Ctl2* __restrict__ ctl, int cond) {
  if (!rhs_active(ctl, cond)) return;
  extern __shared__ double2 sm[];
  constexpr int NT = kThr2;
  const int Nx = tb.nx, Ny = tb.ny;
  const Pair P = row_pair(blockIdx.x, Ny);
  row_load<M, NT>(sm, 0, 1, w.WP, P, (size_t)tb.n);
  fft_slices<M, NT>(sm, 0, 2, tb.twx, -1);
  for (int k = 0; k < 2; ++k) {
    const int r = P.row(k);
    for (int j = threadIdx.x; j < Nx; j += NT) {
      double2 X, Y;   // F(divC2u wallchar), F(Flux . grad wallchar)
      split2(slot(sm, M, k, j), slot(sm, M, k ^ P.flip, (Nx - j) % Nx), X, Y);
      w.H1[(size_t)r * Nx + j] = make_double2(X.x - Y.x, X.y - Y.y);
    }
  }
}

}  // namespace hw2d
