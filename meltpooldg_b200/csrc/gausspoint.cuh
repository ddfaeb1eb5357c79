// Cell values at the Gauss points (sum factorisation over one thread's (k+1)^3 register array), shared by the
// operators whose coefficients vary inside a cell: advection, reinitialisation and projections, and the
// temperature-dependent material.
//
// Values at the points are kept without the point weights; the weights sit in the matrices that test back to
// the nodes (gp_test, one per direction, the cell's volume in the last) and, as W^-1 D^T W, in those that test
// a flux with the gradient (gp_divergence).  FE_Q(2) is used by its structure: the middle Gauss point is
// the middle node (its row of B is a unit row), so a line costs 6 instead of 9 operations for B.  Derivatives
// act on differences of neighbouring values along a line (their matrices have zero row sums): N (N - 1)
// operations and N - 1 differences a line instead of N^2.
//
// Differences of values that were interpolated before carry that interpolation's rounding, amplified by
// |u| / (h |grad u|).  So a gradient alone differences the nodal values and interpolates the differences
// (gp_gradient), and an operator that takes values and gradient from one interpolation subtracts the cell's
// middle node first; their tables are products formed in extended precision and rounded once.  Against 80-bit
// values, FE_Q(2) 35x22x27: right-hand side of the reinitialisation 4.9e-14 without the three, 2.9e-15 with them
// (plain sums over the 27 nodes: 1.8e-14), normal 2.8e-15 and 2.5e-16 (1.1e-15), at the same time per apply.
#pragma once

#include "tables.h"

namespace mpdg
{
  // out (N x (N - 1)) = scale M (N x N, zero row sums) as it acts on u_1 - u_0, u_2 - u_1, ...
  template <typename T, int N, typename R>
  inline void
  gp_on_differences(const R *M, R scale, T *out)
  {
    for (int r = 0; r < N; ++r)
      {
        R s = 0.0;
        for (int k = N - 2; k >= 0; --k)
          {
            s += M[r * N + k + 1];
            out[r * (N - 1) + k] = (T)(scale * s);
          }
      }
  }

  // 1-D matrices of degree N - 1, row-major N x N unless stated
  template <typename T, int N>
  struct GaussTab
  {
    T B[N * N];     // nodal values -> Gauss points (rows: points)
    T Bt[3][N * N]; // test: Gauss points -> nodes, weighted (rows: nodes); the volume in [2]
    T D[3][N * (N - 1)]; // derivative at the points, 1 / h_d D, on differences
    T P[3][N * N];       // flux test, W^-1 D^T W / h_d
    T G[3][N * (N - 1)]; // derivative of the nodal values at the points, 1 / h_d G, on differences
    T Gzt[N * N];        // weighted transpose of the z derivative (rows: nodes), with the volume

    // from B, G, Dq and qw of Tables1D, entries computed in R and rounded (from long double: once)
    template <typename R>
    void
    fill(const R *tB, const R *tG, const R *tD, const R *tw, const double h[3])
    {
      for (int q = 0; q < N; ++q)
        for (int r = 0; r < N; ++r)
          {
            B[q * N + r]   = (T)tB[q * N + r];
            Gzt[r * N + q] = (T)((R)h[0] * h[1] * tw[q] * tG[q * N + r]);
            for (int d = 0; d < 3; ++d)
              {
                Bt[d][r * N + q] = (T)((d == 2 ? (R)h[0] * h[1] * h[2] : R(1)) * tw[q] * tB[q * N + r]);
                P[d][q * N + r]  = (T)(tD[r * N + q] * tw[r] / tw[q] / h[d]);
              }
          }
      for (int d = 0; d < 3; ++d)
        {
          gp_on_differences<T, N>(tD, R(1) / h[d], D[d]);
          gp_on_differences<T, N>(tG, R(1) / h[d], G[d]);
        }
    }
  };

  // v = M v along direction DIR with a point matrix whose middle row (N = 3) is a unit row.  SHORT: the array
  // holds only N - 1 values along that direction (differences).
  template <typename T, int N, int DIR, int SHORT = -1>
  __device__ __forceinline__ void
  gp_interpolate(T *v, const T *M)
  {
    constexpr int S  = DIR == 0 ? 1 : (DIR == 1 ? N : N * N);
    constexpr int DA = DIR == 2 ? 1 : 2, DC = DIR == 0 ? 1 : 0; // the directions of a and c
#pragma unroll
    for (int a = 0; a < N - (DA == SHORT); ++a)
#pragma unroll
      for (int c = 0; c < N - (DC == SHORT); ++c)
        {
          T *p = v + (DIR == 0 ? (a * N + c) * N : (DIR == 1 ? a * N * N + c : a * N + c));
          T  in[N];
#pragma unroll
          for (int k = 0; k < N; ++k)
            in[k] = p[k * S];
#pragma unroll
          for (int r = 0; r < N; ++r)
            {
              if (N == 3 && r == 1)
                continue;
              T s = M[r * N] * in[0];
#pragma unroll
              for (int k = 1; k < N; ++k)
                s = fma(M[r * N + k], in[k], s);
              p[r * S] = s;
            }
        }
  }

  // v = M v along direction DIR, M from Gauss points to nodes (N = 3: the middle point only enters the
  // middle node)
  template <typename T, int N, int DIR>
  __device__ __forceinline__ void
  gp_test(T *v, const T *M)
  {
    constexpr int S = DIR == 0 ? 1 : (DIR == 1 ? N : N * N);
#pragma unroll
    for (int a = 0; a < N; ++a)
#pragma unroll
      for (int c = 0; c < N; ++c)
        {
          T *p = v + (DIR == 0 ? (a * N + c) * N : (DIR == 1 ? a * N * N + c : a * N + c));
          T  in[N];
#pragma unroll
          for (int k = 0; k < N; ++k)
            in[k] = p[k * S];
#pragma unroll
          for (int r = 0; r < N; ++r)
            {
              T s = M[r * N] * in[0];
#pragma unroll
              for (int k = 1; k < N; ++k)
                if (!(N == 3 && k == 1 && r != 1))
                  s = fma(M[r * N + k], in[k], s);
              p[r * S] = s;
            }
        }
  }

  // One direction of a flux tested with the gradient: S += P f along the lines, P = W^-1 D^T W / h (the
  // middle point of N = 3 does not act on itself).  flux(q): the flux component at point q.
  template <typename T, int N, int DIR, class Flux>
  __device__ __forceinline__ void
  gp_divergence(T *S, const T *P, const Flux &flux)
  {
    constexpr int ST = DIR == 0 ? 1 : (DIR == 1 ? N : N * N);
#pragma unroll
    for (int a = 0; a < N; ++a)
#pragma unroll
      for (int c = 0; c < N; ++c)
        {
          const int b = DIR == 0 ? (a * N + c) * N : (DIR == 1 ? a * N * N + c : a * N + c);
          T         t[N];
#pragma unroll
          for (int r = 0; r < N; ++r)
            t[r] = flux(b + r * ST);
#pragma unroll
          for (int r = 0; r < N; ++r)
#pragma unroll
            for (int k = 0; k < N; ++k)
              if (!(N == 3 && r == 1 && k == 1))
                S[b + r * ST] = fma(P[r * N + k], t[k], S[b + r * ST]);
        }
  }

  // Nodal values v to their derivative in direction DIR at the Gauss points (G: the nodal derivative on
  // differences)
  template <typename T, int N, int DIR>
  __device__ __forceinline__ void
  gp_gradient(T *v, const T *B, const T *G)
  {
    constexpr int S = DIR == 0 ? 1 : (DIR == 1 ? N : N * N), ND = N - 1;
    auto          line = [](int a, int c) { return DIR == 0 ? (a * N + c) * N : (DIR == 1 ? a * N * N + c : a * N + c); };
#pragma unroll
    for (int a = 0; a < N; ++a)
#pragma unroll
      for (int c = 0; c < N; ++c)
        {
          T *p = v + line(a, c);
#pragma unroll
          for (int k = 0; k < ND; ++k)
            p[k * S] = p[(k + 1) * S] - p[k * S];
        }
    gp_interpolate<T, N, (DIR + 1) % 3, DIR>(v, B);
    gp_interpolate<T, N, (DIR + 2) % 3, DIR>(v, B);
#pragma unroll
    for (int a = 0; a < N; ++a)
#pragma unroll
      for (int c = 0; c < N; ++c)
        {
          T *p = v + line(a, c);
          T  d[ND];
#pragma unroll
          for (int k = 0; k < ND; ++k)
            d[k] = p[k * S];
#pragma unroll
          for (int r = 0; r < N; ++r)
            {
              T g = G[r * ND] * d[0];
#pragma unroll
              for (int k = 1; k < ND; ++k)
                g = fma(G[r * ND + k], d[k], g);
              p[r * S] = g;
            }
        }
  }

  // Derivative of u at point q in direction DIR: row of D times the differences of the line through q
  template <typename T, int N, int DIR>
  __device__ __forceinline__ T
  gp_derivative(const T *u, const T *D, const int q)
  {
    constexpr int ST = DIR == 0 ? 1 : (DIR == 1 ? N : N * N);
    const int     r = DIR == 0 ? q % N : (DIR == 1 ? q / N % N : q / (N * N)), b = q - r * ST;
    T             g = D[r * (N - 1)] * (u[b + ST] - u[b]);
#pragma unroll
    for (int k = 1; k < N - 1; ++k)
      g = fma(D[r * (N - 1) + k], u[b + (k + 1) * ST] - u[b + k * ST], g);
    return g;
  }

  // ---- one plane of Gauss points (fixed z point), N x N values.  An operator with several coefficient fields
  // walks its cell plane by plane in a rolled loop: it re-reads the nodal values (shared memory, L1) for
  // each plane instead of holding the fields at all N^3 points, and only its N^3 results stay in registers.

  // values or z derivatives of a plane before its x and y interpolation, from nodes(l, j, i)
  template <typename T, int N, class Nodes>
  __device__ __forceinline__ void
  pl_value(const Nodes &nodes, const T *bz, T *v)
  {
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
      for (int i = 0; i < N; ++i)
        {
          T s = bz[0] * nodes(0, j, i);
#pragma unroll
          for (int l = 1; l < N; ++l)
            s = fma(bz[l], nodes(l, j, i), s);
          v[j * N + i] = s;
        }
  }
  template <typename T, int N, class Nodes>
  __device__ __forceinline__ void
  pl_zderivative(const Nodes &nodes, const T *gz, T *v)
  {
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
      for (int i = 0; i < N; ++i)
        {
          T g = gz[0] * (nodes(1, j, i) - nodes(0, j, i));
#pragma unroll
          for (int l = 1; l < N - 1; ++l)
            g = fma(gz[l], nodes(l + 1, j, i) - nodes(l, j, i), g);
          v[j * N + i] = g;
        }
  }
  // v = M v along the lines of direction DIR (0 or 1) of a plane; MID: the middle row of N = 3 is a unit row
  template <typename T, int N, int DIR, bool MID>
  __device__ __forceinline__ void
  pl_apply(T *v, const T *M)
  {
    constexpr int ST = DIR == 0 ? 1 : N, LN = DIR == 0 ? N : 1;
#pragma unroll
    for (int c = 0; c < N; ++c)
      {
        T in[N];
#pragma unroll
        for (int k = 0; k < N; ++k)
          in[k] = v[c * LN + k * ST];
#pragma unroll
        for (int r = 0; r < N; ++r)
          {
            if (MID && N == 3 && r == 1)
              continue;
            T s = M[r * N] * in[0];
#pragma unroll
            for (int k = 1; k < N; ++k)
              s = fma(M[r * N + k], in[k], s);
            v[c * LN + r * ST] = s;
          }
      }
  }
  template <typename T, int N>
  __device__ __forceinline__ void
  pl_interpolate(T *v, const T *B)
  {
    pl_apply<T, N, 0, true>(v, B);
    pl_apply<T, N, 1, true>(v, B);
  }
  // S += P f along the lines of direction DIR (0 or 1) of a plane
  template <typename T, int N, int DIR, class Flux>
  __device__ __forceinline__ void
  pl_divergence(T *S, const T *P, const Flux &flux)
  {
    constexpr int ST = DIR == 0 ? 1 : N, LN = DIR == 0 ? N : 1;
#pragma unroll
    for (int c = 0; c < N; ++c)
      {
        T t[N];
#pragma unroll
        for (int k = 0; k < N; ++k)
          t[k] = flux(c * LN + k * ST);
#pragma unroll
        for (int r = 0; r < N; ++r)
#pragma unroll
          for (int k = 0; k < N; ++k)
            if (!(N == 3 && r == 1 && k == 1))
              S[c * LN + r * ST] = fma(P[r * N + k], t[k], S[c * LN + r * ST]);
      }
  }
  // Tests the plane's values S and z fluxes F back to the nodes: R(l, j, i) += bt[l] S' + gt[l] F'
  template <typename T, int N>
  __device__ __forceinline__ void
  pl_test(T *S, T *F, const GaussTab<T, N> &t, int qz, T *R)
  {
    pl_apply<T, N, 0, false>(S, t.Bt[0]);
    pl_apply<T, N, 1, false>(S, t.Bt[1]);
    pl_apply<T, N, 0, false>(F, t.Bt[0]);
    pl_apply<T, N, 1, false>(F, t.Bt[1]);
#pragma unroll
    for (int l = 0; l < N; ++l)
      {
        const T bt = t.Bt[2][l * N + qz], gt = t.Gzt[l * N + qz];
#pragma unroll
        for (int p = 0; p < N * N; ++p)
          R[l * N * N + p] = fma(bt, S[p], fma(gt, F[p], R[l * N * N + p]));
      }
  }
} // namespace mpdg
