// Conservative level-set reinitialisation operator (Olsson), FE_Q(1..3).
//
// Reference: source/level_set/olsson_CG_operator.cpp, default configuration (no wetting boundary
// faces, no interface penalty):
//   tangent  (:438-470)  val = dpsi / dt,  grad = eps_n (grad dpsi . n) n + eps_t (grad dpsi - (grad dpsi . n) n)
//   rhs      (:197-260)  dst = int [c(psi) n - eps_n (grad psi . n) n - eps_t (grad psi - (grad psi . n) n)] . grad phi,
//                        c(psi) = (1 - psi^2) / 2 (:24-29), dst overwritten, constrained rows 0
// with the unit normal n = normalize(n_h(x_q), tol) of the normal field n_h (three FE_Q components
// on the same lattice, read plainly; normalize divides by |n_h| above tol and by tol otherwise,
// include/meltpooldg/utilities/dealii_tensor.hpp:175-191).  The reference caches n at the Gauss
// points while it assembles the rhs and reuses the cache in vmult; here it is evaluated from the
// normal field at every apply (the same as long as the field does not change in between).
//
// The applies and right-hand sides run in the column-marching frame (march.cuh), one thread per cell, by sum
// factorisation on the Gauss points (gausspoint.cuh).  With v = n_h at the points, D grad u = eps_t grad u +
// c v, c = (eps_n - eps_t) (v . grad u) / |v|^2.  The tangent and the right-hand side walk the cell one plane of
// points at a time: the three components of v, u and its derivatives at all (k+1)^3 points would not fit the
// registers.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "brick.cuh"
#include "gausspoint.cuh"
#include "kernels.h"
#include "march.cuh"

namespace mpdg
{
  namespace
  {
    template <typename T, int N>
    struct ReinitArgs
    {
      GridDesc      g;
      T             scale, inv_dt, eps_n, eps_t, tol, det, ih[3];
      T             B[N * N], G[N * N], w[N];
      const T      *src;
      const double *n[3];
      T            *dst;
      double       *diag;
      int           mode; // wetting faces: 0 tangent apply, 1 rhs (src = psi_old, plain), 2 diagonal
      int           mask_src;
      const double *band_ls; // narrow band (include/meltpooldg/level_set/level_set_tools.hpp:357-368)
      T             band;
      unsigned      wetting; // wetting boundary faces (bit 2d low / 2d+1 high face of dim d)
      T             Vend[2 * N], Dend[2 * N]; // basis values / derivatives at x = 0 and x = 1
    };

    // cell of a lane (a lane outside the mesh reads the fields of the nearest cell), and the values of a
    // plainly read field at the cell's nodes or Gauss points
    struct PointCell
    {
      int c[3];
    };
    __device__ __forceinline__ PointCell
    point_cell(const GridDesc &g, int cx, int cy, int cz)
    {
      return PointCell{{min(cx, g.m[0] - 1), min(cy, g.m[1] - 1), cz}};
    }
    template <typename T, int N>
    __device__ __forceinline__ void
    field_nodes(const double *f, const GridDesc &g, const PointCell &c, T *v)
    {
      constexpr int K  = N - 1;
      const int     sy = g.n[0], sz = g.n[0] * g.n[1];
      f += K * c.c[0] + (long long)sy * (K * c.c[1]) + (long long)sz * (K * c.c[2]);
#pragma unroll
      for (int l = 0; l < N; ++l)
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
          for (int i = 0; i < N; ++i)
            v[(l * N + j) * N + i] = (T)__ldg(f + (j * sy + l * sz + i));
    }
    template <typename T, int N>
    __device__ __forceinline__ void
    interpolate(T *v, const T *B)
    {
      gp_interpolate<T, N, 0>(v, B);
      gp_interpolate<T, N, 1>(v, B);
      gp_interpolate<T, N, 2>(v, B);
    }
    template <typename T, int N>
    __device__ __forceinline__ void
    test(T *S, const GaussTab<T, N> &t)
    {
      gp_test<T, N, 2>(S, t.Bt[2]);
      gp_test<T, N, 1>(S, t.Bt[1]);
      gp_test<T, N, 0>(S, t.Bt[0]);
    }
    __device__ __forceinline__ double
    point_rsqrt(double x)
    {
      return rsqrt(x);
    }
    __device__ __forceinline__ float
    point_rsqrt(float x)
    {
      return 1.0f / sqrtf(x);
    }
    // Points of the narrow band, one bit per Gauss point.  The apply, the right-hand sides and the diagonal all ask
    // here: a point within rounding of the threshold has to be in all of them or in none.
    template <typename T, int N>
    __device__ __forceinline__ unsigned long long
    band_bits(const double *ls, T band, const T *B, const GridDesc &g, const PointCell &c)
    {
      T v[N * N * N];
      field_nodes<T, N>(ls, g, c, v);
      interpolate<T, N>(v, B);
      unsigned long long bits = 0;
#pragma unroll
      for (int q = 0; q < N * N * N; ++q)
        bits |= (unsigned long long)(fabs(v[q]) < band ? 1u : 0u) << q;
      return bits;
    }

    // Diagonal of the tangent (and of the banded isotropic form), one thread per cell, point by point
    template <int K, typename T>
    __global__ void __launch_bounds__(128)
    reinit_diag_kernel(const __grid_constant__ ReinitArgs<T, K + 1> a)
    {
      constexpr int   N     = K + 1, N3 = N * N * N;
      const int       m0    = a.g.m[0], m1 = a.g.m[1];
      const long long ncell = (long long)m0 * m1 * a.g.m[2];
      for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x)
        {
          const int cx = (int)(c % m0), cy = (int)((c / m0) % m1), cz = (int)(c / ((long long)m0 * m1));
          long long idx[N3];
          bool      con[N3];
          T         R[N3];
#pragma unroll
          for (int l = 0; l < N; ++l)
#pragma unroll
            for (int j = 0; j < N; ++j)
#pragma unroll
              for (int i = 0; i < N; ++i)
                {
                  const int       q  = (l * N + j) * N + i;
                  const int       I = K * cx + i, J = K * cy + j, L = K * cz + l;
                  const long long id = (long long)I + (long long)a.g.n[0] * ((long long)J + (long long)a.g.n[1] * L);
                  idx[q]             = id;
                  con[q]             = is_constrained(a.g, I, J, L, id);
                  R[q]               = T(0);
                }
          const unsigned long long bits =
            a.band_ls ? band_bits<T, N>(a.band_ls, a.band, a.B, a.g, PointCell{{cx, cy, cz}}) : ~0ull;
          for (int qz = 0; qz < N; ++qz)
            for (int qy = 0; qy < N; ++qy)
              for (int qx = 0; qx < N; ++qx)
                {
                  // the normal field (none in the isotropic form) at the Gauss point
                  T          nv[3] = {T(0), T(0), T(0)};
                  const bool has_n = a.n[0] != nullptr;
#pragma unroll
                  for (int l = 0; l < N; ++l)
#pragma unroll
                    for (int j = 0; j < N; ++j)
#pragma unroll
                      for (int i = 0; i < N; ++i)
                        {
                          const int q   = (l * N + j) * N + i;
                          const T   phi = a.B[qx * N + i] * a.B[qy * N + j] * a.B[qz * N + l];
                          if (has_n)
#pragma unroll
                            for (int d = 0; d < 3; ++d)
                              nv[d] += phi * (T)a.n[d][idx[q]];
                        }
                  if (has_n)
                    {
                      const T nn  = sqrt(nv[0] * nv[0] + nv[1] * nv[1] + nv[2] * nv[2]);
                      const T inv = nn > a.tol ? T(1) / nn : T(1) / a.tol;
#pragma unroll
                      for (int d = 0; d < 3; ++d)
                        nv[d] *= inv;
                    }
                  const bool in = (bits >> ((qz * N + qy) * N + qx)) & 1u; // narrow band
                  const T    jw = in ? a.det * a.w[qx] * a.w[qy] * a.w[qz] : T(0);
                  // int phi_i^2 / dt + grad phi_i . D grad phi_i
#pragma unroll
                  for (int l = 0; l < N; ++l)
#pragma unroll
                    for (int j = 0; j < N; ++j)
#pragma unroll
                      for (int i = 0; i < N; ++i)
                        {
                          const T bx = a.B[qx * N + i], by = a.B[qy * N + j], bz = a.B[qz * N + l];
                          const T p[3] = {a.G[qx * N + i] * a.ih[0] * by * bz, bx * a.G[qy * N + j] * a.ih[1] * bz,
                                          bx * by * a.G[qz * N + l] * a.ih[2]};
                          const T phi = bx * by * bz;
                          const T pn  = p[0] * nv[0] + p[1] * nv[1] + p[2] * nv[2];
                          const T pp  = p[0] * p[0] + p[1] * p[1] + p[2] * p[2];
                          R[(l * N + j) * N + i] += jw * (a.inv_dt * phi * phi + a.eps_t * pp + (a.eps_n - a.eps_t) * pn * pn);
                        }
                }
#pragma unroll
          for (int q = 0; q < N3; ++q)
            if (!con[q])
              atomicAdd(a.diag + idx[q], (double)R[q]);
        }
    }

    // Wetting boundary faces of the reinitialisation operator (olsson_CG_operator.cpp:550-716), one
    // thread per boundary cell face: at the face's Gauss points the flux D grad u . n_f with
    // D = eps_n n n^T + eps_t (I - n n^T) (tangent, src read with constraints; diagonal: per basis
    // function), or -(-c(psi) n + D grad psi) . n_f with c(psi) = (1 - psi^2) / 2 (rhs, plain reads),
    // tested with the basis values on the face.
    template <int K, typename T>
    __global__ void __launch_bounds__(128)
    wetting_kernel(const __grid_constant__ ReinitArgs<T, K + 1> a)
    {
      constexpr int N = K + 1, N3 = N * N * N;
      const int     m[3] = {a.g.m[0], a.g.m[1], a.g.m[2]};
      long long     count[6], total = 0;
      for (int f = 0; f < 6; ++f)
        {
          const int d = f >> 1;
          count[f]    = ((a.wetting >> f) & 1u) ? (long long)m[(d + 1) % 3] * m[(d + 2) % 3] : 0;
          total += count[f];
        }
      const T hl[3] = {T(1) / a.ih[0], T(1) / a.ih[1], T(1) / a.ih[2]};
      for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x)
        {
          int       f = 0;
          long long r = t;
          while (r >= count[f])
            r -= count[f++];
          const int d = f >> 1, side = f & 1, ea = (d + 1) % 3, eb = (d + 2) % 3;
          int       c[3];
          c[d]  = side ? m[d] - 1 : 0;
          c[ea] = (int)(r % m[ea]);
          c[eb] = (int)(r / m[ea]);
          long long idx[N3];
          bool      con[N3];
          T         u[N3], R[N3], nn[3][N3];
#pragma unroll
          for (int l = 0; l < N; ++l)
#pragma unroll
            for (int j = 0; j < N; ++j)
#pragma unroll
              for (int i = 0; i < N; ++i)
                {
                  const int       q = (l * N + j) * N + i;
                  const int       I = K * c[0] + i, J = K * c[1] + j, L = K * c[2] + l;
                  const long long id = (long long)I + (long long)a.g.n[0] * ((long long)J + (long long)a.g.n[1] * L);
                  idx[q]            = id;
                  con[q]            = is_constrained(a.g, I, J, L, id);
                  u[q]              = (a.mode == 2 || (a.mode == 0 && a.mask_src && con[q])) ? T(0) : a.src[id];
                  R[q]              = T(0);
#pragma unroll
                  for (int e = 0; e < 3; ++e)
                    nn[e][q] = (T)a.n[e][id];
                }
          const T *Vd = a.Vend + side * N, *Dd = a.Dend + side * N;
          const T  W0 = hl[0] * hl[1] * hl[2] / hl[d], sgn = side ? T(1) : T(-1);
          for (int qb = 0; qb < N; ++qb)
            for (int qa = 0; qa < N; ++qa)
              {
                // per node: value and the three derivative factors at this face point
                auto factors = [&](int i, int j, int l, T &val, T gr[3]) {
                  const int ii[3] = {i, j, l};
                  T         v[3], dv[3];
#pragma unroll
                  for (int e = 0; e < 3; ++e)
                    {
                      if (e == d)
                        {
                          v[e]  = Vd[ii[e]];
                          dv[e] = Dd[ii[e]] * a.ih[e];
                        }
                      else
                        {
                          const int qe = e == ea ? qa : qb;
                          v[e]         = a.B[qe * N + ii[e]];
                          dv[e]        = a.G[qe * N + ii[e]] * a.ih[e];
                        }
                    }
                  val   = v[0] * v[1] * v[2];
                  gr[0] = dv[0] * v[1] * v[2];
                  gr[1] = v[0] * dv[1] * v[2];
                  gr[2] = v[0] * v[1] * dv[2];
                };
                T uv = T(0), g[3] = {T(0), T(0), T(0)}, nv[3] = {T(0), T(0), T(0)};
#pragma unroll
                for (int l = 0; l < N; ++l)
#pragma unroll
                  for (int j = 0; j < N; ++j)
#pragma unroll
                    for (int i = 0; i < N; ++i)
                      {
                        const int q = (l * N + j) * N + i;
                        T         val, gr[3];
                        factors(i, j, l, val, gr);
                        uv += val * u[q];
#pragma unroll
                        for (int e = 0; e < 3; ++e)
                          {
                            g[e] += gr[e] * u[q];
                            nv[e] += val * nn[e][q];
                          }
                      }
                const T nrm = sqrt(nv[0] * nv[0] + nv[1] * nv[1] + nv[2] * nv[2]);
                const T inv = nrm > a.tol ? T(1) / nrm : T(1) / a.tol;
#pragma unroll
                for (int e = 0; e < 3; ++e)
                  nv[e] *= inv;
                const T W  = W0 * a.w[qa] * a.w[qb];
                const T gn = g[0] * nv[0] + g[1] * nv[1] + g[2] * nv[2];
                T       integrand;
                if (a.mode == 1)
                  integrand = -sgn * (-T(0.5) * (T(1) - uv * uv) * nv[d] + a.eps_t * g[d] + (a.eps_n - a.eps_t) * gn * nv[d]);
                else
                  integrand = sgn * (a.eps_t * g[d] + (a.eps_n - a.eps_t) * gn * nv[d]);
#pragma unroll
                for (int l = 0; l < N; ++l)
#pragma unroll
                  for (int j = 0; j < N; ++j)
#pragma unroll
                    for (int i = 0; i < N; ++i)
                      {
                        const int q = (l * N + j) * N + i;
                        T         val, gr[3];
                        factors(i, j, l, val, gr);
                        if (a.mode == 2)
                          {
                            const T pn = gr[0] * nv[0] + gr[1] * nv[1] + gr[2] * nv[2];
                            R[q] += W * sgn * (a.eps_t * gr[d] + (a.eps_n - a.eps_t) * pn * nv[d]) * val;
                          }
                        else
                          R[q] += W * integrand * val;
                      }
              }
#pragma unroll
          for (int q = 0; q < N3; ++q)
            if (!con[q])
              {
                if (a.mode == 2)
                  atomicAdd(a.diag + idx[q], (double)R[q]);
                else
                  atomicAdd(a.dst + idx[q], (a.mode == 0 ? a.scale : T(1)) * R[q]);
              }
        }
    }

    // Parameters of the marching kernels
    template <typename T, int N>
    struct PointArgs
    {
      GridDesc       g;
      SyncDesc       s;
      GaussTab<T, N> t;
      T              eps_t, eps;   // scale eps_t, scale (eps_n - eps_t) (scale = -1 in the right-hand side)
      T              mass;         // scale / dt (0 in the right-hand side)
      T              tol2, inv_tol; // normalisation: 1 / |n| where |n|^2 > tol2, else inv_tol
      const T       *src, *b;
      T             *dst;
      const double  *n[3];
      const double  *band_ls;
      T              band;
      int            mask_src;
    };

    // reinitialisation tangent (RHS = false) and right-hand side (RHS = true: src = psi_old, the flux
    // (1 - psi^2) / 2 n - D grad psi, eps_t and eps with a minus sign), one plane of Gauss points at a time
    template <int K, typename T, bool RHS>
    struct ReinitCellOp
    {
      static constexpr int  N = K + 1, N2 = N * N, N3 = N * N * N;
      static constexpr bool HEAVY = true, NODES = true, SPLIT = false;
      using Args = PointArgs<T, N>;
      const Args &a;
      __device__ __forceinline__ PointCell
      load(bool, int cx, int cy, int cz) const
      {
        return point_cell(a.g, cx, cy, cz);
      }
      __device__ __forceinline__ void
      apply(T *R, const MarchNodes<K, T> &nodes, const PointCell &c) const
      {
        const int       sy = a.g.n[0], sz = a.g.n[0] * a.g.n[1];
        const long long first = K * c.c[0] + (long long)sy * (K * c.c[1]) + (long long)sz * (K * c.c[2]);
        // values and gradient of u - ref, ref the middle node: interpolated values of nearly equal size cancel
        const T    ref  = nodes.row[(K / 2) * N + K / 2][K / 2];
        const auto node = [&](int l, int j, int i) { return nodes.row[l * N + j][i] - ref; };
#pragma unroll
        for (int q = 0; q < N3; ++q)
          R[q] = T(0);
#pragma unroll(K == 1 ? 2 : 1)
        for (int qz = 0; qz < N; ++qz)
          {
            const T *bz = a.t.B + qz * N, *gz = a.t.G[2] + qz * (N - 1);
            T        v[3][N2], u[N2], F[N2], S[N2], G[N2];
#pragma unroll
            for (int d = 0; d < 3; ++d)
              {
                const double *f = a.n[d] + first;
                pl_value<T, N>([&](int l, int j, int i) { return (T)__ldg(f + (j * sy + l * sz + i)); }, bz, v[d]);
                pl_interpolate<T, N>(v[d], a.t.B);
              }
            pl_value<T, N>(node, bz, u);
            pl_zderivative<T, N>(node, gz, F);
            pl_interpolate<T, N>(u, a.t.B);
            pl_interpolate<T, N>(F, a.t.B);
            // the flux's factor of n_h: c = eps (n_h . grad u) / |n_h|^2, in the right-hand side with the
            // compressive part (1 - psi^2) / (2 |n_h|)
#pragma unroll
            for (int p = 0; p < N2; ++p)
              {
                const T gx = gp_derivative<T, N, 0>(u, a.t.D[0], p), gy = gp_derivative<T, N, 1>(u, a.t.D[1], p);
                const T nn = fma(v[2][p], v[2][p], fma(v[1][p], v[1][p], v[0][p] * v[0][p]));
                const T inv = nn > a.tol2 ? point_rsqrt(nn) : a.inv_tol;
                const T an  = a.eps * (fma(v[2][p], F[p], fma(v[1][p], gy, v[0][p] * gx)) * inv);
                const T w   = u[p] + ref;
                G[p]        = RHS ? inv * (T(0.5) * (T(1) - w * w) + an) : inv * an;
                S[p]        = a.mass * w;
                F[p]        = fma(a.eps_t, F[p], G[p] * v[2][p]);
              }
            pl_divergence<T, N, 0>(S, a.t.P[0], [&](int p) { return fma(a.eps_t, gp_derivative<T, N, 0>(u, a.t.D[0], p), G[p] * v[0][p]); });
            pl_divergence<T, N, 1>(S, a.t.P[1], [&](int p) { return fma(a.eps_t, gp_derivative<T, N, 1>(u, a.t.D[1], p), G[p] * v[1][p]); });
            pl_test<T, N>(S, F, a.t, qz, R);
          }
      }
    };

    // M / dt + eps K in a narrow band (isotropic, no normal field): value and flux masked per Gauss point
    template <int K, typename T>
    struct BandCellOp
    {
      static constexpr bool HEAVY = false, NODES = false, SPLIT = false;
      static constexpr int N = K + 1, N3 = N * N * N;
      using Args = PointArgs<T, N>;
      const Args &a;
      __device__ __forceinline__ PointCell
      load(bool, int cx, int cy, int cz) const
      {
        return point_cell(a.g, cx, cy, cz);
      }
      template <bool DOT>
      __device__ __forceinline__ double
      apply(T *u, const PointCell &c) const
      {
        T                        S[N3];
        const unsigned long long bits = band_bits<T, N>(a.band_ls, a.band, a.t.B, a.g, c);
        auto in = [&](int q, T x) { return (bits >> q) & 1u ? x : T(0); };
        // u - ref as in ReinitCellOp
        const T ref = u[((K / 2) * N + K / 2) * N + K / 2];
#pragma unroll
        for (int q = 0; q < N3; ++q)
          u[q] -= ref;
        interpolate<T, N>(u, a.t.B);
#pragma unroll
        for (int q = 0; q < N3; ++q)
          S[q] = in(q, a.mass * (u[q] + ref));
        // t.D carries the diffusivity
        gp_divergence<T, N, 0>(S, a.t.P[0], [&](int q) { return in(q, gp_derivative<T, N, 0>(u, a.t.D[0], q)); });
        gp_divergence<T, N, 1>(S, a.t.P[1], [&](int q) { return in(q, gp_derivative<T, N, 1>(u, a.t.D[1], q)); });
        gp_divergence<T, N, 2>(S, a.t.P[2], [&](int q) { return in(q, gp_derivative<T, N, 2>(u, a.t.D[2], q)); });
        test<T, N>(S, a.t);
#pragma unroll
        for (int q = 0; q < N3; ++q)
          u[q] = S[q];
        return 0.0;
      }
    };

    // int grad psi phi, in the band if there is one, to three vectors; NORMALIZED: the unit gradient
    // (|.| > 1e-16).  One launch, the components finished one after the other, or (SPLIT: unit gradient at
    // k = 3, whose 192 values do not fit the registers) by CTAs of their own.  FE_Q(1) 33x66x80: gradient 33 us as three launches, 19 as one; unit gradient,
    // which each of the three formed anew, 62 and 30; FE_Q(2) 80x64x48: 66 and 52, 225 and 125.
    template <int K>
    struct GradientArgs : PointArgs<double, K + 1>
    {
      double *out[3];
    };
    template <int K, bool NORMALIZED>
    struct GradientCellOp
    {
      static constexpr bool HEAVY = NORMALIZED, NODES = true, SPLIT = NORMALIZED && K == 3;
      static constexpr int  N = K + 1, N3 = N * N * N, OUT = SPLIT ? 1 : 3;
      using Args = GradientArgs<K>;
      struct State
      {
        unsigned long long bits;
        double             g[NORMALIZED && !SPLIT ? 3 : 1][NORMALIZED && !SPLIT ? N3 : 1]; // the unit gradient
      };
      const Args &a;
      __device__ __forceinline__ PointCell
      load(bool, int cx, int cy, int cz) const
      {
        return point_cell(a.g, cx, cy, cz);
      }
      __device__ __forceinline__ double *
      out(int m) const
      {
        return a.out[m];
      }
      // put(q, gx, gy, gz): the unit gradient at the points, from u - ref as in ReinitCellOp
      template <class Put>
      __device__ __forceinline__ void
      unit_gradient(const MarchNodes<K, double> &nodes, const Put &put) const
      {
        const double ref = nodes.row[(K / 2) * N + K / 2][K / 2];
        double       v[N3];
#pragma unroll
        for (int r = 0; r < N * N; ++r)
#pragma unroll
          for (int i = 0; i < N; ++i)
            v[r * N + i] = nodes.row[r][i] - ref;
        interpolate<double, N>(v, a.t.B);
#pragma unroll
        for (int q = 0; q < N3; ++q)
          {
            const double gx = gp_derivative<double, N, 0>(v, a.t.D[0], q), gy = gp_derivative<double, N, 1>(v, a.t.D[1], q),
                         gz = gp_derivative<double, N, 2>(v, a.t.D[2], q);
            const double nn = sqrt(fma(gz, gz, fma(gy, gy, gx * gx))), f = nn > 1e-16 ? 1.0 / nn : 1e16;
            put(q, f * gx, f * gy, f * gz);
          }
      }
      __device__ __forceinline__ unsigned long long
      band(const PointCell &c) const
      {
        return a.band_ls ? band_bits<double, N>(a.band_ls, a.band, a.t.B, a.g, c) : ~0ull;
      }
      __device__ __forceinline__ void
      prepare(const MarchNodes<K, double> &nodes, const PointCell &c, State &s) const
      {
        s.bits = band(c);
        if constexpr (NORMALIZED)
          unit_gradient(nodes, [&](int q, double gx, double gy, double gz) {
            s.g[0][q] = gx;
            s.g[1][q] = gy;
            s.g[2][q] = gz;
          });
      }
      template <int DIR>
      __device__ __forceinline__ void
      component(double *u, const MarchNodes<K, double> &nodes, State &s) const
      {
        if constexpr (!NORMALIZED)
          {
#pragma unroll
            for (int r = 0; r < N * N; ++r)
#pragma unroll
              for (int i = 0; i < N; ++i)
                u[r * N + i] = nodes.row[r][i];
            gp_gradient<double, N, DIR>(u, a.t.B, a.t.G[DIR]);
          }
#pragma unroll
        for (int q = 0; q < N3; ++q)
          {
            if constexpr (NORMALIZED)
              u[q] = s.g[DIR][q];
            u[q] = (s.bits >> q) & 1u ? u[q] : 0.0;
          }
        test<double, N>(u, a.t);
      }
      // SPLIT: the component of the CTA
      __device__ __forceinline__ void
      apply(double *u, const MarchNodes<K, double> &nodes, const PointCell &c) const
      {
        const unsigned long long bits = band(c);
        const unsigned           dir  = blockIdx.y;
        unit_gradient(nodes, [&](int q, double gx, double gy, double gz) {
          u[q] = (bits >> q) & 1u ? (dir == 0 ? gx : dir == 1 ? gy : gz) : 0.0;
        });
        test<double, N>(u, a.t);
      }
    };

    // -int div(n) phi, n = normalize(n_i, tol) at every DoF; the marching input is n_x.  t.G carries the sign.
    template <int K>
    struct DivergenceCellOp
    {
      static constexpr bool HEAVY = false, NODES = false, SPLIT = false;
      static constexpr int N = K + 1, N3 = N * N * N;
      using Args = PointArgs<double, N>;
      const Args &a;
      __device__ __forceinline__ PointCell
      load(bool, int cx, int cy, int cz) const
      {
        return point_cell(a.g, cx, cy, cz);
      }
      template <bool DOT>
      __device__ __forceinline__ double
      apply(double *u, const PointCell &c) const
      {
        double S[N3], inv[N3], v[N3];
#pragma unroll
        for (int q = 0; q < N3; ++q)
          inv[q] = u[q] * u[q];
        field_nodes<double, N>(a.n[1], a.g, c, v);
#pragma unroll
        for (int q = 0; q < N3; ++q)
          inv[q] = fma(v[q], v[q], inv[q]);
        field_nodes<double, N>(a.n[2], a.g, c, v);
#pragma unroll
        for (int q = 0; q < N3; ++q)
          {
            const double nn = fma(v[q], v[q], inv[q]);
            inv[q]          = nn > a.tol2 ? point_rsqrt(nn) : a.inv_tol;
            v[q] *= inv[q];
            u[q] *= inv[q];
          }
        gp_gradient<double, N, 2>(v, a.t.B, a.t.G[2]);
        gp_gradient<double, N, 0>(u, a.t.B, a.t.G[0]);
#pragma unroll
        for (int q = 0; q < N3; ++q)
          S[q] = v[q] + u[q];
        field_nodes<double, N>(a.n[1], a.g, c, v);
#pragma unroll
        for (int q = 0; q < N3; ++q)
          v[q] *= inv[q];
        gp_gradient<double, N, 1>(v, a.t.B, a.t.G[1]);
#pragma unroll
        for (int q = 0; q < N3; ++q)
          S[q] += v[q];
        if (a.band_ls)
          {
            const unsigned long long bits = band_bits<double, N>(a.band_ls, a.band, a.t.B, a.g, c);
#pragma unroll
            for (int q = 0; q < N3; ++q)
              S[q] = (bits >> q) & 1u ? S[q] : 0.0;
          }
        test<double, N>(S, a.t);
#pragma unroll
        for (int q = 0; q < N3; ++q)
          u[q] = S[q];
        return 0.0;
      }
    };

    // CTAs (of 128 threads) per SM the register allocation is held to; tangent and rhs, 72x56x64 FE_Q(2) FP64: 288 us at
    // 2 (1250 before, point by point over the nodes), 343 at 3; normal, curvature and banded apply 310 at 3, 348 at 4
    template <int K, typename T, bool HEAVY>
    struct PointMinBlocks
    {
      static constexpr int value = K == 1 ? 6 : (K == 2 ? (sizeof(T) == 8 ? (HEAVY ? 2 : 3) : 4) : 2);
    };

    template <int K, typename T, OutMode MODE, class Op, int BX>
    __global__ void __launch_bounds__(MARCH_NT, PointMinBlocks<K, T, Op::HEAVY>::value)
    reinit_march_kernel(const __grid_constant__ typename Op::Args a)
    {
      extern __shared__ __align__(16) unsigned char smem_raw[];
      __shared__ unsigned                        s_ticket;
      __shared__ __align__(8) unsigned long long s_bars[2];
      Op                                         op{a};
      T                                         *dst = a.dst;
      if constexpr (Op::SPLIT)
        dst = a.out[blockIdx.y];
      march_body<K, T, MODE, Op, false, true, BX>(a.g, a.s, a.src, dst, a.b, a.mask_src != 0, op,
                                              reinterpret_cast<T *>(smem_raw), &s_ticket, s_bars);
    }

    template <int K, typename T, OutMode MODE, class Op, int BX>
    cudaError_t
    launch_point_columns(typename Op::Args &a, cudaStream_t s)
    {
      auto                                   kern = reinit_march_kernel<K, T, MODE, Op, BX>;
      static std::atomic<unsigned long long> devices{0};
      constexpr size_t                       bytes = MarchLayout<K, T, BX>::bytes;
      if (cudaError_t e = ensure_smem(kern, bytes, devices); e != cudaSuccess)
        return e;
      const unsigned ctas = march_grid(a.g, BX, MarchShape<K, T>::BZ, PointMinBlocks<K, T, Op::HEAVY>::value);
      kern<<<dim3(ctas, Op::SPLIT ? 3 : 1), MARCH_NT, bytes, s>>>(a);
      return cudaGetLastError();
    }

    template <int K, typename T, OutMode MODE, class Op>
    cudaError_t
    launch_point_kernel(typename Op::Args &a, cudaStream_t s)
    {
      if constexpr (MODE != OutMode::BPlus) // b + A x is formed once a solve: one width
        if (march_bx(a.g.m) != MARCH_BX)
          return launch_point_columns<K, T, MODE, Op, MARCH_BX_NARROW>(a, s);
      return launch_point_columns<K, T, MODE, Op, MARCH_BX>(a, s);
    }

    // the tangent (mode 0), the banded isotropic form (mode 0 without a normal field) or the rhs (mode 1)
    template <int K, typename T>
    cudaError_t
    launch_reinit_march(const ReinitLaunch<T> &h, int mode, cudaStream_t s)
    {
      constexpr int       N = K + 1;
      PointArgs<T, N>     a{};
      const Tables1D     &t = tables(K);
      const bool          banded = h.band > 0.0 && h.band_ls != nullptr;
      a.g                        = h.grid;
      a.s                        = h.sync;
      a.t.fill(t.ext.B, t.ext.G, t.ext.Dq, t.ext.qw, h.hlen);
      if (h.normal[0] == nullptr) // the banded form's flux: D carries the diffusivity
        for (int d = 0; d < 3; ++d)
          gp_on_differences<T, N>(t.ext.Dq, (long double)h.scale * h.eps_tangential / h.hlen[d], a.t.D[d]);
      a.eps_t    = (T)((mode == 1 ? -1.0 : h.scale) * h.eps_tangential);
      a.eps      = (T)((mode == 1 ? -1.0 : h.scale) * (h.eps_normal - h.eps_tangential));
      a.mass     = mode == 1 ? T(0) : (T)(h.scale / h.dt);
      a.tol2     = (T)(h.normal_tolerance * h.normal_tolerance);
      a.inv_tol  = (T)(1.0 / h.normal_tolerance);
      a.src      = h.src;
      a.dst      = h.dst;
      a.b        = h.b;
      a.mask_src = mode == 1 ? 0 : h.mask_src;
      a.band_ls  = banded ? h.band_ls : nullptr;
      a.band     = (T)h.band;
      for (int d = 0; d < 3; ++d)
        a.n[d] = h.normal[d];
      if (mode == 1)
        return launch_point_kernel<K, T, OutMode::Set, ReinitCellOp<K, T, true>>(a, s);
      if (h.normal[0] == nullptr)
        switch (h.out_mode)
          {
            case 0: return launch_point_kernel<K, T, OutMode::Set, BandCellOp<K, T>>(a, s);
            case 1: return launch_point_kernel<K, T, OutMode::Add, BandCellOp<K, T>>(a, s);
            default: return launch_point_kernel<K, T, OutMode::BPlus, BandCellOp<K, T>>(a, s);
          }
      switch (h.out_mode)
        {
          case 0: return launch_point_kernel<K, T, OutMode::Set, ReinitCellOp<K, T, false>>(a, s);
          case 1: return launch_point_kernel<K, T, OutMode::Add, ReinitCellOp<K, T, false>>(a, s);
          default: return launch_point_kernel<K, T, OutMode::BPlus, ReinitCellOp<K, T, false>>(a, s);
        }
    }

    template <int K, typename T>
    cudaError_t
    launch_reinit(const ReinitLaunch<T> &h, int mode, cudaStream_t s)
    {
      constexpr int     N = K + 1;
      ReinitArgs<T, N> a{};
      a.g      = h.grid;
      a.scale  = (T)h.scale;
      a.inv_dt = (T)(1.0 / h.dt);
      a.eps_n  = (T)h.eps_normal;
      a.eps_t  = (T)h.eps_tangential;
      a.tol    = (T)h.normal_tolerance;
      a.det    = (T)(h.hlen[0] * h.hlen[1] * h.hlen[2]);
      for (int d = 0; d < 3; ++d)
        {
          a.ih[d] = (T)(1.0 / h.hlen[d]);
          a.n[d]  = h.normal[d];
        }
      const Tables1D &t = tables(K);
      for (int i = 0; i < N * N; ++i)
        {
          a.B[i] = (T)t.ext.B[i]; // as in GaussTab (band_bits)
          a.G[i] = (T)t.G[i];
        }
      for (int q = 0; q < N; ++q)
        a.w[q] = (T)t.qw[q];
      a.src      = h.src;
      a.dst      = h.dst;
      a.diag     = h.diag;
      a.mode     = mode;
      a.mask_src = h.mask_src;
      a.band_ls  = h.band > 0.0 ? h.band_ls : nullptr;
      a.band     = (T)h.band;
      a.wetting  = h.wetting;
      // basis values and derivatives at the end points of [0, 1] (Lagrange on the Gauss-Lobatto
      // nodes: the values are the unit rows of the first and last node; the derivatives are the rows
      // of the nodal differentiation matrix there, from the barycentric weights)
      for (int side = 0; side < 2; ++side)
        {
          const int jn = side ? N - 1 : 0;
          for (int i = 0; i < N; ++i)
            {
              a.Vend[side * N + i] = i == jn ? T(1) : T(0);
              double wi = 1.0, wj = 1.0;
              for (int k = 0; k < N; ++k)
                {
                  if (k != i)
                    wi /= (t.nodes[i] - t.nodes[k]);
                  if (k != jn)
                    wj /= (t.nodes[jn] - t.nodes[k]);
                }
              double dji = 0.0;
              if (i != jn)
                dji = wi / wj / (t.nodes[jn] - t.nodes[i]);
              else
                for (int k = 0; k < N; ++k)
                  if (k != jn)
                    {
                      double wk = 1.0;
                      for (int kk = 0; kk < N; ++kk)
                        if (kk != k)
                          wk /= (t.nodes[k] - t.nodes[kk]);
                      dji -= wk / wj / (t.nodes[jn] - t.nodes[k]);
                    }
              a.Dend[side * N + i] = (T)dji;
            }
        }
      const long long ncell  = (long long)h.grid.m[0] * h.grid.m[1] * h.grid.m[2];
      const int       blocks = (int)std::max<long long>(1, std::min<long long>((ncell + 127) / 128, 148LL * 16));
      if (mode == 2)
        reinit_diag_kernel<K, T><<<blocks, 128, 0, s>>>(a);
      else if (cudaError_t e = launch_reinit_march<K, T>(h, mode, s); e != cudaSuccess)
        return e;
      if (h.wetting && a.n[0] != nullptr)
        {
          cudaError_t e = cudaGetLastError();
          if (e != cudaSuccess)
            return e;
          wetting_kernel<K, T><<<148, 128, 0, s>>>(a);
        }
      return cudaGetLastError();
    }
  } // namespace

  namespace
  {
    template <int K>
    cudaError_t
    launch_level_set_rhs(const GridDesc &g, const SyncDesc &sync, const double hlen[3], int mode, int normalized, double tol,
                         const double *const in[3], double *const out[3], cudaStream_t s, const double *band_ls,
                         double band)
    {
      constexpr int        N = K + 1;
      GradientArgs<K> a{};
      a.g = g;
      a.s = sync;
      const Tables1D &t = tables(K);
      a.t.fill(t.ext.B, t.ext.G, t.ext.Dq, t.ext.qw, hlen);
      a.src      = in[0];
      a.mask_src = 0;
      a.band_ls  = band > 0.0 ? band_ls : nullptr;
      a.band     = band;
      if (mode == 0)
        {
          for (int d = 0; d < 3; ++d)
            a.out[d] = out[d];
          return normalized ? launch_point_kernel<K, double, OutMode::Add, GradientCellOp<K, true>>(a, s) :
                              launch_point_kernel<K, double, OutMode::Add, GradientCellOp<K, false>>(a, s);
        }
      for (int d = 0; d < 3; ++d)
        {
          a.n[d] = in[d];
          for (int i = 0; i < N * (N - 1); ++i)
            a.t.G[d][i] = -a.t.G[d][i];
        }
      a.tol2    = tol * tol;
      a.inv_tol = 1.0 / tol;
      a.dst     = out[0];
      return launch_point_kernel<K, double, OutMode::Set, DivergenceCellOp<K>>(a, s);
    }
  } // namespace

  // Right-hand sides of the normal-vector and curvature projections:
  //   mode 0: dst_d += int g_d phi, g = grad psi, or normalize(grad psi, 1e-16) when normalized
  //           (normal_vector_operator.cpp:160-240)
  //   mode 1: dst   = -int div(n) phi with n = normalize(n_i, tol) at every DoF
  //           (curvature_operator.cpp:190-255)
  // Narrow band (normal_vector_operator.cpp:184-191, curvature_operator.cpp:209-214): the gradient or the
  // divergence is masked by |level set| < band at the Gauss point.
  cudaError_t
  level_set_rhs(const GridDesc &g, const SyncDesc &sync, int K, const double hlen[3], int mode, int normalized, double tol,
                const double *in0, const double *in1, const double *in2, double *out0, double *out1, double *out2,
                cudaStream_t s, const double *band_ls, double band)
  {
    const double *in[3]  = {in0, in1, in2};
    double       *out[3] = {out0, out1, out2};
    switch (K)
      {
        case 1: return launch_level_set_rhs<1>(g, sync, hlen, mode, normalized, tol, in, out, s, band_ls, band);
        case 2: return launch_level_set_rhs<2>(g, sync, hlen, mode, normalized, tol, in, out, s, band_ls, band);
        case 3: return launch_level_set_rhs<3>(g, sync, hlen, mode, normalized, tol, in, out, s, band_ls, band);
        default: return cudaErrorInvalidValue;
      }
  }

  template <int K>
  static long long
  launch_bricks(const int m[3], bool banded)
  {
    return march_bricks(m, march_bx(m), MarchShape<K, double>::BZ,
                        banded ? PointMinBlocks<K, double, BandCellOp<K, double>::HEAVY>::value :
                                 PointMinBlocks<K, double, ReinitCellOp<K, double, false>::HEAVY>::value);
  }

  long long
  reinit_launch_bricks(int K, const int m[3], bool banded)
  {
    return K == 1 ? launch_bricks<1>(m, banded) : (K == 2 ? launch_bricks<2>(m, banded) : launch_bricks<3>(m, banded));
  }

  template <typename T>
  cudaError_t
  reinit_integrate(const ReinitLaunch<T> &h, int mode, cudaStream_t s)
  {
    switch (h.degree)
      {
        case 1: return launch_reinit<1, T>(h, mode, s);
        case 2: return launch_reinit<2, T>(h, mode, s);
        case 3: return launch_reinit<3, T>(h, mode, s);
        default: return cudaErrorInvalidValue;
      }
  }

  template cudaError_t reinit_integrate<double>(const ReinitLaunch<double> &, int, cudaStream_t);
  template cudaError_t reinit_integrate<float>(const ReinitLaunch<float> &, int, cudaStream_t);
} // namespace mpdg
