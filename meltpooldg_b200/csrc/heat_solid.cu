// Heat operator with temperature-dependent material (solid / liquid phases), FE_Q(1..3).
//
// Reference: source/heat/heat_diffuse_operator.cpp, tangent_local_cell_operation :1029-1050 with
// do_solidification (material of Material::compute_parameters, MaterialTypes::liquid_solid,
// include/meltpooldg/core/material.templates.hpp:296-360, :540-620, :748-765):
//   tangent   val  = (rho c_p(T) / dt + d(rho c_p)/dT (T - T_old) / dt) u
//             grad = k(T) grad u + dk/dT grad T u
//   residual  (rhs_cell_loop :485-527)  val = rho c_p(T) (T - T_old) / dt,  grad = k(T) grad T,
//             submitted with a minus sign (the heat source enters through the mass apply)
// T and T_old are read plainly (read_dof_values_plain), u with constraints.  Solid fraction
// f_s = clamp((T_liquidus - T) / (T_liquidus - T_solidus), 0, 1) (mushy zone) or T < T_solidus
// (sharp); a property is the cubic blend v_l + (v_s - v_l)(3 f_s^2 - 2 f_s^3) (f_s = 0 / 1 give
// v_l / v_s), its temperature derivative -(v_s - v_l)(6 f_s - 6 f_s^2) / (T_liquidus - T_solidus)
// (0 at f_s = 0 or 1).
//
// One thread per cell in the column-marching frame (march.cuh), sum factorisation on the Gauss points, one plane
// of points at a time (gausspoint.cuh): T, T - T_old and u at the plane, the material point by point, the
// flux k grad u + dk/dT u grad T tested with the gradient.  The cell arrays of the fields at all 27 points
// (FE_Q(2)) do not fit the registers, and in local memory they overrun L1; a rolled loop over the planes holds
// nine points of each field and keeps a third of the code.  The slopes and reciprocals of the capacity's ramp are
// constants (its divisions were two thirds of the FP64 work of a quadrature with 10,069 instructions per
// 32 cells).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "brick.cuh"
#include "gausspoint.cuh"
#include "kernels.h"
#include "march.cuh"

#include <type_traits>

namespace mpdg
{
  namespace
  {
    template <typename T>
    struct SolidMat
    {
      T   rho_l, cp_l, k_l, rho_s, cp_s, k_s, t_liquidus, t_solidus, inv_mushy;
      int sharp;
      T   latent;   // latent heat of fusion (0: none)
      int cap_type; // apparent capacity: 0 quadratic-linear-quadratic, 1 quartic bell, 2 constant
      // constants of the capacity shapes: width and mid temperature of the mushy zone; the tent's peak, its
      // half width, the width delta of its flat ends, its slope and slope / delta; L / dT, L 2 / dT and
      // L (2 / dT)^2
      T   width, t_mid, peak, half, delta, slope, slope_delta, c_const, c_bell, dc_bell;
    };

    // Apparent specific heat of the latent heat and its temperature derivative at solid fraction fs in the
    // open mushy zone (include/meltpooldg/core/material.templates.hpp:561-614,
    // source/heat/apparent_capacity.cpp:157-300), each shape integrating to L over [T_solidus, T_liquidus]:
    // constant L / dT; quartic bell L (2 / dT) 15/16 (1 - x^2)^2 with x = 1 - 2 fs; the default tent of
    // peak 2 L / dT at the mid temperature whose flanks are ramps with zero slope at both ends (quadratic over
    // dT / 6, linear in between), evaluated at T = T_liquidus - fs dT.
    template <typename T>
    __device__ __forceinline__ void
    apparent_capacity(const SolidMat<T> &m, T fs, T &c, T &dc)
    {
      if (m.cap_type == 2)
        {
          c  = m.c_const;
          dc = T(0);
        }
      else if (m.cap_type == 1)
        {
          const T x = T(1) - T(2) * fs, y = T(1) - x * x;
          c         = m.c_bell * T(15.0 / 16.0) * y * y;
          dc        = -m.dc_bell * T(15.0 / 4.0) * y * x;
        }
      else
        {
          const T t = m.t_liquidus - fs * m.width;
          const T x = t <= m.t_mid ? t - m.t_solidus : m.t_liquidus - t, y = m.half - x; // from the nearer end / the peak
          T       d;
          if (x < m.delta)
            {
              c = T(0.5) * m.slope_delta * x * x;
              d = m.slope_delta * x;
            }
          else if (y < m.delta)
            {
              c = m.peak - T(0.5) * m.slope_delta * y * y;
              d = m.slope_delta * y;
            }
          else
            {
              c = m.slope * (x - T(0.5) * m.delta);
              d = m.slope;
            }
          dc = t <= m.t_mid ? d : -d;
        }
    }

    // rho c_p, k and their temperature derivatives at temperature t
    template <typename T>
    __device__ __forceinline__ void
    solid_material(const SolidMat<T> &m, T t, T &rc, T &k, T &drc, T &dk)
    {
      const T fs = m.sharp ? (t < m.t_solidus ? T(1) : T(0)) : fmin(fmax((m.t_liquidus - t) * m.inv_mushy, T(0)), T(1));
      drc = dk = T(0);
      if (fs == T(0))
        {
          rc = m.rho_l * m.cp_l;
          k  = m.k_l;
        }
      else if (fs == T(1))
        {
          rc = m.rho_s * m.cp_s;
          k  = m.k_s;
        }
      else
        {
          const T w = (T(3) - T(2) * fs) * fs * fs, dw = -m.inv_mushy * (T(6) * fs - T(6) * fs * fs);
          T       ca = T(0), dca = T(0);
          if (m.latent > T(0))
            apparent_capacity(m, fs, ca, dca);
          const T rho = m.rho_l + (m.rho_s - m.rho_l) * w, cp = m.cp_l + (m.cp_s - m.cp_l) * w + ca;
          rc          = rho * cp;
          k           = m.k_l + (m.k_s - m.k_l) * w;
          drc         = (m.rho_s - m.rho_l) * dw * cp + rho * ((m.cp_s - m.cp_l) * dw + dca);
          dk          = (m.k_s - m.k_l) * dw;
        }
    }

    template <typename T, int N>
    struct SolidArgs
    {
      GridDesc       g;
      SyncDesc       s;
      SolidMat<T>    m;
      GaussTab<T, N> t;       // Bt[2] with the volume and the scale
      T              inv_dt;
      // diagonal: w_q B_qi^2, w_q (G_qi / h)^2 and w_q B_qi G_qi / h per direction (rows: nodes)
      T              BB[3][N * N], GG[3][N * N], BG[3][N * N];
      const T       *src;
      const double  *temp, *temp_old;
      T             *dst;
      const T       *b;
      int            mask_src;
      const int     *skip;
    };

    // A cell's temperatures at one plane of Gauss points: T, its z derivative and T - T_old (the difference
    // taken in double at the nodes), read plainly.
    struct SolidCell
    {
      long long first; // the cell's first lattice point
    };
    template <int N>
    __device__ __forceinline__ SolidCell
    solid_cell(const GridDesc &g, int cx, int cy, int cz)
    {
      // a lane outside the mesh reads the temperatures of the nearest cell
      constexpr int K = N - 1;
      return SolidCell{K * min(cx, g.m[0] - 1) + (long long)g.n[0] * (K * min(cy, g.m[1] - 1) + (long long)g.n[1] * (K * cz))};
    }
    template <typename T, int N>
    __device__ __forceinline__ void
    solid_plane(const SolidArgs<T, N> &a, const SolidCell &c, const T *bz, const T *gz, T *t, T *tz, T *d)
    {
      const int     sy = a.g.n[0], sz = a.g.n[0] * a.g.n[1];
      const double *ft = a.temp + c.first, *fo = a.temp_old + c.first;
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 0; i < N; ++i)
          {
            T x[N], y[N];
#pragma unroll
            for (int l = 0; l < N; ++l)
              {
                const int    p = j * sy + l * sz + i;
                const double v = __ldg(ft + p);
                x[l]           = (T)v;
                y[l]           = (T)(v - __ldg(fo + p));
              }
            T s = bz[0] * x[0], e = bz[0] * y[0], g = gz[0] * (x[1] - x[0]);
#pragma unroll
            for (int l = 1; l < N; ++l)
              {
                s = fma(bz[l], x[l], s);
                e = fma(bz[l], y[l], e);
              }
#pragma unroll
            for (int l = 1; l < N - 1; ++l)
              g = fma(gz[l], x[l + 1] - x[l], g);
            t[j * N + i]  = s;
            tz[j * N + i] = g;
            d[j * N + i]  = e;
          }
      pl_interpolate<T, N>(t, a.t.B);
      pl_interpolate<T, N>(tz, a.t.B);
      pl_interpolate<T, N>(d, a.t.B);
    }

    // tangent (src read with constraints) and residual (RHS: src unused, the result subtracted by Bt, Gzt)
    template <int K, typename T, bool RHS>
    struct SolidCellOp
    {
      static constexpr int  N = K + 1, N2 = N * N, N3 = N * N * N;
      static constexpr bool NODES = true, TANGENT = !RHS;
      const SolidArgs<T, N> &a;
      __device__ __forceinline__ SolidCell
      load(bool, int cx, int cy, int cz) const
      {
        return solid_cell<N>(a.g, cx, cy, cz);
      }
      __device__ __forceinline__ void
      apply(T *R, const MarchNodes<K, T> &nodes, const SolidCell &c) const
      {
#pragma unroll
        for (int q = 0; q < N3; ++q)
          R[q] = T(0);
#pragma unroll(K == 1 ? 2 : 1)
        for (int qz = 0; qz < N; ++qz)
          {
            const T *bz = a.t.B + qz * N, *gz = a.t.G[2] + qz * (N - 1);
            T        t[N2], tz[N2], S[N2], k[N2], F[N2];
            solid_plane<T, N>(a, c, bz, gz, t, tz, S);
            if constexpr (RHS)
              {
#pragma unroll
                for (int p = 0; p < N2; ++p)
                  {
                    T rc, drc, dk;
                    solid_material(a.m, t[p], rc, k[p], drc, dk);
                    S[p] *= a.inv_dt * rc;
                    F[p] = k[p] * tz[p];
                  }
                pl_divergence<T, N, 0>(S, a.t.P[0], [&](int p) { return k[p] * gp_derivative<T, N, 0>(t, a.t.D[0], p); });
                pl_divergence<T, N, 1>(S, a.t.P[1], [&](int p) { return k[p] * gp_derivative<T, N, 1>(t, a.t.D[1], p); });
              }
            else
              {
                T u[N2], e[N2];
                pl_value<T, N>([&](int l, int j, int i) { return nodes.row[l * N + j][i]; }, bz, u);
                pl_zderivative<T, N>([&](int l, int j, int i) { return nodes.row[l * N + j][i]; }, gz, F);
                pl_interpolate<T, N>(u, a.t.B);
                pl_interpolate<T, N>(F, a.t.B);
#pragma unroll
                for (int p = 0; p < N2; ++p)
                  {
                    T rc, drc, dk;
                    solid_material(a.m, t[p], rc, k[p], drc, dk);
                    S[p] = a.inv_dt * fma(drc, S[p], rc) * u[p];
                    e[p] = dk * u[p];
                    F[p] = fma(k[p], F[p], e[p] * tz[p]);
                  }
                pl_divergence<T, N, 0>(S, a.t.P[0], [&](int p) {
                  return fma(k[p], gp_derivative<T, N, 0>(u, a.t.D[0], p), e[p] * gp_derivative<T, N, 0>(t, a.t.D[0], p));
                });
                pl_divergence<T, N, 1>(S, a.t.P[1], [&](int p) {
                  return fma(k[p], gp_derivative<T, N, 1>(u, a.t.D[1], p), e[p] * gp_derivative<T, N, 1>(t, a.t.D[1], p));
                });
              }
            pl_test<T, N>(S, F, a.t, qz, R);
          }
      }
    };

    // out (+)= M in along the lines of direction DIR (0 or 1) of a plane (in: a function of the point)
    template <typename T, int N, int DIR, bool ACC, class In>
    __device__ __forceinline__ void
    solid_contract(T *out, const T *M, const In &in)
    {
      constexpr int ST = DIR == 0 ? 1 : N, LN = DIR == 0 ? N : 1;
#pragma unroll
      for (int c = 0; c < N; ++c)
        {
          T v[N];
#pragma unroll
          for (int k = 0; k < N; ++k)
            v[k] = in(c * LN + k * ST);
#pragma unroll
          for (int r = 0; r < N; ++r)
            {
              T &o = out[c * LN + r * ST];
              T  s = ACC ? fma(M[r * N], v[0], o) : M[r * N] * v[0];
#pragma unroll
              for (int k = 1; k < N; ++k)
                s = fma(M[r * N + k], v[k], s);
              o = s;
            }
        }
    }

    // Diagonal of the tangent: entry i of a cell is the sum over the points of
    //   JxW [cap phi_i^2 + k |grad phi_i|^2 + dk/dT (grad T . grad phi_i) phi_i],
    // a sum of tensor products of the squared 1-D tables BB, GG and BG: 11 plane sweeps and 3 in z instead of
    // (k+1)^6 terms.
    template <int K, typename T>
    struct SolidDiagCellOp
    {
      static constexpr int  N = K + 1, N2 = N * N, N3 = N * N * N;
      static constexpr bool NODES = true, TANGENT = false;
      const SolidArgs<T, N> &a;
      __device__ __forceinline__ SolidCell
      load(bool, int cx, int cy, int cz) const
      {
        return solid_cell<N>(a.g, cx, cy, cz);
      }
      __device__ __forceinline__ void
      apply(T *R, const MarchNodes<K, T> &, const SolidCell &c) const
      {
#pragma unroll
        for (int q = 0; q < N3; ++q)
          R[q] = T(0);
#pragma unroll(K == 1 ? 2 : 1)
        for (int qz = 0; qz < N; ++qz)
          {
            T t[N2], tz[N2], cap[N2], k[N2], dk[N2], x[N2] = {}, y[N2];
            solid_plane<T, N>(a, c, a.t.B + qz * N, a.t.G[2] + qz * (N - 1), t, tz, cap);
#pragma unroll
            for (int p = 0; p < N2; ++p)
              {
                T rc, drc;
                solid_material(a.m, t[p], rc, k[p], drc, dk[p]);
                cap[p] = a.inv_dt * fma(drc, cap[p], rc);
              }
            auto into = [&](const T *M) {
#pragma unroll
              for (int l = 0; l < N; ++l)
                {
                  const T w = M[l * N + qz];
#pragma unroll
                  for (int p = 0; p < N2; ++p)
                    R[l * N2 + p] = fma(w, y[p], R[l * N2 + p]);
                }
            };
            const auto from_x = [&x](int p) { return x[p]; };
            // z derivatives of the mixed and of the stiffness part
            solid_contract<T, N, 0, false>(x, a.BB[0], [&](int p) { return dk[p] * tz[p]; });
            solid_contract<T, N, 1, false>(y, a.BB[1], from_x);
            into(a.BG[2]);
            solid_contract<T, N, 0, false>(x, a.BB[0], [&](int p) { return k[p]; });
            solid_contract<T, N, 1, false>(y, a.BB[1], from_x);
            into(a.GG[2]);
            // y derivatives, then the x derivatives and the capacity, all with BB in z
            solid_contract<T, N, 1, false>(y, a.GG[1], from_x);
            solid_contract<T, N, 0, false>(x, a.BB[0], [&](int p) { return dk[p] * gp_derivative<T, N, 1>(t, a.t.D[1], p); });
            solid_contract<T, N, 1, true>(y, a.BG[1], from_x);
            solid_contract<T, N, 0, false>(x, a.BB[0], [&](int p) { return cap[p]; });
            solid_contract<T, N, 0, true>(x, a.GG[0], [&](int p) { return k[p]; });
            solid_contract<T, N, 0, true>(x, a.BG[0], [&](int p) { return dk[p] * gp_derivative<T, N, 0>(t, a.t.D[0], p); });
            solid_contract<T, N, 1, true>(y, a.BB[1], from_x);
            into(a.BB[2]);
          }
      }
    };

    // CTAs (of 128 threads) per SM the register allocation is held to.  FE_Q(2) FP64 at 2 and 3: tangent 72^3 273 and
    // 318 us, 80x64x48 206 and 209, 33x33x40 77 and 75 (1.2 KB of spills per thread at 3); residual 80x64x48 176
    // and 171, diagonal 201 and 197
    template <int K, typename T, bool TANGENT>
    struct SolidMinBlocks
    {
      static constexpr int value = K == 1 ? 6 : (K == 2 ? (sizeof(T) == 8 ? (TANGENT ? 2 : 3) : 4) : 2);
    };

    template <int K, typename T, OutMode MODE, class Op, int BX>
    __global__ void __launch_bounds__(MARCH_NT, SolidMinBlocks<K, T, Op::TANGENT>::value)
    heat_solid_kernel(const __grid_constant__ SolidArgs<T, K + 1> a)
    {
      extern __shared__ __align__(16) unsigned char smem_raw[];
      __shared__ unsigned                        s_ticket;
      __shared__ __align__(8) unsigned long long s_bars[2];
      if (a.skip != nullptr && *a.skip != 0)
        return;
      Op op{a};
      march_body<K, T, MODE, Op, false, true, BX>(a.g, a.s, a.src, a.dst, a.b, a.mask_src != 0, op,
                                              reinterpret_cast<T *>(smem_raw), &s_ticket, s_bars);
    }

    template <typename T>
    SolidMat<T>
    solid_mat(const SolidMaterial &m)
    {
      SolidMat<T> s;
      s.rho_l = (T)m.rho_l, s.cp_l = (T)m.cp_l, s.k_l = (T)m.k_l;
      s.rho_s = (T)m.rho_s, s.cp_s = (T)m.cp_s, s.k_s = (T)m.k_s;
      s.t_liquidus = (T)m.t_liquidus, s.t_solidus = (T)m.t_solidus;
      s.inv_mushy  = m.t_liquidus > m.t_solidus ? (T)(1.0 / (m.t_liquidus - m.t_solidus)) : T(0);
      s.sharp      = m.sharp;
      s.latent     = (T)m.latent_heat;
      s.cap_type   = m.capacity_type;
      const double L = m.latent_heat, dT = m.t_liquidus > m.t_solidus ? m.t_liquidus - m.t_solidus : 1.0;
      const double delta = dT / 6.0, slope = 2.0 * L / dT / (0.5 * dT - delta);
      s.width       = (T)dT;
      s.t_mid       = (T)(0.5 * (m.t_solidus + m.t_liquidus));
      s.peak        = (T)(2.0 * L / dT);
      s.half        = (T)(0.5 * dT);
      s.delta       = (T)delta;
      s.slope       = (T)slope;
      s.slope_delta = (T)(slope / delta);
      s.c_const     = (T)(L / dT);
      s.c_bell      = (T)(L * 2.0 / dT);
      s.dc_bell     = (T)(L * 4.0 / (dT * dT));
      return s;
    }

    template <int K, typename T, OutMode MODE, class Op, int BX>
    cudaError_t
    launch_solid_columns(SolidArgs<T, K + 1> &a, cudaStream_t stream)
    {
      auto                                   kern = heat_solid_kernel<K, T, MODE, Op, BX>;
      static std::atomic<unsigned long long> devices{0};
      constexpr size_t                       bytes = MarchLayout<K, T, BX>::bytes;
      if (cudaError_t e = ensure_smem(kern, bytes, devices); e != cudaSuccess)
        return e;
      const unsigned ctas = march_grid(a.g, BX, MarchShape<K, T>::BZ, SolidMinBlocks<K, T, Op::TANGENT>::value);
      kern<<<ctas, MARCH_NT, bytes, stream>>>(a);
      return cudaGetLastError();
    }

    template <int K, typename T, OutMode MODE, class Op>
    cudaError_t
    launch_solid(SolidArgs<T, K + 1> &a, cudaStream_t stream)
    {
      if constexpr (MODE != OutMode::BPlus) // b + A x is formed once a solve: one width
        if (march_bx(a.g.m) != MARCH_BX)
          return launch_solid_columns<K, T, MODE, Op, MARCH_BX_NARROW>(a, stream);
      return launch_solid_columns<K, T, MODE, Op, MARCH_BX>(a, stream);
    }

    template <int K, typename T>
    cudaError_t
    solid_mode(const HeatSolidLaunch<T> &h, cudaStream_t s)
    {
      constexpr int   N = K + 1;
      SolidArgs<T, N> a{};
      a.g = h.grid;
      a.s = h.sync;
      a.m = solid_mat<T>(h.mat);
      // tables from doubles, as the diagonal's: the gradient of a temperature of 1e3 K rounds far above them
      const Tables1D &t = tables(K);
      a.t.fill(t.B, t.G, t.Dq, t.qw, h.hlen);
      const double scale = h.rhs ? -1.0 : h.scale;
      for (int i = 0; i < N * N; ++i)
        {
          a.t.Bt[2][i] = (T)(scale * (double)a.t.Bt[2][i]);
          a.t.Gzt[i]   = (T)(scale * (double)a.t.Gzt[i]);
        }
      a.inv_dt   = (T)(1.0 / h.dt);
      a.src      = h.src;
      a.temp     = h.temp;
      a.temp_old = h.temp_old;
      a.dst      = h.dst;
      a.b        = h.b;
      a.mask_src = h.mask_src;
      a.skip     = h.skip;
      if (h.rhs)
        {
          // the residual takes its values from T alone: the marching input only paces the march
          if constexpr (std::is_same<T, double>::value)
            {
              a.src      = h.temp;
              a.mask_src = 0;
              return launch_solid<K, T, OutMode::Add, SolidCellOp<K, T, true>>(a, s);
            }
          return cudaErrorInvalidValue;
        }
      switch (h.mode)
        {
          case 0: return launch_solid<K, T, OutMode::Set, SolidCellOp<K, T, false>>(a, s);
          case 1: return launch_solid<K, T, OutMode::Add, SolidCellOp<K, T, false>>(a, s);
          default: return launch_solid<K, T, OutMode::BPlus, SolidCellOp<K, T, false>>(a, s);
        }
    }

    template <int K>
    cudaError_t
    solid_diagonal(const GridDesc &g, const SyncDesc &sync, const SolidMaterial &mat, double dt, const double hlen[3],
                   const double *temp, const double *temp_old, double *diag, cudaStream_t s)
    {
      constexpr int        N = K + 1;
      SolidArgs<double, N> a{};
      const Tables1D      &t = tables(K);
      a.g = g;
      a.s = sync;
      a.m = solid_mat<double>(mat);
      a.t.fill(t.B, t.G, t.Dq, t.qw, hlen);
      a.inv_dt = 1.0 / dt;
      for (int d = 0; d < 3; ++d)
        for (int q = 0; q < N; ++q)
          for (int i = 0; i < N; ++i)
            {
              const double w = t.qw[q] * (d == 2 ? hlen[0] * hlen[1] * hlen[2] : 1.0), B = t.B[q * N + i],
                           G = t.G[q * N + i] / hlen[d];
              a.BB[d][i * N + q] = w * B * B;
              a.GG[d][i * N + q] = w * G * G;
              a.BG[d][i * N + q] = w * B * G;
            }
      a.src      = temp;
      a.temp     = temp;
      a.temp_old = temp_old;
      a.dst      = diag;
      a.mask_src = 0;
      return launch_solid<K, double, OutMode::Set, SolidDiagCellOp<K, double>>(a, s);
    }
  } // namespace

  long long
  heat_solid_launch_bricks(int K, const int m[3])
  {
    return K == 1 ? march_bricks(m, march_bx(m), MarchShape<1, double>::BZ, SolidMinBlocks<1, double, true>::value) :
                    (K == 2 ? march_bricks(m, march_bx(m), MarchShape<2, double>::BZ, SolidMinBlocks<2, double, true>::value) :
                              march_bricks(m, march_bx(m), MarchShape<3, double>::BZ, SolidMinBlocks<3, double, true>::value));
  }

  template <typename T>
  cudaError_t
  heat_solid_apply(const HeatSolidLaunch<T> &h, cudaStream_t s)
  {
    switch (h.degree)
      {
        case 1: return solid_mode<1, T>(h, s);
        case 2: return solid_mode<2, T>(h, s);
        case 3: return solid_mode<3, T>(h, s);
        default: return cudaErrorInvalidValue;
      }
  }

  cudaError_t
  heat_solid_diagonal(const GridDesc &g, const SyncDesc &sync, int K, const SolidMaterial &mat, double dt, const double hlen[3],
                      const double *temp, const double *temp_old, double *diag, cudaStream_t s)
  {
    switch (K)
      {
        case 1: return solid_diagonal<1>(g, sync, mat, dt, hlen, temp, temp_old, diag, s);
        case 2: return solid_diagonal<2>(g, sync, mat, dt, hlen, temp, temp_old, diag, s);
        case 3: return solid_diagonal<3>(g, sync, mat, dt, hlen, temp, temp_old, diag, s);
        default: return cudaErrorInvalidValue;
      }
  }

  template cudaError_t heat_solid_apply<double>(const HeatSolidLaunch<double> &, cudaStream_t);
  template cudaError_t heat_solid_apply<float>(const HeatSolidLaunch<float> &, cudaStream_t);
} // namespace mpdg
