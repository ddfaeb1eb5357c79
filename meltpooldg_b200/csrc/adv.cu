// Advection-diffusion operator kernels.  Reference: source/level_set/advection_diffusion_operator.cpp
//   vmult :236-272 (cell_loop, zero dst), tangent_local_cell_operation :448-495
//     val = u/dt + theta v.grad u,  grad = theta eps grad u
//   create_rhs :274-358: val = u_old/dt - (1-theta) v.grad u_old, grad = -(1-theta) eps grad u_old
//     (the same kernel with theta replaced by theta - 1, plain reads)
//   compute_inverse_diagonal_from_matrixfree :399-446
// The velocity is an affine field v(x) = v0 + G x evaluated analytically at the Gauss points (the
// reference evaluates a dealii::Function there, :475-479); rigid rotations are affine.
//
// Per cell (one thread), sum factorisation in registers on the Gauss points, in the column-marching
// frame of march.cuh.  With u_q = (B(x)B(x)B) u the operator's values are kept without the point weights,
//   S = u_q / dt + sum_d [ v_d (theta D_d / h_d) u_q + L_d u_q ],   L_d = theta eps / h_d^2 W^-1 D^T W D
// (D the 1-D collocation derivative on the Gauss points, W its weights), so that a point costs one addition
// for its velocity and one fused multiply-add, and out = (B^T W (x) B^T W (x) B^T W) S.  For an affine velocity
// v_d at a point is the cell's value plus three per-direction offsets.  D, L and E act on the differences of
// neighbouring values (gausspoint.cuh).
//
// SUPG (ConvectionStabilizationType::SUPG, :455-457, :486-490, stabilisation parameter :497-533):
// the strong residual s = u/dt + theta v.grad u - theta eps lap u at the Gauss points (E_d = theta eps /
// h_d^2 D D: exact for the degree-k interpolant), tested with tau_c v.grad phi; tau_c = (coefficient < 0 ?
// 1 / max_q |v| (0 below 1e-6) : coefficient) times the cell size diameter / sqrt(3)
// (source/core/scratch_data.cpp:262-277).  The rhs uses the same form with theta replaced by theta - 1
// (:322-345).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "brick.cuh"
#include "gausspoint.cuh"
#include "kernels.h"
#include "march.cuh"

namespace mpdg
{
  constexpr int ADV_KMAX = 3;

  // out = M in along a line (in place), M[a*N+b], TR: transpose
  template <typename T, int N, int S, bool TR>
  __device__ __forceinline__ void
  line_mat(T *v, const int base, const T *M)
  {
    T in[N];
#pragma unroll
    for (int k = 0; k < N; ++k)
      in[k] = v[base + k * S];
#pragma unroll
    for (int a = 0; a < N; ++a)
      {
        T s = (TR ? M[a] : M[a * N]) * in[0];
#pragma unroll
        for (int k = 1; k < N; ++k)
          s = fma(TR ? M[k * N + a] : M[a * N + k], in[k], s);
        v[base + a * S] = s;
      }
  }

  template <typename T, int N, int D, bool TR>
  __device__ __forceinline__ void
  sweep(T *v, const T *M)
  {
    constexpr int S = D == 0 ? 1 : (D == 1 ? N : N * N);
#pragma unroll
    for (int a = 0; a < N; ++a)
#pragma unroll
      for (int c = 0; c < N; ++c)
        {
          const int base = D == 0 ? (a * N + c) * N : (D == 1 ? a * N * N + c : a * N + c);
          line_mat<T, N, S, TR>(v, base, M);
        }
  }

  // tau_c of the cell with lower corner (x0, y0, z0)
  template <typename T, int N>
  __device__ __forceinline__ T
  supg_tau(const T *vel, const T *h, const T *tqp, T x0, T y0, T z0, T coef, T cell_size)
  {
    T tau = coef;
    if (coef < T(0))
      {
        T vmax = T(0);
#pragma unroll
        for (int qz = 0; qz < N; ++qz)
#pragma unroll
          for (int qy = 0; qy < N; ++qy)
#pragma unroll
            for (int qx = 0; qx < N; ++qx)
              {
                const T x = x0 + h[0] * tqp[qx], y = y0 + h[1] * tqp[qy], z = z0 + h[2] * tqp[qz];
                T       n2 = T(0);
#pragma unroll
                for (int d = 0; d < 3; ++d)
                  {
                    const T v = vel[d] + vel[3 + 3 * d] * x + vel[4 + 3 * d] * y + vel[5 + 3 * d] * z;
                    n2        = fma(v, v, n2);
                  }
                vmax = fmax(vmax, sqrt(n2));
              }
        tau = vmax >= T(1e-6) ? T(1) / vmax : T(0);
      }
    return tau * cell_size;
  }

  // Velocity component d of a DoF-vector field at the cell's Gauss points: the cell's nodal values
  // read plainly (advection_diffusion_operator.cpp:461-466), interpolated by three sweeps of B.
  template <typename T, int N>
  __device__ __forceinline__ void
  field_at_points(const double *f, const GridDesc &g, int cx, int cy, int cz, const T *tB, T *vq)
  {
    constexpr int K = N - 1;
#pragma unroll
    for (int l = 0; l < N; ++l)
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 0; i < N; ++i)
          vq[(l * N + j) * N + i] =
            (T)f[(long long)(K * cx + i) + (long long)g.n[0] * ((long long)(K * cy + j) + (long long)g.n[1] * (K * cz + l))];
    sweep<T, N, 0, false>(vq, tB);
    sweep<T, N, 1, false>(vq, tB);
    sweep<T, N, 2, false>(vq, tB);
  }

  // Kernel parameters of the apply; the 1-D matrices are row-major N x N (point first).
  template <typename T, int N>
  struct AdvArgs
  {
    GridDesc      g;
    SyncDesc      s;
    const T      *src;
    T            *dst;
    const T      *b;
    int           mask_src, dif;
    const int    *skip;
    const double *vfield[3];  // velocity as a DoF vector (three FE_Q(k) components), else affine
    T             B[N * N];   // nodal values -> Gauss points
    T             Bt[3][N * N]; // tests back to the nodes per direction, weighted (rows: nodes); det in [2]
    T             mass;         // scale / dt
    // on the differences of neighbouring values (N x (N - 1)), times scale:
    T             D[3][N * (N - 1)]; // theta / h_d D
    T             L[3][N * (N - 1)]; // theta eps / h_d^2 W^-1 D^T W D
    T             E[3][N * (N - 1)]; // SUPG: theta eps / h_d^2 D D
    T             P[3][N * N];       // SUPG: W^-1 D^T W / h_d
    double        vel[12], origin[3], h[3]; // affine velocity: the cell's value in double, rounded once
    T             voff[3][3][N];   // v_d at the Gauss points minus v_d at the cell's origin, per direction
    T             supg_coef, cell_size;
  };

  // One direction of the operator, line by line on the differences of u: g = D u, S += v g + L u, and with
  // SUPG s += v g - E u.  FIRST: S and s start from mass u.  vel(q): the velocity component at point q.
  template <typename T, int N, int DIR, bool FIRST, bool SUPG, class Vel>
  __device__ __forceinline__ void
  adv_direction(const T *u, T *S, T *s, const T *D, const T *L, const T *E, T mass, bool dif, const Vel &vel)
  {
    constexpr int ST = DIR == 0 ? 1 : (DIR == 1 ? N : N * N), ND = N - 1;
#pragma unroll
    for (int a = 0; a < N; ++a)
#pragma unroll
      for (int c = 0; c < N; ++c)
        {
          const int b = DIR == 0 ? (a * N + c) * N : (DIR == 1 ? a * N * N + c : a * N + c);
          T         du[ND];
#pragma unroll
          for (int k = 0; k < ND; ++k)
            du[k] = u[b + (k + 1) * ST] - u[b + k * ST];
#pragma unroll
          for (int r = 0; r < N; ++r)
            {
              const int q = b + r * ST;
              T         g = D[r * ND] * du[0];
#pragma unroll
              for (int k = 1; k < ND; ++k)
                g = fma(D[r * ND + k], du[k], g);
              const T v = vel(q), from = FIRST ? mass * u[q] : S[q];
              S[q]      = fma(v, g, from);
              if constexpr (SUPG)
                s[q] = FIRST ? S[q] : fma(v, g, s[q]);
            }
          if (dif)
#pragma unroll
            for (int r = 0; r < N; ++r)
#pragma unroll
              for (int k = 0; k < ND; ++k)
                {
                  const int q = b + r * ST;
                  S[q]        = fma(L[r * ND + k], du[k], S[q]);
                  if constexpr (SUPG)
                    s[q] = fma(-E[r * ND + k], du[k], s[q]);
                }
        }
  }

  template <int K, typename T, bool SUPG, bool VDOF>
  struct AdvCellOp
  {
    static constexpr int  N = K + 1, N3 = N * N * N;
    static constexpr bool NODES = false;
    const AdvArgs<T, N> &a;
    struct Cell
    {
      int c[3];
    };
    __device__ __forceinline__ Cell
    load(bool, int cx, int cy, int cz) const
    {
      // a lane outside the mesh reads the field of the nearest cell
      return Cell{{min(cx, a.g.m[0] - 1), min(cy, a.g.m[1] - 1), cz}};
    }
    // component d of a DoF-vector velocity at the cell's Gauss points (read plainly, :461-466)
    __device__ __forceinline__ void
    field(int d, const Cell &c, T *v) const
    {
      const double *f = a.vfield[d] + ((long long)(K * c.c[0]) + (long long)a.g.n[0] * ((long long)(K * c.c[1]) + (long long)a.g.n[1] * (K * c.c[2])));
      const int sy = a.g.n[0], sz = a.g.n[0] * a.g.n[1];
#pragma unroll
      for (int l = 0; l < N; ++l)
#pragma unroll
        for (int j = 0; j < N; ++j)
#pragma unroll
          for (int i = 0; i < N; ++i)
            v[(l * N + j) * N + i] = (T)__ldg(f + (j * sy + l * sz + i));
      gp_interpolate<T, N, 0>(v, a.B);
      gp_interpolate<T, N, 1>(v, a.B);
      gp_interpolate<T, N, 2>(v, a.B);
    }
    __device__ __forceinline__ T
    tau_of(T speed2) const
    {
      if (a.supg_coef >= T(0))
        return a.supg_coef * a.cell_size;
      const T vmax = sqrt(speed2);
      return (vmax >= T(1e-6) ? T(1) / vmax : T(0)) * a.cell_size;
    }
    template <bool DOT>
    __device__ __forceinline__ double
    apply(T *u, const Cell &c) const
    {
      T    S[N3], s[SUPG ? N3 : 1];
      const bool dif = a.dif != 0;
      gp_interpolate<T, N, 0>(u, a.B);
      gp_interpolate<T, N, 1>(u, a.B);
      gp_interpolate<T, N, 2>(u, a.B);
      if constexpr (VDOF)
        {
          // FP32 keeps the three components for the SUPG test (81 registers); FP64 interpolates them
          // twice, with |v|^2 summed over the first pass
          constexpr bool KEEP = SUPG && sizeof(T) == 4 && K <= 2;
          T              v[KEEP ? 3 : 1][N3], n2[SUPG && !KEEP ? N3 : 1];
          auto           at = [&](int d) { return KEEP ? d : 0; };
#define MPDG_ADV_DIR(d)                                                                                         \
  {                                                                                                             \
    T *vd = v[at(d)];                                                                                          \
    field(d, c, vd);                                                                                           \
    adv_direction<T, N, d, d == 0, SUPG>(u, S, s, a.D[d], a.L[d], a.E[d], a.mass, dif, [&](int q) { return vd[q]; });  \
    if constexpr (SUPG && !KEEP)                                                                                \
      _Pragma("unroll") for (int q = 0; q < N3; ++q) n2[q] = d == 0 ? vd[q] * vd[q] : fma(vd[q], vd[q], n2[q]); \
  }
          MPDG_ADV_DIR(0)
          MPDG_ADV_DIR(1)
          MPDG_ADV_DIR(2)
#undef MPDG_ADV_DIR
          if constexpr (SUPG)
            {
              T most = T(0);
#pragma unroll
              for (int q = 0; q < N3; ++q)
                {
                  if constexpr (KEEP)
                    most = fmax(most, fma(v[2][q], v[2][q], fma(v[1][q], v[1][q], v[0][q] * v[0][q])));
                  else
                    most = fmax(most, n2[q]);
                }
              const T tau = tau_of(most);
#pragma unroll
              for (int q = 0; q < N3; ++q)
                s[q] *= tau;
#define MPDG_ADV_TEST(d)                                                                                        \
  {                                                                                                             \
    T *vd = v[at(d)];                                                                                          \
    if constexpr (!KEEP)                                                                                        \
      field(d, c, vd);                                                                                         \
    gp_divergence<T, N, d>(S, a.P[d], [&](int q) { return vd[q] * s[q]; });                                        \
  }
              MPDG_ADV_TEST(2)
              MPDG_ADV_TEST(1)
              MPDG_ADV_TEST(0)
#undef MPDG_ADV_TEST
            }
        }
      else
        {
          T v0[3];
#pragma unroll
          for (int d = 0; d < 3; ++d)
            {
              double t = a.vel[d];
#pragma unroll
              for (int e = 0; e < 3; ++e)
                t = fma(a.vel[3 + 3 * d + e], fma(a.h[e], (double)c.c[e], a.origin[e]), t);
              v0[d] = (T)t;
            }
          auto velocity = [&](int d, int q) {
            return ((v0[d] + a.voff[d][2][q / (N * N)]) + a.voff[d][1][q / N % N]) + a.voff[d][0][q % N];
          };
          adv_direction<T, N, 0, true, SUPG>(u, S, s, a.D[0], a.L[0], a.E[0], a.mass, dif, [&](int q) { return velocity(0, q); });
          adv_direction<T, N, 1, false, SUPG>(u, S, s, a.D[1], a.L[1], a.E[1], a.mass, dif, [&](int q) { return velocity(1, q); });
          adv_direction<T, N, 2, false, SUPG>(u, S, s, a.D[2], a.L[2], a.E[2], a.mass, dif, [&](int q) { return velocity(2, q); });
          if constexpr (SUPG)
            {
              T most = T(0);
              if (a.supg_coef < T(0))
#pragma unroll
                for (int q = 0; q < N3; ++q)
                  {
                    const T v1 = velocity(0, q), v2 = velocity(1, q), v3 = velocity(2, q);
                    most = fmax(most, fma(v3, v3, fma(v2, v2, v1 * v1)));
                  }
              const T tau = tau_of(most);
#pragma unroll
              for (int q = 0; q < N3; ++q)
                s[q] *= tau;
              gp_divergence<T, N, 0>(S, a.P[0], [&](int q) { return velocity(0, q) * s[q]; });
              gp_divergence<T, N, 1>(S, a.P[1], [&](int q) { return velocity(1, q) * s[q]; });
              gp_divergence<T, N, 2>(S, a.P[2], [&](int q) { return velocity(2, q) * s[q]; });
            }
        }
      gp_test<T, N, 2>(S, a.Bt[2]);
      gp_test<T, N, 1>(S, a.Bt[1]);
      gp_test<T, N, 0>(S, a.Bt[0]);
#pragma unroll
      for (int q = 0; q < N3; ++q)
        u[q] = S[q];
      return 0.0;
    }
  };

  // CTAs (of 128 threads) per SM the register allocation is held to; measured on 80^3 FE_Q(2) FP64: affine 67 us
  // at 3, 73 at 4; SUPG 138 at 2, 186 at 3; SUPG with a field 291 at 2, 345 at 3; FP32 affine 49 at 5; 128^3
  // FE_Q(1) FP64 affine 77 at 5
  template <int K, typename T, bool SUPG, bool VDOF>
  struct AdvMinBlocks
  {
    static constexpr bool f64 = sizeof(T) == 8;
    static constexpr int  value = K == 1 ? (SUPG ? (f64 ? 3 : 5) : 5) :
                                 K == 2 ? (SUPG && VDOF ? 2 : SUPG ? (f64 ? 2 : 4) : VDOF ? (f64 ? 2 : 3) : (f64 ? 3 : 5)) : 2;
  };

  template <int K, typename T, OutMode MODE, bool SUPG, bool VDOF, int BX>
  __global__ void __launch_bounds__(MARCH_NT, AdvMinBlocks<K, T, SUPG, VDOF>::value)
  adv_apply_kernel(const __grid_constant__ AdvArgs<T, K + 1> a)
  {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned                        s_ticket;
    __shared__ __align__(8) unsigned long long s_bars[2];
    if (a.skip != nullptr && *a.skip != 0)
      return;
    AdvCellOp<K, T, SUPG, VDOF> op{a};
    march_body<K, T, MODE, AdvCellOp<K, T, SUPG, VDOF>, false, true, BX>(a.g, a.s, a.src, a.dst, a.b, a.mask_src != 0, op,
                                                                     reinterpret_cast<T *>(smem_raw), &s_ticket, s_bars);
  }

  template <int K, typename T, OutMode MODE, bool SUPG, bool VDOF, int BX>
  static cudaError_t
  launch_adv_columns(AdvArgs<T, K + 1> &a, cudaStream_t stream)
  {
    auto                                   kern = adv_apply_kernel<K, T, MODE, SUPG, VDOF, BX>;
    static std::atomic<unsigned long long> devices{0};
    constexpr size_t                       bytes = MarchLayout<K, T, BX>::bytes;
    if (cudaError_t e = ensure_smem(kern, bytes, devices); e != cudaSuccess)
      return e;
    const unsigned ctas = march_grid(a.g, BX, MarchShape<K, T>::BZ, AdvMinBlocks<K, T, SUPG, VDOF>::value);
    kern<<<ctas, MARCH_NT, bytes, stream>>>(a);
    return cudaGetLastError();
  }

  template <int K, typename T, OutMode MODE, bool SUPG, bool VDOF>
  static cudaError_t
  launch_adv_kernel(AdvArgs<T, K + 1> &a, cudaStream_t stream)
  {
    if constexpr (MODE != OutMode::BPlus) // b + A x is formed once a solve: one width
      if (march_bx(a.g.m) != MARCH_BX)
        return launch_adv_columns<K, T, MODE, SUPG, VDOF, MARCH_BX_NARROW>(a, stream);
    return launch_adv_columns<K, T, MODE, SUPG, VDOF, MARCH_BX>(a, stream);
  }

  template <int K, typename T, OutMode MODE>
  static cudaError_t
  launch_adv(const AdvLaunch<T> &h, cudaStream_t stream)
  {
    constexpr int   N = K + 1;
    AdvArgs<T, N>   a{};
    const Tables1D &t = tables(K);
    a.g        = h.grid;
    a.s        = h.sync;
    a.src      = h.src;
    a.dst      = h.dst;
    a.b        = h.b;
    a.mask_src = h.mask_src;
    a.skip     = h.skip;
    const double ta = h.scale * h.p.theta_adv, td = h.scale * h.p.theta_dif, ti = h.scale * h.p.inv_dt;
    const double det = h.p.h[0] * h.p.h[1] * h.p.h[2];
    a.dif            = td != 0.0;
    double dwd[N * N], dd[N * N]; // W^-1 D^T W D, D D
    for (int q = 0; q < N; ++q)
      for (int r = 0; r < N; ++r)
        {
          a.B[q * N + r]  = (T)t.B[q * N + r];
          dwd[q * N + r] = dd[q * N + r] = 0.0;
          for (int k = 0; k < N; ++k)
            {
              dwd[q * N + r] += t.Dq[k * N + q] * t.qw[k] * t.Dq[k * N + r] / t.qw[q];
              dd[q * N + r] += t.Dq[q * N + k] * t.Dq[k * N + r];
            }
          for (int d = 0; d < 3; ++d)
            {
              a.Bt[d][r * N + q] = (T)((d == 2 ? det : 1.0) * t.qw[q] * t.B[q * N + r]);
              a.P[d][q * N + r]  = (T)(t.Dq[r * N + q] * t.qw[r] / t.qw[q] / h.p.h[d]);
            }
        }
    for (int d = 0; d < 3; ++d)
      {
        const double hd = h.p.h[d];
        gp_on_differences<T, N>(t.Dq, ta / hd, a.D[d]);
        gp_on_differences<T, N>(dwd, td / (hd * hd), a.L[d]);
        gp_on_differences<T, N>(dd, td / (hd * hd), a.E[d]);
      }
    a.mass = (T)ti;
    for (int d = 0; d < 3; ++d)
      {
        a.vfield[d] = h.p.vfield[d];
        a.origin[d] = h.p.origin[d];
        a.h[d]      = h.p.h[d];
        for (int e = 0; e < 3; ++e)
          for (int q = 0; q < N; ++q)
            a.voff[d][e][q] = (T)(h.p.vel[3 + 3 * d + e] * h.p.h[e] * t.qp[q]);
      }
    for (int i = 0; i < 12; ++i)
      a.vel[i] = h.p.vel[i];
    a.supg_coef = (T)h.p.supg_coef;
    a.cell_size = (T)(std::sqrt(h.p.h[0] * h.p.h[0] + h.p.h[1] * h.p.h[1] + h.p.h[2] * h.p.h[2]) / std::sqrt(3.0));
    const bool vdof = h.p.vfield[0] != nullptr;
    if (h.p.supg)
      return vdof ? launch_adv_kernel<K, T, MODE, true, true>(a, stream) : launch_adv_kernel<K, T, MODE, true, false>(a, stream);
    return vdof ? launch_adv_kernel<K, T, MODE, false, true>(a, stream) : launch_adv_kernel<K, T, MODE, false, false>(a, stream);
  }

  template <int K, typename T>
  static cudaError_t
  adv_mode(const AdvLaunch<T> &h, cudaStream_t s)
  {
    switch (h.mode)
      {
        case 0: return launch_adv<K, T, OutMode::Set>(h, s);
        case 1: return launch_adv<K, T, OutMode::Add>(h, s);
        default: return launch_adv<K, T, OutMode::BPlus>(h, s);
      }
  }

  template <typename T>
  cudaError_t
  adv_apply(const AdvLaunch<T> &h, cudaStream_t s)
  {
    switch (h.degree)
      {
        case 1: return adv_mode<1, T>(h, s);
        case 2: return adv_mode<2, T>(h, s);
        case 3: return adv_mode<3, T>(h, s);
        default: return cudaErrorInvalidValue;
      }
  }

  template <typename T>
  void
  adv_brick_shape(int K, int shape[3])
  {
    shape[0] = MARCH_BX;
    shape[1] = MARCH_NT / MARCH_BX;
    shape[2] = K == 1 ? MarchShape<1, T>::BZ : (K == 2 ? MarchShape<2, T>::BZ : MarchShape<3, T>::BZ);
  }

  long long
  adv_flags(int K, const int m[3])
  {
    int shape[3]; // FP64: the shorter full-length segments
    adv_brick_shape<double>(K, shape);
    return std::max(march_flags(m, MARCH_BX, shape[2]), march_flags(m, march_bx(m), shape[2]));
  }

  template <int K>
  static long long
  launch_bricks(const int m[3], bool supg, bool field)
  {
    return march_bricks(m, march_bx(m), MarchShape<K, double>::BZ,
                        supg ? (field ? AdvMinBlocks<K, double, true, true>::value : AdvMinBlocks<K, double, true, false>::value) :
                               (field ? AdvMinBlocks<K, double, false, true>::value : AdvMinBlocks<K, double, false, false>::value));
  }

  long long
  adv_launch_bricks(int K, const int m[3], bool supg, bool field)
  {
    return K == 1 ? launch_bricks<1>(m, supg, field) : (K == 2 ? launch_bricks<2>(m, supg, field) : launch_bricks<3>(m, supg, field));
  }

  // ---- diagonal in closed form (MatrixFreeTools::compute_diagonal of the tangent).
  // With phi_i = phi_a(x) phi_b(y) phi_c(z) and an affine velocity, every term of
  //   A_ii = int phi_i^2 / dt + theta v . grad(phi_i) phi_i + theta eps |grad phi_i|^2
  // over a box cell is a sum of products of 1-D quadrature moments of the local indices (a, b, c):
  //   m   = h S[a],  mX = h (x0 S[a] + h S1[a])        (int phi^2,   int x phi^2)
  //   t   = T[a],    tX = x0 T[a] + h T1[a]            (int phi' phi, int x phi' phi)
  //   dd  = D[a] / h                                     (int phi'^2)
  // with S = sum w B^2, S1 = sum w q B^2, T = sum w G B, T1 = sum w q G B, D = sum w G^2 on the
  // reference Gauss rule.  One thread per DoF sums the (<= 8) cells sharing it; constrained -> 1.
  template <typename T>
  struct AdvDiagArgs
  {
    GridDesc g;
    T        S[MAX_N], S1[MAX_N], T0[MAX_N], T1[MAX_N], D[MAX_N];
    T        inv_dt, th_adv, th_dif;
    T        vel[12], origin[3], h[3];
    T       *diag;
  };

  template <int K, typename T>
  __global__ void
  adv_diag_kernel(const __grid_constant__ AdvDiagArgs<T> a)
  {
    const int       n0 = a.g.n[0], n1 = a.g.n[1];
    const long long rows = (long long)n1 * a.g.n[2];
    for (long long row = blockIdx.x; row < rows; row += gridDim.x)
      {
        const int             J = (int)(row % n1), L = (int)(row / n1);
        const Neighbours1D<K> ny(J, a.g.m[1]), nz(L, a.g.m[2]);
        for (int I = threadIdx.x; I < n0; I += blockDim.x)
          {
            const long long idx = (long long)I + (long long)n0 * row;
            if (is_constrained(a.g, I, J, L, idx))
              {
                a.diag[idx] = T(1);
                continue;
              }
            const Neighbours1D<K> nx(I, a.g.m[0]);
            const Neighbours1D<K> *nb[3] = {&nx, &ny, &nz};
            T                      d     = T(0);
#pragma unroll
            for (int z = 0; z < 2; ++z)
#pragma unroll
              for (int y = 0; y < 2; ++y)
#pragma unroll
                for (int x = 0; x < 2; ++x)
                  {
                    if (!(nx.v[x] && ny.v[y] && nz.v[z]))
                      continue;
                    const int sel[3] = {x, y, z};
                    T         m[3], mX[3], t[3], tX[3], dd[3];
#pragma unroll
                    for (int e = 0; e < 3; ++e)
                      {
                        const int li = nb[e]->l[sel[e]];
                        const T   h  = a.h[e], x0 = a.origin[e] + h * (T)nb[e]->c[sel[e]];
                        m[e]         = h * a.S[li];
                        mX[e]        = h * (x0 * a.S[li] + h * a.S1[li]);
                        t[e]         = a.T0[li];
                        tX[e]        = x0 * a.T0[li] + h * a.T1[li];
                        dd[e]        = a.D[li] / h;
                      }
                    T v = a.inv_dt * m[0] * m[1] * m[2] +
                          a.th_dif * (dd[0] * m[1] * m[2] + m[0] * dd[1] * m[2] + m[0] * m[1] * dd[2]);
                    T adv = T(0);
#pragma unroll
                    for (int dir = 0; dir < 3; ++dir)
                      {
                        const int e1 = (dir + 1) % 3, e2 = (dir + 2) % 3;
                        // int v_dir (d phi / d x_dir) phi, v_dir = vel[dir] + sum_e G[dir][e] x_e
                        T term = a.vel[dir] * t[dir] * m[e1] * m[e2];
                        term += a.vel[3 + 3 * dir + dir] * tX[dir] * m[e1] * m[e2];
                        term += a.vel[3 + 3 * dir + e1] * t[dir] * mX[e1] * m[e2];
                        term += a.vel[3 + 3 * dir + e2] * t[dir] * m[e1] * mX[e2];
                        adv += term;
                      }
                    d += v + a.th_adv * adv;
                  }
            a.diag[idx] = d;
          }
      }
  }

  template <typename T>
  cudaError_t
  adv_diagonal(const GridDesc &g, int K, const AdvParams &p, T *diag, cudaStream_t s)
  {
    if (K < 1 || K > ADV_KMAX)
      return cudaErrorInvalidValue;
    AdvDiagArgs<T>   a{};
    const Tables1D &t = tables(K);
    const int       n = t.n;
    for (int i = 0; i < n; ++i)
      {
        double S = 0, S1 = 0, T0 = 0, T1 = 0, D = 0;
        for (int q = 0; q < n; ++q)
          {
            const double w = t.qw[q], b = t.B[q * n + i], gq = t.G[q * n + i];
            S += w * b * b;
            S1 += w * t.qp[q] * b * b;
            T0 += w * gq * b;
            T1 += w * t.qp[q] * gq * b;
            D += w * gq * gq;
          }
        a.S[i] = (T)S, a.S1[i] = (T)S1, a.T0[i] = (T)T0, a.T1[i] = (T)T1, a.D[i] = (T)D;
      }
    a.g      = g;
    a.inv_dt = (T)p.inv_dt;
    a.th_adv = (T)p.theta_adv;
    a.th_dif = (T)p.theta_dif;
    for (int i = 0; i < 12; ++i)
      a.vel[i] = (T)p.vel[i];
    for (int d = 0; d < 3; ++d)
      {
        a.origin[d] = (T)p.origin[d];
        a.h[d]      = (T)p.h[d];
      }
    a.diag                  = diag;
    const long long rows    = (long long)g.n[1] * g.n[2];
    const int       blocks  = (int)std::min<long long>(rows, 148LL * 32);
    const int       threads = std::min(1024, std::max(32, (g.n[0] + 31) / 32 * 32));
    if (K == 1)
      adv_diag_kernel<1, T><<<blocks, threads, 0, s>>>(a);
    else if (K == 2)
      adv_diag_kernel<2, T><<<blocks, threads, 0, s>>>(a);
    else
      adv_diag_kernel<3, T><<<blocks, threads, 0, s>>>(a);
    return cudaGetLastError();
  }

  // ---- SUPG part of the diagonal: one thread per cell; for each free local DoF i
  //   tau_c sum_q JxW (v.grad phi_i)(phi_i / dt + theta v.grad phi_i - theta eps lap phi_i)
  // with the 1-D values B, derivatives G and second derivatives H of the basis at the Gauss points.
  template <typename T>
  struct AdvSupgDiagArgs
  {
    GridDesc g;
    T        B[MAX_N * MAX_N], G[MAX_N * MAX_N], H[MAX_N * MAX_N], qp[MAX_N], qw[MAX_N];
    T        inv_dt, th_adv, th_dif, coef, cell_size, det;
    T        vel[12], origin[3], h[3];
    const double *f[3]; // DoF-vector velocity (FIELD kernels)
    T       *diag;
  };

  // FIELD: the velocity is a DoF vector, evaluated at the cell's Gauss points from its nodal values
  template <int K, typename T, bool FIELD>
  __global__ void
  adv_supg_diag_kernel(const __grid_constant__ AdvSupgDiagArgs<T> a)
  {
    constexpr int   N     = K + 1, N3 = N * N * N;
    const int       m0    = a.g.m[0], m1 = a.g.m[1];
    const long long ncell = (long long)m0 * m1 * a.g.m[2];
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x)
      {
        const int cx = (int)(c % m0), cy = (int)((c / m0) % m1), cz = (int)(c / ((long long)m0 * m1));
        const T   x0 = a.origin[0] + a.h[0] * cx, y0 = a.origin[1] + a.h[1] * cy, z0 = a.origin[2] + a.h[2] * cz;
        T         vq[FIELD ? 3 : 1][FIELD ? N3 : 1];
        T         tau;
        if constexpr (FIELD)
          {
#pragma unroll
            for (int d = 0; d < 3; ++d)
              field_at_points<T, N>(a.f[d], a.g, cx, cy, cz, a.B, vq[d]);
            tau = a.coef;
            if (tau < T(0))
              {
                T vmax = T(0);
#pragma unroll
                for (int q = 0; q < N3; ++q)
                  vmax = fmax(vmax, sqrt(vq[0][q] * vq[0][q] + vq[1][q] * vq[1][q] + vq[2][q] * vq[2][q]));
                tau = vmax >= T(1e-6) ? T(1) / vmax : T(0);
              }
            tau *= a.cell_size;
          }
        else
          tau = supg_tau<T, N>(a.vel, a.h, a.qp, x0, y0, z0, a.coef, a.cell_size);
        if (tau == T(0))
          continue;
        const T ih[3] = {T(1) / a.h[0], T(1) / a.h[1], T(1) / a.h[2]};
        for (int l = 0; l < N; ++l)
          for (int j = 0; j < N; ++j)
            for (int i = 0; i < N; ++i)
              {
                const int       I = K * cx + i, J = K * cy + j, L = K * cz + l;
                const long long idx = (long long)I + (long long)a.g.n[0] * ((long long)J + (long long)a.g.n[1] * L);
                if (is_constrained(a.g, I, J, L, idx))
                  continue;
                T sum = T(0);
                for (int qz = 0; qz < N; ++qz)
                  for (int qy = 0; qy < N; ++qy)
#pragma unroll
                    for (int qx = 0; qx < N; ++qx)
                      {
                        const T bx = a.B[qx * N + i], by = a.B[qy * N + j], bz = a.B[qz * N + l];
                        const T gx = a.G[qx * N + i] * ih[0], gy = a.G[qy * N + j] * ih[1], gz = a.G[qz * N + l] * ih[2];
                        const T hx = a.H[qx * N + i] * ih[0] * ih[0], hy = a.H[qy * N + j] * ih[1] * ih[1],
                                hz = a.H[qz * N + l] * ih[2] * ih[2];
                        const T phi = bx * by * bz;
                        const T dp[3] = {gx * by * bz, bx * gy * bz, bx * by * gz};
                        const T lap   = hx * by * bz + bx * hy * bz + bx * by * hz;
                        const T x = x0 + a.h[0] * a.qp[qx], y = y0 + a.h[1] * a.qp[qy], z = z0 + a.h[2] * a.qp[qz];
                        T       vg = T(0);
#pragma unroll
                        for (int d = 0; d < 3; ++d)
                          {
                            T vd;
                            if constexpr (FIELD)
                              vd = vq[d][(qz * N + qy) * N + qx];
                            else
                              vd = a.vel[d] + a.vel[3 + 3 * d] * x + a.vel[4 + 3 * d] * y + a.vel[5 + 3 * d] * z;
                            vg += vd * dp[d];
                          }
                        sum += a.qw[qx] * a.qw[qy] * a.qw[qz] * vg * (a.inv_dt * phi + a.th_adv * vg - a.th_dif * lap);
                      }
                atomicAdd(a.diag + idx, tau * a.det * sum);
              }
      }
  }

  template <typename T>
  cudaError_t
  adv_supg_diagonal(const GridDesc &g, int K, const AdvParams &p, T *diag, cudaStream_t s)
  {
    if (!p.supg)
      return cudaSuccess;
    if (K < 1 || K > ADV_KMAX)
      return cudaErrorInvalidValue;
    AdvSupgDiagArgs<T> a{};
    const Tables1D    &t = tables(K);
    const int          n = t.n;
    for (int q = 0; q < n; ++q)
      {
        a.qp[q] = (T)t.qp[q];
        a.qw[q] = (T)t.qw[q];
        for (int i = 0; i < n; ++i)
          {
            double hsum = 0.0; // second derivative: collocation derivative of G on the Gauss points
            for (int r = 0; r < n; ++r)
              hsum += t.Dq[q * n + r] * t.G[r * n + i];
            a.B[q * n + i] = (T)t.B[q * n + i];
            a.G[q * n + i] = (T)t.G[q * n + i];
            a.H[q * n + i] = (T)hsum;
          }
      }
    a.g         = g;
    a.inv_dt    = (T)p.inv_dt;
    a.th_adv    = (T)p.theta_adv;
    a.th_dif    = (T)p.theta_dif;
    a.coef      = (T)p.supg_coef;
    a.cell_size = (T)(std::sqrt(p.h[0] * p.h[0] + p.h[1] * p.h[1] + p.h[2] * p.h[2]) / std::sqrt(3.0));
    a.det       = (T)(p.h[0] * p.h[1] * p.h[2]);
    for (int i = 0; i < 12; ++i)
      a.vel[i] = (T)p.vel[i];
    for (int d = 0; d < 3; ++d)
      {
        a.origin[d] = (T)p.origin[d];
        a.h[d]      = (T)p.h[d];
      }
    a.diag                 = diag;
    for (int d = 0; d < 3; ++d)
      a.f[d] = p.vfield[d];
    const bool      field  = p.vfield[0] != nullptr;
    const long long ncell  = (long long)g.m[0] * g.m[1] * g.m[2];
    const int       blocks = (int)std::max<long long>(1, std::min<long long>((ncell + 127) / 128, 148LL * 16));
    if (K == 1)
      (field ? adv_supg_diag_kernel<1, T, true> : adv_supg_diag_kernel<1, T, false>)<<<blocks, 128, 0, s>>>(a);
    else if (K == 2)
      (field ? adv_supg_diag_kernel<2, T, true> : adv_supg_diag_kernel<2, T, false>)<<<blocks, 128, 0, s>>>(a);
    else
      (field ? adv_supg_diag_kernel<3, T, true> : adv_supg_diag_kernel<3, T, false>)<<<blocks, 128, 0, s>>>(a);
    return cudaGetLastError();
  }

  // ---- diagonal with a DoF-vector velocity: one thread per cell; the velocity at the Gauss points
  // from the cell's nodal values, then for each free local DoF i
  //   sum_q JxW (phi_i^2 / dt + theta_adv (v.grad phi_i) phi_i + theta_dif |grad phi_i|^2)
  // (MatrixFreeTools::compute_diagonal of the tangent, advection_diffusion_operator.cpp:399-446)
  struct AdvFieldDiagArgs
  {
    GridDesc      g;
    double        B[MAX_N * MAX_N], G[MAX_N * MAX_N], qw[MAX_N];
    double        inv_dt, th_adv, th_dif, det, h[3];
    const double *f[3];
    double       *diag;
  };

  template <int K>
  __global__ void
  adv_field_diag_kernel(const __grid_constant__ AdvFieldDiagArgs a)
  {
    constexpr int   N = K + 1, N3 = N * N * N;
    const int       m0 = a.g.m[0], m1 = a.g.m[1];
    const long long ncell = (long long)m0 * m1 * a.g.m[2];
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < ncell; c += (long long)gridDim.x * blockDim.x)
      {
        const int cx = (int)(c % m0), cy = (int)((c / m0) % m1), cz = (int)(c / ((long long)m0 * m1));
        double    vq[3][N3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
          field_at_points<double, N>(a.f[d], a.g, cx, cy, cz, a.B, vq[d]);
        const double ih[3] = {1.0 / a.h[0], 1.0 / a.h[1], 1.0 / a.h[2]};
        for (int l = 0; l < N; ++l)
          for (int j = 0; j < N; ++j)
            for (int i = 0; i < N; ++i)
              {
                const int       I = K * cx + i, J = K * cy + j, L = K * cz + l;
                const long long idx = (long long)I + (long long)a.g.n[0] * ((long long)J + (long long)a.g.n[1] * L);
                if (is_constrained(a.g, I, J, L, idx))
                  continue;
                double sum = 0.0;
                for (int qz = 0; qz < N; ++qz)
                  for (int qy = 0; qy < N; ++qy)
#pragma unroll
                    for (int qx = 0; qx < N; ++qx)
                      {
                        const int    q  = (qz * N + qy) * N + qx;
                        const double bx = a.B[qx * N + i], by = a.B[qy * N + j], bz = a.B[qz * N + l];
                        const double dp[3] = {a.G[qx * N + i] * ih[0] * by * bz, bx * a.G[qy * N + j] * ih[1] * bz,
                                              bx * by * a.G[qz * N + l] * ih[2]};
                        const double phi = bx * by * bz;
                        const double vg  = vq[0][q] * dp[0] + vq[1][q] * dp[1] + vq[2][q] * dp[2];
                        const double pp  = dp[0] * dp[0] + dp[1] * dp[1] + dp[2] * dp[2];
                        sum += a.qw[qx] * a.qw[qy] * a.qw[qz] * (a.inv_dt * phi * phi + a.th_adv * vg * phi + a.th_dif * pp);
                      }
                atomicAdd(a.diag + idx, a.det * sum);
              }
      }
  }

  cudaError_t
  adv_field_diagonal(const GridDesc &g, int K, const AdvParams &p, double *diag, cudaStream_t s)
  {
    if (K < 1 || K > ADV_KMAX || !p.vfield[0] || !p.vfield[1] || !p.vfield[2])
      return cudaErrorInvalidValue;
    AdvFieldDiagArgs a{};
    const Tables1D  &t = tables(K);
    const int        n = t.n;
    for (int q = 0; q < n; ++q)
      {
        a.qw[q] = t.qw[q];
        for (int i = 0; i < n; ++i)
          {
            a.B[q * n + i] = t.B[q * n + i];
            a.G[q * n + i] = t.G[q * n + i];
          }
      }
    a.g      = g;
    a.inv_dt = p.inv_dt;
    a.th_adv = p.theta_adv;
    a.th_dif = p.theta_dif;
    a.det    = p.h[0] * p.h[1] * p.h[2];
    for (int d = 0; d < 3; ++d)
      {
        a.h[d] = p.h[d];
        a.f[d] = p.vfield[d];
      }
    a.diag                 = diag;
    const long long ncell  = (long long)g.m[0] * g.m[1] * g.m[2];
    const int       blocks = (int)std::max<long long>(1, std::min<long long>((ncell + 127) / 128, 148LL * 16));
    if (K == 1)
      adv_field_diag_kernel<1><<<blocks, 128, 0, s>>>(a);
    else if (K == 2)
      adv_field_diag_kernel<2><<<blocks, 128, 0, s>>>(a);
    else
      adv_field_diag_kernel<3><<<blocks, 128, 0, s>>>(a);
    return cudaGetLastError();
  }

  template cudaError_t adv_supg_diagonal<double>(const GridDesc &, int, const AdvParams &, double *, cudaStream_t);
  template cudaError_t adv_supg_diagonal<float>(const GridDesc &, int, const AdvParams &, float *, cudaStream_t);
  template cudaError_t adv_apply<double>(const AdvLaunch<double> &, cudaStream_t);
  template cudaError_t adv_apply<float>(const AdvLaunch<float> &, cudaStream_t);
  template cudaError_t adv_diagonal<double>(const GridDesc &, int, const AdvParams &, double *, cudaStream_t);
  template cudaError_t adv_diagonal<float>(const GridDesc &, int, const AdvParams &, float *, cudaStream_t);
  template void adv_brick_shape<double>(int, int[3]);
  template void adv_brick_shape<float>(int, int[3]);
} // namespace mpdg
