// Column-marching apply for low degrees: one thread per cell, no shared-memory reduction.
//
// A CTA of 4 warps owns a column of 32 x 4 cells (x, y; march_bx: or 16 x 8) and marches through a segment of
// bz cell layers in z, a cell per thread in rows along x.  Per layer:
//   1. the K new lattice planes of the layer arrive in a ring of 2 K + 1 planes by bulk copies
//      (cp.async.bulk, one per lattice row, issued by the lanes of warp 0 two layers ahead); the plane
//      shared with the layer below stays in the ring;
//   2. each thread applies the cell operator to its cell's (K+1)^3 values in registers;
//   3. x-neighbours combine their common face with warp shuffles (a cell adds its lower neighbour's x = K
//      face into its x = 0 face), y-neighbours through a small shared exchange buffer (two buffers taken in
//      turn: one barrier per layer), z-neighbours by carrying the z = K face in registers;
//   4. each thread then owns the points i, j, l in [0, K) of its cell and writes them with coalesced
//      stores; points on the faces shared with neighbouring columns / segments are combined with global
//      atomics, initialised by their owner through the ticket / flag handshake of brick.cuh.  The
//      column's high x face and high y face add straight from the values of the cells there,
//      so neither the exchange nor the carry handles them.
//
// Staging.  A lattice row of n points starts at any element, a bulk copy at a 16-byte boundary: the copy
// starts at the boundary below the row's first point, and the row sits in its slot shifted by the
// elements in between, (address / sizeof(T)) mod (16 / sizeof(T)), which every reader computes from the
// row's index.  Granules that would reach outside the vector (its first and last row only) are fetched
// point by point.  Against per-element copies (cp.async of all K + 1 planes by every thread, with the
// row and bounds arithmetic of each point) this took the FE_Q(2) FP64 apply from 1439 to about 1100 warp
// instructions per 32 cells (96^3: 93.7 -> 60.2 us, FP32 128^3: 141 -> 96 us); the kernel is bound by
// instruction issue and latency, not by bandwidth.
//
// Segment length.  bz is chosen per mesh by march_plan (below).
#pragma once

#include <type_traits>

#include "brick.cuh"

namespace mpdg
{
  constexpr int MARCH_BX = 32, MARCH_BX_NARROW = 16, MARCH_NT = 128;
  // segments of any mesh: at most the full-length ones or this many (brick flags, dot partials)
  constexpr long long MARCH_MIN_FLAGS = 8192;

  // Cell layers of a full-length segment (the handle's brick count, and the bound of the flags on
  // large meshes).
  template <int K, typename T>
  struct MarchShape
  {
    static constexpr int BZ = K == 1 ? 16 : (sizeof(T) == 4 ? 16 : 8);
  };

  inline long long
  march_columns(const int m[3], int bx)
  {
    const int by = MARCH_NT / bx;
    return (long long)((m[0] + bx - 1) / bx) * ((m[1] + by - 1) / by);
  }

  // Column width of the operators with coefficients inside the cells (the heat apply always takes 32 x 4): 16 x 8
  // cells where they leave at most 4/5 of the threads that 32 x 4 cells take and the mesh fills the chip (two CTAs
  // per SM in segments of one layer).  A row of lanes outside the mesh costs as much as one inside: FE_Q(3) FP64
  // 48^3 (3/4) temperature-dependent tangent 360 -> 303 us, advection 70 -> 56, reinitialisation 315 -> 262;
  // FE_Q(1) 8x40x160 (1/2) advection 14.5 -> 11.3, tangent 28.9 -> 21.2.  At 5/6 the wider column still wins on
  // small meshes (FE_Q(2) 33x33x40 reinitialisation 43 against 48 us), at equal counts by up to 5 % (FE_Q(1)
  // 192x160x72 advection 71.6 against 74.1), and where a launch takes one CTA's time by its shorter chain, half as many
  // rows to stage (FE_Q(2) 12^3, 2/3: reinitialisation 16.5 against 17.5, banded FP32 10.4 against 12.3).
  inline int
  march_bx(const int m[3])
  {
    const long long wide = march_columns(m, MARCH_BX);
    return 5 * march_columns(m, MARCH_BX_NARROW) <= 4 * wide && wide * m[2] >= 2 * 148 ? MARCH_BX_NARROW : MARCH_BX;
  }

  // Segment length for a mesh: the bz whose CTAs take the least time on the resident slots.  In units of
  // a layer at full occupancy a CTA costs its layers plus about one (two, where it starts on an idle
  // slot: handshake and the first planes' latency); the last wave, of which only a part of the slots is
  // in use, takes 0.57 + 0.43 part of that per layer (fitted to the FE_Q(2) FP64 heat apply at five CTAs per
  // SM: 5.6 us a layer at 4.9 CTAs per SM, 4.5 at 2.9, 3.9 at 1.5).  What it picks, and its neighbours, heat
  // apply: FE_Q(2) FP64 (592 slots) 96^3 58.0 us at bz = 12 (one wave of 576), 68 at 8, 64 at 16, 80 at 24;
  // 64^3 24.7 at 4, 27.7 at 2, 31.0 at 8; 32^3 10.6 at 1, 16.8 at 4; FP32 128^3 91.7 at 16, 93.7 at 8, 103 at
  // 12; FE_Q(1) FP64 192^3 143 us, 149 to 153 at 8 to 24.  The other operators take the same rule.
  inline int
  march_plan(const int m[3], int bx, int bz_full, int slots, int *nseg)
  {
    const long long cols = march_columns(m, bx);
    const long long cap  = cols * ((m[2] + bz_full - 1) / bz_full);
    double          best = 0.0;
    int             bz   = bz_full;
    for (int b = 1; b <= 32 && (b <= m[2] || b == 1); ++b)
      {
        const long long nb = cols * ((m[2] + b - 1) / b);
        if (nb > cap && nb > MARCH_MIN_FLAGS)
          continue;
        const long long full = nb / slots;
        const double    part = (double)(nb % slots) / slots;
        const double    cost = (b + 1.0) * (double)full + (part > 0.0 ? (b + 2.0) * (0.57 + 0.43 * part) : 0.0);
        if (best == 0.0 || cost < best)
          {
            best = cost;
            bz   = b;
          }
      }
    *nseg = (m[2] + bz - 1) / bz;
    return bz;
  }

  // The column counts and the segment length of a launch on 148 SMs with per_sm resident CTAs; returns
  // the number of CTAs.
  inline unsigned
  march_grid(GridDesc &g, int bx, int bz_full, int per_sm)
  {
    g.nbr[0] = (g.m[0] + bx - 1) / bx;
    g.nbr[1] = (g.m[1] + MARCH_NT / bx - 1) / (MARCH_NT / bx);
    g.bz     = march_plan(g.m, bx, bz_full, 148 * per_sm, &g.nbr[2]);
    return (unsigned)g.nbr[0] * g.nbr[1] * g.nbr[2];
  }

  // CTAs that a launch has at least, in columns of width bx or (its b + A x form) MARCH_BX
  inline long long
  march_bricks(const int m[3], int bx, int bz_full, int per_sm)
  {
    GridDesc g{};
    for (int d = 0; d < 3; ++d)
      g.m[d] = m[d];
    const unsigned n = march_grid(g, bx, bz_full, per_sm), wide = march_grid(g, MARCH_BX, bz_full, per_sm);
    return n < wide ? n : wide;
  }

  // flags / dot partials an operator must hold for the segments of any of its marching applies
  inline long long
  march_flags(const int m[3], int bx, int bz_full)
  {
    const long long cap = march_columns(m, bx) * ((m[2] + bz_full - 1) / bz_full);
    return cap > MARCH_MIN_FLAGS ? cap : MARCH_MIN_FLAGS;
  }

  template <int K, typename T, int BX = MARCH_BX>
  struct MarchLayout
  {
    static constexpr int N = K + 1, G = 16 / (int)sizeof(T), BY = MARCH_NT / BX;
    static constexpr int PX = K * BX + 1, PY = K * BY + 1, NRING = 2 * K + 1;
    static constexpr int PITCH = (PX + G - 1 + G - 1) / G * G; // row of a slot: shift + points
    static constexpr int PLANE = PY * PITCH;
    static constexpr int YX    = N * K * MARCH_NT;             // y-exchange, one buffer
    static constexpr size_t bytes = sizeof(T) * (NRING * (size_t)PLANE + 2 * (size_t)YX);
  };

  // Geometry of one column segment (K points per cell; bz layers)
  template <int K, int BX>
  struct Column
  {
    int      c0[3], g0[3], nv[3];
    int      lo_sh[3], hi_sh[3], con_lo[3], con_hi[3], any_con;
    int      sy, sz, layers;
    unsigned id;
    __device__ __forceinline__ void
    set(const GridDesc &g, unsigned t)
    {
      id           = t;
      const int B[3] = {BX, MARCH_NT / BX, g.bz};
      c0[0]        = (int)(t % (unsigned)g.nbr[0]) * B[0];
      c0[1]        = (int)((t / (unsigned)g.nbr[0]) % (unsigned)g.nbr[1]) * B[1];
      c0[2]        = (int)(t / (unsigned)(g.nbr[0] * g.nbr[1])) * g.bz;
      any_con      = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d)
        {
          g0[d]     = K * c0[d];
          nv[d]     = min(K * B[d] + 1, g.n[d] - g0[d]);
          lo_sh[d]  = c0[d] > 0;
          hi_sh[d]  = c0[d] + B[d] < g.m[d];
          con_lo[d] = ((g.faces >> (2 * d)) & 1u) && g0[d] == 0;
          con_hi[d] = ((g.faces >> (2 * d + 1)) & 1u) && g0[d] + nv[d] == g.n[d];
          any_con |= con_lo[d] | con_hi[d];
        }
      sy     = g.n[0];
      sz     = g.n[0] * g.n[1];
      layers = min(g.bz, g.m[2] - c0[2]);
    }
    __device__ __forceinline__ int
    index(int px, int py, int pz) const
    {
      return (g0[0] + px) + sy * (g0[1] + py) + sz * (g0[2] + pz);
    }
    __device__ __forceinline__ bool
    has_lower_neighbour() const
    {
      return lo_sh[0] || lo_sh[1] || lo_sh[2];
    }
  };

  // Initialise the face points the segment owns (Set: 0, BPlus: b) and publish the flag: its high faces
  // and, at the domain's low boundary, its low faces (edge points are visited up to three times with the
  // same value).  acc_lo_z: the lattice's low z plane holds the previous slab's values and stays.
  template <int K, typename T, OutMode MODE, int BX>
  __device__ __forceinline__ void
  column_init_publish(const Column<K, BX> &br, const SyncDesc &s, T *dst, const T *bvec, unsigned acc_lo_z)
  {
    static_assert(MODE != OutMode::Add, "Add mode needs no initialisation");
    auto put = [&](int px, int py, int pz) {
      if ((px == 0 && br.lo_sh[0]) || (py == 0 && br.lo_sh[1]) || (pz == 0 && br.lo_sh[2]))
        return;
      if (acc_lo_z && pz == 0 && br.g0[2] == 0)
        return;
      const int idx = br.index(px, py, pz);
      dst[idx]      = (MODE == OutMode::BPlus) ? bvec[idx] : T(0);
    };
    constexpr int PX = K * BX + 1, PY = K * (MARCH_NT / BX) + 1;
    const int     lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int side = br.lo_sh[0] ? 1 : 0; side < 2; ++side)
      for (int pz = warp; pz < br.nv[2]; pz += MARCH_NT / 32)
#pragma unroll
        for (int c = 0; c < (PY + 31) / 32; ++c)
          if (lane + 32 * c < br.nv[1])
            put(side ? br.nv[0] - 1 : 0, lane + 32 * c, pz);
    for (int side = br.lo_sh[1] ? 1 : 0; side < 2; ++side)
      for (int pz = warp; pz < br.nv[2]; pz += MARCH_NT / 32)
#pragma unroll
        for (int c = 0; c < (PX + 31) / 32; ++c)
          if (lane + 32 * c < br.nv[0])
            put(lane + 32 * c, side ? br.nv[1] - 1 : 0, pz);
    for (int side = br.lo_sh[2] ? 1 : 0; side < 2; ++side)
      for (int py = warp; py < br.nv[1]; py += MARCH_NT / 32)
#pragma unroll
        for (int c = 0; c < (PX + 31) / 32; ++c)
          if (lane + 32 * c < br.nv[0])
            put(lane + 32 * c, py, side ? br.nv[2] - 1 : 0);
    __syncthreads();
    if (threadIdx.x == 0)
      {
        __threadfence();
        st_release(s.flags + br.id, s.epoch);
      }
  }

  // Bounded wait of threads 0..6 for the flags of the lower neighbour segments; the caller's next
  // barrier orders the other threads.
  template <int K, int BX>
  __device__ __forceinline__ void
  column_wait_lower(const Column<K, BX> &br, const GridDesc &g, const SyncDesc &s)
  {
    if (threadIdx.x < 7)
      {
        const unsigned t  = threadIdx.x + 1; // offsets (ox,oy,oz) in {0,1}^3 minus (0,0,0)
        const int      ox = (t & 1u) ? 1 : 0, oy = (t & 2u) ? 1 : 0, oz = (t & 4u) ? 1 : 0;
        if ((!ox || br.lo_sh[0]) && (!oy || br.lo_sh[1]) && (!oz || br.lo_sh[2]))
          {
            const unsigned nb = br.id - (unsigned)ox - (unsigned)g.nbr[0] * ((unsigned)oy + (unsigned)g.nbr[1] * (unsigned)oz);
            unsigned       it = 0;
            while (ld_acquire(s.flags + nb) != s.epoch)
              {
                if (++it > s.spin_limit)
                  {
                    atomicExch(s.error, ERR_FLAG_WAIT);
                    break;
                  }
                __nanosleep(32);
              }
          }
      }
  }

  // ---- bulk copies of lattice rows (sm_90+ PTX)
  __device__ __forceinline__ void
  march_bar_init(unsigned long long *bar, unsigned count)
  {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)), "r"(count)
                 : "memory");
  }
  __device__ __forceinline__ void
  march_bar_expect(unsigned long long *bar, unsigned bytes)
  {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)),
                 "r"(bytes)
                 : "memory");
  }
  // bounded wait for the phase with the given parity (about 2^20 tries, each of which may suspend)
  __device__ __forceinline__ bool
  march_bar_wait(unsigned long long *bar, unsigned parity)
  {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    for (unsigned it = 0; it < (1u << 20); ++it)
      {
        unsigned ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(a), "r"(parity)
                     : "memory");
        if (ok)
          return true;
      }
    return false;
  }

  // One lattice row: points [idx, idx + n) of src (n_src points in all) into the slot row, shifted by the
  // row's misalignment; the caller has computed base = src's own misalignment in elements.  Returns the
  // bytes copied in bulk.  issue = false only returns them.
  template <typename T>
  __device__ __forceinline__ unsigned
  march_row(const T *src, int n_src, int base, int idx, int n, T *slot, unsigned long long *bar, bool issue)
  {
    constexpr int G  = 16 / (int)sizeof(T);
    const int     sh = (base + idx) & (G - 1), first = idx - sh, len = (sh + n + G - 1) / G * G;
    const int     beg = first < 0 ? G : 0, end = (long long)first + len > n_src ? len - G : len;
    const unsigned bytes = end > beg ? (unsigned)((end - beg) * (int)sizeof(T)) : 0u;
    if (issue)
      {
        if (bytes)
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         (unsigned)__cvta_generic_to_shared(slot + beg)),
                       "l"(src + (first + beg)), "r"(bytes), "r"((unsigned)__cvta_generic_to_shared(bar))
                       : "memory");
      }
    else
      {
        // granules that reach outside the vector, point by point
        if (beg)
          for (int i = sh; i < min(G, sh + n); ++i)
            slot[i] = src[first + i];
        if (end < len && !(beg && len == G))
          for (int i = max(end, sh); i < sh + n; ++i)
            slot[i] = src[first + i];
      }
    return bytes;
  }

  // Warp 0: the planes [p0, p1) of the segment into their ring slots (slot = plane mod NRING); every
  // lane arrives on the barrier once (count 32), with the bytes of its rows.
  template <int K, typename T, int BX>
  __device__ __forceinline__ void
  march_stage(const Column<K, BX> &br, const T *src, int n_src, int base, int p0, int p1, T *ring, unsigned long long *bar)
  {
    using LAY = MarchLayout<K, T, BX>;
    const int lane = threadIdx.x;
    const int rows = (p1 - p0) * LAY::PY;
    auto      row  = [&](int r, bool issue) -> unsigned {
      const int py = r % LAY::PY, pz = p0 + r / LAY::PY;
      if (py >= br.nv[1] || pz >= br.nv[2])
        return 0u;
      return march_row<T>(src, n_src, base, br.index(0, py, pz), br.nv[0],
                          ring + (pz % LAY::NRING) * LAY::PLANE + py * LAY::PITCH, bar, issue);
    };
    unsigned bytes = 0;
    for (int r = lane; r < rows; r += 32)
      bytes += row(r, false);
    // the slots were read by every thread before the CTA's last barrier; order those reads before the
    // copies of the asynchronous proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    march_bar_expect(bar, bytes);
    for (int r = lane; r < rows; r += 32)
      row(r, true);
  }

  // The cell's nodal values in the ring, for operators that read them several times instead of holding them:
  // row (l, j) of the cell, N values.  Constrained values are zeroed in the ring before.
  template <int K, typename T>
  struct MarchNodes
  {
    const T *row[(K + 1) * (K + 1)];
  };

  // Results of a cell operator: 1, or Op::OUT of them
  template <class Op, class = void>
  struct MarchOutputs
  {
    static constexpr int value = 1;
    struct State
    {};
  };
  template <class Op>
  struct MarchOutputs<Op, std::void_t<decltype(Op::OUT)>>
  {
    static constexpr int value = Op::OUT;
    using State                = typename Op::State;
  };
  template <int M, int OUT, class Op, typename T, class Nodes, class State, class Finish>
  __device__ __forceinline__ void
  march_components(const Op &op, T *u, const Nodes &nodes, State &state, const Finish &finish)
  {
    if constexpr (M < OUT)
      {
        op.template component<M>(u, nodes, state);
        finish(M, op.out(M));
        march_components<M + 1, OUT>(op, u, nodes, state, finish);
      }
  }

  // The marching body.  Cell operator: op.apply<DOT>(u, op.load(valid, cx, cy, cz)) in place on (K+1)^3 values.
  // With DOT the cell operator returns the cell's form src_c^T A src_c and the sum over the segment goes
  // to the fused dot product (release_ticket_dot).
  // An operator with Op::NODES instead has op.apply(u, nodes, op.load(...)): it reads its input through
  // MarchNodes and only writes u.
  // An operator with Op::OUT results (NODES) has op.prepare(nodes, pre, state), op.component<m>(u, nodes, state)
  // and the output vectors op.out(m) instead: result after result of a layer is exchanged and written.
  // MASKABLE: the operator may carry per-DoF constraint flags (GridDesc::cmask) besides the faces.
  template <int K, typename T, OutMode MODE, class Op, bool DOT = false, bool MASKABLE = false, int BX = MARCH_BX>
  __device__ __forceinline__ void
  march_body(const GridDesc &g, const SyncDesc &s, const T *src, T *dst, const T *bvec, bool mask_src, const Op &op,
             T *smem, unsigned *s_ticket, unsigned long long *bars, const DotSink &dot = DotSink{},
             double *s_red = nullptr)
  {
    double dsum = 0.0;
    using LAY   = MarchLayout<K, T, BX>;
    constexpr int N = K + 1, G = LAY::G, PITCH = LAY::PITCH, NRING = LAY::NRING;
    T *ring = smem, *yx0 = smem + NRING * LAY::PLANE;
    const int     lx = threadIdx.x % BX, row = threadIdx.x / BX; // the thread's cell in the column
    Column<K, BX> br;
    if (threadIdx.x == 0)
      {
        march_bar_init(&bars[0], 32);
        march_bar_init(&bars[1], 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      }
    if constexpr (MODE != OutMode::Add)
      {
        const unsigned t = take_ticket(s, s_ticket);
        if (t >= (unsigned)(g.nbr[0] * g.nbr[1] * g.nbr[2]))
          {
            // stale counter: never index past the flag array; report and keep the count
            if (threadIdx.x == 0)
              atomicExch(s.error, ERR_TICKET);
            release_ticket(s);
            return;
          }
        br.set(g, t);
      }
    else
      {
        br.set(g, blockIdx.x);
        __syncthreads(); // barriers initialised
      }
    const int n_src = g.n[0] * g.n[1] * g.n[2];
    const int base  = (int)((reinterpret_cast<unsigned long long>(src) / sizeof(T)) & (G - 1));
    const int nlayers = br.layers;
    if (row < 32 / BX) // warp 0
      {
        march_stage<K, T, BX>(br, src, n_src, base, 0, K + 1, ring, &bars[0]);
        if (nlayers > 1)
          march_stage<K, T, BX>(br, src, n_src, base, K + 1, 2 * K + 1, ring, &bars[1]);
      }
    if constexpr (MODE != OutMode::Add)
      column_init_publish<K, T, MODE, BX>(br, s, dst, bvec, g.acc_lo_z);
    const int  cx = br.c0[0] + lx, cy = br.c0[1] + row;
    const bool vxy       = cx < g.m[0] && cy < g.m[1];
    const bool x_last = cx == min(br.c0[0] + BX, g.m[0]) - 1;
    const bool y_last = cy == min(br.c0[1] + LAY::BY, g.m[1]) - 1;
    const bool do_mask   = mask_src && br.any_con; // only segments on a constrained face pay for masking
    // Dirichlet planes through the cell
    const bool cI0 = br.con_lo[0] && cx == 0, cIK = br.con_hi[0] && cx == g.m[0] - 1;
    const bool cJ0 = br.con_lo[1] && cy == 0, cJK = br.con_hi[1] && cy == g.m[1] - 1;
    constexpr int OUT = MarchOutputs<Op>::value;
    T             carry[OUT][K * K];
#pragma unroll
    for (int m = 0; m < OUT; ++m)
#pragma unroll
      for (int q = 0; q < K * K; ++q)
        carry[m][q] = T(0);
    const int wbase  = br.index(0, K * row, 0); // first point of the cell row
    int       slot0  = 0;                          // ring slot of the layer's low plane
    for (int lz = 0; lz < nlayers; ++lz)
      {
        // lanes outside the mesh compute on whatever the slot holds: their values only reach lanes and
        // warps outside the mesh, too
        const int  cz  = br.c0[2] + lz;
        const auto pre = op.load(vxy, cx, cy, cz); // per-cell coefficients, in flight during the wait
        if (!march_bar_wait(&bars[lz & 1], (unsigned)(lz >> 1) & 1u) && lx == 0)
          atomicExch(s.error, ERR_FLAG_WAIT);
        const bool last_layer = lz == nlayers - 1;
        const bool cL0 = br.con_lo[2] && cz == 0, cLK = br.con_hi[2] && cz == g.m[2] - 1;
        T                u[N * N * N];
        MarchNodes<K, T> nodes;
        typename MarchOutputs<Op>::State state;
#pragma unroll
        for (int l = 0; l < N; ++l)
          {
            int sl = slot0 + l;
            if (sl >= NRING)
              sl -= NRING;
            const T  *pl = ring + sl * LAY::PLANE + (K * row) * PITCH + K * lx;
            const int e  = base + wbase + br.sz * (K * lz + l);
#pragma unroll
            for (int j = 0; j < N; ++j)
              nodes.row[l * N + j] = pl + j * PITCH + ((e + j * br.sy) & (G - 1));
          }
        slot0 += K;
        if (slot0 >= NRING)
          slot0 -= NRING;
        // exchange of result m (u) with the neighbouring cells and write-out to out
        auto finish = [&](const int m, T *out) {
          // x: a cell adds its lower neighbour's x = K face
#pragma unroll
          for (int q = 0; q < N * N; ++q)
            {
              const T v = __shfl_up_sync(0xffffffffu, u[q * N + K], 1);
              if (lx > 0)
                u[q * N] += v;
            }
          // y: a cell row hands its y = K face to the next (the last adds its own to dst below)
          T *yx = yx0 + ((OUT * lz + m) & 1) * LAY::YX;
#pragma unroll
          for (int l = 0; l < N; ++l)
#pragma unroll
            for (int i = 0; i < K; ++i)
              yx[((row * N + l) * K + i) * BX + lx] = u[(l * N + K) * N + i];
          if constexpr (MODE != OutMode::Add)
            if (lz == 0 && m == 0 && br.has_lower_neighbour())
              column_wait_lower<K, BX>(br, g, s);
          __syncthreads();
          // every thread has read the layer's planes: those that the layer after next needs not are free
          if (m == OUT - 1 && row < 32 / BX && lz + 2 < nlayers)
            march_stage<K, T, BX>(br, src, n_src, base, K * (lz + 2) + 1, K * (lz + 3) + 1, ring, &bars[lz & 1]);
          if (row > 0)
#pragma unroll
            for (int l = 0; l < N; ++l)
#pragma unroll
              for (int i = 0; i < K; ++i)
                u[(l * N) * N + i] += yx[(((row - 1) * N + l) * K + i) * BX + lx];
          // z: add the carried face, carry this layer's z = K face
#pragma unroll
          for (int j = 0; j < K; ++j)
#pragma unroll
            for (int i = 0; i < K; ++i)
              {
                u[j * N + i] += carry[m][j * K + i];
                carry[m][j * K + i] = u[(K * N + j) * N + i];
              }
          // ---- write-out.  Every face point of the segment was initialised by its owner
          // (column_init_publish), so a face point is an atomic add (skipped on constrained rows) and an
          // interior point a plain store; interior points are never constrained (Dirichlet planes are
          // domain faces).
          auto write_out = [&](auto flagged) {
              constexpr bool CM    = decltype(flagged)::value;
              const int      cbase = wbase + K * lx + br.sz * (K * lz);
              T             *d0    = out + cbase;
              const bool     x_low = lx == 0;
              auto store = [&](int i, int j, int l) {
                const int off = j * br.sy + l * br.sz + i;
                const T   v   = u[(l * N + j) * N + i];
                bool con = false;
                if constexpr (CM)
                  con = g.cmask[cbase + off] != 0;
                if constexpr (MODE == OutMode::Set)
                  d0[off] = con ? T(0) : v;
                else if constexpr (MODE == OutMode::Add)
                  {
                    // a reduction without a return value: nothing waits for the old value
                    if (!con)
                      atomicAdd(d0 + off, v);
                  }
                else
                  d0[off] = con ? bvec[cbase + off] : bvec[cbase + off] + v;
              };
              auto add = [&](int i, int j, int l) {
                const int off = j * br.sy + l * br.sz + i;
                if constexpr (CM)
                  if (g.cmask[cbase + off])
                    return;
                atomicAdd(d0 + off, u[(l * N + j) * N + i]);
              };
#pragma unroll
              for (int l = 0; l < K; ++l)
#pragma unroll
                for (int j = 0; j < K; ++j)
                  {
                    if ((j == 0 && row == 0) || (l == 0 && lz == 0))
                      {
                        if (!((j == 0 && cJ0) || (l == 0 && cL0)))
#pragma unroll
                          for (int i = 0; i < K; ++i)
                            if (!(i == 0 && cI0))
                              add(i, j, l);
                      }
                    else
                      {
                        if (!x_low)
                          store(0, j, l);
#pragma unroll
                        for (int i = 1; i < K; ++i)
                          store(i, j, l);
                      }
                  }
              if (x_low && !cI0)
#pragma unroll
                for (int l = 0; l < K; ++l)
#pragma unroll
                  for (int j = 0; j < K; ++j)
                    if (!((j == 0 && row == 0) || (l == 0 && lz == 0)))
                      add(0, j, l);
              if (x_last && !cIK)
#pragma unroll
                for (int l = 0; l < N; ++l)
#pragma unroll
                  for (int j = 0; j < N; ++j)
                    if (!((j == 0 && cJ0) || (j == K && cJK) || (l == 0 && cL0) || (l == K && cLK)))
                      add(K, j, l);
              if (y_last && !cJK)
#pragma unroll
                for (int l = 0; l < N; ++l)
                  if (!((l == 0 && cL0) || (l == K && cLK)))
#pragma unroll
                    for (int i = 0; i < K; ++i)
                      if (!(i == 0 && cI0))
                        add(i, K, l);
              if (last_layer && !cLK)
#pragma unroll
                for (int j = 0; j < K; ++j)
                  if (!(j == 0 && cJ0))
#pragma unroll
                    for (int i = 0; i < K; ++i)
                      if (!(i == 0 && cI0))
                        add(i, j, K);
          };
          if (vxy)
            {
              if constexpr (MASKABLE)
                {
                  if (g.cmask != nullptr)
                    write_out(std::true_type());
                  else
                    write_out(std::false_type());
                }
              else
                write_out(std::false_type());
            }
        };
        if constexpr (Op::NODES)
          {
            // constrained entry (i, j, l) of the cell: Dirichlet planes, per-DoF flags
            auto constrained = [&](int i, int j, int l) {
              bool con = (l == 0 && cL0) || (l == K && cLK) || (j == 0 && cJ0) || (j == K && cJK) || (i == 0 && cI0) ||
                         (i == K && cIK);
              if constexpr (MASKABLE)
                con = con || (g.cmask != nullptr && g.cmask[wbase + K * lx + i + j * br.sy + br.sz * (K * lz + l)]);
              return con;
            };
            const bool masked = do_mask || (MASKABLE && mask_src && g.cmask != nullptr); // the same for the whole CTA
            if (masked)
              {
                // every thread zeroes its cell's constrained values (cells that share one write the same)
                if (vxy)
#pragma unroll
                  for (int l = 0; l < N; ++l)
#pragma unroll
                    for (int j = 0; j < N; ++j)
#pragma unroll
                      for (int i = 0; i < N; ++i)
                        if (constrained(i, j, l))
                          const_cast<T *>(nodes.row[l * N + j])[i] = T(0);
                __syncthreads();
              }
            if constexpr (OUT == 1)
              op.apply(u, nodes, pre);
            else
              op.prepare(nodes, pre, state);
          }
        else
          {
#pragma unroll
            for (int r = 0; r < N * N; ++r)
#pragma unroll
              for (int i = 0; i < N; ++i)
                u[r * N + i] = nodes.row[r][i];
            if (do_mask)
              {
#pragma unroll
                for (int l = 0; l < N; ++l)
#pragma unroll
                  for (int j = 0; j < N; ++j)
                    {
                      const bool cr = (l == 0 && cL0) || (l == K && cLK) || (j == 0 && cJ0) || (j == K && cJK);
#pragma unroll
                      for (int i = 0; i < N; ++i)
                        if (cr || (i == 0 && cI0) || (i == K && cIK))
                          u[(l * N + j) * N + i] = T(0);
                    }
              }
            if constexpr (MASKABLE)
              if (g.cmask != nullptr && mask_src && vxy)
                {
                  const uint8_t *cm = g.cmask + (wbase + K * lx + br.sz * (K * lz));
#pragma unroll
                  for (int l = 0; l < N; ++l)
#pragma unroll
                    for (int j = 0; j < N; ++j)
#pragma unroll
                      for (int i = 0; i < N; ++i)
                        if (cm[j * br.sy + l * br.sz + i])
                          u[(l * N + j) * N + i] = T(0);
                }
            if constexpr (DOT)
              dsum += vxy ? op.template apply<true>(u, pre) : 0.0;
            else
              op.template apply<false>(u, pre);
          }
        if constexpr (OUT == 1)
          finish(0, dst);
        else
          march_components<0, OUT>(op, u, nodes, state, finish);
      }
    if constexpr (DOT)
      release_ticket_dot<MARCH_NT>(s, dot, br.id, dsum, s_red, s_ticket);
    else if constexpr (MODE != OutMode::Add)
      release_ticket(s);
  }
} // namespace mpdg
