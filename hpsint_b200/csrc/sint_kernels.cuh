// Cell kernels of the sintering operator (templates; instantiated per
// dimension, number of grains and mobility type in sint_inst_*.cu).
#pragma once

#include "sint_cellfact.cuh"
#include "sint_common.cuh"
#include "sint_launch.h"
#include "sint_physics.cuh"

namespace sint
{
  // Park a lane's node contribution in shared memory (zero for cells outside the mesh).
  template <int DIM, typename R>
  __device__ __forceinline__ void store_contrib(R *s_con, int comp, R r, bool valid)
  {
    using T = Tile<DIM>;
    s_con[comp * T::CS + (threadIdx.x & (T::NQ - 1)) * T::CP + threadIdx.x / T::NQ] = valid ? r : R(0);
  }

  // -------------------------------------------------------------------------
  // Three-phase cell kernels (Jacobian-vector product and residual).
  //
  // Per tile: phase 1 evaluates every needed component at all points of a cell
  // (one thread per (cell, component), per-cell sum factorisation) into the
  // point-field buffer F[slot][cell]; phase 2 runs the point physics (one
  // thread per (point, cell)) and writes the point results to P[res][q][cell];
  // phase 3 integrates each residual row of a cell (one thread per (cell,
  // row)) into the node contributions K[row][l][cell] (aliasing F); the node
  // sum and the tile-face partials follow.  Warps always work on 32
  // consecutive cells of one component/point/row, so the shared-memory
  // accesses of the three phases are free of bank conflicts.
  //
  // Only the c row has a point-dependent gradient flux (mobility); the mu and
  // eta rows' gradient terms (-kappa_c grad c, L kappa_p grad eta) have
  // constant coefficients and are applied with the exact element stiffness to
  // the nodal values, so those rows integrate point values only.

  // Components evaluated in phase 1, in slot order.  Jacobian product:
  //   tensorial: [lin c, lin mu, lin eta_i] (value + gradient),
  //              [src c, src mu] (value + gradient), [src eta_i] (value)
  //   scalar:    [lin mu, src mu] (value + gradient),
  //              [lin c, lin eta_i, src c, src eta_i] (value)
  // Residual (u = the state, h = the weighted history):
  //   tensorial: [c, mu, eta_i] (value + gradient), [h c, h eta_i] (value)
  //   scalar:    [mu] (value + gradient), [c, eta_i] (value), [h c, h eta_i] (value)
  template <int DIM, int G, bool TENS, bool JVP, bool HIST, bool IN_PLACE = false>
  struct FieldMap
  {
    using SL = Slots<DIM>;
    static constexpr int NVG    = JVP ? (TENS ? 4 + G : 2) : (TENS ? 2 + G : 1);
    static constexpr int NV     = JVP ? (TENS ? G : 2 + 2 * G) : ((TENS ? 0 : 1 + G) + (HIST ? 1 + G : 0));
    static constexpr int NITEMS = NVG + NV;
    // slots: the values of all items first, then the gradients of the first
    // NVG; with IN_PLACE at least as many value slots as there are point results
    static constexpr int NRES  = DIM + 2 + G;
    static constexpr int NVAL  = IN_PLACE && NRES > NITEMS ? NRES : NITEMS;
    static constexpr int NSLOT = NVAL * SL::V + NVG * (SL::VG - SL::V);

    __host__ __device__ static constexpr int base(int item) { return item * SL::V; }
    __host__ __device__ static constexpr int gbase(int item) { return NVAL * SL::V + item * (SL::VG - SL::V); }
    // Value slot (in units of NQ) of point result res.  IN_PLACE: results
    // replace values that only the same (point, cell) thread reads: the eta_i
    // row eta_i's own, the others (written last) the values before the first
    // and behind the last eta_i; together the first NRES slots.
    __host__ __device__ static constexpr int result(int res)
    {
      return !IN_PLACE ? res : (res >= DIM + 2 ? lin_eta(res - DIM - 2) : (res < lin_eta(0) ? res : G + res));
    }
    // item index of each quantity (residual: "lin" is the state itself)
    static constexpr int lin_c  = TENS ? 0 : (JVP ? 2 : 1);
    static constexpr int lin_mu = TENS ? 1 : 0;
    __host__ __device__ static constexpr int lin_eta(int i) { return TENS ? 2 + i : (JVP ? 3 + i : 2 + i); }
    static constexpr int src_c  = TENS ? 2 + G : 3 + G;
    static constexpr int src_mu = TENS ? 3 + G : 1;
    __host__ __device__ static constexpr int src_eta(int i) { return 4 + G + i; }
    static constexpr int h_c = 2 + G;
    __host__ __device__ static constexpr int h_eta(int i) { return 3 + G + i; }
    // grain of a phase-1 item (-1 for c and mu items)
    __host__ __device__ static constexpr int grain(int it)
    {
      return (it >= lin_eta(0) && it < lin_eta(0) + G) ? it - lin_eta(0)
             : (JVP && it >= src_eta(0)) ? it - src_eta(0)
             : (!JVP && HIST && it >= h_eta(0)) ? it - h_eta(0)
                                               : -1;
    }

    // phase 1 item -> (buffer 0 = lin / state, 1 = src / history; component; value+gradient?)
    __device__ static void source(int it, int &buf, int &comp)
    {
      if constexpr (JVP)
        {
          if constexpr (TENS)
            {
              if (it < 2 + G) { buf = 0; comp = it; }
              else if (it < 4 + G) { buf = 1; comp = it - 2 - G; }
              else { buf = 1; comp = 2 + (it - 4 - G); }
            }
          else
            {
              if (it == 0) { buf = 0; comp = 1; }
              else if (it == 1) { buf = 1; comp = 1; }
              else if (it == 2) { buf = 0; comp = 0; }
              else if (it < 3 + G) { buf = 0; comp = 2 + (it - 3); }
              else if (it == 3 + G) { buf = 1; comp = 0; }
              else { buf = 1; comp = 2 + (it - 4 - G); }
            }
        }
      else
        {
          if constexpr (TENS)
            {
              if (it < 2 + G) { buf = 0; comp = it; }
              else if (it == 2 + G) { buf = 1; comp = 0; }
              else { buf = 1; comp = 2 + (it - 3 - G); }
            }
          else
            {
              if (it == 0) { buf = 0; comp = 1; }
              else if (it == 1) { buf = 0; comp = 0; }
              else if (it < 2 + G) { buf = 0; comp = 2 + (it - 2); }
              else if (it == 2 + G) { buf = 1; comp = 0; }
              else { buf = 1; comp = 2 + (it - 3 - G); }
            }
        }
    }
  };

  // Phase 1: evaluate all items of the tile.  With the grain cut-off (CUT),
  // the items of a grain absent on this thread's cell (bit clear in m) are
  // zero; a warp that has no lane needing an item writes the zeros without
  // evaluating.
  template <int DIM, int G, bool TENS, bool JVP, bool HIST, typename R, bool CUT = false, bool IN_PLACE = false>
  __device__ __forceinline__ void phase_evaluate(const R *box0, const R *box1, R *F, const CellConsts<DIM, R> &k,
                                                 unsigned m = ~0u)
  {
    using T            = Tile<DIM>;
    using SL           = Slots<DIM>;
    using FM           = FieldMap<DIM, G, TENS, JVP, HIST, IN_PLACE>;
    constexpr int NGRP = T::THREADS / T::CELLS;
    const int     cell = threadIdx.x % T::CELLS;
    const int     b0   = cell_box_base<DIM>(cell);
    for (int it = threadIdx.x / T::CELLS; it < FM::NITEMS; it += NGRP)
      {
        bool absent = false;
        if constexpr (CUT)
          {
            const int gr = FM::grain(it);
            absent       = gr >= 0 && ((m >> gr) & 1u) == 0u;
            if (!__any_sync(0xffffffffu, !absent))
              {
                for (int sl = 0; sl < SL::V; ++sl)
                  F[(FM::base(it) + sl) * T::CELLS + cell] = R(0);
                if (it < FM::NVG)
                  for (int sl = 0; sl < SL::VG - SL::V; ++sl)
                    F[(FM::gbase(it) + sl) * T::CELLS + cell] = R(0);
                continue;
              }
          }
        int buf = 0, comp = 0;
        FM::source(it, buf, comp);
        R u[1 << DIM];
        cell_nodes<DIM>((buf == 0 ? box0 : box1) + comp * T::BOXS, b0, u);
        if constexpr (CUT)
          if (absent)
#pragma unroll
            for (int l = 0; l < (1 << DIM); ++l)
              u[l] = R(0);
        if (it < FM::NVG)
          cell_eval_vg<DIM>(u, k, F, FM::base(it), FM::gbase(it), cell);
        else
          cell_eval_v<DIM>(u, k, F, FM::base(it), cell);
      }
  }

  // point-field accessors for phase 2 (thread = (point q, cell))
  template <int DIM, typename R>
  __device__ __forceinline__ R fval(const R *F, int base, int q, int cell)
  {
    return F[(base + q) * Tile<DIM>::CELLS + cell];
  }
  template <int DIM, typename R>
  __device__ __forceinline__ void fgrad(const R *F, int gbase, int q, int cell, R (&g)[DIM])
  {
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      g[d] = F[(gbase + d * Slots<DIM>::NG1 + grad_slot<DIM>(d, q)) * Tile<DIM>::CELLS + cell];
  }

  // point results: P[(FieldMap::result(res) * NQ + q) * CELLS + cell]; res 0 = c row value,
  // 1..DIM = c row flux, DIM + 1 = mu row value, DIM + 2 + i = eta_i row value
  template <int DIM, typename R>
  __device__ __forceinline__ void pstore(R *P, int res, int q, int cell, nd<R> v)
  {
    P[(res * Slots<DIM>::NQ + q) * Tile<DIM>::CELLS + cell] = v;
  }

  // Point terms of the Jacobian product (SinteringOperatorGenericQuad::
  // operator(), generic.h:101-190) from the fields at one point: the state
  // (c, eta and their gradients, grad mu), and the direction (d*).  Every
  // result goes to emit(res, value) with pstore's numbering: res 0 = c row
  // value, 1..DIM = c row flux, DIM + 1 = mu row value, DIM + 2 + i = eta_i
  // row value.
  template <int DIM, int G, bool TENS, typename R, typename Emit>
  __device__ __forceinline__ void jvp_terms(const PhysR<R> &p, const R &c, const R (&gc)[DIM], const R (&gmu)[DIM],
                                            const R (&eta)[gdim(G)], const R (*geta)[DIM], const R &dc,
                                            const R (&gdc)[DIM], const R &dmu, const R (&gdmu)[DIM],
                                            const R (&deta)[gdim(G)], unsigned m, Emit emit)
  {
    // free energy second derivatives at the linearisation point (free_energy.h:143-161)
    R s2 = R(0);
#pragma unroll
    for (int i = 0; i < G; ++i)
      s2 += eta[i] * eta[i];
    const R omc = R(1) - c;
    // f_cc = 2 A c^2 + 4 A c (2 c - 2) + 2 A (1 - c)^2 + 2 B = 2 (A + B) - 12 A c (1 - c)
    const R fcc = R(2) * (p.A + p.B) - (R(12) * p.A) * c * omc;
    const R B12 = p.B * R(12);
    // f_{c eta_i} = 12 B eta_i (eta_i - 1) (free_energy.h:150-152), shared by the mu
    // and eta rows
    R fce[gdim(G)];
#pragma unroll
    for (int i = 0; i < G; ++i)
      {
        const R be = B12 * eta[i];
        fce[i]     = be * eta[i] - be;
      }

    // 1) c row (generic.h:120-134)
    {
      R gres[DIM];
      apply_M_derivative<DIM, G, TENS>(p, c, gc, gmu, eta, geta, dc, gdc, gdmu, deta, gres, m);
      emit(0, dc * p.w0);
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        emit(1 + d, gres[d]);
    }
    // 2) mu row value (generic.h:138-144)
    {
      R v = p.walg * dmu - fcc * dc;
#pragma unroll
      for (int i = 0; i < G; ++i)
        v -= fce[i] * deta[i];
      emit(DIM + 1, v);
    }
    // 3) eta row values (generic.h:150-163, free_energy.h:233-252)
    {
      R S = R(0);
#pragma unroll
      for (int i = 0; i < G; ++i)
        S += eta[i] * deta[i];
      // w0 deta_i + L (f_{c eta_i} dc + f_{eta_i eta_i} deta_i) + 24 B L eta_i (S -
      // eta_i deta_i) with f_{eta_i eta_i} = B (12 - 12 c + 2 eta_i (12 c - 24) + 24
      // eta_i^2 + 12 sum eta^2) (free_energy.h:154-158): the 24 B L eta_i^2 deta_i
      // of the last two cancel
      const R al0 = p.w0 + p.L * (B12 * (omc + s2)), al1 = (p.L * p.B) * (R(24) * c - R(48));
      const R Ldc = p.L * dc, gS = (p.L * R(24) * p.B) * S;
#pragma unroll
      for (int i = 0; i < G; ++i)
        {
          const R al = al0 + eta[i] * al1;
          R       v  = deta[i] * al + fce[i] * Ldc;
          v += gS * eta[i];
          emit(DIM + 2 + i, v);
        }
    }
  }

  // Phase 2 of the Jacobian product at point q of cell `cell`.
  template <int DIM, int G, bool TENS, typename FM, typename R>
  __device__ __forceinline__ void jvp_point(const PhysR<R> &p, const R *F, R *P, int q, int cell, unsigned m = ~0u)
  {
    R c, gc[DIM], gmu[DIM];
    c = fval<DIM>(F, FM::base(FM::lin_c), q, cell);
    if constexpr (TENS)
      fgrad<DIM>(F, FM::gbase(FM::lin_c), q, cell, gc);
    fgrad<DIM>(F, FM::gbase(FM::lin_mu), q, cell, gmu);
    R eta[gdim(G)];
    R geta[TENS ? gdim(G) : 1][DIM];
#pragma unroll
    for (int i = 0; i < G; ++i)
      {
        eta[i] = fval<DIM>(F, FM::base(FM::lin_eta(i)), q, cell);
        if constexpr (TENS)
          fgrad<DIM>(F, FM::gbase(FM::lin_eta(i)), q, cell, geta[i]);
      }
    R dc, gdc[DIM], dmu, gdmu[DIM];
    dc = fval<DIM>(F, FM::base(FM::src_c), q, cell);
    if constexpr (TENS)
      fgrad<DIM>(F, FM::gbase(FM::src_c), q, cell, gdc);
    dmu = fval<DIM>(F, FM::base(FM::src_mu), q, cell);
    fgrad<DIM>(F, FM::gbase(FM::src_mu), q, cell, gdmu);
    R deta[gdim(G)];
#pragma unroll
    for (int i = 0; i < G; ++i)
      deta[i] = fval<DIM>(F, FM::base(FM::src_eta(i)), q, cell);
    jvp_terms<DIM, G, TENS, R>(p, c, gc, gmu, eta, geta, dc, gdc, dmu, gdmu, deta, m,
                               [&](int res, R v) { pstore<DIM>(P, FM::result(res), q, cell, v); });
  }

  // Point terms of the residual (SinteringOperatorGenericResidualQuad::
  // operator(), generic.h:254-308) from the fields at one point;
  // time(i, v) adds the time-derivative term of c (i = -1) or eta_i to v,
  // emit(res, value) as in jvp_terms.
  template <int DIM, int G, bool TENS, typename R, typename Time, typename Emit>
  __device__ __forceinline__ void residual_terms(const PhysR<R> &p, const R &c, const R (&gc)[DIM], const R &mu,
                                                 const R (&gmu)[DIM], const R (&eta)[gdim(G)], const R (*geta)[DIM],
                                                 unsigned m, Time time, Emit emit)
  {
    R s2 = R(0), s3 = R(0);
#pragma unroll
    for (int i = 0; i < G; ++i)
      {
        const R e2 = eta[i] * eta[i];
        s2 += e2;
        s3 += e2 * eta[i];
      }
    const R omc = R(1) - c;
    const R LB12 = p.L * (p.B * R(12)), os = omc + s2;
    // 1) c row (generic.h:275-285)
    {
      const R v = time(-1, R(0));
      R       gres[DIM];
      apply_M<DIM, G, TENS>(p, c, eta, gc, geta, gmu, gres, m);
      emit(0, v);
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        emit(1 + d, gres[d]);
    }
    // 2) mu row value (generic.h:288, free_energy.h:124-134)
    {
      // A c^2 (2 c - 2) + 2 A c (1 - c)^2 = 2 A c (1 - c) (1 - 2 c)
      const R df_dc = (R(2) * p.A) * c * omc * (R(1) - R(2) * c) + p.B * (R(2) * c - R(6) * s2 + R(4) * s3);
      emit(DIM + 1, p.walg * mu - df_dc);
    }
    // 3) eta row values (generic.h:293-302, free_energy.h:136-141)
#pragma unroll
    for (int i = 0; i < G; ++i)
      {
        const R e = eta[i];
        emit(DIM + 2 + i, time(i, (LB12 * e) * (e * (c - R(2)) + os)));
      }
  }

  // Phase 2 of the residual at point q of cell `cell`.
  template <int DIM, int G, bool TENS, int WTD, typename FM, typename R>
  __device__ __forceinline__ void residual_point(const PhysR<R> &p, const R *F, R *P, int q, int cell,
                                                 unsigned m = ~0u)
  {
    R c, gc[DIM], mu, gmu[DIM];
    c = fval<DIM>(F, FM::base(FM::lin_c), q, cell);
    if constexpr (TENS)
      fgrad<DIM>(F, FM::gbase(FM::lin_c), q, cell, gc);
    mu = fval<DIM>(F, FM::base(FM::lin_mu), q, cell);
    fgrad<DIM>(F, FM::gbase(FM::lin_mu), q, cell, gmu);
    R eta[gdim(G)];
    R geta[TENS ? gdim(G) : 1][DIM];
#pragma unroll
    for (int i = 0; i < G; ++i)
      {
        eta[i] = fval<DIM>(F, FM::base(FM::lin_eta(i)), q, cell);
        if constexpr (TENS)
          fgrad<DIM>(F, FM::gbase(FM::lin_eta(i)), q, cell, geta[i]);
      }
    residual_terms<DIM, G, TENS, R>(
      p, c, gc, mu, gmu, eta, geta, m,
      [&](int i, R v) {
        if constexpr (WTD >= 1)
          v += (i < 0 ? c : eta[i < 0 ? 0 : i]) * p.w0;
        if constexpr (WTD == 2)
          v += fval<DIM>(F, FM::base(i < 0 ? FM::h_c : FM::h_eta(i)), q, cell);
        return v;
      },
      [&](int res, R v) { pstore<DIM>(P, FM::result(res), q, cell, v); });
  }

  // ---- the residual of many grains in 3D: pair sums streamed from shared memory
  // With more than 5 grains the state of a point does not fit 128 registers,
  // and one block of 256 threads per SM (8 warps) left the residual waiting on
  // latency (9 grains: issue in 24 % of the cycles).  Here a point thread
  // keeps a block of pair_block grains in registers and streams the others
  // past it, and the results replace values in the point-field buffer
  // (FieldMap IN_PLACE), so that two blocks fit an SM's registers and shared
  // memory: 96^3 cells, BDF2, 9 grains 1794 -> 1203 us (tensorial), 1450 ->
  // 864 us (scalar).  The FP64 Jacobian product was not faster this way (9
  // grains 1178 -> 1231 us: the streamed operands are 40 % more) and keeps
  // its registers.
  template <int G>
  __host__ __device__ constexpr int pair_block()
  {
    return G % 3 == 0 && G % 4 != 0 ? 3 : 4;
  }

  template <int DIM, typename R>
  struct PairGrain
  {
    R e, g[DIM];

    template <typename FM>
    __device__ __forceinline__ void load(const R *F, int i, int q, int cell)
    {
      e = fval<DIM>(F, FM::base(FM::lin_eta(i)), q, cell);
      fgrad<DIM>(F, FM::gbase(FM::lin_eta(i)), q, cell, g);
    }
  };

  // s1 = sum_{i>j} eta_i eta_j and acc = -sum_{i>j} eta_i eta_j f_ij d_ij (d_ij .
  // grad mu), the projected part of the pair mobility (mobility.h:785-804)
  template <int DIM, int G, typename FM, typename R>
  __device__ __forceinline__ void pair_sums(const R *F, int q, int cell, const R (&gmu)[DIM], unsigned m, R &s1,
                                            R (&acc)[DIM])
  {
    constexpr int BI = pair_block<G>();
    s1               = R(0);
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      acc[d] = R(0);
    auto pair = [&](const PairGrain<DIM, R> &x, const PairGrain<DIM, R> &y) {
      R dd[DIM];
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        dd[d] = x.g[d] - y.g[d];
      const R p1 = x.e * y.e;
      s1 += p1;
      const R t = p1 * unit_vector_filter_2<DIM>(dd) * dotv<DIM>(dd, gmu);
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        acc[d] -= t * dd[d];
    };
#pragma unroll 1
    for (int i0 = 0; i0 < G; i0 += BI)
      {
        PairGrain<DIM, R> x[BI];
#pragma unroll
        for (int b = 0; b < BI; ++b)
          if (G % BI == 0 || i0 + b < G)
            x[b].template load<FM>(F, i0 + b, q, cell);
#pragma unroll
        for (int b = 1; b < BI; ++b)
          if (G % BI == 0 || i0 + b < G)
#pragma unroll
            for (int c = 0; c < b; ++c)
              if (pair_needed(m, i0 + b, i0 + c))
                pair(x[b], x[c]);
#pragma unroll 1
        for (int j = 0; j < i0; ++j)
          {
            PairGrain<DIM, R> y;
            y.template load<FM>(F, j, q, cell);
#pragma unroll
            for (int b = 0; b < BI; ++b)
              if (G % BI == 0 || i0 + b < G)
                if (pair_needed(m, i0 + b, j))
                  pair(x[b], y);
          }
      }
  }

  // residual_point with the pair sums streamed and the results in place.
  template <int DIM, int G, bool TENS, int WTD, typename FM, typename R>
  __device__ __forceinline__ void residual_point_streamed(const PhysR<R> &p, R *F, int q, int cell, unsigned m)
  {
    const R c = fval<DIM>(F, FM::base(FM::lin_c), q, cell), mu = fval<DIM>(F, FM::base(FM::lin_mu), q, cell);
    R       flux[DIM];
    {
      R gc[DIM], gmu[DIM], none[1] = {R(0)};
      const R(*gnone)[DIM] = nullptr;
      fgrad<DIM>(F, FM::gbase(FM::lin_mu), q, cell, gmu);
      if constexpr (TENS)
        {
          R s1, acc[DIM];
          pair_sums<DIM, G, FM>(F, q, cell, gmu, m, s1, acc);
          fgrad<DIM>(F, FM::gbase(FM::lin_c), q, cell, gc);
          apply_M<DIM, 1, TENS>(p, c, none, gc, gnone, gmu, flux); // the c part
          const R m2 = R(2) * p.Mgb;
#pragma unroll
          for (int d = 0; d < DIM; ++d)
            flux[d] += m2 * (s1 * gmu[d] + acc[d]);
        }
      else
        {
          R etaij = R(0), sum = R(0); // sum_i eta_i (eta_0 + .. + eta_{i-1})
#pragma unroll 3
          for (int i = 0; i < G; ++i)
            {
              const R e = fval<DIM>(F, FM::base(FM::lin_eta(i)), q, cell);
              etaij += e * sum;
              sum += e;
            }
          apply_M<DIM, 1, TENS>(p, c, none, gc, gnone, gmu, flux);
#pragma unroll
          for (int d = 0; d < DIM; ++d)
            flux[d] += ((R(2) * p.Mgb) * etaij) * gmu[d];
        }
    }
    R v0 = R(0);
    if constexpr (WTD >= 1)
      v0 = c * p.w0;
    if constexpr (WTD == 2)
      v0 += fval<DIM>(F, FM::base(FM::h_c), q, cell);
    R s2 = R(0), s3 = R(0);
#pragma unroll 3
    for (int i = 0; i < G; ++i)
      {
        const R e = fval<DIM>(F, FM::base(FM::lin_eta(i)), q, cell);
        const R e2 = e * e;
        s2 += e2;
        s3 += e2 * e;
      }
    const R omc = R(1) - c;
    const R LB12 = p.L * (p.B * R(12)), os = omc + s2;
#pragma unroll 3
    for (int i = 0; i < G; ++i)
      {
        const R e = fval<DIM>(F, FM::base(FM::lin_eta(i)), q, cell);
        R       v = (LB12 * e) * (e * (c - R(2)) + os);
        if constexpr (WTD >= 1)
          v += e * p.w0;
        if constexpr (WTD == 2)
          v += fval<DIM>(F, FM::base(FM::h_eta(i)), q, cell);
        pstore<DIM>(F, FM::result(DIM + 2 + i), q, cell, v);
      }
    const R df_dc = (R(2) * p.A) * c * omc * (R(1) - R(2) * c) + p.B * (R(2) * c - R(6) * s2 + R(4) * s3);
    pstore<DIM>(F, FM::result(0), q, cell, v0);
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      pstore<DIM>(F, FM::result(1 + d), q, cell, flux[d]);
    pstore<DIM>(F, FM::result(DIM + 1), q, cell, p.walg * mu - df_dc);
  }

  // Global coordinates of local cell `cell` of tile tc; false outside the mesh.
  template <int DIM>
  __device__ __forceinline__ bool cell_global(int cell, const TileCoord &tc, const Grid &g, int (&cc)[3])
  {
    using T = Tile<DIM>;
    cc[0]   = tc.o[0] + cell % T::TX;
    cc[1]   = tc.o[1] + (cell / T::TX) % T::TY;
    cc[2]   = DIM == 3 ? tc.o[2] + cell / (T::TX * T::TY) : 0;
    return cc[0] < g.n[0] && cc[1] < g.n[1] && (DIM == 2 || cc[2] < g.n[2]);
  }

  // Advection coefficients of one tile, staged once per tile before phase 1
  // (AdvectionVelocityData::reinit, sintering/advection.h:185-222): for
  // grain k (the tile's k-th grain under the cut-off) and local cell `cell`,
  // item i = k * CELLS + cell: vel[6 i ..] = the velocity at the cell's lower
  // corner and the angular velocity, has[i] = 1 when the grain has a segment
  // on the cell.  The velocity at point q is then vel + w x (x_q - corner).
  template <int DIM, int G, typename R, bool CUT>
  __device__ __forceinline__ void adv_stage(const AdvData &a, const Grid &g, const TileCoord &tc,
                                            unsigned long long gl, R *vel, unsigned char *has)
  {
    using T                 = Tile<DIM>;
    const long long n_cells = (long long)g.n[0] * g.n[1] * g.n[2];
    for (int it = threadIdx.x; it < G * T::CELLS; it += T::THREADS)
      {
        const int k = it / T::CELLS, cell = it % T::CELLS;
        int       cc[3];
        int       s = -1;
        if (cell_global<DIM>(cell, tc, g, cc))
          {
            const int b = CUT ? int((gl >> (4 * k)) & 15ull) : k;
            s           = a.cell_segments[b * n_cells + cc[0] + (long long)g.n[0] * (cc[1] + (long long)g.n[1] * cc[2])];
            if (s >= a.n_segments)
              s = -1;
          }
        has[it] = s >= 0;
        if (s >= 0)
          {
            const double *d    = a.segments + 9 * (long long)s;
            double        r[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int e = 0; e < DIM; ++e)
              r[e] = a.origin[e] + cc[e] * g.h[e] - d[6 + e];
            R *o = vel + 6 * it;
            o[0] = R(d[0] + d[4] * r[2] - d[5] * r[1]);
            o[1] = R(d[1] + d[5] * r[0] - d[3] * r[2]);
            o[2] = R(d[2] + d[3] * r[1] - d[4] * r[0]);
            o[3] = R(d[3]);
            o[4] = R(d[4]);
            o[5] = R(d[5]);
          }
      }
  }

  // Velocity of staged item `it` at point q (offset dq from the cell corner).
  template <int DIM, typename R>
  __device__ __forceinline__ void adv_velocity(const R *vel, int it, const R (&dq)[3], R (&v)[DIM])
  {
    const R *w = vel + 6 * it;
    v[0]       = w[0] + (w[4] * dq[2] - w[5] * dq[1]);
    v[1]       = w[1] + (w[5] * dq[0] - w[3] * dq[2]);
    if constexpr (DIM == 3)
      v[2] = w[2] + (w[3] * dq[1] - w[4] * dq[0]);
  }

  template <int DIM, typename R>
  __device__ __forceinline__ void adv_offset(const CellConsts<DIM, R> &k, const Grid &g, int q, R (&dq)[3])
  {
#pragma unroll
    for (int e = 0; e < 3; ++e)
      dq[e] = e < DIM ? (((q >> e) & 1) ? k.x1 : k.x0) * R(g.h[e]) : R(0);
  }

  // Advection of the c row at point q (phase 2, after the point physics):
  // the c flux loses v_i c for every grain i with a velocity on the cell, one
  // grain after the other (operator_sintering_generic.h:1015-1036 for the
  // residual, :167-177 for J v, where c is the direction's value).  With the
  // grain cut-off only the cell's relevant grains move it (AdvectionVelocityData
  // maps order parameters through the relevant-grain table,
  // sintering/advection.h:225-245).
  template <int DIM, int G, typename R, bool CUT>
  __device__ __forceinline__ void advect_c_point(const CellConsts<DIM, R> &k, const Grid &g, const R *F, int c_base,
                                                 R *P, int q, int cell, unsigned m, const R *vel,
                                                 const unsigned char *has)
  {
    using T = Tile<DIM>;
    R     dq[3];
    adv_offset<DIM>(k, g, q, dq);
    const R c = fval<DIM>(F, c_base, q, cell);
    R       flux[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      flux[d] = P[((1 + d) * Slots<DIM>::NQ + q) * T::CELLS + cell];
#pragma unroll 1
    for (int i = 0; i < G; ++i)
      {
        if ((CUT && ((m >> i) & 1u) == 0u) || !has[i * T::CELLS + cell])
          continue;
        R v[DIM];
        adv_velocity<DIM>(vel, i * T::CELLS + cell, dq, v);
#pragma unroll
        for (int d = 0; d < DIM; ++d)
          flux[d] = flux[d] - v[d] * c;
      }
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      P[((1 + d) * Slots<DIM>::NQ + q) * T::CELLS + cell] = flux[d];
  }

  // Phase 3, 3D: the c row's contributions to the local nodes with z bit HZ
  // (K rows l = lx + 2 ly + 4 HZ) from the point values and fluxes in P.
  // FM: the kernel's FieldMap (where the point results are).
  template <int HZ, typename FM, typename R>
  __device__ __forceinline__ void integrate_c_row_half(const R *P, const CellConsts<3, R> &k, int cell, bool in,
                                                       bool in_b, R *K)
  {
    using T          = Tile<3>;
    constexpr int NQ = 8;
    R v[NQ], gg[3][NQ], r[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      {
        v[q] = P[(FM::result(0) * NQ + q) * T::CELLS + cell];
#pragma unroll
        for (int d = 0; d < 3; ++d)
          gg[d][q] = P[(FM::result(1 + d) * NQ + q) * T::CELLS + cell];
      }
    cell_integrate_vg_half<HZ>(v, gg, k, r);
#pragma unroll
    for (int l = 4 * HZ; l < 4 * HZ + 4; ++l)
      K[l * T::CP + cell] = (in && in_b) ? r[l] : lane_keep(r[l], in, in_b);
  }

  // Phase 3: integrate every row of every cell into K[(row * NQ + l) * CP + cell];
  // contributions of cells outside the mesh (partial tiles) are zero.  `stiff`
  // holds the nodal values the constant-coefficient gradient terms act on
  // (component 0 = c for the mu row, component 2 + i = eta_i for the eta rows).
  // With the grain cut-off (CUT) the row of a grain absent on the cell is zero
  // (do_vmult_range_no_template / do_evaluate_nonlinear_residual_nt,
  // operator_sintering_generic.h:456-537, :1008-1081, assemble the relevant
  // grains' rows only).  ADV: the eta_i row of a grain with a velocity on the
  // cell gains the flux -v_i eta_i (operator_sintering_generic.h:1015-1036,
  // :167-177), eta_i interpolated from the same nodal values `stiff` holds;
  // warps in which no cell of the row moves keep the value-only integration.
  // tc_b (packed pairs only): the tile of lane y, whose cells outside the
  // mesh are zeroed lane by lane.
  template <int DIM, int G, typename FM, typename R, bool CUT = false, bool ADV = false>
  __device__ __forceinline__ void phase_integrate(const PhysR<R> &p, const Grid &g, const CellConsts<DIM, R> &k,
                                                  const TileCoord &tc, const R *P, const R *stiff, R *K,
                                                  unsigned m = ~0u, const R *vel = nullptr,
                                                  const unsigned char *has = nullptr,
                                                  const TileCoord *tc_b = nullptr)
  {
    using T            = Tile<DIM>;
    constexpr int NQ   = 1 << DIM;
    constexpr int C    = G + 2;
    constexpr int NGRP = T::THREADS / T::CELLS;
    // In 3D with fewer rows than thread groups, the c row (the only one with
    // a point-dependent flux, the longest) is shared by two groups, one per
    // layer of local nodes (z bit 0 / 1): C + 1 tasks instead of C rows.
    constexpr bool SPLIT0 = DIM == 3 && C + 1 <= NGRP;
    constexpr int  NTASK  = C + (SPLIT0 ? 1 : 0);
    const int     cell = threadIdx.x % T::CELLS;
    const int     b0   = cell_box_base<DIM>(cell);
    const bool    in   = cell_in_mesh<DIM>(cell, tc, g);
    const bool    in_b = tc_b ? cell_in_mesh<DIM>(cell, *tc_b, g) : in;
    for (int task = threadIdx.x / T::CELLS; task < NTASK; task += NGRP)
      {
        const int row = SPLIT0 ? (task < 2 ? 0 : task - 1) : task;
        if constexpr (SPLIT0)
          if (task < 2)
            {
              if (task == 0)
                integrate_c_row_half<0, FM>(P, k, cell, in, in_b, K);
              else
                integrate_c_row_half<1, FM>(P, k, cell, in, in_b, K);
              continue;
            }
        bool keep = in;
        if constexpr (CUT)
          if (row >= 2)
            {
              keep = keep && ((m >> (row - 2)) & 1u) != 0u;
              if (!__any_sync(0xffffffffu, keep))
                {
#pragma unroll
                  for (int l = 0; l < NQ; ++l)
                    K[(row * NQ + l) * T::CP + cell] = R(0);
                  continue;
                }
            }
        R r[NQ];
        if (row == 0)
          {
            R v[NQ], gg[DIM][NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q)
              {
                v[q] = P[(FM::result(0) * NQ + q) * T::CELLS + cell];
#pragma unroll
                for (int d = 0; d < DIM; ++d)
                  gg[d][q] = P[(FM::result(1 + d) * NQ + q) * T::CELLS + cell];
              }
            cell_integrate_vg<DIM>(v, gg, k, r);
          }
        else if (ADV && row >= 2 && __any_sync(0xffffffffu, has[(row - 2) * T::CELLS + cell] != 0))
          {
            R v[NQ], u[NQ], gg[DIM][NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q)
              {
                v[q] = P[((DIM + row) * NQ + q) * T::CELLS + cell];
#pragma unroll
                for (int d = 0; d < DIM; ++d)
                  gg[d][q] = R(0);
              }
            cell_nodes<DIM>(stiff + row * T::BOXS, b0, u);
            const int it = (row - 2) * T::CELLS + cell;
            if (has[it])
              {
                R e[NQ];
                cell_values<DIM>(u, k, e);
#pragma unroll
                for (int q = 0; q < NQ; ++q)
                  {
                    R dq[3], vq[DIM];
                    adv_offset<DIM>(k, g, q, dq);
                    adv_velocity<DIM>(vel, it, dq, vq);
#pragma unroll
                    for (int d = 0; d < DIM; ++d)
                      gg[d][q] = -(vq[d] * e[q]);
                  }
              }
            cell_integrate_vg<DIM>(v, gg, k, r);
            cell_stiffness_add<DIM, 1>(u, g, r);
          }
        else
          {
            // mu row: result DIM + 1, eta_i row (row = 2 + i): DIM + 2 + i
            const int res = FM::result(DIM + row);
            R         v[NQ];
#pragma unroll
            for (int q = 0; q < NQ; ++q)
              v[q] = P[(res * NQ + q) * T::CELLS + cell];
            cell_integrate_v<DIM>(v, k, r);
            R u[NQ];
            cell_nodes<DIM>(stiff + (row == 1 ? 0 : row) * T::BOXS, b0, u);
            if (row == 1)
              cell_stiffness_add<DIM, 0>(u, g, r);
            else
              cell_stiffness_add<DIM, 1>(u, g, r);
          }
        // a branch, not a select per value: in tiles inside the mesh every
        // cell keeps its row
        if (keep && in_b)
          {
#pragma unroll
            for (int l = 0; l < NQ; ++l)
              K[(row * NQ + l) * T::CP + cell] = r[l];
          }
        else
          {
#pragma unroll
            for (int l = 0; l < NQ; ++l)
              K[(row * NQ + l) * T::CP + cell] = lane_keep(r[l], keep, in_b);
          }
      }
  }

  // Grain-cut-off mask of local cell `cell` of tile tc (one bit per grain,
  // n[0] x n[1] x n[2] cells in lexicographic order); cells outside the mesh
  // have no relevant grain.
  template <int DIM>
  __device__ __forceinline__ unsigned cell_mask(const uint16_t *__restrict__ mask, const Grid &g,
                                                const TileCoord &tc, int cell)
  {
    using T      = Tile<DIM>;
    const int cx = cell % T::TX, cy = (cell / T::TX) % T::TY, cz = cell / (T::TX * T::TY);
    const int i = tc.o[0] + cx, j = tc.o[1] + cy, k = DIM == 3 ? tc.o[2] + cz : 0;
    if (i >= g.n[0] || j >= g.n[1] || (DIM == 3 && k >= g.n[2]))
      return 0u;
    return mask[i + (long long)g.n[0] * (j + (long long)g.n[1] * k)];
  }

  // Cell mask m (bits = grains of the full operator) in the numbering of a
  // tile's compacted grain list gl: bit k set when grain gl[k] is relevant.
  template <int G>
  __device__ __forceinline__ unsigned local_mask(unsigned m, unsigned long long gl)
  {
    unsigned r = 0;
#pragma unroll
    for (int kk = 0; kk < G; ++kk)
      r |= ((m >> unsigned((gl >> (4 * kk)) & 15ull)) & 1u) << kk;
    return r;
  }

  // Shared memory of a block (in elements) with NBUF box buffers.  IN_PLACE:
  // the point results take the first FM::NRES value slots and the node
  // contributions follow them, all inside the point-field buffer.
  template <int DIM, int G, bool TENS, bool JVP, bool HIST, bool ADV, bool IN_PLACE, int NBUF>
  struct ThreePhaseLayout
  {
    using T                     = Tile<DIM>;
    using FM                    = FieldMap<DIM, G, TENS, JVP, HIST, IN_PLACE>;
    static constexpr int C      = G + 2;
    static constexpr int NQ     = 1 << DIM;
    static constexpr int BOXES  = 2 * C * T::BOXS; // both inputs of one tile
    static constexpr int K_SIZE = C * NQ * T::CP;
    static constexpr int P_AT   = IN_PLACE ? 0 : FM::NSLOT * T::CELLS;
    static constexpr int K_AT   = IN_PLACE ? FM::NRES * NQ * T::CELLS : 0; // else aliases the dead point fields
    static constexpr int FIELDS = FM::NSLOT * T::CELLS;
    static constexpr int F_SIZE = IN_PLACE && K_AT + K_SIZE > FIELDS ? K_AT + K_SIZE : FIELDS;
    static constexpr int P_SIZE = IN_PLACE ? 0 : FM::NRES * NQ * T::CELLS;
    static_assert(IN_PLACE || K_SIZE <= F_SIZE, "node contributions must fit in the point-field buffer");
    // staged advection coefficients (adv_stage): 6 values and one flag byte
    // per (grain, cell); the flags are counted in 4-byte elements
    static constexpr int ADV_VEL = ADV ? 6 * G * T::CELLS : 0;
    static constexpr int ADV_HAS = ADV ? (G * T::CELLS + 3) / 4 : 0;
    static constexpr int BUFFERS = NBUF;
    static constexpr int TOTAL   = NBUF * BOXES + F_SIZE + P_SIZE + ADV_VEL + ADV_HAS;
  };

  // Bytes a block may take for two blocks to fit an SM (228 KB, 1 KB reserved
  // per block).
  constexpr int TWO_BLOCK_BYTES = (228 * 1024) / 2 - 1024;

  // The layout a kernel uses.  RB = bytes per value (8 for FP64 and packed
  // FP32).  More than 5 grains in 3D: in place where two blocks then fit an SM
  // (FP32: three), with the next tile's boxes double-buffered if they fit too;
  // not for the tensorial Jacobian product, which is bound by registers.  J v
  // of 9 grains, scalar, at 96^3 cells: FP64 701 -> 602 us, FP32 500 -> 417 us.
  template <int DIM, int G, bool TENS, bool JVP, bool HIST, bool ADV, int RB>
  struct ThreePhasePlan
  {
    template <int NBUF>
    using InPlace = ThreePhaseLayout<DIM, G, TENS, JVP, HIST, ADV, true, NBUF>;
    static constexpr bool IN_PLACE =
      DIM == 3 && G > 5 && !ADV && !(JVP && TENS) && InPlace<1>::TOTAL * RB <= TWO_BLOCK_BYTES;
    static constexpr int  NBUF =
      JVP && (!IN_PLACE || InPlace<2>::TOTAL * RB <= TWO_BLOCK_BYTES) ? 2 : 1;
    using type = ThreePhaseLayout<DIM, G, TENS, JVP, HIST, ADV, IN_PLACE, NBUF>;
  };
  template <int DIM, int G, bool TENS, bool JVP, bool HIST, bool ADV, int RB>
  using ThreePhaseSmem = typename ThreePhasePlan<DIM, G, TENS, JVP, HIST, ADV, RB>::type;

  // -------------------------------------------------------------------------
  // Jacobian-vector product: dst = J(lin) src.
  // SinteringOperatorGenericQuad::operator() (operator_sintering_generic.h:101-190)
  // inside do_vmult_range (:539-577), with the linearisation point evaluated
  // from the nodal state instead of a quadrature-point cache.  Persistent and
  // software pipelined: block b handles tiles b, b + grid, ...; the node boxes
  // of the next tile are copied (cp.async) into the second half of a double
  // buffer while the current tile is computed.
  // Two resident blocks per SM (<= 128 registers) unless the 3D FP64 grain
  // state of large G would spill (one block, up to 255 registers; two where
  // the point results are in place); the light 2D FP32 product runs three (<=
  // 85 registers), and the grain cut-off's G = 0 class (c and mu only) four
  // (<= 64 registers).
  template <int DIM, int G, bool TENS, typename R, bool ADV>
  constexpr int jvp_blocks_per_sm()
  {
    return G == 0                                                               ? 4 :
           ThreePhasePlan<DIM, G, TENS, true, false, ADV, sizeof(R)>::IN_PLACE  ? (sizeof(R) == 4 ? 3 : 2) :
           (DIM == 3 && sizeof(R) == 8 && G > 5)                                ? 1 :
           (DIM == 2 && sizeof(R) == 4)                                         ? 3 :
                                                                                  2;
  }
  template <int DIM, int G, bool TENS, bool HIST, bool ADV>
  constexpr int residual_blocks_per_sm()
  {
    return G == 0                                                         ? 4 :
           ThreePhasePlan<DIM, G, TENS, false, HIST, ADV, 8>::IN_PLACE    ? 2 :
           (DIM == 3 && G > 5)                                            ? 1 :
                                                                            2;
  }

  // CUT: grain cut-off.  The kernel instantiated for G grains runs over the
  // tiles of class G, ct.tiles[ct.range[G] .. ct.range[G + 1]), on their
  // compacted components (c, mu and the tile's G grains); a cell lacking one
  // of the tile's grains treats it as absent.  The tile ids, grain lists and
  // masks of the next tile are read one tile ahead, so their latency hides
  // behind the current tile.
  // ADV: with the advection terms of the grains' rigid-body velocities.
  template <int DIM, int G, bool TENS, typename R, bool CUT, bool ADV = false>
  __global__ void __launch_bounds__(Tile<DIM>::THREADS, jvp_blocks_per_sm<DIM, G, TENS, R, ADV>())
    jvp_kernel(const Grid g, const Phys ph, const R *__restrict__ lin, const R *__restrict__ src,
               R *__restrict__ dst, R *__restrict__ partial, const CutTiles ct, const AdvData adv)
  {
    using T  = Tile<DIM>;
    using SM = ThreePhaseSmem<DIM, G, TENS, true, false, ADV, sizeof(R)>;
    using FM = typename SM::FM;
    using PL = ThreePhasePlan<DIM, G, TENS, true, false, ADV, sizeof(R)>;
    constexpr int C = G + 2, NBUF = SM::BUFFERS;
    if constexpr (CUT)
      siblings_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R *s_buf = reinterpret_cast<R *>(smem_raw); // NBUF x BOXES
    R *F     = s_buf + NBUF * SM::BOXES;
    R *P     = F + SM::P_AT;
    R *K     = F + SM::K_AT;
    R *A_vel = F + SM::F_SIZE + SM::P_SIZE;
    unsigned char *A_has = reinterpret_cast<unsigned char *>(A_vel + SM::ADV_VEL);

    const PhysR<R>           p(ph);
    const CellConsts<DIM, R> k(g);
    const NodePlan<DIM>      np(g);
    const int                cell = threadIdx.x % T::CELLS;
    const long long          i0   = CUT ? (long long)ct.range[G] : 0;
    const long long          i1   = CUT ? (long long)ct.range[G + 1] : g.n_tiles;
    long long                idx  = i0 + blockIdx.x;
    // node boxes of both inputs of tile tcx into buffer bb
    auto prefetch = [&](R *bb, const TileCoord &tcx, unsigned long long glx) {
      if (tile_interior<DIM>(g, tcx))
        {
          const long long n0 = tile_node0(g, tcx);
          load_box_async_interior<DIM>(bb, lin, C, g, np, n0, glx, CUT);
          load_box_async_interior<DIM>(bb + C * T::BOXS, src, C, g, np, n0, glx, CUT);
        }
      else
        {
          const BoxNode<DIM> bn(g, tcx);
          load_box_async<DIM>(bb, lin, C, g, bn, glx, CUT);
          load_box_async<DIM>(bb + C * T::BOXS, src, C, g, bn, glx, CUT);
        }
    };
    // current and next tile: id, grain list, union mask, this thread's cell mask
    long long          tile = 0, t_next = 0;
    unsigned long long gl = 0, gl_next = 0;
    unsigned           tm = 0, tm_next = 0, m_glob = ~0u, m_glob_next = ~0u;
    if constexpr (CUT)
      {
        if (idx < i1)
          {
            tile = ct.tiles[idx];
            gl   = ct.tile_grains[idx];
            tm   = ct.tile_mask[idx];
          }
        if (idx + gridDim.x < i1)
          {
            t_next  = ct.tiles[idx + gridDim.x];
            gl_next = ct.tile_grains[idx + gridDim.x];
            tm_next = ct.tile_mask[idx + gridDim.x];
          }
      }
    else
      tile = idx;
    if (idx < i1)
      {
        const TileCoord tc0 = tile_coord_of<DIM>(g, tile);
        prefetch(s_buf, tc0, gl);
        if constexpr (CUT)
          m_glob = cell_mask<DIM>(ct.cell_mask, g, tc0, cell);
      }
    cp_async_commit();
    for (int it = 0; idx < i1; ++it, idx += gridDim.x)
      {
        const long long nidx = idx + gridDim.x;
        R              *nb   = s_buf + (NBUF == 2 ? ((it + 1) & 1) * SM::BOXES : 0);
        long long       t_nn = 0; // the tile after next (CUT)
        unsigned long long gl_nn = 0;
        unsigned           tm_nn = 0;
        const TileCoord    tcn = tile_coord_of<DIM>(g, CUT ? t_next : (nidx < i1 ? nidx : idx));
        if (nidx < i1)
          {
            if constexpr (NBUF == 2)
              prefetch(nb, tcn, gl_next);
            if constexpr (CUT)
              {
                m_glob_next = cell_mask<DIM>(ct.cell_mask, g, tcn, cell);
                if (nidx + gridDim.x < i1)
                  {
                    t_nn  = ct.tiles[nidx + gridDim.x];
                    gl_nn = ct.tile_grains[nidx + gridDim.x];
                    tm_nn = ct.tile_mask[nidx + gridDim.x];
                  }
              }
          }
        if constexpr (NBUF == 2)
          {
            cp_async_commit();
            cp_async_wait<1>(); // this tile's group has landed (only the prefetch may be pending)
          }
        else
          cp_async_wait<0>();
        __syncthreads();
        const TileCoord tc = tile_coord_of<DIM>(g, tile);
        const R        *cb = s_buf + (NBUF == 2 ? (it & 1) * SM::BOXES : 0);
        const unsigned  m  = CUT ? local_mask<G>(m_glob, gl) : ~0u;
        if constexpr (ADV)
          adv_stage<DIM, G, R, CUT>(adv, g, tc, gl, A_vel, A_has);
        phase_evaluate<DIM, G, TENS, true, false, R, CUT, PL::IN_PLACE>(cb, cb + C * T::BOXS, F, k, m);
        __syncthreads();
        jvp_point<DIM, G, TENS, FM, R>(p, F, P, threadIdx.x / T::CELLS, cell, m);
        if constexpr (ADV)
          {
            advect_c_point<DIM, G, R, CUT>(k, g, F, FM::base(FM::src_c), P, threadIdx.x / T::CELLS, cell, m, A_vel,
                                           A_has);
          }
        __syncthreads();
        phase_integrate<DIM, G, FM, R, CUT, ADV>(p, g, k, tc, P, cb + C * T::BOXS, K, m, A_vel, A_has);
        __syncthreads();
        if constexpr (NBUF == 1)
          {
            // one box buffer: its last readers have passed, the next tile's
            // copies run behind the stores below
            if (nidx < i1)
              prefetch(nb, tcn, gl_next);
            cp_async_commit();
          }
        if (tile_interior<DIM>(g, tc))
          sum_and_store_interior<DIM>(K, C, g, tc.linear, np, tile_node0(g, tc), dst, partial, gl, CUT, ct.c_all, tm);
        else
          sum_and_store<DIM>(K, C, g, tc, BoxNode<DIM>(g, tc), dst, partial, gl, CUT, ct.c_all, tm);
        // No further barrier: the next tile's prefetch writes a box buffer whose
        // last readers (phases 1 and 3) have passed the barrier after phase 3,
        // and K (inside F) is next written in phase 1, after the barrier that
        // follows the next cp.async wait.
        if constexpr (CUT)
          {
            tile    = t_next;
            gl      = gl_next;
            tm      = tm_next;
            m_glob  = m_glob_next;
            t_next  = t_nn;
            gl_next = gl_nn;
            tm_next = tm_nn;
          }
        else
          tile = nidx;
      }
    cp_async_wait<0>();
    if constexpr (CUT)
      siblings_end();
  }

  // -------------------------------------------------------------------------
  // FP32 Jacobian-vector product of few grains on tile pairs.  sm_100 executes
  // FP32 add, multiply and fused multiply-add on two values held in a 64-bit
  // register pair with one instruction (FADD2 / FMUL2 / FFMA2); the FP32
  // product is bound by instruction issue, so the block computes tiles 2j and
  // 2j + 1 together: every shared-memory value is a pair (lane x of tile 2j,
  // lane y of tile 2j + 1), phases 1-3 run once on F2 for both tiles, and the
  // node sums are stored per lane.  Each lane rounds exactly as the scalar FP32
  // arithmetic of the same expression does.  The full 3D operator without
  // advection, up to four grains (launch_jvp_full says why); shared memory and
  // registers as the FP64 product.
  // CUT (2D, G = 0 only): the grain cut-off's class of tiles without a relevant
  // grain, ct.tiles[ct.range[0] .. ct.range[1]), on c and mu; their owned nodes
  // get zero grain rows.
  // Resident blocks per SM: as the FP64 product (pairs take the FP64 product's
  // registers), but three for the class without grains, whose pairs need
  // ~70 registers (four blocks would cap them at 64 and spill).
  template <int DIM, int G, bool TENS>
  constexpr int jvp_pair_blocks_per_sm()
  {
    return G == 0 ? 3 : jvp_blocks_per_sm<DIM, G, TENS, double, false>();
  }

  template <int DIM, int G, bool TENS, bool CUT = false>
  __global__ void __launch_bounds__(Tile<DIM>::THREADS, jvp_pair_blocks_per_sm<DIM, G, TENS>())
    jvp_pair_kernel(const Grid g, const Phys ph, const float *__restrict__ lin, const float *__restrict__ src,
                    float *__restrict__ dst, float *__restrict__ partial, const CutTiles ct)
  {
    static_assert(!CUT || G == 0, "the cut-off pair kernel serves the class without grains");
    using T  = Tile<DIM>;
    using SM = ThreePhaseSmem<DIM, G, TENS, true, false, false, sizeof(F2)>;
    using FM = typename SM::FM;
    static_assert(G <= 4 && SM::BUFFERS == 2, "pairs serve few grains");
    constexpr int C = G + 2;
    if constexpr (CUT)
      siblings_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    F2 *s_buf = reinterpret_cast<F2 *>(smem_raw); // 2 x BOXES pairs
    F2 *F     = s_buf + 2 * SM::BOXES;
    F2 *P     = F + SM::P_AT;
    F2 *K     = F + SM::K_AT;

    const PhysR<F2>           p(ph);
    const CellConsts<DIM, F2> k(g);
    const NodePlan<DIM>       np(g);
    const int                 cell   = threadIdx.x % T::CELLS;
    // the tiles served: all of them, or the class-0 list of the cut-off
    const long long           i0     = CUT ? (long long)ct.range[0] : 0;
    const long long           nt     = CUT ? (long long)ct.range[1] - i0 : g.n_tiles;
    const long long           npairs = (nt + 1) / 2;
    auto tile_id = [&](long long i) -> long long { return CUT ? (long long)ct.tiles[i0 + i] : i; };
    long long                 idx    = blockIdx.x;
    // node boxes of both inputs of the tiles of pair j into buffer bb (a
    // missing second tile leaves its lane stale: computed, never stored)
    auto prefetch = [&](F2 *bb, long long j) {
#pragma unroll
      for (int lane = 0; lane < 2; ++lane)
        {
          if (2 * j + lane >= nt)
            break;
          const long long tile = tile_id(2 * j + lane);
          const TileCoord tcx  = tile_coord_of<DIM>(g, tile);
          float          *fb  = reinterpret_cast<float *>(bb) + lane;
          if (tile_interior<DIM>(g, tcx))
            {
              const long long n0 = tile_node0(g, tcx);
              load_box_async_interior<DIM, float, 2>(fb, lin, C, g, np, n0);
              load_box_async_interior<DIM, float, 2>(fb + 2 * C * T::BOXS, src, C, g, np, n0);
            }
          else
            {
              const BoxNode<DIM> bn(g, tcx);
              load_box_async<DIM, float, 2>(fb, lin, C, g, bn);
              load_box_async<DIM, float, 2>(fb + 2 * C * T::BOXS, src, C, g, bn);
            }
        }
    };
    if (idx < npairs)
      prefetch(s_buf, idx);
    cp_async_commit();
    for (int it = 0; idx < npairs; ++it, idx += gridDim.x)
      {
        const long long nidx = idx + gridDim.x;
        if (nidx < npairs)
          prefetch(s_buf + ((it + 1) & 1) * SM::BOXES, nidx);
        cp_async_commit();
        cp_async_wait<1>(); // this pair's group has landed (only the prefetch may be pending)
        __syncthreads();
        const bool      has_b  = 2 * idx + 1 < nt;
        const long long tile_a = tile_id(2 * idx), tile_b = has_b ? tile_id(2 * idx + 1) : tile_a;
        const TileCoord tca    = tile_coord_of<DIM>(g, tile_a);
        const TileCoord tcb    = tile_coord_of<DIM>(g, tile_b);
        const F2       *cb     = s_buf + (it & 1) * SM::BOXES;
        phase_evaluate<DIM, G, TENS, true, false, F2, false>(cb, cb + C * T::BOXS, F, k);
        __syncthreads();
        jvp_point<DIM, G, TENS, FM, F2>(p, F, P, threadIdx.x / T::CELLS, cell);
        __syncthreads();
        phase_integrate<DIM, G, FM, F2, false, false>(p, g, k, tca, P, cb + C * T::BOXS, K, ~0u, nullptr, nullptr,
                                                  &tcb);
        __syncthreads();
#pragma unroll
        for (int lane = 0; lane < 2; ++lane)
          {
            if (lane == 1 && !has_b)
              break;
            const TileCoord &tc = lane ? tcb : tca;
            const float     *kf = reinterpret_cast<const float *>(K) + lane;
            // CUT: c and mu are components 0 and 1 of the c_all-component
            // layout; no grain is relevant on the tile (union mask 0)
            if (tile_interior<DIM>(g, tc))
              sum_and_store_interior<DIM, float, 2>(kf, C, g, tc.linear, np, tile_node0(g, tc), dst, partial, 0, CUT,
                                                    ct.c_all, 0u);
            else
              sum_and_store<DIM, float, 2>(kf, C, g, tc, BoxNode<DIM>(g, tc), dst, partial, 0, CUT, ct.c_all, 0u);
          }
      }
    cp_async_wait<0>();
    if constexpr (CUT)
      siblings_end();
  }

  // -------------------------------------------------------------------------
  // Nonlinear residual: dst = R(src), SinteringOperatorGenericResidualQuad
  // (operator_sintering_generic.h:254-308) with the history of
  // do_evalute_history (:927-975) for WTD == 2: the weighted sum of the old
  // solutions is formed at the nodes while staging and evaluated at the points.
  // CUT: the kernel for G grains runs over the tiles of class G on their
  // compacted components, as the Jacobian product does.
  // ADV: with the advection terms of the grains' rigid-body velocities.
  template <int DIM, int G, bool TENS, int WTD, bool CUT, bool ADV = false>
  __global__ void __launch_bounds__(Tile<DIM>::THREADS, residual_blocks_per_sm<DIM, G, TENS, WTD == 2, ADV>())
    residual_kernel(const Grid g, const Phys ph, const double *__restrict__ src, const double *__restrict__ h0,
                    const double *__restrict__ h1, const double *__restrict__ h2, double *__restrict__ dst,
                    double *__restrict__ partial, const CutTiles ct, const AdvData adv)
  {
    using R  = double;
    using T  = Tile<DIM>;
    using SM = ThreePhaseSmem<DIM, G, TENS, false, WTD == 2, ADV, sizeof(double)>;
    using FM = typename SM::FM;
    using PL = ThreePhasePlan<DIM, G, TENS, false, WTD == 2, ADV, sizeof(double)>;
    constexpr int C = G + 2;
    if constexpr (CUT)
      siblings_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R *s_u = reinterpret_cast<R *>(smem_raw);
    R *s_h = s_u + C * T::BOXS;
    R *F   = s_u + SM::BOXES;
    R *P   = F + SM::P_AT;
    R *K   = F + SM::K_AT;
    R *A_vel = F + SM::F_SIZE + SM::P_SIZE;
    unsigned char *A_has = reinterpret_cast<unsigned char *>(A_vel + SM::ADV_VEL);

    const PhysR<R>           p(ph);
    const CellConsts<DIM, R> k(g);
    const NodePlan<DIM>      np(g);
    const long long          i0 = CUT ? (long long)ct.range[G] : 0;
    const long long          i1 = CUT ? (long long)ct.range[G + 1] : g.n_tiles;
    // The next tile's nodal values (this thread's box node, every NG-th
    // component) wait in registers while this tile's sums are stored: the
    // history is combined with arithmetic, so cp.async cannot stage it.  Not
    // with at most one grain, where finding the next tile ahead costs more than
    // the few loads it hides (one grain, scalar, no history, 96^3 cells: 178 us
    // ahead, 168 at the tile; cut-off class without grains, with advection, 136
    // and 125 us).
    constexpr bool AHEAD = G > 1;
    constexpr int  NV    = (C + T::NG - 1) / T::NG;
    R              rv[NV], rh[WTD == 2 ? NV : 1][3];
    auto           load = [&](const TileCoord &tc, bool interior, long long node0, unsigned long long gl) {
      if (!np.active)
        return;
      // in an interior tile the box node exists and reads itself
      bool      inside = true;
      long long lidx   = node0 + np.off;
      if (!interior)
        {
          const BoxNode<DIM> bn(g, tc);
          inside = bn.inside;
          lidx   = bn.lidx;
        }
#pragma unroll
      for (int n = 0; n < NV; ++n)
        {
          const int  comp = np.grp + n * T::NG;
          const bool on   = inside && comp < C;
          const long long off = on ? (CUT ? comp_of(comp, gl) : comp) * g.ld + lidx : 0;
          rv[n]               = on ? src[off] : R(0);
          if (on && ph.hooks.perturb) // the residual's perturbation hook: src + a x
            rv[n] += ph.hooks.perturb_scale * ph.hooks.perturb[off];
          if constexpr (WTD == 2)
            {
              // mu has no history
              const bool h = on && comp != 1;
              rh[n][0]     = h ? h0[off] : R(0);
              rh[n][1]     = h && ph.order > 1 ? h1[off] : R(0);
              rh[n][2]     = h && ph.order > 2 ? h2[off] : R(0);
            }
        }
    };
    auto load_ahead = [&](long long idx) {
      if (idx >= i1)
        return;
      const TileCoord tc = tile_coord_of<DIM>(g, CUT ? (long long)ct.tiles[idx] : idx);
      load(tc, tile_interior<DIM>(g, tc), tile_node0(g, tc), CUT ? ct.tile_grains[idx] : 0ull);
    };
    if constexpr (AHEAD)
      load_ahead(i0 + blockIdx.x);
    for (long long idx = i0 + blockIdx.x; idx < i1; idx += gridDim.x)
      {
        const long long          tile = CUT ? (long long)ct.tiles[idx] : idx;
        const unsigned long long gl   = CUT ? ct.tile_grains[idx] : 0ull;
        const unsigned           tm   = CUT ? ct.tile_mask[idx] : 0u;
        const TileCoord          tc   = tile_coord_of<DIM>(g, tile);
        const bool               interior = tile_interior<DIM>(g, tc);
        const long long          node0    = tile_node0(g, tc);
        const unsigned m = CUT ? local_mask<G>(cell_mask<DIM>(ct.cell_mask, g, tc, threadIdx.x % T::CELLS), gl) : ~0u;
        if constexpr (!AHEAD)
          load(tc, interior, node0, gl);
        if (np.active)
#pragma unroll
          for (int n = 0; n < NV; ++n)
            {
              const int comp = np.grp + n * T::NG;
              if (comp >= C)
                break;
              s_u[comp * T::BOXS + np.sb] = rv[n];
              // sum_i w_{i+1} u_old_i at the nodes (generic.h:947-966)
              if constexpr (WTD == 2)
                {
                  R hv = rh[n][0] * ph.w_hist[0];
                  if (ph.order > 1)
                    hv += rh[n][1] * ph.w_hist[1];
                  if (ph.order > 2)
                    hv += rh[n][2] * ph.w_hist[2];
                  s_h[comp * T::BOXS + np.sb] = hv;
                }
            }
        if constexpr (ADV)
          adv_stage<DIM, G, R, CUT>(adv, g, tc, gl, A_vel, A_has);
        __syncthreads();
        phase_evaluate<DIM, G, TENS, false, WTD == 2, R, CUT, PL::IN_PLACE>(s_u, s_h, F, k, m);
        __syncthreads();
        if constexpr (PL::IN_PLACE)
          residual_point_streamed<DIM, G, TENS, WTD, FM, R>(p, F, threadIdx.x / T::CELLS, threadIdx.x % T::CELLS, m);
        else
          residual_point<DIM, G, TENS, WTD, FM, R>(p, F, P, threadIdx.x / T::CELLS, threadIdx.x % T::CELLS, m);
        if constexpr (ADV)
          {
            advect_c_point<DIM, G, R, CUT>(k, g, F, FM::base(FM::lin_c), P, threadIdx.x / T::CELLS,
                                           threadIdx.x % T::CELLS, m, A_vel, A_has);
          }
        __syncthreads();
        phase_integrate<DIM, G, FM, R, CUT, ADV>(p, g, k, tc, P, s_u, K, m, A_vel, A_has);
        __syncthreads();
        if constexpr (AHEAD)
          load_ahead(idx + gridDim.x);
        if (interior)
          sum_and_store_interior<DIM>(K, C, g, tc.linear, np, node0, dst, partial, gl, CUT, ct.c_all, tm, &ph.hooks);
        else
          sum_and_store<DIM>(K, C, g, tc, BoxNode<DIM>(g, tc), dst, partial, gl, CUT, ct.c_all, tm, &ph.hooks);
        // no barrier: the next tile's staging writes the boxes, read last in
        // phase 3 before the barrier above; K (aliasing F) is next written in
        // phase 1, after the barrier that follows the staging
      }
    if constexpr (CUT)
      siblings_end();
  }

  // -------------------------------------------------------------------------
  // Preconditioner diagonals at the linearisation point (FP64), G + 4 outputs:
  //   [0..3] node-diagonal 2x2 block of the Cahn-Hilliard tangent
  //          (OperatorCahnHilliard, sintering/preconditioners.h:110-168):
  //          J_cc, J_c,mu, J_mu,c, J_mu,mu
  //   [4..]  diagonal of OperatorAllenCahn (preconditioners.h:364-394)
  // Each thread first computes its point's coefficients (mobility matrix M,
  // dM/dc grad mu, dM/dgrad c, f_cc, f_eta_i eta_i), then, as the owner of
  // local node l, sums phi_l / grad phi_l weighted terms over the cell's points.
  template <int DIM, int G, bool TENS, bool ADV = false>
  struct DiagLayout
  {
    static constexpr int NOUT  = G + 4;
    static constexpr int NADV  = ADV ? G * DIM : 0; // the grains' velocities at the point
    static constexpr int NCOEF = DIM * DIM + DIM + DIM * DIM + 1 + G + NADV;
  };

  // CUT: the grains absent on a cell (mask bit clear) have zero values there
  // and no Allen-Cahn diagonal contribution from it (preconditioners.h:787-817).
  // ADV: the advection terms of the preconditioner's operators
  // (precondition_advection_ch / _ac, operator_sintering_generic.h:800-850):
  // J_cc gains -(phi_l sum_i v_i, grad phi_l) and grain i's diagonal
  // -(phi_l v_i, grad phi_l), with the velocities of the current table.
  template <int DIM, int G, bool TENS, bool CUT, bool ADV = false>
  __global__ void __launch_bounds__(Tile<DIM>::THREADS)
    diag_kernel(const Grid g, const Phys ph, const double *__restrict__ lin, double *__restrict__ dst,
                double *__restrict__ partial, const uint16_t *__restrict__ mask, const AdvData adv)
  {
    using R          = double;
    using T          = Tile<DIM>;
    using LY         = DiagLayout<DIM, G, TENS, ADV>;
    constexpr int C  = G + 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R *s_lin  = reinterpret_cast<R *>(smem_raw);
    R *s_coef = s_lin + C * T::BOXS;
    R *s_con  = s_coef + LY::NCOEF * T::THREADS; // NOUT * CS

    const TileCoord    tc = tile_coord<DIM>(g);
    const BoxNode<DIM> bn(g, tc);
    load_box<DIM>(s_lin, lin, C, g, bn);
    __syncthreads();

    const PhysR<R>   p(ph);
    const QP<DIM, R> w(g);
    const int        cell  = threadIdx.x / T::NQ;
    const int        b0    = cell_box_base<DIM>(cell);
    const bool       valid = cell_in_mesh<DIM>(cell, tc, g);
    const unsigned   gmask = CUT ? cell_mask<DIM>(mask, g, tc, cell) : ~0u;

    {
      R c, gc[DIM], mu_unused, gmu[DIM];
      eval_vg<DIM>(s_lin, b0, w, c, gc);
      eval_vg<DIM>(s_lin + T::BOXS, b0, w, mu_unused, gmu);
      R eta[G];
      R geta[G][DIM];
#pragma unroll
      for (int i = 0; i < G; ++i)
        {
          eval_vg<DIM>(s_lin + (2 + i) * T::BOXS, b0, w, eta[i], geta[i]);
          if (CUT && ((gmask >> i) & 1u) == 0u)
            {
              eta[i] = R(0);
#pragma unroll
              for (int d = 0; d < DIM; ++d)
                geta[i][d] = R(0);
            }
        }
      R *cf = s_coef + threadIdx.x * LY::NCOEF;
      // mobility matrix (M grad mu = apply_M(grad mu)) in one pass over the
      // grain pairs; absent grains (CUT) enter with zero values
      {
        R Mm[DIM][DIM];
        mobility_matrix<DIM, G, TENS>(p, c, eta, gc, geta, Mm);
#pragma unroll
        for (int a = 0; a < DIM; ++a)
#pragma unroll
          for (int b = 0; b < DIM; ++b)
            cf[a * DIM + b] = Mm[a][b];
      }
      R m[DIM];
      dM_dc_times<DIM, TENS>(p, c, gc, gmu, m);
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        cf[DIM * DIM + d] = m[d];
      R K[DIM][DIM];
      dM_dgrad_c<DIM, TENS>(p, c, gc, gmu, K);
#pragma unroll
      for (int a = 0; a < DIM; ++a)
#pragma unroll
        for (int b = 0; b < DIM; ++b)
          cf[DIM * DIM + DIM + a * DIM + b] = K[a][b];
      const R omc = R(1) - c;
      R       s2  = R(0);
#pragma unroll
      for (int i = 0; i < G; ++i)
        s2 += eta[i] * eta[i];
      cf[2 * DIM * DIM + DIM] =
        R(2) * p.A * (c * c) + R(4) * p.A * c * (R(2) * c - R(2)) + R(2) * p.A * (omc * omc) + R(2) * p.B;
#pragma unroll
      for (int i = 0; i < G; ++i)
        {
          const R e = eta[i];
          cf[2 * DIM * DIM + DIM + 1 + i] =
            p.B * (R(12) - R(12) * c + R(2) * e * (R(12) * c - R(24)) + R(24) * (e * e) + R(12) * s2);
        }
      if constexpr (ADV)
        {
          // velocity of every grain at this thread's point (zero without a segment)
          R        *vc = cf + 2 * DIM * DIM + DIM + 1 + G;
          int       cc[3];
          const int q  = threadIdx.x & (T::NQ - 1);
          const bool in = cell_global<DIM>(cell, tc, g, cc);
          const long long n_cells = (long long)g.n[0] * g.n[1] * g.n[2];
          const long long lin_cell = cc[0] + (long long)g.n[0] * (cc[1] + (long long)g.n[1] * cc[2]);
          const double gp0 = 0.5 - 0.5 / sqrt(3.0), gp1 = 0.5 + 0.5 / sqrt(3.0);
#pragma unroll 1
          for (int i = 0; i < G; ++i)
            {
              int s = -1;
              if (in && (!CUT || ((gmask >> i) & 1u)))
                {
                  s = adv.cell_segments[i * n_cells + lin_cell];
                  if (s >= adv.n_segments)
                    s = -1;
                }
              R v[3] = {R(0), R(0), R(0)};
              if (s >= 0)
                {
                  const double *d    = adv.segments + 9 * (long long)s;
                  double        r[3] = {0.0, 0.0, 0.0};
#pragma unroll
                  for (int e = 0; e < DIM; ++e)
                    r[e] = adv.origin[e] + (cc[e] + (((q >> e) & 1) ? gp1 : gp0)) * g.h[e] - d[6 + e];
                  v[0] = d[0] + d[4] * r[2] - d[5] * r[1];
                  v[1] = d[1] + d[5] * r[0] - d[3] * r[2];
                  v[2] = d[2] + d[3] * r[1] - d[4] * r[0];
                }
#pragma unroll
              for (int e = 0; e < DIM; ++e)
                vc[i * DIM + e] = v[e];
            }
        }
    }
    __syncthreads();

    {
      // this thread is the owner of local node l = lane bits
      const int l = threadIdx.x & (T::NQ - 1);
      R         acc[LY::NOUT];
#pragma unroll
      for (int k = 0; k < LY::NOUT; ++k)
        acc[k] = R(0);
      for (int q = 0; q < T::NQ; ++q)
        {
          const R *cf = s_coef + (cell * T::NQ + q) * LY::NCOEF;
          // phi_l(x_q) and grad phi_l(x_q)
          R phi = R(1), dphi[DIM];
#pragma unroll
          for (int d = 0; d < DIM; ++d)
            {
              const int ld = (l >> d) & 1, qd = (q >> d) & 1;
              phi *= (ld == qd) ? w.g1 : w.g0;
            }
#pragma unroll
          for (int d = 0; d < DIM; ++d)
            {
              R v = (((l >> d) & 1) ? R(1) : R(-1)) * w.ih[d];
#pragma unroll
              for (int e = 0; e < DIM; ++e)
                if (e != d)
                  v *= (((l >> e) & 1) == ((q >> e) & 1)) ? w.g1 : w.g0;
              dphi[d] = v;
            }
          const R *Mm = cf;
          const R *mv = cf + DIM * DIM;
          const R *Km = cf + DIM * DIM + DIM;
          const R  fcc = cf[2 * DIM * DIM + DIM];
          R        gg = R(0), MphiPhi = R(0), KphiPhi = R(0), mphi = R(0);
#pragma unroll
          for (int a = 0; a < DIM; ++a)
            {
              gg += dphi[a] * dphi[a];
              mphi += mv[a] * dphi[a];
#pragma unroll
              for (int b = 0; b < DIM; ++b)
                {
                  MphiPhi += dphi[a] * Mm[a * DIM + b] * dphi[b];
                  KphiPhi += dphi[a] * Km[a * DIM + b] * dphi[b];
                }
            }
          const R pp = phi * phi;
          acc[0] += w.JxW * (p.w0 * pp + phi * mphi + KphiPhi);
          acc[1] += w.JxW * MphiPhi;
          acc[2] += w.JxW * (-fcc * pp - p.kc * gg);
          acc[3] += w.JxW * (p.walg * pp);
#pragma unroll
          for (int i = 0; i < G; ++i)
            acc[4 + i] += w.JxW * ((p.w0 + p.L * cf[2 * DIM * DIM + DIM + 1 + i]) * pp + p.L * p.kp * gg);
          if constexpr (ADV)
            {
              const R *vc = cf + 2 * DIM * DIM + DIM + 1 + G;
#pragma unroll
              for (int i = 0; i < G; ++i)
                {
                  R vd = R(0);
#pragma unroll
                  for (int e = 0; e < DIM; ++e)
                    vd += vc[i * DIM + e] * dphi[e];
                  acc[0] -= w.JxW * phi * vd;
                  acc[4 + i] -= w.JxW * phi * vd;
                }
            }
        }
#pragma unroll
      for (int i = 0; i < G; ++i)
        if (CUT && ((gmask >> i) & 1u) == 0u)
          acc[4 + i] = R(0);
#pragma unroll
      for (int k = 0; k < LY::NOUT; ++k)
        store_contrib<DIM>(s_con, k, acc[k], valid);
    }
    __syncthreads();
    sum_and_store<DIM>(s_con, LY::NOUT, g, tc, bn, dst, partial);
  }
} // namespace sint
