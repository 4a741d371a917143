// One-kernel 2D cell loop of the full operator (no grain cut-off, no
// advection): Jacobian-vector product and residual.
//
// The tiled kernels of sint_kernels.cuh share a cell's work among threads
// through shared memory in three barrier-separated phases and leave the
// tile-face nodes to a second launch.  In 2D a cell has four nodes and four
// points, so one thread can carry a whole cell in registers, and overlapping
// the tiles by one row and one column of cells costs less than the second
// launch and its partial sums: a block of TX x TY threads computes TX x TY
// cells and owns the (TX - 1) x (TY - 1) nodes whose four cells it has.
//
// What bounds it: instruction issue (FP32) and the FP64 pipe (57 % and 63 %
// busy at 512 x 512 cells, the rest is the ramp of each block's loads and the
// last wave).  16 x 8 threads recompute 22 % of the cells; 16 x 16 recompute
// 14 % but balance worse over the SMs and overlap loads and arithmetic less
// (two blocks per SM instead of four): when the tile was chosen, 512 x 512, FP32
// scalar J v of 8 grains 35.1 us against 39.9 us; 256 x 128, FP64 tensorial J v
// of 3 grains 10.6 us against 12.6 us.  Those two take 31.5 and 7.1 us today;
// the tiled kernels with their combine launch took 55.3 and 11.8 us.
#pragma once

#include "sint_kernels.cuh"
#include "sint_launch.h"

namespace sint
{
  // MODE: -1 = Jacobian-vector product, 0..2 = residual with_time_derivative.
  template <int G, int MODE>
  struct Fused2D
  {
    static constexpr int  TX = 16, TY = 8;
    static constexpr int  C   = G + 2;
    static constexpr bool JVP = MODE < 0;
    static constexpr int  P   = TX + 1;            // row pitch of a staged field
    static constexpr int  BOX = P * (TY + 1);      // nodes of the cells' box
    // staged fields: the state (C), then the direction (C), or for
    // with_time_derivative 2 the time term w0 u + sum_i w_i u_old_i of c and
    // the eta_i (1 + G)
    static constexpr int NF = C + (JVP ? C : (MODE == 2 ? 1 + G : 0));
    static constexpr int T0 = C; // first field of the second group
    __host__ __device__ static constexpr int t_of(int comp) { return JVP ? T0 + comp : T0 + (comp == 0 ? 0 : comp - 1); }
    static constexpr int ROWS    = C * TX * TY;    // upper-node sums handed to the next cell row
    static constexpr int THREADS = TX * TY;
    template <typename R>
    static constexpr size_t smem()
    {
      return size_t(NF * BOX + ROWS) * sizeof(R);
    }
  };

  // Input vectors of one launch: a = the linearisation point or the state,
  // b = the direction (J v), h = the old solutions (residual).
  template <typename R>
  struct Fused2DArgs
  {
    const R *a, *b, *h[3];
    R       *dst;
    int      blocks_x; // blocks per row of blocks
  };

  // Resident blocks per SM the registers are shared out for.  Four blocks leave
  // 128 registers a thread, and the point physics of more grains spill there
  // (bytes stored per thread: FP32 J v tensorial from 28 for 7 grains to 536 for
  // 12, scalar from 16 for 8 to 136 for 12; FP64 tensorial 56 for 3, scalar 80
  // and 152 for 4 and 5).  Spills cost most on meshes of about one block per
  // SM, where nothing hides them.  Device time in us of the FP32 tensorial J v,
  // four / three blocks: 128 x 128 cells 14.7 / 11.5 (8 grains), 27.9 / 22.2
  // (12), where the tiled kernels take 14.8 and 26.9; 512 x 512 64.8 / 62.6 and
  // 140.8 / 126.8; 7 grains 1024 x 1024 202 / 205.  Of the FP64 tensorial J v
  // of 3 grains, four / two blocks: 136 x 136 9.1 / 5.3 (tiled 8.7), 1024 x
  // 1024 134.7 / 132.1; its residual 124.1 / 129.7 there, so it keeps four.
  template <int G, bool TENS, typename R, int MODE>
  constexpr int fused2d_blocks()
  {
    return sizeof(R) == 4 ? (TENS && G >= 8 ? 3 : 4) : G <= (TENS ? (MODE < 0 ? 2 : 3) : 5) ? 4 : 2;
  }

  template <int G, bool TENS, typename R, int MODE>
  __global__ void __launch_bounds__(Fused2D<G, MODE>::THREADS, fused2d_blocks<G, TENS, R, MODE>())
    fused2d_kernel(const Grid g, const Phys ph, const Fused2DArgs<R> args)
  {
    using L = Fused2D<G, MODE>;
    constexpr int  C = L::C, P = L::P, TX = L::TX, TY = L::TY;
    constexpr bool JVP = L::JVP;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    dependent_start();
    R *box = reinterpret_cast<R *>(smem_raw); // [field][node]
    R *up  = box + L::NF * L::BOX;            // [row][cell]: sums of the cell's upper nodes

    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int bx = blockIdx.x % args.blocks_x, by = blockIdx.x / args.blocks_x;
    // cell (0, 0) of the block: one before the first owned node
    const int ox = bx * (TX - 1) - 1, oy = by * (TY - 1) - 1;

    // node box, all loads of a thread in flight together; nodes outside the
    // mesh read as zero, periodic slaves read their master
#pragma unroll
    for (int it = 0; it < (L::BOX + L::THREADS - 1) / L::THREADS; ++it)
      {
        const int n = threadIdx.x + it * L::THREADS;
        if (n < L::BOX)
          {
            int        i  = ox + n % P, j = oy + n / P;
            const bool in = i >= 0 && j >= 0 && i < g.nn[0] && j < g.nn[1];
            if ((g.periodic & 1) && i == g.n[0])
              i = 0;
            if ((g.periodic & 2) && j == g.n[1])
              j = 0;
            const long long node = in ? node_index(g, i, j, 0) : 0;
            R               v[L::NF];
#pragma unroll
            for (int f = 0; f < C; ++f)
              {
                v[f] = in ? args.a[f * g.ld + node] : R(0);
                if constexpr (JVP)
                  v[L::T0 + f] = in ? args.b[f * g.ld + node] : R(0);
              }
            if constexpr (!JVP)
              {
                if (ph.hooks.perturb) // the residual's perturbation hook: src + a x
                  {
#pragma unroll
                    for (int f = 0; f < C; ++f)
                      if (in)
                        v[f] += ph.hooks.perturb_scale * ph.hooks.perturb[f * g.ld + node];
                  }
                // the time term at the nodes (generic.h:947-966); mu has none
                if constexpr (MODE == 2)
                  {
#pragma unroll
                    for (int f = 0; f < C; ++f)
                      if (f != 1)
                        {
                          R h = in ? args.h[0][f * g.ld + node] * ph.w_hist[0] : R(0);
                          if (in && ph.order > 1)
                            h += args.h[1][f * g.ld + node] * ph.w_hist[1];
                          if (in && ph.order > 2)
                            h += args.h[2][f * g.ld + node] * ph.w_hist[2];
                          v[L::t_of(f)] = v[f] * ph.w0 + h;
                        }
                  }
              }
#pragma unroll
            for (int f = 0; f < L::NF; ++f)
              box[f * L::BOX + n] = v[f];
          }
      }
    __syncthreads();

    const PhysR<R>         p(ph);
    const CellConsts<2, R> k(g);
    const R               *cell = box + ty * P + tx; // the cell's lower left node

    // row r of the cell's four nodes, l = lx + 2 ly
    R acc[C][4];
#pragma unroll
    for (int r = 0; r < C; ++r)
#pragma unroll
      for (int l = 0; l < 4; ++l)
        acc[r][l] = R(0);

    // the point loops stay loops: unrolled, the compiler holds both columns of
    // points (and their interpolated fields) in registers at once
#pragma unroll 1
    for (int qx = 0; qx < 2; ++qx)
      {
        asm volatile("" ::: "memory"); // reread the box: hoisted loads would live across the whole loop
        // phi_1 and phi_0 of the 1D shape functions at x_qx
        const R px1 = qx ? k.x1 : k.x0, px0 = qx ? k.x0 : k.x1;
        // every field interpolated to x_qx: on the lower cell edge, and the
        // difference of the upper edge to it
        R a0[L::NF], ad[L::NF];
#pragma unroll
        for (int f = 0; f < L::NF; ++f)
          {
            const R *u = cell + f * L::BOX;
            a0[f]      = u[0] + px1 * (u[1] - u[0]);
            ad[f]      = u[P] + px1 * (u[P + 1] - u[P]) - a0[f];
          }
#pragma unroll 1
        for (int qy = 0; qy < 2; ++qy)
          {
            asm volatile("" ::: "memory");
            const R py1 = qy ? k.x1 : k.x0, py0 = qy ? k.x0 : k.x1;
            auto    val = [&](int f) -> R { return a0[f] + py1 * ad[f]; };
            auto    grad = [&](int f, R(&o)[2]) {
              const R *u  = cell + f * L::BOX;
              const R  d0 = u[1] - u[0], d1 = u[P + 1] - u[P];
              o[0]        = (d0 + py1 * (d1 - d0)) * k.ih[0];
              o[1]        = ad[f] * k.ih[1];
            };
            // weights of the four nodes: JxW phi_l and JxW d phi_l / dx_d
            R w[4], wd[2][4];
#pragma unroll
            for (int l = 0; l < 4; ++l)
              {
                const R px = (l & 1) ? px1 : px0, py = (l >> 1) ? py1 : py0;
                w[l]       = px * py * k.JxW;
                wd[0][l]   = ((l & 1) ? k.ih[0] : -k.ih[0]) * py * k.JxW;
                wd[1][l]   = ((l >> 1) ? k.ih[1] : -k.ih[1]) * px * k.JxW;
              }
            auto emit = [&](int res, R v) {
#pragma unroll
              for (int l = 0; l < 4; ++l)
                if (res >= 1 && res <= 2)
                  acc[0][l] += wd[res == 2][l] * v;
                else
                  acc[res == 0 ? 0 : res - 2][l] += w[l] * v;
            };
            R c = val(0), gc[2], gmu[2], eta[gdim(G)], geta[TENS ? gdim(G) : 1][2];
            grad(1, gmu);
            if constexpr (TENS)
              grad(0, gc);
#pragma unroll
            for (int i = 0; i < G; ++i)
              {
                eta[i] = val(2 + i);
                if constexpr (TENS)
                  grad(2 + i, geta[i]);
              }
            if constexpr (JVP)
              {
                R gdc[2], gdmu[2], deta[gdim(G)];
                if constexpr (TENS)
                  grad(L::T0, gdc);
                grad(L::T0 + 1, gdmu);
#pragma unroll
                for (int i = 0; i < G; ++i)
                  deta[i] = val(L::T0 + 2 + i);
                jvp_terms<2, G, TENS, R>(p, c, gc, gmu, eta, geta, val(L::T0), gdc, val(L::T0 + 1), gdmu, deta, ~0u,
                                         emit);
              }
            else
              residual_terms<2, G, TENS, R>(
                p, c, gc, val(1), gmu, eta, geta, ~0u,
                [&](int i, R v) {
                  if constexpr (MODE == 1)
                    v += (i < 0 ? c : eta[i < 0 ? 0 : i]) * p.w0;
                  if constexpr (MODE == 2)
                    v += val(L::t_of(i < 0 ? 0 : 2 + i));
                  return v;
                },
                emit);
          }
      }
    // constant-coefficient gradient terms with the exact element Laplacian:
    // -kappa_c on c for the mu row, L kappa_p on eta_i for the eta_i row
#pragma unroll
    for (int r = 1; r < C; ++r)
      {
        const R *s = cell + ((JVP ? L::T0 : 0) + (r == 1 ? 0 : r)) * L::BOX;
        const R  u[4] = {s[0], s[1], s[P], s[P + 1]};
        if (r == 1)
          cell_stiffness_add<2, 0>(u, g, acc[r]);
        else
          cell_stiffness_add<2, 1>(u, g, acc[r]);
      }

    const int  cx = ox + tx, cy = oy + ty;
    const bool valid = cx >= 0 && cy >= 0 && cx < g.n[0] && cy < g.n[1];
    const bool owner = tx > 0 && ty > 0 && cx < g.nn[0] && cy < g.nn[1];
    const long long node = owner ? node_index(g, cx, cy, 0) : 0;
    // node (cx, cy) = this cell's node 0, the left cell's node 1 and the
    // lower cells' nodes 2 and 3: x neighbours by shuffle, y through `up`
    R low[C];
#pragma unroll
    for (int r = 0; r < C; ++r)
      {
#pragma unroll
        for (int l = 0; l < 4; ++l)
          if (!valid)
            acc[r][l] = R(0);
        low[r] = acc[r][0] + __shfl_up_sync(0xffffffffu, acc[r][1], 1, TX);
        up[r * L::THREADS + threadIdx.x] = acc[r][2] + __shfl_up_sync(0xffffffffu, acc[r][3], 1, TX);
      }
    __syncthreads();
    if (!owner)
      return;
#pragma unroll
    for (int r = 0; r < C; ++r)
      {
        R v = up[r * L::THREADS + threadIdx.x - TX] + low[r];
        if constexpr (!JVP)
          if (ph.hooks.epilogue) // (R - subtract) * scale
            v = (v - (ph.hooks.subtract ? R(ph.hooks.subtract[r * g.ld + node]) : R(0))) * R(ph.hooks.scale);
        args.dst[r * g.ld + node] = v;
      }
  }
} // namespace sint
