// The grain cut-off's class of 3D tiles without a relevant grain (c and mu
// only, most of a packing): one warp per tile, one lane per cell.
//
// The block kernels spread a cell over eight threads and pay barriers,
// shared-memory round trips of the point fields and a per-item dispatch for
// two rows of output.  Four fields of a cell fit a thread's registers, so here
// a lane evaluates its whole cell and only the nodes pass through shared
// memory; warps share nothing, so there is no block barrier and the next
// tile's nodes are copied (cp.async) while this tile is computed.
#pragma once

#include "sint_kernels.cuh"

namespace sint
{
  // MODE: -1 = Jacobian-vector product, 0..2 = residual with_time_derivative.
  template <int MODE>
  struct LightTile
  {
    using T = Tile<3>;
    static constexpr bool JVP = MODE < 0;
    // staged fields: c and mu of the state, then c and mu of the direction, or
    // the time term w0 c + sum_i w_i c_old_i (with_time_derivative 2)
    static constexpr int NF    = JVP ? 4 : (MODE == 2 ? 3 : 2);
    static constexpr int NBUF  = JVP ? 2 : 1; // the product double-buffers its boxes
    static constexpr int BOX   = NF * T::BOXS;
    static constexpr int KSZ   = 2 * T::CS; // node contributions of the two rows
    static constexpr int WARPS = 4;
    static constexpr int SLOTS = (T::BOX + 31) / 32; // box nodes per lane
    template <typename R>
    static constexpr size_t smem()
    {
      return size_t(WARPS) * (NBUF * BOX + KSZ) * sizeof(R);
    }
  };

  template <typename R>
  struct LightArgs
  {
    const R      *a, *b; // state (or linearisation point), direction
    const double *h[3];  // old solutions (residual)
    R            *dst, *partial;
  };

  // The box nodes a lane serves: node lane + 32 s of the tile's box.
  template <int SLOTS>
  struct LightPlan
  {
    int      sb[SLOTS], off[SLOTS], cbase[SLOTS];
    unsigned ok[SLOTS];
    bool     inner[SLOTS];

    __device__ __forceinline__ explicit LightPlan(const Grid &g)
    {
      using T = Tile<3>;
#pragma unroll
      for (int s = 0; s < SLOTS; ++s)
        {
          const int b  = (threadIdx.x & 31) + 32 * s;
          const int bx = b % T::BX, by = (b / T::BX) % T::BY, bz = b / (T::BX * T::BY);
          sb[s]    = bx + T::SY * by + T::SZ * bz;
          off[s]   = bx + g.nn[0] * (by + g.nn[1] * bz);
          cbase[s] = bx + T::TX * (by + T::TY * bz);
          inner[s] = bx > 0 && bx < T::TX && by > 0 && by < T::TY && bz > 0 && bz < T::TZ;
          ok[s]    = 0u;
#pragma unroll
          for (int l = 0; l < T::NQ; ++l)
            {
              const int cx = bx - (l & 1), cy = by - ((l >> 1) & 1), cz = bz - (l >> 2);
              if (b < T::BOX && cx >= 0 && cx < T::TX && cy >= 0 && cy < T::TY && cz >= 0 && cz < T::TZ)
                ok[s] |= 1u << l;
            }
        }
    }
  };

  // Resident blocks per SM: the FP32 product takes 128 registers, the FP64
  // product 239, the FP64 residual fits 168.  (Tried on the FP32 product of a
  // 256^3 packing, all classes together: packed FP32 pairs of tiles, 255
  // registers, 2.41 ms, 168 with spills 2.48 ms; one line of two points at a
  // time, 96 registers, 2.36 ms; this form 2.21 ms, and 2.09 ms since the classes
  // run beside one another.)
  template <typename R, int MODE>
  constexpr int light_blocks()
  {
    return sizeof(R) == 4 ? 4 : (MODE < 0 ? 2 : 3);
  }

  template <bool TENS, typename R, int MODE>
  __global__ void __launch_bounds__(LightTile<MODE>::WARPS * 32, light_blocks<R, MODE>())
    light_kernel(const Grid g, const Phys ph, const LightArgs<R> args, const CutTiles ct)
  {
    using T             = Tile<3>;
    using L             = LightTile<MODE>;
    constexpr bool JVP  = L::JVP;
    constexpr int  S    = L::SLOTS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    siblings_begin();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    R        *buf  = reinterpret_cast<R *>(smem_raw) + warp * (L::NBUF * L::BOX + L::KSZ);
    R        *K    = buf + L::NBUF * L::BOX;

    const LightPlan<S>     np(g);
    const PhysR<R>         p(ph);
    const CellConsts<3, R> k(g);
    const int              b0     = cell_box_base<3>(lane);
    const int              i0     = ct.range[0], i1 = ct.range[1];
    const int              stride = gridDim.x * L::WARPS;
    int                    idx    = i0 + blockIdx.x * L::WARPS + warp;

    // node s of the lane in tile tc: whether it exists, and where it is read
    auto node_of = [&](const TileCoord &tc, int s, bool &inside) -> long long {
      const int b  = lane + 32 * s;
      const int gi = tc.o[0] + b % T::BX, gj = tc.o[1] + (b / T::BX) % T::BY, gk = tc.o[2] + b / (T::BX * T::BY);
      inside       = b < T::BOX && gi < g.nn[0] && gj < g.nn[1] && gk < g.nn[2];
      if (!inside)
        return 0;
      return node_index(g, ((g.periodic & 1) && gi == g.n[0]) ? 0 : gi, ((g.periodic & 2) && gj == g.n[1]) ? 0 : gj,
                        ((g.periodic & 4) && gk == g.n[2]) ? 0 : gk);
    };
    auto prefetch = [&](R *bb, int tile) {
      const TileCoord tc       = tile_coord_of<3>(g, tile);
      const bool      interior = tile_interior<3>(g, tc);
      const long long n0       = tile_node0(g, tc);
#pragma unroll
      for (int s = 0; s < S; ++s)
        {
          bool      in   = lane + 32 * s < T::BOX;
          long long node = in ? n0 + np.off[s] : 0;
          if (!interior)
            node = node_of(tc, s, in);
          if (lane + 32 * s < T::BOX)
            {
              cp_async_elem(bb + np.sb[s], args.a + node, in);
              cp_async_elem(bb + T::BOXS + np.sb[s], args.a + g.ld + node, in);
              cp_async_elem(bb + 2 * T::BOXS + np.sb[s], args.b + node, in);
              cp_async_elem(bb + 3 * T::BOXS + np.sb[s], args.b + g.ld + node, in);
            }
        }
    };
    // this warp's tile and the next one, read ahead
    int tile = idx < i1 ? ct.tiles[idx] : 0;
    int next = idx + stride < i1 ? ct.tiles[idx + stride] : 0;
    if constexpr (JVP)
      {
        if (idx < i1)
          prefetch(buf, tile);
        cp_async_commit();
      }
    for (int it = 0; idx < i1; ++it, idx += stride)
      {
        const int       next2    = idx + 2 * stride < i1 ? ct.tiles[idx + 2 * stride] : 0;
        const TileCoord tc       = tile_coord_of<3>(g, tile);
        const bool      interior = tile_interior<3>(g, tc);
        const long long n0       = tile_node0(g, tc);
        const R *cb = buf + (JVP ? (it & 1) * L::BOX : 0);
        if constexpr (JVP)
          {
            if (idx + stride < i1)
              prefetch(buf + ((it + 1) & 1) * L::BOX, next);
            cp_async_commit();
            cp_async_wait<1>(); // this tile's copies have landed (only the prefetch may be pending)
          }
        else
          {
#pragma unroll
            for (int s = 0; s < S; ++s)
              {
                bool      in   = lane + 32 * s < T::BOX;
                long long node = in ? n0 + np.off[s] : 0;
                if (!interior)
                  node = node_of(tc, s, in);
                if (lane + 32 * s < T::BOX)
                  {
                    R c = in ? args.a[node] : R(0), mu = in ? args.a[g.ld + node] : R(0);
                    if (ph.hooks.perturb && in) // the residual's perturbation hook: src + a x
                      {
                        c += ph.hooks.perturb_scale * ph.hooks.perturb[node];
                        mu += ph.hooks.perturb_scale * ph.hooks.perturb[g.ld + node];
                      }
                    buf[np.sb[s]]           = c;
                    buf[T::BOXS + np.sb[s]] = mu;
                    if constexpr (MODE == 2)
                      {
                        // the time term at the nodes (operator_sintering_generic.h:947-966)
                        R h = in ? args.h[0][node] * ph.w_hist[0] : R(0);
                        if (in && ph.order > 1)
                          h += args.h[1][node] * ph.w_hist[1];
                        if (in && ph.order > 2)
                          h += args.h[2][node] * ph.w_hist[2];
                        buf[2 * T::BOXS + np.sb[s]] = c * ph.w0 + h;
                      }
                  }
              }
          }
        __syncwarp();

        // the lane's cell: rows c and mu at its eight nodes
        R acc[2][8];
#pragma unroll
        for (int l = 0; l < 8; ++l)
          acc[0][l] = acc[1][l] = R(0);
        const R *u = cb + b0;
        auto     nv = [&](int f, int l) { // nodal value
          return u[f * T::BOXS + (l & 1) + T::SY * ((l >> 1) & 1) + T::SZ * (l >> 2)];
        };
#pragma unroll 1
        for (int qz = 0; qz < 2; ++qz)
          {
            asm volatile("" ::: "memory"); // reread the box: hoisted loads would live across the loop
            const R pz1 = qz ? k.x1 : k.x0, pz0 = qz ? k.x0 : k.x1;
            // per field the four x-y corners at z_qz, and their z differences
            R a[L::NF][4], dz[L::NF][4];
#pragma unroll
            for (int f = 0; f < L::NF; ++f)
#pragma unroll
              for (int c = 0; c < 4; ++c)
                {
                  const R lo = nv(f, c);
                  dz[f][c]   = nv(f, c + 4) - lo;
                  a[f][c]    = lo + pz1 * dz[f][c];
                }
            // this layer's sums to the x-y corners: values with x and y fluxes, z flux, mu row
            R cv[4], cz[4], mv[4];
#pragma unroll
            for (int c = 0; c < 4; ++c)
              cv[c] = cz[c] = mv[c] = R(0);
#pragma unroll
            for (int qy = 0; qy < 2; ++qy)
              {
                const R py1 = qy ? k.x1 : k.x0, py0 = qy ? k.x0 : k.x1;
                // sums of this line of two points, to its ends in x: values, x flux,
                // y flux, z flux, mu row
                R lv[2], lx = R(0), ly[2], lz[2], lm[2];
                lv[0] = lv[1] = ly[0] = ly[1] = lz[0] = lz[1] = lm[0] = lm[1] = R(0);
#pragma unroll
                for (int qx = 0; qx < 2; ++qx)
                  {
                    const R px1 = qx ? k.x1 : k.x0, px0 = qx ? k.x0 : k.x1;
                    auto    xy  = [&](const R(&v)[4]) -> R { // bilinear at the point
                      const R v0 = v[0] + py1 * (v[2] - v[0]), v1 = v[1] + py1 * (v[3] - v[1]);
                      return v0 + px1 * (v1 - v0);
                    };
                    auto grad = [&](int f, R(&o)[3]) {
                      const R x0 = a[f][1] - a[f][0], x1 = a[f][3] - a[f][2];
                      const R y0 = a[f][2] - a[f][0], y1 = a[f][3] - a[f][1];
                      o[0] = (x0 + py1 * (x1 - x0)) * k.ih[0];
                      o[1] = (y0 + px1 * (y1 - y0)) * k.ih[1];
                      o[2] = xy(dz[f]) * k.ih[2];
                    };
                    auto emit = [&](int res, R v) {
                      if (res == 1)
                        lx += v;
                      else
                        {
                          R(&o)[2] = res == 0 ? lv : (res == 2 ? ly : (res == 3 ? lz : lm));
                          o[0] += px0 * v;
                          o[1] += px1 * v;
                        }
                    };
                    const R c = xy(a[0]);
                    R       gc[3], gmu[3], none[1] = {R(0)};
                    const R(*gnone)[3] = nullptr;
                    if constexpr (TENS)
                      grad(0, gc);
                    grad(1, gmu);
                    if constexpr (JVP)
                      {
                        R gdc[3], gdmu[3];
                        if constexpr (TENS)
                          grad(2, gdc);
                        grad(3, gdmu);
                        jvp_terms<3, 0, TENS, R>(p, c, gc, gmu, none, gnone, xy(a[2]), gdc, xy(a[3]), gdmu, none, ~0u,
                                                 emit);
                      }
                    else
                      residual_terms<3, 0, TENS, R>(
                        p, c, gc, xy(a[1]), gmu, none, gnone, ~0u,
                        [&](int, R v) {
                          if constexpr (MODE == 1)
                            v += c * p.w0;
                          if constexpr (MODE == 2)
                            v += xy(a[2]);
                          return v;
                        },
                        emit);
                  }
                lv[0] -= k.ih[0] * lx;
                lv[1] += k.ih[0] * lx;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                  {
                    const R py = (c >> 1) ? py1 : py0;
                    cv[c] += py * lv[c & 1] + ((c >> 1) ? k.ih[1] : -k.ih[1]) * ly[c & 1];
                    cz[c] += py * lz[c & 1];
                    mv[c] += py * lm[c & 1];
                  }
              }
            const R w0 = pz0 * k.JxW, w1 = pz1 * k.JxW, wz = k.ih[2] * k.JxW;
#pragma unroll
            for (int c = 0; c < 4; ++c)
              {
                acc[0][c] += w0 * cv[c] - wz * cz[c];
                acc[0][c + 4] += w1 * cv[c] + wz * cz[c];
                acc[1][c] += w0 * mv[c];
                acc[1][c + 4] += w1 * mv[c];
              }
          }
        // -kappa_c grad c of the mu row with the exact element Laplacian
        {
          R s[8];
#pragma unroll
          for (int l = 0; l < 8; ++l)
            s[l] = nv(JVP ? 2 : 0, l);
          cell_stiffness_add<3, 0>(s, g, acc[1]);
        }
        const bool valid = interior || cell_in_mesh<3>(lane, tc, g);
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
          for (int l = 0; l < 8; ++l)
            K[r * T::CS + l * T::CP + lane] = valid ? acc[r][l] : R(0);
        __syncwarp();

        // sums per node in a fixed order: owned nodes to dst (their grain rows
        // are zero), the others to the tile's partials
#pragma unroll
        for (int s = 0; s < S; ++s)
          {
            if (lane + 32 * s >= T::BOX)
              break;
            bool      owned = np.inner[s];
            long long node  = n0 + np.off[s];
            if (!interior)
              {
                const int b  = lane + 32 * s;
                const int bx = b % T::BX, by = (b / T::BX) % T::BY, bz = b / (T::BX * T::BY);
                const int gi = tc.o[0] + bx, gj = tc.o[1] + by, gk = tc.o[2] + bz;
                if (gi >= g.nn[0] || gj >= g.nn[1] || gk >= g.nn[2])
                  continue;
                owned = (bx > 0 || gi == 0) && (bx < T::TX || gi == g.n[0]) && (by > 0 || gj == 0) &&
                        (by < T::TY || gj == g.n[1]) && (bz > 0 || gk == 0) && (bz < T::TZ || gk == g.n[2]);
              }
            R sum[2] = {R(0), R(0)};
            const R *kc = K + np.cbase[s];
#pragma unroll
            for (int l = 0; l < 8; ++l)
              if ((np.ok[s] >> l) & 1u)
                {
                  const int o = l * T::CP - ((l & 1) + T::TX * ((l >> 1) & 1) + T::TX * T::TY * (l >> 2));
                  sum[0] += kc[o];
                  sum[1] += kc[o + T::CS];
                }
            if (owned)
              {
                for (int cc = 0; cc < ct.c_all; ++cc)
                  {
                    R v = cc == 0 ? sum[0] : (cc == 1 ? sum[1] : R(0));
                    if constexpr (!JVP)
                      if (ph.hooks.epilogue) // (R - subtract) * scale
                        v = (v - (ph.hooks.subtract ? R(ph.hooks.subtract[cc * g.ld + node]) : R(0))) *
                            R(ph.hooks.scale);
                    args.dst[cc * g.ld + node] = v;
                  }
              }
            else
              {
                R *out      = args.partial + (long long)tile * ct.c_all * T::BOX + lane + 32 * s;
                out[0]      = sum[0];
                out[T::BOX] = sum[1];
              }
          }
        __syncwarp(); // K and, for the residual, the box are rewritten by the next tile
        tile = next;
        next = next2;
      }
    if constexpr (JVP)
      cp_async_wait<0>();
    siblings_end();
  }
} // namespace sint
