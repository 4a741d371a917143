// Definitions of the launchers declared in sint_launch.h; included by the
// sint_inst_*.cu translation units, each of which instantiates one
// (dimension, mobility) combination for all grain counts.
#pragma once
#include <type_traits>

#include "sint_fused2d.cuh"
#include "sint_kernels.cuh"
#include "sint_launch.h"
#include "sint_light.cuh"

namespace sint
{
  // Dynamic shared memory above the 48 KB default, and a shared-memory
  // carveout just large enough for `blocks` resident blocks (the rest of the
  // unified storage stays L1).
  template <typename Kernel>
  inline cudaError_t prepare_smem(Kernel k, size_t bytes, int blocks = 2)
  {
    cudaError_t e = cudaSuccess;
    if (bytes > 48 * 1024 && (e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes))) !=
                               cudaSuccess)
      return e;
    int                dev = 0, per_sm = 0;
    cudaFuncAttributes fa{};
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess ||
        (e = cudaFuncGetAttributes(&fa, k)) != cudaSuccess)
      return e;
    // dynamic + static shared memory + the per-block reservation
    const size_t need = size_t(blocks) * (bytes + fa.sharedSizeBytes + 1024);
    const int    pct  = need >= size_t(per_sm) ? 100 : int((need * 100 + per_sm - 1) / per_sm);
    return cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
  }

  // Persistent grid of kernel k on the current device: its shared-memory
  // attributes set, as many blocks as are resident at once (once per device).
  template <typename Kernel>
  inline cudaError_t persistent_grid(DeviceCache &cache, Kernel k, size_t smem, int blocks_per_sm, int threads,
                                     int &grid_cap)
  {
    return per_device(cache, grid_cap, [&](int dev, int &cap) {
      cudaError_t e = prepare_smem(k, smem, blocks_per_sm);
      int         sms = 0, per_sm = 0;
      if (e != cudaSuccess || (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
          (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem)) != cudaSuccess)
        return e;
      cap = sms * (per_sm > 0 ? per_sm : 1);
      return cudaSuccess;
    });
  }

  // sibling: a class kernel of the cut-off that may run beside the one before it
  template <int DIM, int G, bool TENS, typename R, bool CUT, bool ADV>
  cudaError_t launch_jvp_g(const Grid &g, const Phys &p, const R *lin, const R *src, R *dst, R *partial,
                           const CutTiles &ct, const AdvData &adv, cudaStream_t s, bool sibling = false)
  {
    const size_t smem = ThreePhaseSmem<DIM, G, TENS, true, false, ADV, sizeof(R)>::TOTAL * sizeof(R);
    auto         k    = jvp_kernel<DIM, G, TENS, R, CUT, ADV>;
    static DeviceCache cache;
    int                grid_cap = 0;
    if (const cudaError_t e =
          persistent_grid(cache, k, smem, jvp_blocks_per_sm<DIM, G, TENS, R, ADV>(), Tile<DIM>::THREADS, grid_cap))
      return e;
    const long long blocks = g.n_tiles < grid_cap ? g.n_tiles : grid_cap;
    return launch_dependent_if(sibling, k, dim3((unsigned)blocks), Tile<DIM>::THREADS, smem, s, g, p, lin, src, dst,
                               partial, ct, adv);
  }

  template <int DIM, int G, bool TENS, bool CUT = false>
  cudaError_t launch_jvp_pair_g(const Grid &g, const Phys &p, const float *lin, const float *src, float *dst,
                                float *partial, cudaStream_t s, const CutTiles &ct = CutTiles(), bool sibling = false)
  {
    const size_t smem = ThreePhaseSmem<DIM, G, TENS, true, false, false, sizeof(F2)>::TOTAL * sizeof(F2);
    auto         k    = jvp_pair_kernel<DIM, G, TENS, CUT>;
    static DeviceCache cache;
    int                grid_cap = 0;
    if (const cudaError_t e =
          persistent_grid(cache, k, smem, jvp_pair_blocks_per_sm<DIM, G, TENS>(), Tile<DIM>::THREADS, grid_cap))
      return e;
    // the class size of the cut-off lives on the device: a full persistent grid
    const long long pairs  = CUT ? (long long)grid_cap : (g.n_tiles + 1) / 2;
    const long long blocks = pairs < grid_cap ? pairs : grid_cap;
    return launch_dependent_if(sibling, k, dim3((unsigned)blocks), Tile<DIM>::THREADS, smem, s, g, p, lin, src, dst,
                               partial, ct);
  }

  template <int DIM, int G, bool TENS, int WTD, bool CUT, bool ADV>
  cudaError_t launch_residual_g(const Grid &g, const Phys &p, const double *src, const double *const *hist,
                                double *dst, double *partial, const CutTiles &ct, const AdvData &adv,
                                cudaStream_t s, bool sibling = false)
  {
    const size_t  smem     = ThreePhaseSmem<DIM, G, TENS, false, WTD == 2, ADV, sizeof(double)>::TOTAL * sizeof(double);
    auto          k        = residual_kernel<DIM, G, TENS, WTD, CUT, ADV>;
    static DeviceCache cache;
    int                grid_cap = 0;
    if (const cudaError_t e =
          persistent_grid(cache, k, smem, residual_blocks_per_sm<DIM, G, TENS, WTD == 2, ADV>(), Tile<DIM>::THREADS, grid_cap))
      return e;
    const double *h0     = WTD == 2 ? hist[0] : nullptr;
    const double *h1     = (WTD == 2 && p.order > 1) ? hist[1] : nullptr;
    const double *h2     = (WTD == 2 && p.order > 2) ? hist[2] : nullptr;
    const long long blocks = g.n_tiles < grid_cap ? g.n_tiles : grid_cap;
    return launch_dependent_if(sibling, k, dim3((unsigned)blocks), Tile<DIM>::THREADS, smem, s, g, p, src, h0, h1, h2, dst,
                               partial, ct, adv);
  }

  // The 3D class of the grain cut-off without a relevant grain (MODE: -1 = J v,
  // 0..2 = residual); the class size lives on the device, so the grid is the
  // persistent one.
  template <bool TENS, typename R, int MODE>
  cudaError_t launch_light(const Grid &g, const Phys &p, const LightArgs<R> &args, const CutTiles &ct, cudaStream_t s,
                           bool sibling)
  {
    using L           = LightTile<MODE>;
    const size_t smem = L::template smem<R>();
    auto         k    = light_kernel<TENS, R, MODE>;
    static DeviceCache cache;
    int                grid_cap = 0;
    if (const cudaError_t e = persistent_grid(cache, k, smem, light_blocks<R, MODE>(), L::WARPS * 32, grid_cap))
      return e;
    const long long need   = (g.n_tiles + L::WARPS - 1) / L::WARPS;
    const long long blocks = need < grid_cap ? need : grid_cap;
    return launch_dependent_if(sibling, k, dim3((unsigned)blocks), L::WARPS * 32, smem, s, g, p, args, ct);
  }

  // The one-kernel 2D cell loop (MODE: -1 = J v, 0..2 = residual).
  template <int G, bool TENS, typename R, int MODE>
  cudaError_t launch_fused2d_g(const Grid &g, const Phys &p, Fused2DArgs<R> args, cudaStream_t s)
  {
    using L           = Fused2D<G, MODE>;
    const size_t smem = L::template smem<R>();
    auto         k    = fused2d_kernel<G, TENS, R, MODE>;
    static DeviceCache cache;
    int                ready = 0;
    if (const cudaError_t e = per_device(cache, ready, [&](int, int &v) {
          v = 1;
          return prepare_smem(k, smem, fused2d_blocks<G, TENS, R, MODE>());
        }))
      return e;
    args.blocks_x          = (g.nn[0] + L::TX - 2) / (L::TX - 1);
    const long long blocks = (long long)args.blocks_x * ((g.nn[1] + L::TY - 2) / (L::TY - 1));
    return launch_dependent(k, dim3((unsigned)blocks), L::THREADS, smem, s, g, p, args);
  }

  template <int DIM, int G, bool TENS, bool CUT, bool ADV>
  cudaError_t launch_diag_g(const Grid &g, const Phys &p, const double *lin, double *dst, double *partial,
                            const uint16_t *mask, const AdvData &adv, cudaStream_t s)
  {
    const size_t smem = smem_diag(DIM, G, ADV);
    auto         k    = diag_kernel<DIM, G, TENS, CUT, ADV>;
    cudaError_t  e    = prepare_smem(k, smem);
    if (e != cudaSuccess)
      return e;
    k<<<dim3((unsigned)g.n_tiles), Tile<DIM>::THREADS, smem, s>>>(g, p, lin, dst, partial, mask, adv);
    count_launches(1);
    return cudaGetLastError();
  }

#define SINT_G_SWITCH(CALL)                                                                                       \
  switch (G)                                                                                                      \
    {                                                                                                             \
      case 1: return CALL(1);                                                                                     \
      case 2: return CALL(2);                                                                                     \
      case 3: return CALL(3);                                                                                     \
      case 4: return CALL(4);                                                                                     \
      case 5: return CALL(5);                                                                                     \
      case 6: return CALL(6);                                                                                     \
      case 7: return CALL(7);                                                                                     \
      case 8: return CALL(8);                                                                                     \
      case 9: return CALL(9);                                                                                     \
      case 10: return CALL(10);                                                                                   \
      case 11: return CALL(11);                                                                                   \
      case 12: return CALL(12);                                                                                   \
      default: return cudaErrorInvalidValue;                                                                      \
    }

  // G = the class of the grain cut-off (0..12 relevant grains)
  template <int DIM, bool TENS, typename R, bool ADV>
  cudaError_t launch_jvp_class(int G, const Grid &g, const Phys &p, const R *lin, const R *src, R *dst, R *partial,
                               const CutTiles &ct, const AdvData &adv, cudaStream_t s, bool sibling)
  {
#define SINT_CALL(GG) launch_jvp_g<DIM, GG, TENS, R, true, ADV>(g, p, lin, src, dst, partial, ct, adv, s, sibling)
    if (G == 0) // without grains: c and mu only, the bulk of a packing's vapour
      {
        if constexpr (DIM == 3 && !ADV)
          return launch_light<TENS, R, -1>(g, p, LightArgs<R>{lin, src, {}, dst, partial}, ct, s, sibling);
        else if constexpr (std::is_same_v<R, float> && !ADV) // on tile pairs
          return launch_jvp_pair_g<DIM, 0, TENS, true>(g, p, lin, src, dst, partial, s, ct, sibling);
        else
          return SINT_CALL(0);
      }
    SINT_G_SWITCH(SINT_CALL)
#undef SINT_CALL
  }

  // The full operator's J v: one kernel in 2D (sint_fused2d.cuh), in 3D packed
  // FP32 tile pairs for few grains, or the tiled kernel.  Pairs take 8 bytes
  // per value: with more grains one block fits an SM's registers, and the
  // scalar FP32 kernel with two (tensorial) or three (scalar mobility) is
  // faster (160^3 cells: 9 grains tensorial 3347 us on pairs, 2967 us here; 5
  // grains 1700 / 1647 us, 4 grains 1367 / 1380 us; scalar mobility, 9 grains
  // 2216 / 1816 us, 5 grains 1264 / 1254 us, 4 grains 1105 / 1116 us).
  template <int DIM, int G, bool TENS, typename R, bool ADV>
  cudaError_t launch_jvp_full(const Grid &g, const Phys &p, const R *lin, const R *src, R *dst, R *partial,
                              const AdvData &adv, cudaStream_t s)
  {
    if constexpr (!ADV && runs_fused2d(DIM, G, TENS, sizeof(R)))
      return launch_fused2d_g<G, TENS, R, -1>(g, p, Fused2DArgs<R>{lin, src, {}, dst, 0}, s);
    else if constexpr (!ADV && std::is_same_v<R, float> && G <= 4)
      return launch_jvp_pair_g<DIM, G, TENS>(g, p, lin, src, dst, partial, s);
    else
      return launch_jvp_g<DIM, G, TENS, R, false, ADV>(g, p, lin, src, dst, partial, CutTiles(), adv, s);
  }

  // cut == nullptr: the full operator; otherwise the grain cut-off, one
  // launch per grain-count class 0..G (classes without tiles return at once).
  // ADV: the kernels with the advection terms.
  template <int DIM, bool TENS, typename R, bool ADV>
  cudaError_t launch_jvp_impl(int G, const Grid &g, const Phys &p, const R *lin, const R *src, R *dst, R *partial,
                              const CutTiles *cut, const AdvData &adv, cudaStream_t s)
  {
    if (cut)
      {
        // the classes of many grains have few tiles and a long time per tile:
        // launched first, they run beside the light ones (siblings_begin)
        for (int K = G; K >= 0; --K)
          if (const cudaError_t e =
                launch_jvp_class<DIM, TENS, R, ADV>(K, g, p, lin, src, dst, partial, *cut, adv, s, K < G))
            return e;
        return cudaSuccess;
      }
#define SINT_CALL(GG) launch_jvp_full<DIM, GG, TENS, R, ADV>(g, p, lin, src, dst, partial, adv, s)
    SINT_G_SWITCH(SINT_CALL)
#undef SINT_CALL
  }

  // The advection kernels are instantiated in their own translation units
  // (launch_jvp_adv, launch_residual_adv).
  template <int DIM, bool TENS, typename R>
  cudaError_t launch_jvp(int G, const Grid &g, const Phys &p, const R *lin, const R *src, R *dst, R *partial,
                         const CutTiles *cut, const AdvData *adv, cudaStream_t s)
  {
    if (adv)
      return launch_jvp_adv<DIM, TENS, R>(G, g, p, lin, src, dst, partial, cut, *adv, s);
    return launch_jvp_impl<DIM, TENS, R, false>(G, g, p, lin, src, dst, partial, cut, AdvData(), s);
  }

  // The full operator's residual: one kernel in 2D, else the tiled kernel.
  template <int DIM, int G, bool TENS, int WTD, bool ADV>
  cudaError_t launch_residual_full(const Grid &g, const Phys &p, const double *src, const double *const *hist,
                                   double *dst, double *partial, const AdvData &adv, cudaStream_t s)
  {
    if constexpr (!ADV && runs_fused2d(DIM, G, TENS, sizeof(double)))
      {
        Fused2DArgs<double> args{src, nullptr, {}, dst, 0};
        for (int i = 0; WTD == 2 && i < p.order; ++i)
          args.h[i] = hist[i];
        return launch_fused2d_g<G, TENS, double, WTD>(g, p, args, s);
      }
    else
      return launch_residual_g<DIM, G, TENS, WTD, false, ADV>(g, p, src, hist, dst, partial, CutTiles(), adv, s);
  }

  // G = the grain count (full operator, 1..12) or the class (grain cut-off, 0..12)
  template <int DIM, bool TENS, bool CUT, int WTD, bool ADV>
  cudaError_t launch_residual_w(int G, const Grid &g, const Phys &p, const double *src, const double *const *hist,
                                double *dst, double *partial, const CutTiles &ct, const AdvData &adv,
                                cudaStream_t s, bool sibling)
  {
    if constexpr (CUT)
      {
#define SINT_CALL(GG) launch_residual_g<DIM, GG, TENS, WTD, true, ADV>(g, p, src, hist, dst, partial, ct, adv, s, sibling)
        if (G == 0)
          {
            if constexpr (DIM == 3 && !ADV)
              {
                LightArgs<double> args{src, nullptr, {}, dst, partial};
                for (int i = 0; WTD == 2 && i < p.order; ++i)
                  args.h[i] = hist[i];
                return launch_light<TENS, double, WTD>(g, p, args, ct, s, sibling);
              }
            else
              return SINT_CALL(0);
          }
        SINT_G_SWITCH(SINT_CALL)
#undef SINT_CALL
      }
    else
      {
#define SINT_CALL(GG) launch_residual_full<DIM, GG, TENS, WTD, ADV>(g, p, src, hist, dst, partial, adv, s)
        SINT_G_SWITCH(SINT_CALL)
#undef SINT_CALL
      }
  }

  template <int DIM, bool TENS, bool CUT, bool ADV>
  cudaError_t launch_residual_c(int G, int wtd, const Grid &g, const Phys &p, const double *src,
                                const double *const *hist, double *dst, double *partial, const CutTiles &ct,
                                const AdvData &adv, cudaStream_t s, bool sibling = false)
  {
    if (wtd == 0)
      return launch_residual_w<DIM, TENS, CUT, 0, ADV>(G, g, p, src, hist, dst, partial, ct, adv, s, sibling);
    if (wtd == 1)
      return launch_residual_w<DIM, TENS, CUT, 1, ADV>(G, g, p, src, hist, dst, partial, ct, adv, s, sibling);
    return launch_residual_w<DIM, TENS, CUT, 2, ADV>(G, g, p, src, hist, dst, partial, ct, adv, s, sibling);
  }

  // With advection in 3D the class without grains is a block kernel that is
  // most of the call.  On large meshes it runs faster by itself than beside the
  // other classes' last blocks, whose shared-memory carveout it inherits (an SM
  // changes it only while idle): 128^3 cells, 2 grains, scalar, with history 474
  // us, beside them 540 to 584; tensorial without history 459 and 505.  On small
  // ones it hides their tails (64 x 56 x 48 cells, 9 grains 116 us, one class
  // after the other 152).
  constexpr long long CLASS0_BESIDE_TILES = 12288;

  template <int DIM, bool TENS, bool ADV>
  cudaError_t launch_residual_impl(int G, int wtd, const Grid &g, const Phys &p, const double *src,
                                   const double *const *hist, double *dst, double *partial, const CutTiles *cut,
                                   const AdvData &adv, cudaStream_t s)
  {
    if (cut)
      {
        for (int K = G; K >= 0; --K) // as the Jacobian product
          {
            const bool beside = K < G && !(ADV && DIM == 3 && K == 0 && g.n_tiles > CLASS0_BESIDE_TILES);
            if (const cudaError_t e =
                  launch_residual_c<DIM, TENS, true, ADV>(K, wtd, g, p, src, hist, dst, partial, *cut, adv, s, beside))
              return e;
          }
        return cudaSuccess;
      }
    return launch_residual_c<DIM, TENS, false, ADV>(G, wtd, g, p, src, hist, dst, partial, CutTiles(), adv, s);
  }

  template <int DIM, bool TENS>
  cudaError_t launch_residual(int G, int wtd, const Grid &g, const Phys &p, const double *src,
                              const double *const *hist, double *dst, double *partial, const CutTiles *cut,
                              const AdvData *adv, cudaStream_t s)
  {
    if (adv)
      return launch_residual_adv<DIM, TENS>(G, wtd, g, p, src, hist, dst, partial, cut, *adv, s);
    return launch_residual_impl<DIM, TENS, false>(G, wtd, g, p, src, hist, dst, partial, cut, AdvData(), s);
  }

  template <int DIM, bool TENS, bool ADV>
  cudaError_t launch_diag_impl(int G, const Grid &g, const Phys &p, const double *lin, double *dst, double *partial,
                               const uint16_t *mask, const AdvData &adv, cudaStream_t s)
  {
    if (mask)
      {
#define SINT_CALL(GG) launch_diag_g<DIM, GG, TENS, true, ADV>(g, p, lin, dst, partial, mask, adv, s)
        SINT_G_SWITCH(SINT_CALL)
#undef SINT_CALL
      }
#define SINT_CALL(GG) launch_diag_g<DIM, GG, TENS, false, ADV>(g, p, lin, dst, partial, nullptr, adv, s)
    SINT_G_SWITCH(SINT_CALL)
#undef SINT_CALL
  }

  template <int DIM, bool TENS>
  cudaError_t launch_diag(int G, const Grid &g, const Phys &p, const double *lin, double *dst, double *partial,
                          const uint16_t *mask, const AdvData *adv, cudaStream_t s)
  {
    if (adv)
      return launch_diag_adv<DIM, TENS>(G, g, p, lin, dst, partial, mask, *adv, s);
    return launch_diag_impl<DIM, TENS, false>(G, g, p, lin, dst, partial, mask, AdvData(), s);
  }
} // namespace sint
