// BLAS-1 on block vectors (DynamicBlockVector, lac/dynamic_block_vector.h:346-516)
// and the fused multi-vector kernels used by GMRES's Gram-Schmidt step.
// Reductions are deterministic: a fixed grid of NB_RED blocks writes block
// partials in FP64, one block sums them in a fixed tree order.
#include <string>
#include <type_traits>

#include "sint_internal.h"
#include "sint_launch.h"

namespace sint
{
  constexpr int RED_THREADS = 256;

  __device__ __forceinline__ double warp_sum(double v)
  {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }

  // Block-wide sum of one value per thread (RED_THREADS threads); result valid in thread 0.
  __device__ __forceinline__ double block_sum(double v, double *s_w)
  {
    v              = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0)
      s_w[wid] = v;
    __syncthreads();
    double r = 0.0;
    if (wid == 0)
      {
        r = lane < RED_THREADS / 32 ? s_w[lane] : 0.0;
        r = warp_sum(r);
      }
    __syncthreads();
    return r;
  }

  // --- 16-byte packs ---------------------------------------------------------
  // The Krylov kernels move 16 bytes per load (2 doubles or 4 floats) when
  // every pointer is 16-byte aligned and n, stride are multiples of the pack;
  // otherwise one element per load (E = 1).  Block vectors of a context
  // always qualify: ld is a multiple of 32.
  template <typename R, int E>
  struct Pack
  {
    R v[E];
  };

  template <typename R, int E>
  __device__ __forceinline__ Pack<R, E> ld_pack(const R *__restrict__ p, long long c)
  {
    Pack<R, E> x;
    if constexpr (E * sizeof(R) == 16 && sizeof(R) == 8)
      {
        const double2 t = reinterpret_cast<const double2 *>(p)[c];
        x.v[0] = t.x, x.v[1] = t.y;
      }
    else if constexpr (E * sizeof(R) == 16 && sizeof(R) == 4)
      {
        const float4 t = reinterpret_cast<const float4 *>(p)[c];
        x.v[0] = t.x, x.v[1] = t.y, x.v[2] = t.z, x.v[3] = t.w;
      }
    else
      {
#pragma unroll
        for (int e = 0; e < E; ++e)
          x.v[e] = p[c * E + e];
      }
    return x;
  }

  template <typename R, int E>
  __device__ __forceinline__ void st_pack(R *__restrict__ p, long long c, const Pack<R, E> &x)
  {
    if constexpr (E * sizeof(R) == 16 && sizeof(R) == 8)
      reinterpret_cast<double2 *>(p)[c] = make_double2(x.v[0], x.v[1]);
    else if constexpr (E * sizeof(R) == 16 && sizeof(R) == 4)
      reinterpret_cast<float4 *>(p)[c] = make_float4(x.v[0], x.v[1], x.v[2], x.v[3]);
    else
      {
#pragma unroll
        for (int e = 0; e < E; ++e)
          p[c * E + e] = x.v[e];
      }
  }

  template <typename R>
  constexpr int pack_of()
  {
    return 16 / int(sizeof(R));
  }

  inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

  // Live chunks (grain cut-off): bit k of live is clear when elements
  // [k * LIVE_CHUNK, (k + 1) * LIVE_CHUNK) of every Krylov vector are known
  // to be zero; nullptr = all live.  A warp's packs never straddle a chunk.
  __device__ __forceinline__ bool chunk_live(const uint32_t *__restrict__ live, long long elem)
  {
    if (!live)
      return true;
    const long long k = elem / LIVE_CHUNK;
    return (live[k >> 5] >> (k & 31)) & 1u;
  }

  template <typename R>
  inline bool can_pack(long long n, long long stride, const void *a, const void *b)
  {
    constexpr int E = pack_of<R>();
    return n % E == 0 && stride % E == 0 && aligned16(a) && aligned16(b);
  }

  // Fused finish of a reduction: every block has written its partials
  // (rows 0..m-1, one column per block, row pitch NB_RED); the block that
  // takes the last ticket sums each row in a fixed order (lane l adds blocks
  // l, l + 32, ..., then a fixed butterfly), writes out[0..m) and resets the
  // ticket.  The result does not depend on which block finishes last.  Returns
  // whether this is that block.
  __device__ __forceinline__ bool finish_if_last(const double *__restrict__ rows, int m, double *__restrict__ out,
                                                 unsigned *ticket)
  {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
      last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last)
      return false;
    __threadfence();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nb = gridDim.x;
    for (int j = warp; j < m; j += RED_THREADS / 32)
      {
        // a row's loads are all in flight together
        constexpr int L = (NB_RED + 31) / 32;
        double        t[L];
#pragma unroll
        for (int i = 0; i < L; ++i)
          t[i] = lane + 32 * i < nb ? __ldcg(rows + (size_t)j * NB_RED + lane + 32 * i) : 0.0;
        double v = 0.0;
#pragma unroll
        for (int i = 0; i < L; ++i)
          v += t[i];
        v = warp_sum(v);
        if (lane == 0)
          out[j] = v;
      }
    if (threadIdx.x == 0)
      *ticket = 0u;
    return true;
  }

  // Blocks of a reduction over nc packs: one pack per thread until NB_RED
  // blocks are reached (a 2D Krylov vector of 130,000 values fills 260).
  static unsigned red_blocks(long long nc)
  {
    const long long b = (nc + RED_THREADS - 1) / RED_THREADS;
    return (unsigned)(b < 1 ? 1 : (b < NB_RED ? b : NB_RED));
  }

  // partial[j * NB_RED + blockIdx.x] = sum over this block's chunks of w . V_j
  // (FP64 products and sums; m <= M).
  template <typename R, int M, int E>
  __global__ void __launch_bounds__(RED_THREADS)
    multidot_kernel(long long nc, const R *__restrict__ w, const R *__restrict__ V, long long stride, int m,
                    double *__restrict__ partial, const int *__restrict__ cond, const double *__restrict__ rows,
                    int m_total, double *__restrict__ out, unsigned *ticket, const uint32_t *__restrict__ live)
  {
    dependent_start();
    if (cond && *cond == 0)
      return;
    constexpr int     NW = RED_THREADS / 32;
    __shared__ double s_w[M][NW];
    double            acc[M];
#pragma unroll
    for (int j = 0; j < M; ++j)
      acc[j] = 0.0;
    for (long long c = (long long)blockIdx.x * RED_THREADS + threadIdx.x; c < nc; c += (long long)gridDim.x * RED_THREADS)
      {
        if (!chunk_live(live, c * E))
          continue;
        const Pack<R, E> wi = ld_pack<R, E>(w, c);
#pragma unroll
        for (int j = 0; j < M; ++j)
          if (j < m)
            {
              const Pack<R, E> vj = ld_pack<R, E>(V + j * stride, c);
#pragma unroll
              for (int e = 0; e < E; ++e)
                acc[j] += double(wi.v[e]) * double(vj.v[e]);
            }
      }
    // all rows through the warps at once: one barrier for the block
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < M; ++j)
      if (j < m)
        {
          const double v = warp_sum(acc[j]);
          if (lane == 0)
            s_w[j][wid] = v;
        }
    __syncthreads();
    for (int j = threadIdx.x; j < m; j += RED_THREADS)
      {
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < NW; ++k)
          v += s_w[j][k];
        partial[(size_t)j * NB_RED + blockIdx.x] = v;
      }
    if (out)
      finish_if_last(rows, m_total, out, ticket);
  }

  // Vectors per multidot / multiaxpy pass, and the instances for few vectors
  // (an instance tests each of its M vectors against m).
  constexpr int MD = 16;
  template <typename F>
  static cudaError_t by_count(int m, F go)
  {
    return m <= 4 ? go(std::integral_constant<int, 4>{}) :
           m <= 8 ? go(std::integral_constant<int, 8>{}) : go(std::integral_constant<int, MD>{});
  }

  template <typename R>
  static int launch_multidot(Ctx *c, long long n, const R *w, const R *V, long long stride, int m, double *out,
                             cudaStream_t s, const int *cond = nullptr, const uint32_t *live = nullptr)
  {
    if (m < 1 || m > MAX_MULTIDOT)
      {
        set_error("multidot: m out of range");
        return SINT_ERR_ARG;
      }
    constexpr int  E    = pack_of<R>();
    const bool     pack = can_pack<R>(n, stride, w, V);
    const unsigned nb   = red_blocks(pack ? n / E : n); // the same for every pass: the last one sums all rows
    for (int j0 = 0; j0 < m; j0 += MD)
      {
        const int         mm   = m - j0 < MD ? m - j0 : MD;
        double           *pp   = c->red + (size_t)j0 * NB_RED;
        double           *outl = j0 + MD >= m ? out : nullptr;
        const cudaError_t e    = by_count(mm, [&](auto k) {
          constexpr int M = decltype(k)::value;
          return pack ? launch_dependent(multidot_kernel<R, M, E>, nb, RED_THREADS, 0, s, n / E, w, V + j0 * stride,
                                            stride, mm, pp, cond, c->red, m, outl, c->red_ticket, live) :
                           launch_dependent(multidot_kernel<R, M, 1>, nb, RED_THREADS, 0, s, n, w, V + j0 * stride,
                                            stride, mm, pp, cond, c->red, m, outl, c->red_ticket, live);
        });
        if (e != cudaSuccess)
          return cuda_fail(e, "multidot");
      }
    return SINT_OK;
  }

  template <typename R>
  int multidot(Ctx *c, long long n, const R *w, const R *V, long long stride, int m, double *out, cudaStream_t s,
               const uint32_t *live)
  {
    return launch_multidot<R>(c, n, w, V, stride, m, out, s, nullptr, live);
  }
  template int multidot<double>(Ctx *, long long, const double *, const double *, long long, int, double *,
                                cudaStream_t, const uint32_t *);
  template int multidot<float>(Ctx *, long long, const float *, const float *, long long, int, double *,
                               cudaStream_t, const uint32_t *);

  template <typename R>
  int multidot_if(Ctx *c, long long n, const R *w, const R *V, long long stride, int m, double *out, const int *cond,
                  cudaStream_t s, const uint32_t *live)
  {
    return launch_multidot<R>(c, n, w, V, stride, m, out, s, cond, live);
  }
  template int multidot_if<double>(Ctx *, long long, const double *, const double *, long long, int, double *,
                                   const int *, cudaStream_t, const uint32_t *);
  template int multidot_if<float>(Ctx *, long long, const float *, const float *, long long, int, double *,
                                  const int *, cudaStream_t, const uint32_t *);

  int dot_f64(Ctx *c, long long n, const double *x, const double *y, double *out, cudaStream_t s)
  {
    return launch_multidot<double>(c, n, x, y, 0, 1, out, s);
  }
  int dot_f32(Ctx *c, long long n, const float *x, const float *y, double *out, cudaStream_t s)
  {
    return launch_multidot<float>(c, n, x, y, 0, 1, out, s);
  }

  // w -= sum_j coef[j] V_j (j < m <= M); with `partial`, also the block
  // partials of |w|^2 after the update (FP64), for the norm that follows, and
  // with chk.H the bookkeeping of an Arnoldi step after its first
  // Gram-Schmidt pass (in the block that finishes the norm): Hessenberg column
  // j = h and deal.II's re-orthogonalisation test (Kelley 1995, as in
  // SolverGMRES): once |w| after the pass falls below 10 sqrt(eps) of |w|
  // before it, every later iteration of this solve takes a second pass (the
  // flag is sticky).  thresh2 = 100 eps of the Krylov vectors' precision;
  // |w|^2 before = |h|^2 + |w'|^2.
  template <typename R, int M, int E>
  __global__ void __launch_bounds__(RED_THREADS)
    multiaxpy_kernel(long long nc, R *__restrict__ w, const R *__restrict__ V, long long stride, int m,
                     const double *__restrict__ coef, double *__restrict__ partial, const int *__restrict__ cond,
                     double *norm2_out, unsigned *ticket, const uint32_t *__restrict__ live, const ArnoldiCheck chk)
  {
    dependent_start();
    if (cond && *cond == 0)
      return;
    __shared__ R      s_c[M];
    __shared__ double s_w[RED_THREADS / 32];
    if (threadIdx.x < M)
      s_c[threadIdx.x] = threadIdx.x < m ? R(coef[threadIdx.x]) : R(0);
    __syncthreads();
    double nrm = 0.0;
    for (long long c = (long long)blockIdx.x * RED_THREADS + threadIdx.x; c < nc; c += (long long)gridDim.x * RED_THREADS)
      {
        if (!chunk_live(live, c * E)) // w and every V_j are zero there: w stays zero
          continue;
        Pack<R, E> acc = ld_pack<R, E>(w, c);
#pragma unroll
        for (int j = 0; j < M; ++j)
          if (j < m)
            {
              const Pack<R, E> vj = ld_pack<R, E>(V + j * stride, c);
#pragma unroll
              for (int e = 0; e < E; ++e)
                acc.v[e] -= s_c[j] * vj.v[e];
            }
        st_pack<R, E>(w, c, acc);
        if (partial)
          {
#pragma unroll
            for (int e = 0; e < E; ++e)
              nrm += double(acc.v[e]) * double(acc.v[e]);
          }
      }
    if (partial)
      {
        const double t = block_sum(nrm, s_w);
        if (threadIdx.x == 0)
          partial[blockIdx.x] = t;
        if (!finish_if_last(partial, 1, norm2_out, ticket) || !chk.H || threadIdx.x >= 32)
          return;
        double *hcol = chk.H + (long long)chk.j * chk.ldh;
        double  hh   = 0.0;
        for (int i = threadIdx.x; i <= chk.j; i += 32)
          {
            const double h = chk.d_s[i];
            hcol[i]        = h;
            hh += h * h;
          }
        hh = warp_sum(hh);
        __syncwarp();
        if (threadIdx.x == 0)
          {
            const double nw2 = *norm2_out; // written by this thread in finish_if_last
            if (nw2 < chk.thresh2 * (hh + nw2))
              *chk.reorth = 1;
          }
      }
  }

  template <typename R>
  static int launch_multiaxpy(Ctx *c, long long n, R *w, const R *V, long long stride, int m, const double *coef,
                              double *norm2_out, cudaStream_t s, const int *cond = nullptr,
                              const uint32_t *live = nullptr, const ArnoldiCheck &chk = ArnoldiCheck())
  {
    constexpr int  E    = pack_of<R>();
    const bool     pack = can_pack<R>(n, stride, w, V);
    const unsigned nb   = red_blocks(pack ? n / E : n);
    for (int j0 = 0; j0 < m; j0 += MD)
      {
        const int         mm   = m - j0 < MD ? m - j0 : MD;
        double           *part = (norm2_out && j0 + MD >= m) ? c->red : nullptr; // norm in the last pass
        unsigned         *tk   = c ? c->red_ticket : nullptr;
        const cudaError_t e    = by_count(mm, [&](auto k) {
          constexpr int M = decltype(k)::value;
          return pack ? launch_dependent(multiaxpy_kernel<R, M, E>, nb, RED_THREADS, 0, s, n / E, w, V + j0 * stride,
                                            stride, mm, coef + j0, part, cond, norm2_out, tk, live, chk) :
                           launch_dependent(multiaxpy_kernel<R, M, 1>, nb, RED_THREADS, 0, s, n, w, V + j0 * stride,
                                            stride, mm, coef + j0, part, cond, norm2_out, tk, live, chk);
        });
        if (e != cudaSuccess)
          return cuda_fail(e, "multiaxpy");
      }
    return SINT_OK;
  }

  template <typename R>
  int multiaxpy(long long n, R *w, const R *V, long long stride, int m, const double *coef, cudaStream_t s)
  {
    return launch_multiaxpy<R>(nullptr, n, w, V, stride, m, coef, nullptr, s);
  }
  template int multiaxpy<double>(long long, double *, const double *, long long, int, const double *, cudaStream_t);
  template int multiaxpy<float>(long long, float *, const float *, long long, int, const double *, cudaStream_t);

  template <typename R>
  int multiaxpy_norm2(Ctx *c, long long n, R *w, const R *V, long long stride, int m, const double *coef,
                      double *norm2_out, cudaStream_t s, const uint32_t *live, const ArnoldiCheck &chk)
  {
    return launch_multiaxpy<R>(c, n, w, V, stride, m, coef, norm2_out, s, nullptr, live, chk);
  }
  template int multiaxpy_norm2<double>(Ctx *, long long, double *, const double *, long long, int, const double *,
                                       double *, cudaStream_t, const uint32_t *, const ArnoldiCheck &);
  template int multiaxpy_norm2<float>(Ctx *, long long, float *, const float *, long long, int, const double *,
                                      double *, cudaStream_t, const uint32_t *, const ArnoldiCheck &);

  template <typename R>
  int multiaxpy_norm2_if(Ctx *c, long long n, R *w, const R *V, long long stride, int m, const double *coef,
                         double *norm2_out, const int *cond, cudaStream_t s, const uint32_t *live)
  {
    return launch_multiaxpy<R>(c, n, w, V, stride, m, coef, norm2_out, s, cond, live);
  }
  template int multiaxpy_norm2_if<double>(Ctx *, long long, double *, const double *, long long, int, const double *,
                                          double *, const int *, cudaStream_t, const uint32_t *);
  template int multiaxpy_norm2_if<float>(Ctx *, long long, float *, const float *, long long, int, const double *,
                                         double *, const int *, cudaStream_t, const uint32_t *);

  // y += sum_j coef[j] V_j
  template <typename R, int M, int E>
  __global__ void __launch_bounds__(256) lincomb_kernel(long long nc, R *__restrict__ y, const R *__restrict__ V,
                                                        long long stride, int m, const double *__restrict__ coef,
                                                        const uint32_t *__restrict__ live)
  {
    __shared__ R s_c[M];
    if (threadIdx.x < M)
      s_c[threadIdx.x] = threadIdx.x < m ? R(coef[threadIdx.x]) : R(0);
    __syncthreads();
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += (long long)gridDim.x * blockDim.x)
      {
        if (!chunk_live(live, c * E)) // y and every V_j are zero there
          continue;
        Pack<R, E> acc = ld_pack<R, E>(y, c);
#pragma unroll
        for (int j = 0; j < M; ++j)
          if (j < m)
            {
              const Pack<R, E> vj = ld_pack<R, E>(V + j * stride, c);
#pragma unroll
              for (int e = 0; e < E; ++e)
                acc.v[e] += s_c[j] * vj.v[e];
            }
        st_pack<R, E>(y, c, acc);
      }
  }

  template <typename R>
  int lincomb(long long n, R *y, const R *V, long long stride, int m, const double *coef, cudaStream_t s,
              const uint32_t *live)
  {
    constexpr int E    = pack_of<R>();
    const bool    pack = can_pack<R>(n, stride, y, V);
    for (int j0 = 0; j0 < m; j0 += MD)
      {
        const int mm = m - j0 < MD ? m - j0 : MD;
        if (pack)
          lincomb_kernel<R, MD, E><<<1184, 256, 0, s>>>(n / E, y, V + j0 * stride, stride, mm, coef + j0, live);
        else
          lincomb_kernel<R, MD, 1><<<1184, 256, 0, s>>>(n, y, V + j0 * stride, stride, mm, coef + j0, live);
        count_launches(1);
      }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? SINT_OK : cuda_fail(e, "lincomb");
  }
  template int lincomb<double>(long long, double *, const double *, long long, int, const double *, cudaStream_t,
                               const uint32_t *);
  template int lincomb<float>(long long, float *, const float *, long long, int, const double *, cudaStream_t,
                              const uint32_t *);

  // y = b y + a x; a term whose factor is 0 is dropped, so NaN in an unused
  // operand does not spread.  Chunks that are not live are written as zero
  // without reading.
  template <typename R, int E>
  __device__ __forceinline__ void axpby_body(long long nc, R a, const R *__restrict__ x, R b, R *__restrict__ y,
                                             const uint32_t *__restrict__ live)
  {
    for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += (long long)gridDim.x * blockDim.x)
      {
        if (!chunk_live(live, c * E))
          {
            st_pack<R, E>(y, c, Pack<R, E>{});
            continue;
          }
        Pack<R, E> xv{}, yv{}, out;
        if (a != R(0))
          xv = ld_pack<R, E>(x, c);
        if (b != R(0))
          yv = ld_pack<R, E>(y, c);
#pragma unroll
        for (int e = 0; e < E; ++e)
          out.v[e] = (b == R(0) ? R(0) : b * yv.v[e]) + (a == R(0) ? R(0) : a * xv.v[e]);
        st_pack<R, E>(y, c, out);
      }
  }

  // Blocks of an element-wise pass of 256 threads over nc packs.
  static unsigned map_blocks(long long nc)
  {
    const long long b = (nc + 255) / 256;
    return (unsigned)(b < 1 ? 1 : (b < 1184 ? b : 1184));
  }

  template <typename R, int E>
  __global__ void __launch_bounds__(256) axpby_kernel(long long nc, R a, const R *__restrict__ x, R b,
                                                      R *__restrict__ y, const uint32_t *__restrict__ live)
  {
    dependent_start();
    axpby_body<R, E>(nc, a, x, b, y, live);
  }

  // A dependent launch hides its set-up (FP64, 1000 to 400,000 values: 1.6 to
  // 2.5 us, 0.2 to 0.3 us less; 1.3 million 3.8 -> 3.6), but its blocks then
  // start on whichever SM is free, and two vectors that only fit the L2 while
  // every block finds its part on its own side of it miss: FP64, 6 million
  // values, 12.4 -> 16.4 us.  2.6 million (40 MiB) take 5.7 us either way, 20
  // million, in HBM, 76.8 and 75.7.
  constexpr long long AXPBY_DEPENDENT_BYTES = 40ll << 20;

  template <typename R>
  int axpby(long long n, double a, const R *x, double b, R *y, cudaStream_t s, const uint32_t *live)
  {
    constexpr int     E   = pack_of<R>();
    const bool        dep = 2 * n * (long long)sizeof(R) <= AXPBY_DEPENDENT_BYTES;
    const cudaError_t e =
      can_pack<R>(n, 0, x, y) ?
        launch_dependent_if(dep, axpby_kernel<R, E>, map_blocks(n / E), 256, 0, s, n / E, R(a), x, R(b), y, live) :
        launch_dependent_if(dep, axpby_kernel<R, 1>, map_blocks(n), 256, 0, s, n, R(a), x, R(b), y, live);
    return e == cudaSuccess ? SINT_OK : cuda_fail(e, "axpby");
  }
  template int axpby<double>(long long, double, const double *, double, double *, cudaStream_t, const uint32_t *);
  template int axpby<float>(long long, double, const float *, double, float *, cudaStream_t, const uint32_t *);

  // End of Arnoldi step j after the (optional) second Gram-Schmidt pass: the
  // next basis vector y = w / |w| by all blocks, and in block 0 the
  // bookkeeping of the step: Hessenberg column, Givens rotations, residual
  // estimate.  out[j] = {|g_{j+1}|, status}: 0 continue, 1 converged, 2
  // breakdown, 3 non-finite.
  template <typename R, int E>
  __global__ void __launch_bounds__(256)
    arnoldi_next_kernel(long long nc, const R *__restrict__ w, R *__restrict__ y, const uint32_t *__restrict__ live,
                        const ArnoldiNext st)
  {
    dependent_start();
    const double nw = sqrt(fmax(st.d_s[MAX_MULTIDOT], 0.0));
    if (blockIdx.x == 0)
      {
        // the column and the rotations in shared memory: the recurrence below
        // is serial, its loads need not be
        __shared__ double s_h[MAX_MULTIDOT + 1], s_c[MAX_MULTIDOT], s_s[MAX_MULTIDOT];
        const int         j    = st.j;
        double           *hcol = st.H + (long long)j * st.ldh;
        if (int(threadIdx.x) <= j)
          {
            s_h[threadIdx.x] = hcol[threadIdx.x] + (*st.reorth ? st.d_s[threadIdx.x] : 0.0);
            if (int(threadIdx.x) < j)
              {
                s_c[threadIdx.x] = st.cs[threadIdx.x];
                s_s[threadIdx.x] = st.sn[threadIdx.x];
              }
          }
        __syncthreads();
        if (threadIdx.x == 0)
          {
            double a = s_h[0];
            for (int i = 0; i < j; ++i)
              {
                const double b = s_h[i + 1];
                s_h[i]         = s_c[i] * a + s_s[i] * b;
                a              = -s_s[i] * a + s_c[i] * b;
              }
            const double rr = hypot(a, nw);
            const double cj = rr == 0.0 ? 1.0 : a / rr, sj = rr == 0.0 ? 0.0 : nw / rr;
            s_h[j]          = rr;
            st.cs[j]        = cj;
            st.sn[j]        = sj;
            const double gj = st.g[j];
            st.g[j + 1]     = -sj * gj;
            st.g[j]         = cj * gj;
            const double res = fabs(sj * gj);
            double       status;
            if (!isfinite(res) || !isfinite(nw))
              status = 3.0;
            else if (res <= *st.tol)
              status = 1.0;
            else if (nw == 0.0)
              status = 2.0;
            else
              status = 0.0;
            st.out[j] = make_double2(res, status);
          }
        __syncthreads();
        if (int(threadIdx.x) <= j)
          hcol[threadIdx.x] = s_h[threadIdx.x];
        if (int(threadIdx.x) == j + 1)
          hcol[j + 1] = 0.0;
      }
    axpby_body<R, E>(nc, R(1.0 / nw), w, R(0), y, live);
  }

  template <typename R>
  int arnoldi_next(long long n, const R *w, R *y, const ArnoldiNext &st, cudaStream_t s, const uint32_t *live)
  {
    constexpr int     E = pack_of<R>();
    const cudaError_t e =
      can_pack<R>(n, 0, w, y) ?
        launch_dependent(arnoldi_next_kernel<R, E>, map_blocks(n / E), 256, 0, s, n / E, w, y, live, st) :
        launch_dependent(arnoldi_next_kernel<R, 1>, map_blocks(n), 256, 0, s, n, w, y, live, st);
    return e == cudaSuccess ? SINT_OK : cuda_fail(e, "Arnoldi step");
  }
  template int arnoldi_next<double>(long long, const double *, double *, const ArnoldiNext &, cudaStream_t,
                                    const uint32_t *);
  template int arnoldi_next<float>(long long, const float *, float *, const ArnoldiNext &, cudaStream_t,
                                   const uint32_t *);

  template <typename S, typename D>
  __global__ void convert_kernel(long long n, const S *__restrict__ x, D *__restrict__ y)
  {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
      y[i] = D(x[i]);
  }

  template <typename S, typename D>
  int convert(long long n, const S *x, D *y, cudaStream_t s)
  {
    convert_kernel<S, D><<<1184, 256, 0, s>>>(n, x, y);
    count_launches(1);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? SINT_OK : cuda_fail(e, "convert");
  }
  template int convert<double, float>(long long, const double *, float *, cudaStream_t);
  template int convert<float, double>(long long, const float *, double *, cudaStream_t);

  __global__ void sqrt_kernel(double *x) { x[0] = sqrt(x[0]); }

  __global__ void select_kernel(long long n, const double *__restrict__ a, const double *__restrict__ b,
                                const double *__restrict__ na, const double *__restrict__ nb, double *out)
  {
    const double *src = *na <= *nb ? a : b;
    if (src == out)
      return;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
      out[i] = src[i];
  }
} // namespace sint

using namespace sint;

static int check_ptrs(const void *a, const void *b, int64_t n)
{
  if (n < 0 || (n > 0 && (!a || !b)))
    {
      set_error("BLAS-1: null pointer or negative size");
      return SINT_ERR_ARG;
    }
  return SINT_OK;
}

extern "C" {

int sint_vec_axpy_f64(int64_t n, double a, const double *x, double *y, sint_stream_t s)
{
  if (int e = check_ptrs(x, y, n))
    return e;
  return n ? axpby<double>(n, a, x, 1.0, y, s) : SINT_OK;
}

int sint_vec_sadd_f64(int64_t n, double sc, double a, const double *x, double *y, sint_stream_t s)
{
  if (int e = check_ptrs(x, y, n))
    return e;
  return n ? axpby<double>(n, a, x, sc, y, s) : SINT_OK;
}

int sint_vec_scale_f64(int64_t n, double a, double *x, sint_stream_t s)
{
  if (int e = check_ptrs(x, x, n))
    return e;
  return n ? axpby<double>(n, 0.0, x, a, x, s) : SINT_OK;
}

int sint_vec_axpy_f32(int64_t n, float a, const float *x, float *y, sint_stream_t s)
{
  if (int e = check_ptrs(x, y, n))
    return e;
  return n ? axpby<float>(n, a, x, 1.0, y, s) : SINT_OK;
}

int sint_vec_dot_f64(sint_ctx *c, int64_t n, const double *x, const double *y, double *result, sint_stream_t s)
{
  if (!c || !result)
    {
      set_error("sint_vec_dot_f64: null context or result");
      return SINT_ERR_ARG;
    }
  if (int e = check_ptrs(x, y, n))
    return e;
  return dot_f64(c, n, x, y, result, s);
}

int sint_vec_norm2_f64(sint_ctx *c, int64_t n, const double *x, double *result, sint_stream_t s)
{
  if (!c || !result)
    {
      set_error("sint_vec_norm2_f64: null context or result");
      return SINT_ERR_ARG;
    }
  if (int e = check_ptrs(x, x, n))
    return e;
  if (int e = dot_f64(c, n, x, x, result, s))
    return e;
  sqrt_kernel<<<1, 1, 0, s>>>(result);
  count_launches(1);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SINT_OK : cuda_fail(e, "sint_vec_norm2_f64");
}

int sint_vec_dot_f32(sint_ctx *c, int64_t n, const float *x, const float *y, double *result, sint_stream_t s)
{
  if (!c || !result)
    {
      set_error("sint_vec_dot_f32: null context or result");
      return SINT_ERR_ARG;
    }
  if (int e = check_ptrs(x, y, n))
    return e;
  return dot_f32(c, n, x, y, result, s);
}

int sint_vec_norm2_f32(sint_ctx *c, int64_t n, const float *x, double *result, sint_stream_t s)
{
  if (!c || !result)
    {
      set_error("sint_vec_norm2_f32: null context or result");
      return SINT_ERR_ARG;
    }
  if (int e = check_ptrs(x, x, n))
    return e;
  if (int e = dot_f32(c, n, x, x, result, s))
    return e;
  sqrt_kernel<<<1, 1, 0, s>>>(result);
  count_launches(1);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SINT_OK : cuda_fail(e, "sint_vec_norm2_f32");
}

int sint_vec_f64_to_f32(int64_t n, const double *x, float *y, sint_stream_t s)
{
  if (int e = check_ptrs(x, y, n))
    return e;
  return n ? convert<double, float>(n, x, y, s) : SINT_OK;
}

int sint_vec_select_f64(int64_t n, const double *a, const double *b, const double *norm_a, const double *norm_b,
                        double *out, sint_stream_t s)
{
  if (int e = check_ptrs(a, b, n))
    return e;
  if (!norm_a || !norm_b || !out)
    {
      set_error("sint_vec_select_f64: null pointer");
      return SINT_ERR_ARG;
    }
  if (n == 0)
    return SINT_OK;
  select_kernel<<<1184, 256, 0, s>>>(n, a, b, norm_a, norm_b, out);
  count_launches(1);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? SINT_OK : cuda_fail(e, "sint_vec_select_f64");
}

int sint_vec_f32_to_f64(int64_t n, const float *x, double *y, sint_stream_t s)
{
  if (int e = check_ptrs(x, y, n))
    return e;
  return n ? convert<float, double>(n, x, y, s) : SINT_OK;
}

} // extern "C"
