// 3D convolution of the learned Newton guess for inference, in one pass.
//
// The 3D network works on depth-padded windows [S][D + 2][C][H][W]: slices 1
// .. D hold the data, slices 0 and D + 1 are zero (the depth padding).  The
// training path evaluates a 3x3x3 convolution as three slice-shifted 3x3
// convolutions (sint_nn.cu), which reads and writes every activation three
// times and needs a separate pass to clear the padding.  This kernel does the
// 27 taps, a second input, the bias, a broadcast addend and the leaky ReLU in
// one pass: every output is written once, the input tile once staged.
//
// Block: 256 threads on a tile of the (x, y) plane whose width (16 to 32) is
// chosen for the window (launch_conv3d); each thread owns a column of ZB
// consecutive output slices at its (x, y) for all COUT output channels (ZB x
// COUT FP32 accumulators).  Per input channel the block stages the ZB + 2
// slices of the tile with its halo (zero outside the window) and that
// channel's 27 x COUT weights in shared memory with cp.async, double-buffered:
// the next channel's copies are in flight while this one is computed.  A
// thread reads, per (dy, dx)
// tap column, ZB + 2 input values and per dz the COUT weights (one broadcast
// read serves the warp), and issues 3 ZB COUT fused multiply-adds, as packed
// FP32 pairs of output channels (FFMA2) when COUT is a multiple of 4.
//
// Bound by issue and the FMA pipe, so what is not a multiply-add is kept out of
// the channel loop: a thread stages the same one or two (x, y) entries of every
// slice, its bounds test and offset serve the whole column, and entries outside
// the window are zeroed once for all channels.  (Row by row with a test per
// entry, staging was a fifth of the instructions at COUT 8 and almost half at
// COUT 1.)  96^3 window, 6 grains, whole guess: 3133 us with 32 x 8 tiles, rows
// and one addend at a time; 3070 us with 16 x 16 tiles where they fit better and
// the addends as here; 2596 us with the staging by columns; 2300 us with the
// width chosen for the window.
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "sint_internal.h"
#include "sint_launch.h"

namespace sint
{
  namespace
  {
    constexpr int C3_THREADS = 256;
    constexpr int C3_BOX     = 340; // largest (x, y) box of a tile with its halo

    struct Conv3dArgs
    {
      int          S, D, H, W;
      const float *x[2];   // inputs, [S][D + 2][c][H][W]
      const float *w[2];   // weights [3 (dz)][cout][c][3 (dy)][3 (dx)]
      int          c[2];   // input channels (c[1] = 0: no second input)
      const float *bias;   // [cout] or nullptr
      const float *addend; // [S / addend_group][D + 2][cout][H][W] or nullptr
      int          addend_group;
      int          leaky;
      float        slope;
      float       *out; // [S][D + 2][cout][H][W]
      int          cout;
      int          accumulate;
      int          tx, ty;   // tile of the (x, y) plane, tx * ty <= C3_THREADS
      unsigned     div_bx;   // ceil(2^16 / (tx + 2))
    };

    // output slices per thread: ZB x COUT accumulators stay within 64 registers,
    // the two staged boxes within the 48 KB of static shared memory
    template <int COUT>
    __host__ __device__ constexpr int conv3d_zb()
    {
      return COUT >= 32 ? 1 : COUT >= 16 ? 4 : COUT >= 8 ? 8 : 12;
    }

    // 4-byte asynchronous global->shared copy; !valid writes zero (source size 0)
    __device__ __forceinline__ void cp_async4(float *dst, const float *src, bool valid)
    {
      const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(sa), "l"(src), "r"(valid ? 4 : 0));
    }
    __device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;\n" ::); }
    template <int N>
    __device__ __forceinline__ void cp_async_wait_group()
    {
      asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
    }

    template <int COUT>
    __global__ void __launch_bounds__(C3_THREADS, COUT <= 2 ? 3 : 2) conv3d_kernel(const Conv3dArgs a)
    {
      constexpr int ZB = conv3d_zb<COUT>();
      constexpr int BZ = ZB + 2;
      const int     BX = a.tx + 2, box = BX * (a.ty + 2);
      // double-buffered input box and weights of one input channel
      __shared__ float s_in[2][BZ][C3_BOX]; // row pitch BX
      __shared__ __align__(16) float s_w[2][27][COUT];

      const int tiles_x = (a.W + a.tx - 1) / a.tx;
      const int x0 = (blockIdx.x % tiles_x) * a.tx, y0 = (blockIdx.x / tiles_x) * a.ty;
      const int z0 = 1 + blockIdx.y * ZB; // first output slice (window slice index)
      const int s  = blockIdx.z;
      // threads beyond the tile compute its first node again and store nothing
      const bool idle = threadIdx.x >= a.tx * a.ty;
      const int  ty = idle ? 0 : threadIdx.x / a.tx, tx = idle ? 0 : threadIdx.x - ty * a.tx;
      const long long hw = (long long)a.H * a.W;
      const int       D2 = a.D + 2;
      const int       nch = a.c[0] + a.c[1];

      // a thread copies the same one or two entries of every slice of the box
      constexpr int NE = (C3_BOX + C3_THREADS - 1) / C3_THREADS;
      // box entries outside the window are zero for all channels
      if (x0 == 0 || y0 == 0 || z0 == 1 || x0 + a.tx >= a.W || y0 + a.ty >= a.H || z0 + ZB > a.D)
        {
          float *z = &s_in[0][0][0];
          for (int i = threadIdx.x; i < 2 * BZ * C3_BOX; i += C3_THREADS)
            z[i] = 0.f;
          __syncthreads();
        }
      // slices of the box inside the window: bz0 <= bz < bz1
      const int bz0 = z0 == 1 ? 1 : 0, bz1 = min(BZ, a.D + 2 - z0);

      // stage input channel g (of x1 then x2) into buffer b
      auto stage = [&](int g, int b) {
        // selects, not a dynamic index into the parameter arrays (which would
        // copy them to local memory)
        const bool   k   = g >= a.c[0];
        const int    ci  = k ? g - a.c[0] : g;
        const int    ck  = k ? a.c[1] : a.c[0];
        const float *xk  = k ? a.x[1] : a.x[0];
        const float *wk  = k ? a.w[1] : a.w[0];
        const long long zstep = ck * hw;
        const float    *src   = xk + ((long long)s * D2 + z0 - 1) * zstep + (long long)ci * hw;
#pragma unroll
        for (int h = 0; h < NE; ++h)
          {
            const int i  = threadIdx.x + C3_THREADS * h;
            const int by = int((unsigned(i) * a.div_bx) >> 16), bx = i - by * BX; // exact: i * BX < 2^16
            const int yy = y0 - 1 + by, xx = x0 - 1 + bx;
            if (i < box && yy >= 0 && yy < a.H && xx >= 0 && xx < a.W)
              {
                const float *sp = src + (long long)yy * a.W + xx;
                float       *dp = &s_in[b][0][i];
#pragma unroll
                for (int bz = 0; bz < BZ; ++bz)
                  if (bz >= bz0 && bz < bz1)
                    cp_async4(dp + bz * C3_BOX, sp + bz * zstep, true);
              }
          }
        for (int i = threadIdx.x; i < 27 * COUT; i += C3_THREADS)
          {
            const int  tap = i / COUT, co = i % COUT, dz = tap / 9, t9 = tap % 9;
            const bool v   = co < a.cout;
            cp_async4(&s_w[b][tap][co], v ? wk + (((long long)dz * a.cout + co) * ck + ci) * 9 + t9 : a.w[0], v);
          }
      };

      // accumulators: scalar, or channel pairs when COUT is a multiple of 4
      constexpr bool PAIRS = COUT % 4 == 0;
      float          acc[PAIRS ? 1 : ZB][PAIRS ? 1 : COUT];
      float2         acc2[PAIRS ? ZB : 1][PAIRS ? COUT / 2 : 1];
#pragma unroll
      for (int z = 0; z < ZB; ++z)
#pragma unroll
        for (int co = 0; co < COUT; ++co)
          {
            if constexpr (PAIRS)
              (co & 1 ? acc2[z][co / 2].y : acc2[z][co / 2].x) = 0.f;
            else
              acc[z][co] = 0.f;
          }

      const int at = ty * BX + tx; // first tap's entry of the thread's column
      stage(0, 0);
      cp_async_commit_group();
      for (int g = 0; g < nch; ++g)
        {
          const int b = g & 1;
          if (g + 1 < nch)
            stage(g + 1, b ^ 1);
          cp_async_commit_group();
          cp_async_wait_group<1>(); // channel g has landed (only g + 1 may be pending)
          __syncthreads();
#pragma unroll
          for (int dy = 0; dy < 3; ++dy)
#pragma unroll
            for (int dx = 0; dx < 3; ++dx)
              {
                float col[BZ];
#pragma unroll
                for (int z = 0; z < BZ; ++z)
                  col[z] = s_in[b][z][at + dy * BX + dx];
                if constexpr (COUT % 4 == 0)
                  {
                    // packed FP32 pairs: two output channels per FFMA2 (each
                    // lane rounds as fmaf does), the input value in both lanes
                    float2 cc[BZ];
#pragma unroll
                    for (int z = 0; z < BZ; ++z)
                      cc[z] = make_float2(col[z], col[z]);
#pragma unroll
                    for (int dz = 0; dz < 3; ++dz)
                      {
                        const float *wr = s_w[b][(dz * 3 + dy) * 3 + dx];
#pragma unroll
                        for (int co = 0; co < COUT; co += 4)
                          {
                            const float4 q  = *reinterpret_cast<const float4 *>(wr + co);
                            const float2 w0 = make_float2(q.x, q.y), w1 = make_float2(q.z, q.w);
#pragma unroll
                            for (int z = 0; z < ZB; ++z)
                              {
                                acc2[z][co / 2]     = __ffma2_rn(w0, cc[z + dz], acc2[z][co / 2]);
                                acc2[z][co / 2 + 1] = __ffma2_rn(w1, cc[z + dz], acc2[z][co / 2 + 1]);
                              }
                          }
                      }
                  }
                else
                  {
#pragma unroll
                    for (int dz = 0; dz < 3; ++dz)
                      {
                        const float *wr = s_w[b][(dz * 3 + dy) * 3 + dx];
                        float        wv[COUT];
#pragma unroll
                        for (int co = 0; co < COUT; ++co)
                          wv[co] = wr[co];
#pragma unroll
                        for (int z = 0; z < ZB; ++z)
#pragma unroll
                          for (int co = 0; co < COUT; ++co)
                            acc[z][co] = fmaf(wv[co], col[z + dz], acc[z][co]);
                      }
                  }
              }
          // the next iteration's copies overwrite the buffer read here
          __syncthreads();
        }
      cp_async_wait_group<0>();

      const int x = x0 + tx, y = y0 + ty;
      if (idle || x >= a.W || y >= a.H)
        return;
      const long long pix = (long long)y * a.W + x;
      // slice z0, channel 0 of this thread's output and addend columns
      const long long zs = (long long)a.cout * hw;
      float          *op = a.out + ((long long)s * D2 + z0) * zs + pix;
      const float    *ap = a.addend ? a.addend + ((long long)(s / a.addend_group) * D2 + z0) * zs + pix : nullptr;
      auto            value = [&](int z, int co) -> float {
        if constexpr (PAIRS)
          return co & 1 ? acc2[z][co / 2].y : acc2[z][co / 2].x;
        else
          return acc[z][co];
      };
      if (!ap && !a.accumulate)
        {
#pragma unroll
          for (int z = 0; z < ZB; ++z)
            {
              if (z0 + z > a.D)
                break;
#pragma unroll
              for (int co = 0; co < COUT; ++co)
                {
                  if (co >= a.cout)
                    break;
                  float v = value(z, co);
                  if (a.bias)
                    v += COUT == 8 ? __ldg(a.bias + co) : a.bias[co];
                  if (a.leaky && v < 0.f)
                    v *= a.slope;
                  op[z * zs + co * hw] = v;
                }
            }
        }
      else
        {
          // the addends of CE channels are loaded together, and read-only so that
          // they may go ahead of the stores before them: one at a time each load
          // waited for its turn behind a store.  (Without addends this form costs
          // up to 3 us a launch: 2 windows of 24 x 64 x 64, 2 to 8 channels 14.2
          // us, 11.6 as above, where the bias through the read-only path gained 3
          // % at 8 output channels and lost up to 5 % at others.)
          constexpr int CE = COUT < 8 ? COUT : 8;
#pragma unroll
          for (int z = 0; z < ZB; ++z)
            {
              if (z0 + z > a.D)
                break;
#pragma unroll
              for (int c0 = 0; c0 < COUT; c0 += CE)
                {
                  float add[CE];
#pragma unroll
                  for (int c = 0; c < CE; ++c)
                    {
                      const int co = c0 + c;
                      add[c]       = ap && co < a.cout ? __ldg(ap + z * zs + co * hw) : 0.f;
                      if (a.accumulate && co < a.cout)
                        add[c] += op[z * zs + co * hw];
                    }
#pragma unroll
                  for (int c = 0; c < CE; ++c)
                    {
                      const int co = c0 + c;
                      if (co >= a.cout)
                        break;
                      float v = value(z, co);
                      if (a.bias)
                        v += __ldg(a.bias + co);
                      v += add[c];
                      if (a.leaky && v < 0.f)
                        v *= a.slope;
                      op[z * zs + co * hw] = v;
                    }
                }
            }
        }
      // the depth padding of the output: slice 0 by the first z tile, D + 1 by the last
      if (blockIdx.y == 0 || blockIdx.y == gridDim.y - 1)
        for (int co = 0; co < a.cout; ++co)
          {
            if (blockIdx.y == 0)
              a.out[(((long long)s * D2 + 0) * a.cout + co) * hw + pix] = 0.f;
            if (blockIdx.y == gridDim.y - 1)
              a.out[(((long long)s * D2 + a.D + 1) * a.cout + co) * hw + pix] = 0.f;
          }
    }

    // Tiles of the window when they are tx wide: as many rows as the threads
    // and the staged box allow.  The width with the fewest tiles is taken: the
    // multiply-adds of threads outside the window are what a kernel bound by its
    // arithmetic can save (97 x 97 nodes: 40 tiles of 25 x 10, 49 of 16 x 16, 52
    // of 32 x 8; 33 x 33: 6 of 23 x 11, 9, 10).  4 windows of 48 x 97 x
    // 97, against tiles of 32 x 8 (COUT 1, 2) or 16 x 16: COUT 2 103 -> 90 us, 4
    // 149 -> 136, 8 218 -> 205, 16 781 -> 621, 32 5454 -> 4458; COUT 1, bound by
    // its shared-memory reads, where a warp on two rows meets some banks twice,
    // 77 -> 78.  Where 32 x 8 fits (2 of 24 x 64 x 64) the pitch in a register
    // instead of a constant costs up to 2 us of 25 to 39 at COUT 2 and 8 and
    // nothing at 1, 4, 16 and 32.
    inline int conv3d_rows(int tx) { return std::min(C3_THREADS / tx, C3_BOX / (tx + 2) - 2); }
    inline long long conv3d_tiles(const Conv3dArgs &a, int tx)
    {
      const int ty = conv3d_rows(tx);
      return (long long)((a.W + tx - 1) / tx) * ((a.H + ty - 1) / ty);
    }
    template <int COUT>
    cudaError_t launch_conv3d(Conv3dArgs a, cudaStream_t st)
    {
      constexpr int ZB = conv3d_zb<COUT>();
      a.tx             = 32;
      for (int tx = 31; tx >= 16; --tx)
        if (conv3d_tiles(a, tx) < conv3d_tiles(a, a.tx))
          a.tx = tx;
      a.ty     = conv3d_rows(a.tx);
      a.div_bx = (65536 + a.tx + 1) / (a.tx + 2);
      const dim3 grid(unsigned(conv3d_tiles(a, a.tx)), unsigned((a.D + ZB - 1) / ZB), unsigned(a.S));
      conv3d_kernel<COUT><<<grid, C3_THREADS, 0, st>>>(a);
      count_launches(1);
      return cudaGetLastError();
    }
  } // namespace
} // namespace sint

using namespace sint;

extern "C" {

int sint_nn_conv3d_f32(int S, int D, int H, int W, const float *x1, int c1, const float *w1, const float *x2, int c2,
                       const float *w2, const float *bias, const float *addend, int addend_group, int leaky,
                       float slope, float *out, int cout, int accumulate, sint_stream_t stream)
{
  if (S < 1 || D < 1 || H < 1 || W < 1 || !x1 || !w1 || c1 < 1 || c2 < 0 || (c2 > 0 && (!x2 || !w2)) || !out ||
      cout < 1 || cout > 32 || (addend && (addend_group < 1 || S % addend_group != 0)) ||
      (long long)((W + 31) / 32) * ((H + 7) / 8) >= (1ll << 31) || S > 65535)
    {
      set_error("sint_nn_conv3d_f32: bad argument");
      return SINT_ERR_ARG;
    }
  Conv3dArgs a{};
  a.S = S, a.D = D, a.H = H, a.W = W;
  a.x[0] = x1, a.x[1] = c2 > 0 ? x2 : nullptr;
  a.w[0] = w1, a.w[1] = c2 > 0 ? w2 : nullptr;
  a.c[0] = c1, a.c[1] = c2;
  a.bias = bias, a.addend = addend, a.addend_group = addend ? addend_group : 1;
  a.leaky = leaky, a.slope = slope, a.out = out, a.cout = cout, a.accumulate = accumulate;
  cudaError_t e;
  if (cout <= 1)
    e = launch_conv3d<1>(a, stream);
  else if (cout <= 2)
    e = launch_conv3d<2>(a, stream);
  else if (cout <= 4)
    e = launch_conv3d<4>(a, stream);
  else if (cout <= 8)
    e = launch_conv3d<8>(a, stream);
  else if (cout <= 16)
    e = launch_conv3d<16>(a, stream);
  else
    e = launch_conv3d<32>(a, stream);
  return e == cudaSuccess ? SINT_OK : cuda_fail(e, "sint_nn_conv3d_f32");
}

} // extern "C"
