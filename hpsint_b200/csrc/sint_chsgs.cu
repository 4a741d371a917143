// Matrix-based preconditioner of the Cahn-Hilliard block.
//
// hpsint's default BlockPreconditioner2 (sintering/preconditioners.h:1222-1283,
// block_0 = "ILU", preconditioner_parameters.h) assembles the Cahn-Hilliard
// block of the tangent (OperatorCahnHilliard::do_vmult_kernel,
// preconditioners.h:85-169, through MyMatrixFreeTools::compute_matrix,
// matrix_free/tools.h:29-175) and factorises it with ILU(0)
// (lac/preconditioners.h:607-1088); the grain block keeps the inverse
// diagonal.  On the GPU the triangular solves of a natural-order ILU are
// sequential, so this build applies the assembled block through a symmetric
// Gauss-Seidel sweep pair in multicolour order instead:
//
//   * the matrix: for every node row the 2x2 blocks (J_cc, J_c,mu, J_mu,c,
//     J_mu,mu) of its 3^dim neighbours.  Two passes over slabs of cell layers:
//     ch_rows_kernel computes every cell's element-matrix rows, ch_gather_kernel
//     sums the rows that meet at a node in a fixed order (no atomics) and
//     writes the matrix in the layout the sweeps read;
//   * the sweeps: nodes coloured by the parity of their index (no two nodes
//     of one colour share a cell, so every colour updates independently);
//     forward y_n = D_n^-1 (r_n - sum_{colour(j) < colour(n)} A_nj y_j) for
//     colours 0 .. 2^dim - 1, backward z_n = y_n - D_n^-1 sum_{colour(j) >
//     colour(n)} A_nj z_j for colours 2^dim - 2 .. 0 (D_n = centre block,
//     inverted as the block-Jacobi preconditioner inverts it).
//
// FP32 copies of the matrix and of the inverted centre blocks serve the FP32
// Krylov solve.  Periodic constraints are not supported by this
// preconditioner (the set-up reports an error).
#include <string>

#include "sint_internal.h"
#include "sint_kernels.cuh"
#include "sint_launch.h"

namespace sint
{
  // Neighbours of a node row in the order the matrix stores them: by the
  // parity flip f of the neighbour's colour (bit d set = offset -1 or +1 in
  // direction d), f = 1, 2, 3, ..; the flips of one highest bit b are the
  // neighbours 3^b - 1 .. 3^(b+1) - 2.  A colour's forward sweep needs the
  // flips whose highest bit is set in the colour (they lead to smaller
  // colours), its backward sweep the others, so each sweep reads whole runs.
  template <int DIM>
  struct ChStencil
  {
    static constexpr int NQ  = 1 << DIM;
    static constexpr int NK  = DIM == 3 ? 27 : 9; // blocks of a node row
    static constexpr int NB  = NK - 1;            // neighbours
    static constexpr int INV = NB;                // slot of the inverted centre block
    static constexpr int CTR = NB + 1;            // slot of the centre block (FP64 only)

    __host__ __device__ static constexpr int slots(bool f64) { return NB + (f64 ? 2 : 1); }
    __host__ __device__ static constexpr int run_begin(int bit) { return bit == 0 ? 0 : (bit == 1 ? 2 : 8); }
    __host__ __device__ static constexpr int run_end(int bit) { return bit == 0 ? 2 : (bit == 1 ? 8 : 26); }
    __host__ __device__ static constexpr int flip(int k)
    {
      return k < 2 ? 1 : (k < 4 ? 2 : (k < 8 ? 3 : (k < 10 ? 4 : (k < 14 ? 5 : (k < 18 ? 6 : 7)))));
    }
    __host__ __device__ static constexpr int first(int f)
    {
      return f == 1 ? 0 : (f == 2 ? 2 : (f == 3 ? 4 : (f == 4 ? 8 : (f == 5 ? 10 : (f == 6 ? 14 : 18)))));
    }
    // offset of neighbour k in direction d
    __host__ __device__ static constexpr int off(int k, int d)
    {
      const int f = flip(k), s = k - first(f);
      int       rank = 0;
      for (int e = 0; e < d; ++e)
        rank += (f >> e) & 1;
      return ((f >> d) & 1) ? (((s >> rank) & 1) ? 1 : -1) : 0;
    }
  };

  // The nodes of colour c (bit d = parity of the index in direction d) form
  // the lattice x = 2 a + p0, y = 2 b + p1 (, z = 2 c + p2) of m[c][d] nodes
  // per direction, t = a + m0 (b + m1 c) their index in it.  The matrix is
  // stored colour by colour in groups of 32 rows, slot-major inside a group:
  // a warp of a sweep reads one contiguous piece, 16 bytes per lane and load.
  struct ColourLattice
  {
    long long cnt[8]; // nodes of the colour
    long long grp[8]; // 32-row groups of the colours before it
    long long groups; // all groups
    int       m[8][3];
  };

  template <int DIM>
  ColourLattice colour_lattice(const Grid &g)
  {
    ColourLattice L{};
    for (int col = 0; col < 8; ++col)
      {
        long long cnt = col < (1 << DIM) ? 1 : 0;
        for (int d = 0; d < 3; ++d)
          {
            L.m[col][d] = d < DIM ? (g.nn[d] - ((col >> d) & 1) + 1) / 2 : 1;
            cnt *= L.m[col][d];
          }
        L.cnt[col] = cnt;
        L.grp[col] = L.groups;
        L.groups += (cnt + 31) / 32;
      }
    return L;
  }

  // Element of entry e of slot k of row t of a colour whose groups start at
  // grp, in a matrix of `slots` slots: [group][slot][4 / V][32 rows][V], V
  // values per 16 bytes.
  template <typename R>
  __device__ __forceinline__ long long ch_index(long long grp, long long t, int slots, int k, int e)
  {
    constexpr int V = 16 / int(sizeof(R));
    return ((grp + (t >> 5)) * slots + k) * 128 + (e / V) * (32 * V) + int(t & 31) * V + e % V;
  }

  // Per-point coefficients of the CH tangent (OperatorCahnHilliard): the
  // symmetric mobility matrix (rows of its upper triangle), dM/dc grad mu minus
  // the grains' summed velocity (ADV), dM/dgrad c, f_cc; then the coefficients
  // w0 + L f_{eta_i eta_i} of the Allen-Cahn diagonal.
  template <int DIM>
  struct ChCoef
  {
    static constexpr int M = 0, MV = DIM * (DIM + 1) / 2, K = MV + DIM, FCC = K + DIM * DIM, AC = FCC + 1;
    __host__ __device__ static constexpr int m(int a, int b)
    {
      return a <= b ? (DIM == 3 ? (a == 0 ? b : a + b + 1) : a + b) : m(b, a);
    }
  };

  // Scratch of the assembly: for local node l of a cell, the values that node
  // gets from the cell, at the node's place: plane p of [planes][ring layers]
  // [layer], p = (l NQ + m) 3 + e for the element matrix (e = cc, c mu, mu c)
  // and 3 NQ^2 + l G + i for the Allen-Cahn diagonal.  A layer is a node layer
  // of the slowest direction, rows padded to an even pitch; ring layers are
  // reused slab after slab.
  struct ChScratch
  {
    double   *s;
    long long plane;  // elements per plane
    long long layer;  // elements per layer
    int       pitch;  // elements per x row
    int       ring;   // layers kept
    int       first, count; // the slab's cell layers
  };

  template <int DIM>
  __device__ __forceinline__ long long ch_place(const ChScratch &sc, int x, int y, int z)
  {
    return DIM == 3 ? (z % sc.ring) * sc.layer + (long long)y * sc.pitch + x : (y % sc.ring) * sc.layer + x;
  }

  // Value and gradient at this thread's point from a cell's 2^dim nodal
  // values u[l] (l = lx + 2 ly + 4 lz), sum-factorised as eval_vg.
  template <int DIM, typename R>
  __device__ __forceinline__ void eval_local(const R *u, const QP<DIM, R> &w, R &val, R (&grad)[DIM])
  {
    if constexpr (DIM == 3)
      {
        R vx[2][2], dx[2][2];
#pragma unroll
        for (int lz = 0; lz < 2; ++lz)
#pragma unroll
          for (int ly = 0; ly < 2; ++ly)
            {
              const R u0 = u[2 * ly + 4 * lz], u1 = u[1 + 2 * ly + 4 * lz];
              vx[lz][ly] = w.wA[0] * u0 + w.wB[0] * u1;
              dx[lz][ly] = (u1 - u0) * w.ih[0];
            }
        R vxy[2], dxy[2], dyy[2];
#pragma unroll
        for (int lz = 0; lz < 2; ++lz)
          {
            vxy[lz] = w.wA[1] * vx[lz][0] + w.wB[1] * vx[lz][1];
            dxy[lz] = w.wA[1] * dx[lz][0] + w.wB[1] * dx[lz][1];
            dyy[lz] = (vx[lz][1] - vx[lz][0]) * w.ih[1];
          }
        val     = w.wA[2] * vxy[0] + w.wB[2] * vxy[1];
        grad[0] = w.wA[2] * dxy[0] + w.wB[2] * dxy[1];
        grad[1] = w.wA[2] * dyy[0] + w.wB[2] * dyy[1];
        grad[2] = (vxy[1] - vxy[0]) * w.ih[2];
      }
    else
      {
        R vx[2], dx[2];
#pragma unroll
        for (int ly = 0; ly < 2; ++ly)
          {
            const R u0 = u[2 * ly], u1 = u[1 + 2 * ly];
            vx[ly]     = w.wA[0] * u0 + w.wB[0] * u1;
            dx[ly]     = (u1 - u0) * w.ih[0];
          }
        val     = w.wA[1] * vx[0] + w.wB[1] * vx[1];
        grad[0] = w.wA[1] * dx[0] + w.wB[1] * dx[1];
        grad[1] = (vx[1] - vx[0]) * w.ih[1];
      }
  }

  // 2x2 inverse of a centre block (entries by rows), the guarded point inverse
  // where it is singular.
  __device__ __forceinline__ void ch_invert(const double (&a)[4], double (&inv)[4])
  {
    const double det   = a[0] * a[3] - a[1] * a[2];
    const double scale = fabs(a[0] * a[3]) + fabs(a[1] * a[2]);
    if (det != 0.0 && isfinite(det) && fabs(det) > 1e-14 * scale)
      {
        inv[0] = a[3] / det;
        inv[1] = -a[1] / det;
        inv[2] = -a[2] / det;
        inv[3] = a[0] / det;
      }
    else
      {
        inv[0] = fabs(a[0]) > 1.0e-10 ? 1.0 / a[0] : 1.0;
        inv[3] = fabs(a[3]) > 1.0e-10 ? 1.0 / a[3] : 1.0;
        inv[1] = inv[2] = 0.0;
      }
  }

  // Element-matrix rows of the slab's cells.  A block takes 256 / 2^dim cells
  // (consecutive in x, then row by row); thread = (point, cell) for the point
  // coefficients, then (row, cell).  A row's contraction with the trial
  // functions at the points is the transposed sum factorisation that phase 3
  // of the cell kernels uses, with the row's coefficient vectors as "fluxes":
  // ~450 FP64 operations a row instead of ~3800 for the double loop over
  // columns and points.  CUT: absent grains have zero values (grain cut-off
  // of the preconditioner) and no Allen-Cahn row.  ADV: J_cc gains
  // -(psi_m sum_i v_i, grad phi_l), the grains' diagonals -(phi_l v_i, grad
  // phi_l) (precondition_advection_ch, operator_sintering_generic.h:800-824).
  template <int DIM, int G, bool TENS, bool CUT, bool ADV>
  __global__ void __launch_bounds__(256, 2)
    ch_rows_kernel(const Grid g, const Phys ph, const double *__restrict__ lin, const ChScratch sc,
                   const uint16_t *__restrict__ mask, const AdvData adv)
  {
    using CF            = ChCoef<DIM>;
    constexpr int NQ    = 1 << DIM;
    constexpr int CELLS = 256 / NQ;
    constexpr int C     = G + 2;
    constexpr int NCOEF = CF::AC + G;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *s_nodes = reinterpret_cast<double *>(smem_raw); // [comp][l][cell]
    double *s_coef  = s_nodes + C * 256;                     // [coef][q][cell]
    double *s_vel   = s_coef + NCOEF * 256;                  // [grain][dim][q][cell] (ADV)

    const int cell = threadIdx.x % CELLS, q = threadIdx.x / CELLS;
    const long long per_layer = DIM == 3 ? (long long)g.n[0] * g.n[1] : g.n[0];
    const long long idx       = (long long)blockIdx.x * CELLS + cell;
    const bool      valid     = idx < per_layer * sc.count;
    int             cc[3]     = {0, 0, 0};
    if (valid)
      {
        const int layer = int(idx / per_layer);
        const int rest  = int(idx - layer * per_layer);
        cc[0]           = rest % g.n[0];
        cc[1]           = DIM == 3 ? rest / g.n[0] : sc.first + layer;
        cc[2]           = DIM == 3 ? sc.first + layer : 0;
      }
    const int       nx = cc[0] + (q & 1), ny = cc[1] + ((q >> 1) & 1), nz = DIM == 3 ? cc[2] + (q >> 2) : 0;
    const long long node = node_index(g, nx, ny, nz); // node q of this cell
    {
      double v[C];
#pragma unroll
      for (int comp = 0; comp < C; ++comp)
        v[comp] = valid ? lin[comp * g.ld + node] : 0.0;
#pragma unroll
      for (int comp = 0; comp < C; ++comp)
        s_nodes[comp * 256 + threadIdx.x] = v[comp];
    }
    const long long n_cells = (long long)g.n[0] * g.n[1] * g.n[2];
    const long long lcell   = cc[0] + (long long)g.n[0] * (cc[1] + (long long)g.n[1] * cc[2]);
    const unsigned  gmask   = (CUT && valid) ? mask[lcell] : ~0u;
    __syncthreads();

    const PhysR<double>   pr(ph);
    const QP<DIM, double> w(g, q);
    auto                  eval = [&](int comp, double &val, double(&grad)[DIM]) {
      double u[NQ];
#pragma unroll
      for (int l = 0; l < NQ; ++l)
        u[l] = s_nodes[comp * 256 + l * CELLS + cell];
      eval_local<DIM>(u, w, val, grad);
    };
    {
      double c, gc[DIM], mu_unused, gmu[DIM];
      eval(0, c, gc);
      eval(1, mu_unused, gmu);
      double eta[gdim(G)];
      double geta[gdim(G)][DIM];
#pragma unroll
      for (int i = 0; i < G; ++i)
        {
          eval(2 + i, eta[i], geta[i]);
          if (CUT && ((gmask >> i) & 1u) == 0u)
            {
              eta[i] = 0.0;
#pragma unroll
              for (int d = 0; d < DIM; ++d)
                geta[i][d] = 0.0;
            }
        }
      double *cf = s_coef + threadIdx.x; // stride 256 per coefficient
      {
        double Mm[DIM][DIM];
        mobility_matrix<DIM, G, TENS>(pr, c, eta, gc, geta, Mm);
#pragma unroll
        for (int a = 0; a < DIM; ++a)
#pragma unroll
          for (int b = a; b < DIM; ++b)
            cf[(CF::M + CF::m(a, b)) * 256] = Mm[a][b];
      }
      double vs[3] = {0.0, 0.0, 0.0};
      if constexpr (ADV)
        {
          const double gp0 = 0.5 - 0.5 / sqrt(3.0), gp1 = 0.5 + 0.5 / sqrt(3.0);
#pragma unroll 1
          for (int i = 0; i < G; ++i)
            {
              double v[3] = {0.0, 0.0, 0.0};
              int    s    = -1;
              if (valid && !(CUT && ((gmask >> i) & 1u) == 0u))
                s = adv.cell_segments[i * n_cells + lcell];
              if (s >= 0 && s < adv.n_segments)
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
                {
                  vs[e] += v[e];
                  s_vel[(i * DIM + e) * 256 + threadIdx.x] = v[e];
                }
            }
        }
      double mv[DIM];
      dM_dc_times<DIM, TENS>(pr, c, gc, gmu, mv);
#pragma unroll
      for (int d = 0; d < DIM; ++d)
        cf[(CF::MV + d) * 256] = ADV ? mv[d] - vs[d] : mv[d];
      double Km[DIM][DIM];
      dM_dgrad_c<DIM, TENS>(pr, c, gc, gmu, Km);
#pragma unroll
      for (int a = 0; a < DIM; ++a)
#pragma unroll
        for (int b = 0; b < DIM; ++b)
          cf[(CF::K + a * DIM + b) * 256] = Km[a][b];
      const double omc = 1.0 - c;
      cf[CF::FCC * 256] = 2.0 * pr.A * (c * c) + 4.0 * pr.A * c * (2.0 * c - 2.0) + 2.0 * pr.A * (omc * omc) + 2.0 * pr.B;
      double s2 = 0.0;
#pragma unroll
      for (int i = 0; i < G; ++i)
        s2 += eta[i] * eta[i];
#pragma unroll
      for (int i = 0; i < G; ++i)
        {
          const double e   = eta[i];
          const double fee = pr.B * (12.0 - 12.0 * c + 2.0 * e * (12.0 * c - 24.0) + 24.0 * (e * e) + 12.0 * s2);
          cf[(CF::AC + i) * 256] = pr.w0 + pr.L * fee;
        }
    }
    __syncthreads();
    if (!valid)
      return;

    // this thread: row of local node l, the same for a whole warp
    const int                     l = q;
    const CellConsts<DIM, double> k(g);
    // phi_l and its gradient at point qq from the 1D factors
    double f1[DIM][2];
#pragma unroll
    for (int d = 0; d < DIM; ++d)
#pragma unroll
      for (int b = 0; b < 2; ++b)
        f1[d][b] = ((l >> d) & 1) == b ? k.x1 : k.x0;
    auto phi = [&](int qq) {
      double v = f1[0][qq & 1] * f1[1][(qq >> 1) & 1];
      if constexpr (DIM == 3)
        v *= f1[2][(qq >> 2) & 1];
      return v;
    };
    auto dphi = [&](int qq, int d) {
      double v = ((l >> d) & 1) ? k.ih[d] : -k.ih[d];
#pragma unroll
      for (int e = 0; e < DIM; ++e)
        if (e != d)
          v *= f1[e][(qq >> e) & 1];
      return v;
    };
    const double   *cf    = s_coef + cell; // coefficient i at point qq: cf[i * 256 + qq * CELLS]
    const long long place = ch_place<DIM>(sc, nx, ny, nz);
    double         *out   = sc.s + (long long)(l * NQ * 3) * sc.plane + place;
    double          gg[DIM][NQ], v[NQ], r[NQ];
    // (c, c): psi_m (w0 phi_l + dM/dc grad mu . grad phi_l) + (dM/dgrad c)^T grad phi_l . grad psi_m
#pragma unroll
    for (int qq = 0; qq < NQ; ++qq)
      {
        const double *cq = cf + qq * CELLS;
        double        dp[DIM];
#pragma unroll
        for (int a = 0; a < DIM; ++a)
          dp[a] = dphi(qq, a);
        double v0 = pr.w0 * phi(qq);
#pragma unroll
        for (int a = 0; a < DIM; ++a)
          v0 += cq[(CF::MV + a) * 256] * dp[a];
        v[qq] = v0;
#pragma unroll
        for (int b = 0; b < DIM; ++b)
          {
            double t = cq[(CF::K + b) * 256] * dp[0];
#pragma unroll
            for (int a = 1; a < DIM; ++a)
              t += cq[(CF::K + a * DIM + b) * 256] * dp[a];
            gg[b][qq] = t;
          }
      }
    cell_integrate_vg<DIM>(v, gg, k, r);
#pragma unroll
    for (int m = 0; m < NQ; ++m)
      out[(m * 3 + 0) * sc.plane] = r[m];
    asm volatile("" ::: "memory"); // one matrix at a time in registers
    // (c, mu): M grad phi_l . grad psi_m
#pragma unroll
    for (int qq = 0; qq < NQ; ++qq)
      {
        const double *cq = cf + qq * CELLS;
        v[qq]            = 0.0;
#pragma unroll
        for (int b = 0; b < DIM; ++b)
          {
            double t = 0.0;
#pragma unroll
            for (int a = 0; a < DIM; ++a)
              t += cq[(CF::M + CF::m(a, b)) * 256] * dphi(qq, a);
            gg[b][qq] = t;
          }
      }
    cell_integrate_vg<DIM>(v, gg, k, r);
#pragma unroll
    for (int m = 0; m < NQ; ++m)
      out[(m * 3 + 1) * sc.plane] = r[m];
    asm volatile("" ::: "memory");
    // (mu, c): -f_cc phi_l psi_m - kappa_c grad phi_l . grad psi_m (exact element Laplacian)
#pragma unroll
    for (int qq = 0; qq < NQ; ++qq)
      v[qq] = -cf[CF::FCC * 256 + qq * CELLS] * phi(qq);
    cell_integrate_v<DIM>(v, k, r);
#pragma unroll
    for (int m = 0; m < NQ; ++m)
      out[(m * 3 + 2) * sc.plane] = r[m] + g.kstd[0][l ^ m];
    // Allen-Cahn diagonal: (w0 + L f_ee) phi_l^2 + L kappa_p |grad phi_l|^2 (- phi_l v_i . grad phi_l)
    double *ac = sc.s + (long long)(3 * NQ * NQ + l * G) * sc.plane + place;
#pragma unroll
    for (int qq = 0; qq < NQ; ++qq)
      v[qq] = k.JxW * phi(qq) * phi(qq);
#pragma unroll 1
    for (int i = 0; i < G; ++i)
      {
        double d = g.kstd[1][0];
#pragma unroll
        for (int qq = 0; qq < NQ; ++qq)
          d += v[qq] * cf[(CF::AC + i) * 256 + qq * CELLS];
        if constexpr (ADV)
#pragma unroll 1
          for (int qq = 0; qq < NQ; ++qq)
            {
              double vd = 0.0;
#pragma unroll
              for (int e = 0; e < DIM; ++e)
                vd += s_vel[(i * DIM + e) * 256 + qq * CELLS + cell] * dphi(qq, e);
              d -= k.JxW * phi(qq) * vd;
            }
        if (CUT && ((gmask >> i) & 1u) == 0u)
          d = 0.0;
        ac[i * sc.plane] = d;
      }
  }

  // Outputs of the assembly.
  struct ChOut
  {
    double *A64;   // the matrix in FP64: neighbours, inverted centre block, centre block
    float  *A32;   // in FP32: neighbours, inverted centre block
    double *raw;   // pc_raw: centre blocks and Allen-Cahn diagonal by node
    double *inv64; // pc_inv64 / pc_inv32: the inverse diagonal (blocks 4 ..)
    float  *inv32;
  };

  // One thread per pair of x-adjacent nodes (one of either colour) of the node
  // layers [first, first + layers) and group of slots (blockIdx.y: GATHER_SPLIT
  // groups of neighbours, then the centre block with the Allen-Cahn diagonal):
  // sums what the pair's cells left in the scratch, 16 bytes per load, and
  // writes the matrix, its inverted centre blocks (guarded as
  // precond_invert_kernel) and the diagonal.
  // Bound by memory: it reads 8 (3 NQ^2 / NQ + G) NQ bytes and writes ~1350
  // bytes per node (3D).
  constexpr int GATHER_SPLIT = 4;

  template <int DIM>
  __global__ void __launch_bounds__(128)
    ch_gather_kernel(const Grid g, double walg, int G, const ChScratch sc, int first, int layers,
                     const ColourLattice cl, const ChOut o)
  {
    using S              = ChStencil<DIM>;
    constexpr int   NQ   = S::NQ;
    const int       half = (g.nn[0] + 1) / 2;
    const long long rows = DIM == 3 ? (long long)g.nn[1] * layers : layers;
    const long long i    = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= half * rows)
      return;
    const long long row = i / half;
    const int       x   = 2 * int(i - row * half);
    const int       y   = DIM == 3 ? int(row % g.nn[1]) : first + int(row);
    const int       z   = DIM == 3 ? first + int(row / g.nn[1]) : 0;
    const bool      two = x + 1 < g.nn[0]; // the second node exists
    // cells around the two nodes, by the local node l they have there
    unsigned ok0 = 0u, ok1 = 0u;
#pragma unroll
    for (int l = 0; l < NQ; ++l)
      {
        const int cx = x - (l & 1), cy = y - ((l >> 1) & 1), cz = DIM == 3 ? z - (l >> 2) : 0;
        const bool yz = cy >= 0 && cy < g.n[1] && (DIM == 2 || (cz >= 0 && cz < g.n[2]));
        if (yz && cx >= 0 && cx < g.n[0])
          ok0 |= 1u << l;
        if (yz && two && cx + 1 < g.n[0])
          ok1 |= 1u << l;
      }
    const double *src = sc.s + ch_place<DIM>(sc, x, y, z);
    auto          add = [&](long long p, int l, double &a, double &b) {
      const double2 t = *reinterpret_cast<const double2 *>(src + p * sc.plane);
      if ((ok0 >> l) & 1u)
        a += t.x;
      if ((ok1 >> l) & 1u)
        b += t.y;
    };
    const int       c0 = ((y & 1) << 1) | ((z & 1) << 2), c1 = c0 | 1;
    const long long yz0 = (y >> 1) + (long long)cl.m[c0][1] * (z >> 1);
    const long long t0 = (x >> 1) + cl.m[c0][0] * yz0, t1 = (x >> 1) + cl.m[c1][0] * yz0;
    const long long node = node_index(g, x, y, z);
    // mass of two local nodes that differ in d directions: JxW sums to h/3 and h/6 per direction
    double cellv = 1.0;
#pragma unroll
    for (int d = 0; d < DIM; ++d)
      cellv *= g.h[d] / 6.0;
    auto store = [&](int k, const double(&a)[4], const double(&b)[4]) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
        {
          if (h && !two)
            break;
          const double(&v)[4] = h ? b : a;
          const long long grp = cl.grp[h ? c1 : c0], t = h ? t1 : t0;
          double         *d64 = o.A64 + ch_index<double>(grp, t, S::slots(true), k, 0);
          *reinterpret_cast<double2 *>(d64)      = make_double2(v[0], v[1]);
          *reinterpret_cast<double2 *>(d64 + 64) = make_double2(v[2], v[3]);
          if (k != S::CTR)
            *reinterpret_cast<float4 *>(o.A32 + ch_index<float>(grp, t, S::slots(false), k, 0)) =
              make_float4(float(v[0]), float(v[1]), float(v[2]), float(v[3]));
        }
    };
    // block of the neighbour at offset (dx, dy, dz): local nodes l of this
    // node and m = l + offset in the cells that hold both
    auto block = [&](int dx, int dy, int dz, double(&a)[4], double(&b)[4]) {
      double mass = walg * cellv;
#pragma unroll
      for (int e = 0; e < 4; ++e)
        a[e] = b[e] = 0.0;
#pragma unroll
      for (int l = 0; l < NQ; ++l)
        {
          const int mx = (l & 1) + dx, my = ((l >> 1) & 1) + dy, mz = (l >> 2) + dz;
          if (mx < 0 || mx > 1 || my < 0 || my > 1 || mz < 0 || mz > 1)
            continue;
          const int m = mx + 2 * my + 4 * mz;
#pragma unroll
          for (int e = 0; e < 3; ++e)
            add((l * NQ + m) * 3 + e, l, a[e], b[e]);
          a[3] += (ok0 >> l) & 1u ? 1.0 : 0.0;
          b[3] += (ok1 >> l) & 1u ? 1.0 : 0.0;
        }
      mass *= (dx ? 1.0 : 2.0) * (dy ? 1.0 : 2.0) * (DIM == 3 ? (dz ? 1.0 : 2.0) : 1.0);
      a[3] *= mass;
      b[3] *= mass;
    };
#pragma unroll
    for (int k = 0; k < S::NB; ++k)
      {
        if (k * GATHER_SPLIT / S::NB != int(blockIdx.y))
          continue;
        double a[4], b[4];
        block(S::off(k, 0), S::off(k, 1), DIM == 3 ? S::off(k, 2) : 0, a, b);
        store(k, a, b);
      }
    if (blockIdx.y < GATHER_SPLIT)
      return;
    {
      double a[4], b[4], ia[4], ib[4];
      block(0, 0, 0, a, b);
      ch_invert(a, ia);
      ch_invert(b, ib);
      store(S::CTR, a, b);
      store(S::INV, ia, ib);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        {
          o.raw[e * g.ld + node] = a[e];
          if (two)
            o.raw[e * g.ld + node + 1] = b[e];
        }
    }
    for (int gr = 0; gr < G; ++gr)
      {
        double a = 0.0, b = 0.0;
#pragma unroll
        for (int l = 0; l < NQ; ++l)
          add(3 * NQ * NQ + l * G + gr, l, a, b);
        const double ia = fabs(a) > 1.0e-10 ? 1.0 / a : 1.0, ib = fabs(b) > 1.0e-10 ? 1.0 / b : 1.0;
        const long long at  = (4 + gr) * g.ld + node;
        o.raw[at]           = a;
        o.inv64[at]         = ia;
        o.inv32[at]         = float(ia);
        if (two)
          {
            o.raw[at + 1]   = b;
            o.inv64[at + 1] = ib;
            o.inv32[at + 1] = float(ib);
          }
      }
  }

  // The FP64 matrix in the interface's order: A[(k * 4 + e) * ld + n],
  // neighbour k = (dx + 1) + 3 (dy + 1) (+ 9 (dz + 1)); zeros behind the last node.
  template <int DIM>
  __global__ void __launch_bounds__(256) ch_export_kernel(const Grid g, const ColourLattice cl,
                                                          const double *__restrict__ A, double *__restrict__ out)
  {
    using S           = ChStencil<DIM>;
    const long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= g.ld)
      return;
    if (n >= g.N)
      {
        for (int i = 0; i < S::NK * 4; ++i)
          out[i * g.ld + n] = 0.0;
        return;
      }
    const int x = int(n % g.nn[0]), y = int((n / g.nn[0]) % g.nn[1]);
    const int z = DIM == 3 ? int(n / ((long long)g.nn[0] * g.nn[1])) : 0;
    const int       col = (x & 1) | ((y & 1) << 1) | ((z & 1) << 2);
    const long long t   = (x >> 1) + (long long)cl.m[col][0] * ((y >> 1) + (long long)cl.m[col][1] * (z >> 1));
#pragma unroll
    for (int k = 0; k < S::NK; ++k)
      {
        const int  kk  = k < S::NB ? k : S::CTR;
        const int  pos = kk == S::CTR ? S::NK / 2
                                      : (S::off(kk, 0) + 1) + 3 * (S::off(kk, 1) + 1) +
                                          (DIM == 3 ? 9 * (S::off(kk, 2) + 1) : 0);
        for (int e = 0; e < 4; ++e)
          out[(pos * 4 + e) * g.ld + n] = A[ch_index<double>(cl.grp[col], t, S::slots(true), kk, e)];
      }
  }

  // One colour of the forward (FWD) or backward sweep; z holds the c and mu
  // blocks of the result (y of the forward sweep, overwritten by the
  // backward one).  Bound by the matrix: 16 bytes per lane and load, a warp's
  // rows contiguous, every neighbour block read in exactly one of the two
  // sweeps.  The colours depend on one another, the matrix does not: every
  // launch but an apply's first is a programmatic dependent launch that loads
  // its FP32 rows while the colour before it ends, and waits only before it
  // reads z (the first launch is an ordinary one, so the matrix and r are
  // complete before any of them starts).  PRE: how many of the three runs
  // (2, 6, 18 neighbours) are loaded before the wait; all of them take 128
  // registers, which pays while the colour is one wave of blocks (FP32 apply
  // at 48^3 cells 36.5 us, PRE = 2 48.7 us, PRE = 0 95.1 us; at 96^3 111.8 /
  // 94.8 / 124.4 us; at 192^3 756 / 655 / 690 us).  With the rule as it stands
  // the apply takes 632 / 661 / 705 us at 192^3 cells with 4 / 6 / 9 grains;
  // entry-major rows without programmatic launches took 951 us with 9.  The
  // first launch of an apply (ac_blocks > 0) also does the grain rows z =
  // inverse diagonal * r in its blocks behind the colour's.
  constexpr int       SGS_THREADS  = 128;
  constexpr long long SGS_WAVE_F32 = 148 * 4 * SGS_THREADS, SGS_WAVE_F64 = 148 * 2 * SGS_THREADS;

  template <int DIM, typename R, bool FWD, int PRE>
  __global__ void __launch_bounds__(SGS_THREADS)
    ch_sgs_kernel(const Grid g, int colour, const ColourLattice cl, const R *__restrict__ A, const R *__restrict__ r,
                  R *__restrict__ z, unsigned colour_blocks, int G, const R *__restrict__ ac_inv)
  {
    using S                 = ChStencil<DIM>;
    constexpr int   V       = 16 / int(sizeof(R));
    constexpr int   SLOTS   = S::slots(sizeof(R) == 8);
    const long long ld      = g.ld;
    cudaTriggerProgrammaticLaunchCompletion();
    if (blockIdx.x >= colour_blocks)
      {
        // V nodes per thread; block vectors start every component 16-byte aligned
        const long long n = ((long long)(blockIdx.x - colour_blocks) * SGS_THREADS + threadIdx.x) * V;
        for (int i = 0; i < G; ++i)
          {
            const R *rv = r + (2 + i) * ld, *dv = ac_inv + i * ld;
            R       *zv = z + (2 + i) * ld;
            if (n + V <= g.N)
              {
                if constexpr (V == 4)
                  {
                    const float4 a = *reinterpret_cast<const float4 *>(rv + n);
                    const float4 d = *reinterpret_cast<const float4 *>(dv + n);
                    *reinterpret_cast<float4 *>(zv + n) = make_float4(d.x * a.x, d.y * a.y, d.z * a.z, d.w * a.w);
                  }
                else
                  {
                    const double2 a = *reinterpret_cast<const double2 *>(rv + n);
                    const double2 d = *reinterpret_cast<const double2 *>(dv + n);
                    *reinterpret_cast<double2 *>(zv + n) = make_double2(d.x * a.x, d.y * a.y);
                  }
              }
            else
              for (long long j = n; j < g.N; ++j)
                zv[j] = dv[j] * rv[j];
          }
        return;
      }
    const long long t = (long long)blockIdx.x * SGS_THREADS + threadIdx.x;
    if (t >= cl.cnt[colour])
      return;
    const int m0 = cl.m[colour][0], m1 = cl.m[colour][1];
    int       a, b, c;
    if (cl.cnt[colour] < (1ll << 31))
      {
        const unsigned ti = unsigned(t), row = ti / unsigned(m0), lay = row / unsigned(m1);
        a = int(ti - row * unsigned(m0)), b = int(row - lay * unsigned(m1)), c = int(lay);
      }
    else
      a = int(t % m0), b = int((t / m0) % m1), c = int(t / ((long long)m0 * m1));
    const int x = 2 * a + (colour & 1), y = 2 * b + ((colour >> 1) & 1), zz = DIM == 3 ? 2 * c + (colour >> 2) : 0;
    const long long n    = node_index(g, x, y, zz);
    const R        *Arow = A + ((cl.grp[colour] + (t >> 5)) * SLOTS) * 128 + (t & 31) * V;
    // which of the neighbours at offsets -1 and +1 exist, per direction
    const bool lo[3] = {x > 0, y > 0, zz > 0}, hi[3] = {x + 1 < g.nn[0], y + 1 < g.nn[1], zz + 1 < g.nn[2]};
    const long long step[3] = {1, g.nn[0], (long long)g.nn[0] * g.nn[1]};
    R               s0 = R(0), s1 = R(0);
    auto            load = [&](int k, R(&e)[4]) {
      if constexpr (V == 4)
        {
          const float4 f = __ldcs(reinterpret_cast<const float4 *>(Arow + k * 128));
          e[0] = f.x, e[1] = f.y, e[2] = f.z, e[3] = f.w;
        }
      else
        {
          const double2 f = __ldcs(reinterpret_cast<const double2 *>(Arow + k * 128));
          const double2 h = __ldcs(reinterpret_cast<const double2 *>(Arow + k * 128 + 64));
          e[0] = f.x, e[1] = f.y, e[2] = h.x, e[3] = h.y;
        }
    };
    // FP32: the row's blocks of every run of this sweep, loaded before the wait
    R row[PRE > 0 ? S::run_end(PRE - 1) : 1][4], inv[4], tmp[4];
    if constexpr (PRE > 0)
      {
#pragma unroll
        for (int bit = PRE - 1; bit >= 0; --bit)
          if ((((colour >> bit) & 1) != 0) == FWD)
            {
#pragma unroll
              for (int k = S::run_begin(bit); k < S::run_end(bit); ++k)
                load(k, row[k]);
            }
      }
    load(S::INV, inv);
    const R r0 = FWD ? r[n] : R(0), r1 = FWD ? r[ld + n] : R(0);
    cudaGridDependencySynchronize();
#pragma unroll
    for (int bit = 0; bit < DIM; ++bit)
      if ((((colour >> bit) & 1) != 0) == FWD)
        {
          // a run's sums by themselves: in one sum over all runs the FP32 apply was
          // 8.2e-8 off in the 2-norm (192^3 cells, 9 grains), so 7.4e-8
          R t0 = R(0), t1 = R(0);
#pragma unroll
          for (int k = S::run_begin(bit); k < S::run_end(bit); ++k)
            {
              bool      in = true;
              long long j  = n;
#pragma unroll
              for (int d = 0; d < DIM; ++d)
                {
                  const int o = S::off(k, d);
                  if (o != 0)
                    in = in && (o < 0 ? lo[d] : hi[d]);
                  j += o * step[d];
                }
              if (bit >= PRE)
                load(k, tmp);
              const R(&e)[4] = bit >= PRE ? tmp : row[bit >= PRE ? 0 : k];
              const R v0 = in ? z[j] : R(0), v1 = in ? z[ld + j] : R(0);
              t0 += e[0] * v0 + e[1] * v1;
              t1 += e[2] * v0 + e[3] * v1;
            }
          s0 += t0;
          s1 += t1;
        }
    if (FWD)
      {
        const R a0 = r0 - s0, a1 = r1 - s1;
        z[n]       = inv[0] * a0 + inv[1] * a1;
        z[ld + n]  = inv[2] * a0 + inv[3] * a1;
      }
    else
      {
        z[n]      = z[n] - (inv[0] * s0 + inv[1] * s1);
        z[ld + n] = z[ld + n] - (inv[2] * s0 + inv[3] * s1);
      }
  }

  template <int DIM, int G, bool TENS, bool CUT, bool ADV>
  static cudaError_t launch_ch_rows_g(const Ctx *c, const ChScratch &sc, const uint16_t *mask, const AdvData &adv,
                                      cudaStream_t s)
  {
    const Grid  &g    = c->grid;
    const size_t smem = size_t(G + 2 + ChCoef<DIM>::AC + G + (ADV ? G * DIM : 0)) * 256 * sizeof(double);
    auto         k    = ch_rows_kernel<DIM, G, TENS, CUT, ADV>;
    if (smem > 48 * 1024)
      if (cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)))
        return e;
    const long long cells = (DIM == 3 ? (long long)g.n[0] * g.n[1] : g.n[0]) * sc.count;
    const long long nb    = (cells + (256 >> DIM) - 1) / (256 >> DIM);
    k<<<dim3((unsigned)nb), 256, smem, s>>>(g, c->phys, c->lin64, sc, mask, adv);
    count_launches(1);
    return cudaGetLastError();
  }

  template <int DIM, bool TENS, bool CUT, bool ADV>
  static cudaError_t launch_ch_rows(const Ctx *c, const ChScratch &sc, const uint16_t *mask, const AdvData &adv,
                                    cudaStream_t s)
  {
    switch (c->G)
      {
#define SINT_CASE(GG)                                                                                             \
  case GG: return launch_ch_rows_g<DIM, GG, TENS, CUT, ADV>(c, sc, mask, adv, s);
        SINT_CASE(1) SINT_CASE(2) SINT_CASE(3) SINT_CASE(4) SINT_CASE(5) SINT_CASE(6)
        SINT_CASE(7) SINT_CASE(8) SINT_CASE(9) SINT_CASE(10) SINT_CASE(11) SINT_CASE(12)
#undef SINT_CASE
      }
    return cudaErrorInvalidValue;
  }

  // Scratch of the assembly: as many cell layers per slab as fit in this many
  // bytes (of a context's own, kept for its later set-ups), at least one, which
  // takes two node layers.  Small slabs that stay in L2 lose more to short
  // launches than they save in HBM traffic: set-up of 118^3 cells, 6 grains,
  // with 64 / 256 / 576 / 1024 MiB 5.13 / 3.56 / 3.35 / 3.41 ms when the bound was
  // chosen, 2.96 ms with these 512 MiB today (eight colour launches that updated
  // the matrix in place, and the separate diagonal kernel: 9.4 ms).
  constexpr size_t CH_SCRATCH_BYTES = size_t(512) << 20;

  template <int DIM>
  static long long scratch_planes(int G)
  {
    constexpr int NQ = 1 << DIM;
    return 3 * NQ * NQ + NQ * G;
  }

  // Layout in `bytes` of scratch; the ring holds at least two layers, even if
  // they take more (scratch_bytes).
  template <int DIM>
  static ChScratch scratch_layout(const Grid &g, int G, size_t bytes)
  {
    ChScratch sc{};
    sc.pitch              = (g.nn[0] + 1) / 2 * 2;
    sc.layer              = DIM == 3 ? (long long)sc.pitch * g.nn[1] : sc.pitch;
    const long long slabs = (long long)(bytes / (size_t(scratch_planes<DIM>(G) * sc.layer) * sizeof(double)));
    const int       layers = g.n[DIM - 1];
    sc.ring               = int(slabs < 2 ? 2 : (slabs < layers + 1 ? slabs : layers + 1));
    sc.plane              = sc.layer * sc.ring;
    return sc;
  }
  template <int DIM>
  static size_t scratch_bytes(const Grid &g, int G, size_t bytes)
  {
    return size_t(scratch_layout<DIM>(g, G, bytes).plane) * size_t(scratch_planes<DIM>(G)) * sizeof(double);
  }

  // The scratch of a context, at its first set-up.  Where the device has no
  // room for it, the set-up works in smaller slabs: in the tile-face partials,
  // which no other call of the context uses meanwhile, if they hold two layers
  // (3D: from 16 cell layers on for 12 grains, from 35 for one; 2D: from 10 and
  // 17 rows), else in an allocation of two layers.
  template <int DIM>
  static cudaError_t scratch_alloc(Ctx *c)
  {
    const size_t want = scratch_bytes<DIM>(c->grid, c->G, CH_SCRATCH_BYTES);
    const size_t two  = scratch_bytes<DIM>(c->grid, c->G, 0);
    cudaError_t  e    = cudaMalloc(&c->ch_scratch, want);
    c->ch_scratch_bytes = want;
    if (e == cudaErrorMemoryAllocation && two <= c->partial_bytes)
      {
        c->ch_scratch       = c->partial;
        c->ch_scratch_bytes = c->partial_bytes;
        e                   = cudaSuccess;
      }
    else if (e == cudaErrorMemoryAllocation && two < want)
      {
        e                   = cudaMalloc(&c->ch_scratch, two);
        c->ch_scratch_bytes = two;
      }
    cudaGetLastError(); // a refused allocation is not the next launch's error
    if (e != cudaSuccess)
      c->ch_scratch = nullptr;
    return e;
  }

  template <int DIM, bool TENS, bool CUT, bool ADV>
  static cudaError_t assemble_dim(const Ctx *c, const uint16_t *mask, const AdvData &adv, cudaStream_t s)
  {
    const Grid         &g  = c->grid;
    const ColourLattice cl = colour_lattice<DIM>(g);
    ChScratch           sc = scratch_layout<DIM>(g, c->G, c->ch_scratch_bytes);
    sc.s                   = c->ch_scratch;
    const ChOut o{c->ch_A64, c->ch_A32, c->pc_raw, c->pc_inv64, c->pc_inv32};
    const int   n = g.n[DIM - 1];
    for (int first = 0; first < n; first += sc.ring - 1)
      {
        sc.first = first;
        sc.count = n - first < sc.ring - 1 ? n - first : sc.ring - 1;
        if (const cudaError_t e = launch_ch_rows<DIM, TENS, CUT, ADV>(c, sc, mask, adv, s))
          return e;
        // node layers whose cells are all done; the last slab also has the last layer
        const int       layers = sc.count + (first + sc.count == n ? 1 : 0);
        const long long pairs  = (long long)((g.nn[0] + 1) / 2) * (DIM == 3 ? g.nn[1] : 1) * layers;
        ch_gather_kernel<DIM><<<dim3((unsigned)((pairs + 127) / 128), GATHER_SPLIT + 1), 128, 0, s>>>(g, c->phys.w_alg, c->G, sc, first,
                                                                                    layers, cl, o);
        count_launches(1);
        if (const cudaError_t e = cudaGetLastError())
          return e;
      }
    return cudaSuccess;
  }
  template <int DIM>
  static cudaError_t assemble_mob(const Ctx *c, cudaStream_t s)
  {
    const uint16_t *m   = preconditioner_mask(c);
    const AdvData  *adv = active_adv(c);
    const bool      t   = c->params.tensorial != 0;
#define SINT_ASM(TT, CC, AA) assemble_dim<DIM, TT, CC, AA>(c, m, adv ? *adv : AdvData(), s)
    if (t)
      return m ? (adv ? SINT_ASM(true, true, true) : SINT_ASM(true, true, false))
               : (adv ? SINT_ASM(true, false, true) : SINT_ASM(true, false, false));
    return m ? (adv ? SINT_ASM(false, true, true) : SINT_ASM(false, true, false))
             : (adv ? SINT_ASM(false, false, true) : SINT_ASM(false, false, false));
#undef SINT_ASM
  }

  int ch_sgs_setup(Ctx *c, cudaStream_t s)
  {
    if (c->grid.periodic)
      {
        set_error("sint_precond_setup: the Cahn-Hilliard Gauss-Seidel preconditioner does not support periodic "
                  "constraints; use the block-Jacobi preconditioner");
        return SINT_ERR_ARG;
      }
    const bool          d3 = c->grid.dim == 3;
    const ColourLattice cl = d3 ? colour_lattice<3>(c->grid) : colour_lattice<2>(c->grid);
    const size_t        n64 = size_t(cl.groups) * 128 * (d3 ? ChStencil<3>::slots(true) : ChStencil<2>::slots(true));
    const size_t        n32 = size_t(cl.groups) * 128 * (d3 ? ChStencil<3>::slots(false) : ChStencil<2>::slots(false));
    cudaError_t         e   = cudaSuccess;
    // the rows that fill up a colour's last group of 32 are never used
    if ((!c->ch_A64 && (e = cudaMalloc(&c->ch_A64, n64 * sizeof(double))) != cudaSuccess) ||
        (!c->ch_A32 && (e = cudaMalloc(&c->ch_A32, n32 * sizeof(float))) != cudaSuccess) ||
        (!c->ch_scratch && (e = d3 ? scratch_alloc<3>(c) : scratch_alloc<2>(c)) != cudaSuccess))
      return cuda_fail(e, "sint_precond_setup: Cahn-Hilliard matrix allocation");
    e = c->grid.dim == 3 ? assemble_mob<3>(c, s) : assemble_mob<2>(c, s);
    return e == cudaSuccess ? SINT_OK : cuda_fail(e, "sint_precond_setup: Cahn-Hilliard matrix");
  }

  template <int DIM, typename R>
  static cudaError_t sweeps(const Ctx *c, const R *A, const R *ac_inv, const R *r, R *z, cudaStream_t s)
  {
    constexpr int       NCOL = 1 << DIM;
    const Grid         &g    = c->grid;
    const ColourLattice cl   = colour_lattice<DIM>(g);
    auto                launch = [&](int colour, bool fwd) -> cudaError_t {
      const long long cnt = cl.cnt[colour];
      if (cnt == 0)
        return cudaSuccess;
      constexpr int  V     = 16 / int(sizeof(R)), T = SGS_THREADS;
      const bool     first = fwd && colour == 0;
      const unsigned nb    = (unsigned)((cnt + T - 1) / T);
      const unsigned ac    = first ? (unsigned)((g.N + T * V - 1) / (T * V)) : 0u;
      auto           go = [&](auto k) {
        return launch_dependent_if(!first, k, dim3(nb + ac), dim3(T), 0, s, g, colour, cl, A, r, z, nb, c->G, ac_inv);
      };
      // the rows of one wave of blocks at the registers all runs take
      const bool all = cnt <= (sizeof(R) == 4 ? SGS_WAVE_F32 : SGS_WAVE_F64);
      return fwd ? (all ? go(ch_sgs_kernel<DIM, R, true, DIM>) : go(ch_sgs_kernel<DIM, R, true, 2>)) :
                   (all ? go(ch_sgs_kernel<DIM, R, false, DIM>) : go(ch_sgs_kernel<DIM, R, false, 2>));
    };
    for (int col = 0; col < NCOL; ++col)
      if (cudaError_t e = launch(col, true))
        return e;
    for (int col = NCOL - 2; col >= 0; --col)
      if (cudaError_t e = launch(col, false))
        return e;
    return cudaSuccess;
  }

  template <typename R>
  cudaError_t ch_sgs_apply(const Ctx *c, const R *r, R *z, cudaStream_t s)
  {
    const R *A = sizeof(R) == 8 ? reinterpret_cast<const R *>(c->ch_A64) : reinterpret_cast<const R *>(c->ch_A32);
    const R *ac_inv = (sizeof(R) == 8 ? reinterpret_cast<const R *>(c->pc_inv64)
                                      : reinterpret_cast<const R *>(c->pc_inv32)) + 4 * c->ld;
    return c->grid.dim == 3 ? sweeps<3, R>(c, A, ac_inv, r, z, s) : sweeps<2, R>(c, A, ac_inv, r, z, s);
  }
  template cudaError_t ch_sgs_apply<double>(const Ctx *, const double *, double *, cudaStream_t);
  template cudaError_t ch_sgs_apply<float>(const Ctx *, const float *, float *, cudaStream_t);

  cudaError_t ch_matrix_export(const Ctx *c, double *A, cudaStream_t s)
  {
    const Grid    &g  = c->grid;
    const unsigned nb = (unsigned)((g.ld + 255) / 256);
    if (g.dim == 3)
      ch_export_kernel<3><<<nb, 256, 0, s>>>(g, colour_lattice<3>(g), c->ch_A64, A);
    else
      ch_export_kernel<2><<<nb, 256, 0, s>>>(g, colour_lattice<2>(g), c->ch_A64, A);
    count_launches(1);
    return cudaGetLastError();
  }
} // namespace sint
