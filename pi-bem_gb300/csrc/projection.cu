// L2 projections onto the continuous Q1 space of the mesh -- the steps pi-BEM
// runs on either side of the solve:
//   BEMProblem::compute_normals            (source/bem_problem.cc:1998-2070)
//   BEMProblem::compute_surface_gradients  (source/bem_problem.cc:1879-1996)
//   BEMProblem::compute_gradients          (source/bem_problem.cc:1747-1877)
// Each solves M u_c = b_c for the three components c: M_ij = sum over cells and
// Gauss points of phi_i phi_j JxW (the consistent Q1 mass matrix, the same for
// every component), b_c,i = sum phi_i g_c JxW with the projected field g =
//   the cell normal n                          (normals),
//   grad_G u = sum_b u_b grad_G phi_b          (surface gradients of u),
//   grad_G phi + n dphi/dn                     (gradients; dphi/dn interpolated),
// where grad_G phi_b = J (J^T J)^-1 grad_ref phi_b is the tangential gradient
// of the shape function through the bilinear map (J = [x_xi, x_eta], 3 x 2), as
// deal.II's FEValues gives it for a codimension-one mesh.
//
// The reference assembles M into a Trilinos matrix and solves with GMRES + AMG to
// the solver tolerance; here M's rows are gathered once from per-cell 4 x 4 blocks
// (merged, in a fixed order) and the 3 R systems are solved together with
// Jacobi-preconditioned CG (M is SPD and well conditioned) to a relative residual
// of 1e-13.
//
// The CG runs on the device: three launches an iteration, each adding the partial
// sums of the one before in a fixed order in every block, so the host only looks
// whether all columns are done, every PROJ_BATCH iterations and while the next ones
// run.  What bounds it: the launches up to about 10^5 nodes, then the FP64 units in
// the mass product (the matrix-free product did 16 FMA a row and component, the
// merged row does 9) and in the loads.  Vectors are node-major with the three
// components of a column together (the output's layout), so a neighbour is one
// 24-byte gather.
//   Measured (GB300), the normals and three columns' gradients at 41,336 nodes through
// the host interface: 9.0 ms with nine launches and two host round trips an iteration ->
// 2.9 ms (2.0 ms of kernels, 32 iterations of 26 us for three columns).
#include <algorithm>
#include <cmath>
#include <vector>

#include "kernels.h"
#include "krylov.h"
#include "pdl.cuh"

namespace pibem
{
  namespace
  {
    enum : int
    {
      PROJ_NORMALS = 0,
      PROJ_SURFACE_GRADIENT = 1,
      PROJ_GRADIENT = 2
    };

    constexpr int PROJ_THREADS = 192;     // a multiple of 3: a thread keeps its component
    constexpr int PROJ_BLOCKS  = 2 * 152; // most blocks (partial sums) per column triple
    constexpr int PROJ_BATCH   = 4;       // iterations between two looks at the columns
    constexpr int PROJ_LONG    = 8;       // nodes in more cells: a warp per row

    // per cell: the 4 x 4 mass block and, for NR columns r0.., the 4 x 3 load vectors
    // rhs[((c R + r) 4 + a) 3 + k].  The geometry of a quadrature point is formed once
    // for the NR columns.
    template <int NR>
    __global__ void proj_cell_kernel(int mode, int64_t n_cells, int nq, int R, int64_t N,
                                     const int32_t *__restrict__ cells,
                                     const double *__restrict__ xyz,
                                     const double *__restrict__ gpts,
                                     const double *__restrict__ qshape,
                                     const double *__restrict__ qjxw,
                                     const double *__restrict__ qnrm,
                                     const double *__restrict__ u, const double *__restrict__ dudn,
                                     double *__restrict__ cellM, double *__restrict__ rhs)
    {
      const int64_t c = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (c >= n_cells)
        return;
      const int r0 = blockIdx.y * NR, nr = min(NR, R - r0);
      double    v[12];
      int       nd[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        {
          nd[j] = cells[4 * c + j];
#pragma unroll
          for (int k = 0; k < 3; ++k)
            v[3 * j + k] = xyz[3 * int64_t(nd[j]) + k];
        }
      double uc[NR][4], dc[NR][4], b[NR][12], M[10];
#pragma unroll
      for (int r = 0; r < NR; ++r)
        {
#pragma unroll
          for (int a = 0; a < 4; ++a)
            {
              uc[r][a] = mode != PROJ_NORMALS && r < nr ? u[int64_t(r0 + r) * N + nd[a]] : 0.0;
              dc[r][a] = mode == PROJ_GRADIENT && r < nr ? dudn[int64_t(r0 + r) * N + nd[a]] : 0.0;
            }
#pragma unroll
          for (int i = 0; i < 12; ++i)
            b[r][i] = 0.0;
        }
#pragma unroll
      for (int i = 0; i < 10; ++i)
        M[i] = 0.0;
      for (int q = 0; q < nq; ++q)
        {
          const int64_t t = c * nq + q;
          const double  w = qjxw[t];
          double        sh[4], sw[4], nv[3];
#pragma unroll
          for (int a = 0; a < 4; ++a)
            {
              sh[a] = qshape[4 * t + a];
              sw[a] = sh[a] * w;
            }
#pragma unroll
          for (int k = 0; k < 3; ++k)
            nv[k] = mode != PROJ_SURFACE_GRADIENT ? qnrm[3 * t + k] : 0.0;
          if (blockIdx.y == 0)
            {
              int i = 0;
#pragma unroll
              for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int e = a; e < 4; ++e, ++i)
                  M[i] = fma(sw[a], sh[e], M[i]);
            }
          if (mode == PROJ_NORMALS)
            {
#pragma unroll
              for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int k = 0; k < 3; ++k)
                  b[0][3 * a + k] = fma(sw[a], nv[k], b[0][3 * a + k]);
              continue;
            }
          const double xi = gpts[2 * q], eta = gpts[2 * q + 1];
          double       tx[3], ty[3];
#pragma unroll
          for (int k = 0; k < 3; ++k)
            {
              tx[k] = (1 - eta) * (v[3 + k] - v[k]) + eta * (v[9 + k] - v[6 + k]);
              ty[k] = (1 - xi) * (v[6 + k] - v[k]) + xi * (v[9 + k] - v[3 + k]);
            }
          const double g11 = tx[0] * tx[0] + tx[1] * tx[1] + tx[2] * tx[2];
          const double g12 = tx[0] * ty[0] + tx[1] * ty[1] + tx[2] * ty[2];
          const double g22 = ty[0] * ty[0] + ty[1] * ty[1] + ty[2] * ty[2];
          const double det = 1.0 / (g11 * g22 - g12 * g12);
#pragma unroll
          for (int r = 0; r < NR; ++r)
            if (r < nr)
              {
                // grad_ref of the interpolated u (lexicographic Q1 shape functions)
                const double sx = (1 - eta) * (uc[r][1] - uc[r][0]) + eta * (uc[r][3] - uc[r][2]);
                const double se = (1 - xi) * (uc[r][2] - uc[r][0]) + xi * (uc[r][3] - uc[r][1]);
                const double cx = (g22 * sx - g12 * se) * det, ce = (g11 * se - g12 * sx) * det;
                double       dn = 0;
                if (mode == PROJ_GRADIENT)
#pragma unroll
                  for (int a = 0; a < 4; ++a)
                    dn = fma(sh[a], dc[r][a], dn);
#pragma unroll
                for (int k = 0; k < 3; ++k)
                  {
                    const double g = fma(tx[k], cx, fma(ty[k], ce, nv[k] * dn));
#pragma unroll
                    for (int a = 0; a < 4; ++a)
                      b[r][3 * a + k] = fma(sw[a], g, b[r][3 * a + k]);
                  }
              }
        }
      if (blockIdx.y == 0)
        {
          int i = 0;
#pragma unroll
          for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int e = a; e < 4; ++e, ++i)
              cellM[16 * c + 4 * a + e] = cellM[16 * c + 4 * e + a] = M[i];
        }
#pragma unroll
      for (int r = 0; r < NR; ++r)
        if (r < nr)
#pragma unroll
          for (int i = 0; i < 12; ++i)
            rhs[(c * R + r0 + r) * 12 + i] = b[r][i];
    }

    // the block's sums of n values per thread into part[(triple n + k) gridDim.x + block]
    // (warp butterfly, then the warps in order)
    template <int n>
    __device__ __forceinline__ void proj_partials(double (&s)[n], double *__restrict__ part)
    {
      __shared__ double red[PROJ_THREADS / 32][n];
      const int         lane = threadIdx.x & 31;
      for (int k = 0; k < n; ++k)
        {
          for (int o = 16; o > 0; o >>= 1)
            s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
          if (lane == 0)
            red[threadIdx.x >> 5][k] = s[k];
        }
      __syncthreads();
      if (threadIdx.x < n)
        {
          double t = 0;
          for (int w = 0; w < PROJ_THREADS / 32; ++w)
            t += red[w][threadIdx.x];
          part[(int64_t(blockIdx.y) * n + threadIdx.x) * gridDim.x + blockIdx.x] = t;
        }
    }

    // tot[k] = the sum of the nb partials of the block's column triple: a warp per
    // value, lanes over the partials, fixed butterfly
    template <int n>
    __device__ __forceinline__ void proj_totals(const double *__restrict__ part, int nb, double *tot)
    {
      const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
      if (k < n)
        {
          double        s = 0;
          const double *v = part + (int64_t(blockIdx.y) * n + k) * nb;
          for (int b0 = lane; b0 - lane < nb; b0 += 8 * 32)
            {
              double a[8];
#pragma unroll
              for (int u = 0; u < 8; ++u)
                a[u] = b0 + 32 * u < nb ? v[b0 + 32 * u] : 0.0;
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (b0 - lane + 32 * u < nb)
                  s += a[u];
            }
          for (int o = 16; o > 0; o >>= 1)
            s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == 0)
            tot[k] = s;
        }
      __syncthreads();
    }

    // For node i, visit its (cell, local vertex) incidences in a fixed order: the
    // node -> cells list is ordered by cell, a cell listed twice for a node that
    // is two vertices of a collapsed cell.
    template <typename F>
    __device__ inline void for_each_incidence(int64_t i, const int32_t *elem_off,
                                              const int32_t *elem_ids, const int32_t *cells, F f)
    {
      int prev = -1, used = -1;
      for (int e = elem_off[i]; e < elem_off[i + 1]; ++e)
        {
          const int c = elem_ids[e];
          int       from = c == prev ? used + 1 : 0, a = -1;
          for (int j = from; j < 4 && a < 0; ++j)
            if (cells[4 * int64_t(c) + j] == int(i))
              a = j;
          prev = c;
          used = a;
          if (a >= 0)
            f(c, a);
        }
    }

    // The rows of M: node i's (column, value) pairs are slot e of its slice of 32
    // nodes, at slice_ptr[i / 32] + 32 e + i % 32 (coalesced over the nodes), cnt[i]
    // of them; entries with the same column merged (not in nodes of many cells).
    // And b, r = b, the inverse diagonal, p = r / diag, x = 0, with the partial sums
    // of b.b and r.z of the three components (blockIdx.y: column triple).
    __global__ void __launch_bounds__(PROJ_THREADS)
      proj_assemble_kernel(int64_t N, int R, const int32_t *__restrict__ elem_off,
                           const int32_t *__restrict__ elem_ids, const int32_t *__restrict__ cells,
                           const double *__restrict__ cellM, const double *__restrict__ rhs,
                           const int64_t *__restrict__ slice_ptr, int32_t *__restrict__ cnt,
                           int32_t *__restrict__ mcol, double *__restrict__ mval,
                           double *__restrict__ dinv, double *__restrict__ x, double *__restrict__ r,
                           double *__restrict__ p, double *__restrict__ part)
    {
      const int rr = blockIdx.y;
      double    s[6] = {0, 0, 0, 0, 0, 0};
      for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N;
           i += int64_t(gridDim.x) * blockDim.x)
        {
          const int64_t base = slice_ptr[i >> 5] + (i & 31);
          const bool    merge = elem_off[i + 1] - elem_off[i] <= PROJ_LONG;
          int           n = 0;
          double        d = 0, b[3] = {0, 0, 0};
          for_each_incidence(i, elem_off, elem_ids, cells, [&](int c, int a) {
            d += cellM[16 * int64_t(c) + 5 * a];
            for (int k = 0; k < 3; ++k)
              b[k] += rhs[(int64_t(c) * R + rr) * 12 + 3 * a + k];
            if (rr == 0)
              for (int e = 0; e < 4; ++e)
                {
                  const int    col = cells[4 * int64_t(c) + e];
                  const double m   = cellM[16 * int64_t(c) + 4 * a + e];
                  int          f   = merge ? 0 : n;
                  while (f < n && mcol[base + 32 * int64_t(f)] != col)
                    ++f;
                  if (f < n)
                    mval[base + 32 * int64_t(f)] += m;
                  else
                    {
                      mcol[base + 32 * int64_t(n)] = col;
                      mval[base + 32 * int64_t(n)] = m;
                      ++n;
                    }
                }
          });
          const double di = 1.0 / d;
          if (rr == 0)
            {
              cnt[i]  = n;
              dinv[i] = di;
            }
          for (int k = 0; k < 3; ++k)
            {
              const int64_t t = (int64_t(rr) * N + i) * 3 + k;
              const double  z = b[k] * di;
              x[t]            = 0;
              r[t]            = b[k];
              p[t]            = z;
              s[k]     = fma(b[k], b[k], s[k]);
              s[3 + k] = fma(b[k], z, s[3 + k]);
            }
        }
      proj_partials<6>(s, part);
    }

    // q = M p of column triple blockIdx.y, and the partial sums of p.q.  Blocks
    // [0, row_blocks): a thread per row of at most PROJ_LONG cells; the others: a
    // warp per long row.
    __global__ void __launch_bounds__(PROJ_THREADS)
      proj_mass_kernel(int64_t N, int row_blocks, int n_long, const int32_t *__restrict__ long_rows,
                       const int32_t *__restrict__ elem_off, const int64_t *__restrict__ slice_ptr,
                       const int32_t *__restrict__ cnt, const int32_t *__restrict__ mcol,
                       const double *__restrict__ mval, const int *__restrict__ act,
                       const double *__restrict__ p, double *__restrict__ q,
                       double *__restrict__ part)
    {
      pdl_entry();
      const int rr = blockIdx.y;
      if (!(act[3 * rr] | act[3 * rr + 1] | act[3 * rr + 2]))
        return;
      const double *pr = p + int64_t(rr) * N * 3;
      double       *qr = q + int64_t(rr) * N * 3;
      double        s[3] = {0, 0, 0};
      if (int(blockIdx.x) < row_blocks)
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N;
             i += int64_t(row_blocks) * blockDim.x)
          {
            if (elem_off[i + 1] - elem_off[i] > PROJ_LONG)
              continue;
            const int64_t base = slice_ptr[i >> 5] + (i & 31);
            const int     n    = cnt[i];
            double        y0 = 0, y1 = 0, y2 = 0;
#pragma unroll 4
            for (int e = 0; e < n; ++e)
              {
                const double  m = mval[base + 32 * int64_t(e)];
                const double *v = pr + 3 * int64_t(mcol[base + 32 * int64_t(e)]);
                y0 = fma(m, v[0], y0);
                y1 = fma(m, v[1], y1);
                y2 = fma(m, v[2], y2);
              }
            qr[3 * i]     = y0;
            qr[3 * i + 1] = y1;
            qr[3 * i + 2] = y2;
            s[0] = fma(pr[3 * i], y0, s[0]);
            s[1] = fma(pr[3 * i + 1], y1, s[1]);
            s[2] = fma(pr[3 * i + 2], y2, s[2]);
          }
      else
        {
          const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
          for (int l = int(blockIdx.x - row_blocks) * nw + int(threadIdx.x >> 5); l < n_long;
               l += int(gridDim.x - row_blocks) * nw)
            {
              const int64_t i = long_rows[l], base = slice_ptr[i >> 5] + (i & 31);
              double        y[3] = {0, 0, 0};
              for (int e = lane; e < cnt[i]; e += 32)
                {
                  const double  m = mval[base + 32 * int64_t(e)];
                  const double *v = pr + 3 * int64_t(mcol[base + 32 * int64_t(e)]);
                  for (int k = 0; k < 3; ++k)
                    y[k] = fma(m, v[k], y[k]);
                }
              for (int k = 0; k < 3; ++k)
                {
                  for (int o = 16; o > 0; o >>= 1)
                    y[k] += __shfl_xor_sync(0xffffffffu, y[k], o);
                  if (lane == 0)
                    {
                      qr[3 * i + k] = y[k];
                      s[k]          = fma(pr[3 * i + k], y[k], s[k]);
                    }
                }
            }
        }
      proj_partials<3>(s, part);
    }

    // x += alpha p, r -= alpha q with alpha = r.z / p.q per component (0 for a
    // component that is done), and the partial sums of r.r and r.z
    __global__ void __launch_bounds__(PROJ_THREADS)
      proj_update_kernel(int64_t N, int mass_blocks, const double *__restrict__ pq_part,
                         const double *__restrict__ rz, const int *__restrict__ act,
                         const double *__restrict__ dinv, const double *__restrict__ p,
                         const double *__restrict__ q, double *__restrict__ x,
                         double *__restrict__ r, double *__restrict__ part)
    {
      pdl_entry();
      const int rr = blockIdx.y;
      if (!(act[3 * rr] | act[3 * rr + 1] | act[3 * rr + 2]))
        return;
      __shared__ double tot[3], alpha[3];
      proj_totals<3>(pq_part, mass_blocks, tot);
      if (threadIdx.x < 3)
        {
          const int c        = 3 * rr + threadIdx.x;
          const double pq    = tot[threadIdx.x];
          alpha[threadIdx.x] = act[c] && pq != 0 ? rz[c] / pq : 0.0;
        }
      __syncthreads();
      // a thread takes the values threadIdx.x, + the grid's, ... of the triple's 3 N
      // (coalesced), all of component threadIdx.x % 3
      // (3 N fits in 32 bits: node ids are below 2^31 / 8)
      const int64_t  o  = int64_t(rr) * N * 3;
      const uint32_t n3 = uint32_t(N) * 3;
      const int      k  = threadIdx.x % 3;
      double         s0 = 0, s1 = 0;
      for (uint32_t t = blockIdx.x * PROJ_THREADS + threadIdx.x; t < n3; t += gridDim.x * PROJ_THREADS)
        {
          x[o + t]       = fma(alpha[k], p[o + t], x[o + t]);
          const double v = fma(-alpha[k], q[o + t], r[o + t]);
          r[o + t]       = v;
          const double w = v * v;
          s0 += w;
          s1 = fma(w, dinv[t / 3], s1);
        }
      __shared__ double red[2][3][PROJ_THREADS / 3];
      red[0][k][threadIdx.x / 3] = s0;
      red[1][k][threadIdx.x / 3] = s1;
      __syncthreads();
      static_assert(PROJ_THREADS == 192, "six warps add six sums of 64 values");
      const int     w = threadIdx.x >> 5, lane = threadIdx.x & 31;
      const double *v = red[w / 3][w % 3];
      double        t = v[lane] + v[lane + 32];
      for (int d = 16; d > 0; d >>= 1)
        t += __shfl_xor_sync(0xffffffffu, t, d);
      if (lane == 0)
        part[(int64_t(rr) * 6 + w) * gridDim.x + blockIdx.x] = t;
    }

    // p = z + beta p with beta = the new r.z over the old one; block 0 keeps the new
    // r.z and drops the components with |r| <= tol |b| (or r.z = 0): they take no
    // further steps, so a column's result does not depend on the others.  First: the
    // sums of the start (part holds b.b and r.z; p is in place).
    template <bool FIRST>
    __global__ void __launch_bounds__(PROJ_THREADS)
      proj_direction_kernel(int64_t N, int blocks, double tol, const double *__restrict__ part,
                            const double *__restrict__ rz_old, double *__restrict__ rz_new,
                            const int *__restrict__ act_old, int *__restrict__ act_new,
                            double *__restrict__ bb, const double *__restrict__ dinv,
                            const double *__restrict__ r, double *__restrict__ p)
    {
      pdl_entry();
      const int rr = blockIdx.y;
      if (!FIRST && !(act_old[3 * rr] | act_old[3 * rr + 1] | act_old[3 * rr + 2]))
        {
          if (blockIdx.x == 0 && threadIdx.x < 3)
            act_new[3 * rr + threadIdx.x] = 0;
          return;
        }
      __shared__ double tot[6], beta[3];
      proj_totals<6>(part, blocks, tot);
      if (threadIdx.x < 3)
        {
          const int    c = 3 * rr + threadIdx.x;
          const double n = tot[3 + threadIdx.x], o = FIRST ? 0.0 : rz_old[c];
          beta[threadIdx.x] = o != 0 ? n / o : 0.0;
          if (blockIdx.x == 0)
            {
              if (FIRST)
                {
                  bb[c]      = tot[threadIdx.x];
                  act_new[c] = n != 0;
                }
              else
                act_new[c] = act_old[c] && n != 0 && !(sqrt(tot[threadIdx.x]) <= tol * sqrt(bb[c]));
              rz_new[c] = n;
            }
        }
      if constexpr (FIRST)
        return;
      __syncthreads();
      const int64_t  o  = int64_t(rr) * N * 3;
      const uint32_t n3 = uint32_t(N) * 3;
      const int      k  = threadIdx.x % 3;
      for (uint32_t t = blockIdx.x * PROJ_THREADS + threadIdx.x; t < n3; t += gridDim.x * PROJ_THREADS)
        p[o + t] = fma(beta[k], p[o + t], r[o + t] * dinv[t / 3]);
    }

    inline unsigned grid_for(int64_t n) { return unsigned((n + PROJ_THREADS - 1) / PROJ_THREADS); }
  } // namespace

  void proj_row_layout(int64_t N, const std::vector<int32_t> &elem_off, std::vector<int64_t> &slice_ptr,
                       std::vector<int32_t> &long_rows)
  {
    slice_ptr.assign(size_t((N + 31) / 32) + 1, 0);
    long_rows.clear();
    for (int64_t i = 0; i < N; ++i)
      {
        const int64_t inc = elem_off[i + 1] - elem_off[i];
        if (inc > PROJ_LONG)
          long_rows.push_back(int32_t(i));
        int64_t &w = slice_ptr[size_t(i >> 5) + 1];
        w          = std::max(w, 32 * 4 * inc);
      }
    for (size_t k = 1; k < slice_ptr.size(); ++k)
      slice_ptr[k] += slice_ptr[k - 1];
  }

  void l2_projection(const ProjectionArgs &a, cudaStream_t s)
  {
    const int64_t N = a.n_nodes, C = a.n_cells;
    const int     R = a.R, ncol = 3 * R;
    const int64_t n = N * ncol;
    const int row_blocks = int(std::min<int64_t>(PROJ_BLOCKS, grid_for(N)));
    const int long_blocks = std::min(PROJ_BLOCKS, (a.n_long + PROJ_THREADS / 32 - 1) / (PROJ_THREADS / 32));
    const int mass_blocks = row_blocks + long_blocks;
    double  *cellM = a.work, *rhs = cellM + 16 * C, *dinv = rhs + 12 * C * R, *r = dinv + N, *p = r + n,
           *q = p + n, *pa = q + n, *pb = pa + int64_t(2) * ncol * PROJ_BLOCKS,
           *rz = pb + int64_t(2) * ncol * PROJ_BLOCKS, *bb = rz + 2 * ncol, *mval = bb + ncol;
    int32_t *mcol = reinterpret_cast<int32_t *>(mval + a.n_slots), *cnt = mcol + a.n_slots;
    int     *act = cnt + N; // [2][ncol]
    auto cell = [&](auto kern, int nr) {
      kern<<<dim3(grid_for(C), unsigned((R + nr - 1) / nr)), PROJ_THREADS, 0, s>>>(
        a.mode, C, a.nq, R, N, a.cells, a.xyz, a.gpts, a.qshape, a.qjxw, a.qnrm, a.u, a.dudn, cellM, rhs);
    };
    if (a.mode == PROJ_NORMALS) // one instantiation per mode: a column has the same bits in any batch
      cell(proj_cell_kernel<1>, 1);
    else
      cell(proj_cell_kernel<3>, 3);
    const dim3 rows(row_blocks, R);
    proj_assemble_kernel<<<rows, PROJ_THREADS, 0, s>>>(N, R, a.elem_off, a.elem_ids, a.cells, cellM, rhs,
                                                       a.slice_ptr, cnt, mcol, mval, dinv, a.out, r, p, pa);
    launch_pdl(proj_direction_kernel<true>, dim3(1, R), PROJ_THREADS, 0, s, N, row_blocks, a.tolerance, pa,
               rz, rz, act, act, bb, dinv, r, p);
    PIBEM_CUDA(cudaGetLastError());
    note_launch(3);
    // Jacobi-preconditioned CG, all 3R columns together, from x = 0.  The columns'
    // flags after a batch of iterations are read while the next batch runs.
    int cur = 0;
    for (int it = 0, look = 0; it < a.max_iterations; look ^= 1)
      {
        for (int e = 0; e < PROJ_BATCH && it < a.max_iterations; ++e, ++it, cur ^= 1)
          {
            const int *ac = act + cur * ncol;
            launch_pdl(proj_mass_kernel, dim3(mass_blocks, R), PROJ_THREADS, 0, s, N, row_blocks, a.n_long,
                       a.long_rows, a.elem_off, a.slice_ptr, cnt, mcol, mval, ac, p, q, pb);
            launch_pdl(proj_update_kernel, rows, PROJ_THREADS, 0, s, N, mass_blocks, pb, rz + cur * ncol, ac,
                       dinv, p, q, a.out, r, pa);
            launch_pdl(proj_direction_kernel<false>, rows, PROJ_THREADS, 0, s, N, row_blocks, a.tolerance,
                       pa, rz + cur * ncol, rz + (cur ^ 1) * ncol, ac, act + (cur ^ 1) * ncol, bb, dinv, r,
                       p);
            note_launch(3);
          }
        PIBEM_CUDA(cudaGetLastError());
        int *h = a.flags + look * ncol;
        PIBEM_CUDA(cudaMemcpyAsync(h, act + cur * ncol, sizeof(int) * ncol, cudaMemcpyDeviceToHost, s));
        PIBEM_CUDA(cudaEventRecord(a.looked[look], s));
        if (it <= PROJ_BATCH)
          continue;
        PIBEM_CUDA(cudaEventSynchronize(a.looked[look ^ 1]));
        const int *prev = a.flags + (look ^ 1) * ncol;
        if (std::none_of(prev, prev + ncol, [](int f) { return f != 0; }))
          break;
      }
    PIBEM_CUDA(cudaStreamSynchronize(s));
  }

  size_t l2_projection_work(int64_t n_nodes, int64_t n_cells, int R, int64_t n_slots)
  {
    const int64_t n = n_nodes * 3 * R, ncol = 3 * R;
    return size_t(16 * n_cells + 12 * n_cells * R + n_nodes + 3 * n + 4 * ncol * PROJ_BLOCKS + 3 * ncol +
                  n_slots + (n_slots + n_nodes + 2 * ncol + 1) / 2);
  }
} // namespace pibem
