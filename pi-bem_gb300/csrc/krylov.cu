// Vector kernels of the device-resident GMRES (FP64 Arnoldi with classical
// Gram-Schmidt applied twice) and of the BEMProblem wrappers (masks, rhs,
// system matrix).  Reductions are two-stage with a fixed order, so results do
// not depend on scheduling.
#include <algorithm>
#include <cmath>

#include "krylov.h"
#include "pdl.cuh"

namespace pibem
{
  namespace
  {
    constexpr int kDotBlock  = 256;
    constexpr int AR_THREADS = 512; // Arnoldi kernels

    // partial[(r * nblk + blk) * ncols + i] = sum over the block's rows of V[r][i][t] w[r][t].
    // Warp k of the block takes columns k, k + 8, ...; its lanes stride over the
    // block's rows (coalesced; the w slice is re-read from L1) and the warp sum is
    // reduced in a fixed order, so the columns proceed in parallel without block
    // barriers.
    __global__ void dots_partial_kernel(int64_t n, int ncols, int64_t ldv, int64_t ldr,
                                        const double *__restrict__ V,
                                        const double *__restrict__ w, int nblk,
                                        double *__restrict__ partial)
    {
      const int     r     = blockIdx.y;
      const int     blk   = blockIdx.x;
      const double *Vr    = V + int64_t(r) * ldr;
      const double *wr    = w + int64_t(r) * n;
      const int64_t chunk = (n + nblk - 1) / nblk;
      const int64_t t0 = int64_t(blk) * chunk, t1 = min(n, t0 + chunk);
      const int     warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
      for (int i = warp; i < ncols; i += nw)
        {
          const double *v = Vr + int64_t(i) * ldv;
          double        s = 0;
#pragma unroll 8
          for (int64_t t = t0 + lane; t < t1; t += 32)
            s += v[t] * wr[t];
          for (int o = 16; o > 0; o >>= 1)
            s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == 0)
            partial[(int64_t(r) * nblk + blk) * ncols + i] = s;
        }
    }

    // one warp per output: lanes stride over the block partials, fixed-order tree
    __global__ void dots_final_kernel(int R, int ncols, int nblk, const double *__restrict__ partial,
                                      double *__restrict__ out)
    {
      const int idx  = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
      const int lane = threadIdx.x & 31;
      if (idx >= R * ncols)
        return;
      const int r = idx / ncols, i = idx % ncols;
      double    s = 0;
      for (int b = lane; b < nblk; b += 32)
        s += partial[(int64_t(r) * nblk + b) * ncols + i];
      for (int o = 16; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0)
        out[idx] = s;
    }

    // w[r][t] -= sum_i V[r][i][t] h[r][i]   (h on the device, layout [r][ldh])
    //   (jvec non-null: column r takes ncols = jvec[r]; sel non-null: selected
    //   columns only)
    __global__ void gemv_sub_kernel(int64_t n, int R, int ncols, int64_t ldv, int64_t ldr,
                                    const double *__restrict__ V, const double *__restrict__ h,
                                    int ldh, double *__restrict__ w, double sign,
                                    const int *__restrict__ jvec, const int *__restrict__ sel)
    {
      int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * R)
        return;
      int64_t r = idx / n, t = idx % n;
      if (sel && !sel[r])
        return;
      if (jvec)
        ncols = jvec[r];
      double  s = 0;
#pragma unroll 8
      for (int i = 0; i < ncols; ++i)
        s += V[r * ldr + int64_t(i) * ldv + t] * h[r * ldh + i];
      w[idx] -= sign * s;
    }

    // ---- one Arnoldi step, four launches ---------------------------------------
    // Classical Gram-Schmidt applied twice (FP64) on the batch's columns, then the
    // normalisation, the preconditioner and the Givens step:
    //   arnoldi_dots    w = the operator's result, dots V_i . w
    //   arnoldi_sub<0>  h1 = the dots' sums; w -= V h1; dots V_i . w
    //   arnoldi_sub<1>  h2 likewise; w -= V h2; |w|^2
    //   arnoldi_finish  V_{j+1} = w / |w|, z = P^-1 V_{j+1}, Givens (below)
    // Column k of the batch is slot act[k] (act[k] >= S: an idle padding column).
    // A column's rows are cut into G chunks, one block each; a block leaves its
    // partial sums in global memory and every block of the next launch adds the G
    // partials itself, in a fixed order: the launch boundary is the only barrier,
    // so nothing waits on a flag and no block is last.  G depends on n alone, so a
    // column's arithmetic depends on nothing but the column.
    //   What bounds it: on large meshes the FP64 units (2 FMA per clock and SM: 4 n j
    // FMA a step), on small ones the four launches' latency.  G = ceil(sqrt(n) / 2),
    // up to one block per SM, balances the chunk's 2 n / G FMA per basis vector against
    // the G additions of the partials (mixed solves at 1.5k / 98k nodes and 16 columns
    // at 24k: 5.83 / 45.0 / 154.7 ms with sqrt(n), 5.86 / 45.0 / 150.9 with half of
    // it, 5.88 / 46.0 / 148.2 with 0.35).  Sums run over groups of eight lanes, so
    // that a warp works on four basis vectors and a sum ends after three shuffles.
    //   Measured (kernel times of a step, warm caches, GB300) against one launch per
    // pass with a last-block reduction, the scatter / gather of the columns, the
    // preconditioner and a one-thread Givens step: 1.5k nodes 45 -> 26 us, 98k
    // nodes 68 -> 47 us; mixed solves to 1e-12 6.95 -> 5.86 ms and 47.2 -> 45.0 ms.

    // partial dots of the block's rows [t0, t1) with the ncols vectors V_i (n
    // apart): out[i * G + blk]; warp = (row part, group of four vectors)
    __device__ __forceinline__ void ar_dots(int64_t n, int ncols, const double *V, const double *w,
                                            int64_t t0, int64_t t1, double (*red)[64], double *out,
                                            int G, int blk)
    {
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      const int part = warp & 3, quad = warp >> 2;
      for (int i0 = 0; i0 < ncols; i0 += 64)
        {
#pragma unroll 1
          for (int q = 0; q < 4 && i0 + 16 * q < ncols; ++q)
            {
              const int l = 16 * q + 4 * quad + (lane >> 3), i = i0 + l;
              double    s = 0;
              if (i < ncols)
                {
                  const double *v = V + int64_t(i) * n;
                  for (int64_t t = t0 + 8 * part + (lane & 7); t < t1; t += 8 * 32)
                    {
                      double a[8], b[8];
#pragma unroll
                      for (int u = 0; u < 8; ++u)
                        if (t + 32 * u < t1)
                          {
                            a[u] = v[t + 32 * u];
                            b[u] = w[t + 32 * u];
                          }
#pragma unroll
                      for (int u = 0; u < 8; ++u)
                        if (t + 32 * u < t1)
                          s = fma(a[u], b[u], s);
                    }
                }
              __syncwarp();
              for (int o = 4; o > 0; o >>= 1)
                s += __shfl_xor_sync(0xffffffffu, s, o);
              if ((lane & 7) == 0)
                red[part][l] = s;
            }
          __syncthreads();
          const int i = i0 + threadIdx.x;
          if (threadIdx.x < 64 && i < ncols)
            out[int64_t(i) * G + blk] = (red[0][threadIdx.x] + red[1][threadIdx.x]) +
                                        (red[2][threadIdx.x] + red[3][threadIdx.x]);
          __syncthreads();
        }
    }

    // w = the operator's result on the batch (FP32 or FP64), the first dots, and
    // jcur = the columns' step for the rest of this step's launches
    template <typename T>
    __global__ void __launch_bounds__(AR_THREADS)
      arnoldi_dots_kernel(int64_t n, int S, int G, int L, int64_t ldr, const int *__restrict__ act,
                          const T *__restrict__ in, const double *__restrict__ V,
                          double *__restrict__ w, const int *__restrict__ jvec,
                          int *__restrict__ jcur, double *__restrict__ partial)
    {
      pdl_entry();
      __shared__ double red[4][64];
      const int k = blockIdx.y, r = act[k], blk = blockIdx.x;
      if (r >= S)
        return;
      const int j = jvec[r];
      if (blk == 0 && threadIdx.x == 0)
        jcur[r] = j;
      if (j < 0)
        return;
      const int64_t chunk = (n + G - 1) / G;
      const int64_t t0 = int64_t(blk) * chunk, t1 = min(n, t0 + chunk);
      double       *wr = w + int64_t(r) * n;
      for (int64_t t = t0 + threadIdx.x; t < t1; t += AR_THREADS)
        wr[t] = double(in[int64_t(k) * n + t]);
      __syncthreads();
      ar_dots(n, j + 1, V + int64_t(r) * ldr, wr, t0, t1, red, partial + int64_t(k) * L * G, G, blk);
    }

    // h_i = the sum of the G partials (block 0 keeps it in hout), w -= V h, then
    // the dots of the next pass (LAST: the partial squared norms).  With chunks of
    // fewer than AR_THREADS rows four warps share a row's sum over i.
    template <bool LAST>
    __global__ void __launch_bounds__(AR_THREADS)
      arnoldi_sub_kernel(int64_t n, int S, int G, int L, int64_t ldr, const int *__restrict__ act,
                         const double *__restrict__ V, double *__restrict__ w,
                         const int *__restrict__ jcur, const double *__restrict__ pin,
                         double *__restrict__ hout, double *__restrict__ pout)
    {
      pdl_entry();
      extern __shared__ double sh[]; // [L]
      __shared__ double red[4][AR_THREADS];
      const int k = blockIdx.y, r = act[k], blk = blockIdx.x;
      if (r >= S)
        return;
      const int j = jcur[r];
      if (j < 0)
        return;
      const int     ncols = j + 1, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      const int64_t chunk = (n + G - 1) / G;
      const int64_t t0 = int64_t(blk) * chunk, t1 = min(n, t0 + chunk);
      const double *Vr = V + int64_t(r) * ldr;
      double       *wr = w + int64_t(r) * n;
      for (int i0 = 0; i0 < ncols; i0 += AR_THREADS / 8)
        {
          const int i = i0 + int(threadIdx.x >> 3);
          double    s = 0;
          if (i < ncols)
            {
              const double *p = pin + (int64_t(k) * L + i) * G;
#pragma unroll 4
              for (int b = lane & 7; b < G; b += 8)
                s += p[b];
            }
          __syncwarp();
          for (int o = 4; o > 0; o >>= 1)
            s += __shfl_xor_sync(0xffffffffu, s, o);
          if (i < ncols && (lane & 7) == 0)
            {
              sh[i] = s;
              if (blk == 0)
                hout[int64_t(r) * L + i] = s;
            }
        }
      __syncthreads();
      double nrm = 0;
      // sum over i = i0, i0 + step, ... of V_i[t] h_i, eight loads in flight
      auto dot_h = [&](int64_t t, int i0, int step) {
        double s = 0;
        for (int i = i0; i < ncols; i += 8 * step)
          {
            double a[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (i + u * step < ncols)
                a[u] = Vr[int64_t(i + u * step) * n + t];
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (i + u * step < ncols)
                s = fma(a[u], sh[i + u * step], s);
          }
        return s;
      };
      if (chunk >= AR_THREADS)
        for (int64_t t = t0 + threadIdx.x; t < t1; t += AR_THREADS)
          {
            const double v = wr[t] - dot_h(t, 0, 1);
            wr[t]          = v;
            nrm            = LAST ? fma(v, v, nrm) : 0;
          }
      else
        {
          const int part = warp & 3, rg = warp >> 2;
          for (int64_t t = t0 + 32 * rg + lane; t < t1; t += 128)
            red[part][t - t0] = dot_h(t, part, 4);
          __syncthreads();
          const int l = threadIdx.x;
          if (t0 + l < t1)
            {
              const double v = wr[t0 + l] - ((red[0][l] + red[1][l]) + (red[2][l] + red[3][l]));
              wr[t0 + l]     = v;
              nrm            = LAST ? v * v : 0;
            }
        }
      __syncthreads(); // w is updated (visible to the block); red is free
      if constexpr (!LAST)
        ar_dots(n, ncols, Vr, wr, t0, t1, reinterpret_cast<double(*)[64]>(&red[0][0]),
                pout + int64_t(k) * L * G, G, blk);
      else
        {
          for (int o = 16; o > 0; o >>= 1)
            nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
          if (lane == 0)
            red[0][warp] = nrm;
          __syncthreads();
          if (threadIdx.x == 0)
            {
              double s = 0;
              for (int q = 0; q < AR_THREADS / 32; ++q)
                s += red[0][q];
              pout[int64_t(k) * G + blk] = s;
            }
        }
    }

    // out[r] = w[r] / sqrt(nrm[r]) (0 for a zero norm) of the columns with sel[r]
    // (column stride ldr); with z also into z[r]
    __global__ void normalize_kernel(int64_t n, int R, const double *__restrict__ w,
                                     const double *__restrict__ nrm, double *__restrict__ out,
                                     int64_t ldr, double *__restrict__ z, const int *__restrict__ sel)
    {
      int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * R)
        return;
      int64_t r = idx / n, t = idx % n;
      if (!sel[r])
        return;
      double       h = sqrt(nrm[r]);
      const double v = h > 0 ? w[idx] / h : 0.0;
      out[r * ldr + t] = v;
      if (z)
        z[idx] = v;
    }

    // ---- device-driven GMRES cycles, one state per column (slot) -------------
    // Per column r: Hessenberg H[r] ((m+1) x m, entry (i, j) at i m + j), Givens
    // cosines / sines cs[r], sn[r] (m), g[r] (m+1), jvec[r] (the column's next
    // Arnoldi step; -1: the column takes no part), kdone[r] (-1, or the step
    // count after which the column met its tolerance), its[r] / maxit[r]
    // (iterations so far / limit), bn[r], tol[r] (stopping test |g_{j+1}| /
    // bn <= tol).  hb: [h1 (R x L) | h2 (R x L)], L = m + 1, the two Gram-Schmidt
    // passes' coefficients of a step.  ctl[0]: 1 while
    // the steps go on; ctl[1]: steps run; ctl[2]: most steps before the host is
    // back (a quantum).

    // cycle start of the selected columns: g[r] = (beta_r, 0, ...) with beta_r =
    // sqrt(nrm2[r]), jvec[r] = 0, kdone[r] = -1
    __global__ void gmres_cycle_init_kernel(int R, int L, const int *__restrict__ sel,
                                            const double *__restrict__ nrm2, double *__restrict__ g,
                                            int *__restrict__ kdone, int *__restrict__ jvec)
    {
      for (int r = threadIdx.x; r < R; r += blockDim.x)
        if (sel[r])
          {
            g[int64_t(r) * L] = sqrt(nrm2[r]);
            kdone[r]          = -1;
            jvec[r]           = 0;
          }
    }

    // End of a column's cycle: y[r] solves its triangular system of k steps (k =
    // kdone[r] if it met its tolerance, else jvec[r]); y[r][i] = 0 for i >= k.
    // Selected columns only.
    __global__ void gmres_lsq_kernel(int R, int m, const int *__restrict__ sel,
                                     const double *__restrict__ H, const double *__restrict__ g,
                                     const int *__restrict__ kdone, const int *__restrict__ jvec,
                                     double *__restrict__ y)
    {
      const int L = m + 1;
      for (int r = threadIdx.x; r < R; r += blockDim.x)
        {
          if (!sel[r])
            continue;
          const int     k  = kdone[r] < 0 ? jvec[r] : kdone[r];
          const double *Hc = H + int64_t(r) * L * m;
          const double *gg = g + int64_t(r) * L;
          double       *yr = y + int64_t(r) * L;
          for (int i = k; i < L; ++i)
            yr[i] = 0.0;
          for (int i = k - 1; i >= 0; --i)
            {
              double sum = gg[i];
              for (int jj = i + 1; jj < k; ++jj)
                sum -= Hc[int64_t(i) * m + jj] * yr[jj];
              yr[i] = sum / Hc[int64_t(i) * m + i];
            }
        }
    }

    // dst[k] = src[cols[k]] (n values a column; source column stride lds)
    __global__ void gather_cols_kernel(int64_t n, int Rc, const int *__restrict__ cols,
                                       const double *__restrict__ src, int64_t lds,
                                       double *__restrict__ dst)
    {
      pdl_entry();
      const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * Rc)
        return;
      const int64_t k = idx / n, t = idx - k * n;
      dst[idx]        = src[int64_t(cols[k]) * lds + t];
    }
    // dst[cols[k]] = src[k]
    __global__ void scatter_cols_kernel(int64_t n, int Rc, const int *__restrict__ cols,
                                        const double *__restrict__ src, double *__restrict__ dst,
                                        int64_t ldd)
    {
      pdl_entry();
      const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * Rc)
        return;
      const int64_t k = idx / n, t = idx - k * n;
      dst[int64_t(cols[k]) * ldd + t] = src[idx];
    }

    // dst[k] = float(src[cols[k]]) and dst[cols[k]] = double(src[k]): the FP32
    // operator's input from the slots and back
    __global__ void gather_d2f_kernel(int64_t n, int Rc, const int *__restrict__ cols,
                                      const double *__restrict__ src, float *__restrict__ dst)
    {
      pdl_entry();
      const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * Rc)
        return;
      const int64_t k = idx / n, t = idx - k * n;
      dst[idx]        = float(src[int64_t(cols[k]) * n + t]);
    }
    __global__ void f2d_scatter_kernel(int64_t n, int Rc, const int *__restrict__ cols,
                                       const float *__restrict__ src, double *__restrict__ dst)
    {
      const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * Rc)
        return;
      const int64_t k = idx / n, t = idx - k * n;
      dst[int64_t(cols[k]) * n + t] = double(src[idx]);
    }

    // y[r] = a x[r] + b y[r] for the selected columns
    __global__ void axpby_sel_kernel(int64_t n, int R, const int *__restrict__ sel, double a,
                                     const double *__restrict__ x, double b, double *__restrict__ y)
    {
      const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * R || !sel[idx / n])
        return;
      y[idx] = a * x[idx] + b * y[idx];
    }

    __global__ void axpby_kernel(int64_t n, double a, const double *__restrict__ x, double b,
                                 double *__restrict__ y)
    {
      int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (i < n)
        y[i] = a * x[i] + b * y[i];
    }

    __global__ void d2f_kernel(int64_t n, const double *__restrict__ a, float *__restrict__ b)
    {
      pdl_entry();
      int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (i < n)
        b[i] = float(a[i]);
    }
    __global__ void f2d_kernel(int64_t n, const float *__restrict__ a, double *__restrict__ b)
    {
      pdl_entry();
      int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (i < n)
        b[i] = double(a[i]);
    }

    // S = N where the column dof is Neumann, -D where Dirichlet, + alpha on the
    // diagonal of Neumann rows (BEMProblem::vmult FMA branch, bem_problem.cc:1199-1209,
    // as one matrix like BEMFMA's init_preconditioner, bem_fma.cc:952-962).
    __global__ void system_matrix_kernel(int64_t n_vals, int n_leaves,
                                         const int64_t *__restrict__ val_ptr,
                                         const int64_t *__restrict__ col_ptr,
                                         const int64_t *__restrict__ row_ptr,
                                         const int32_t *__restrict__ rows,
                                         const int32_t *__restrict__ cols,
                                         const uint8_t *__restrict__ dir,
                                         const double *__restrict__ alpha,
                                         const double *__restrict__ Nv,
                                         const double *__restrict__ Dv, double *__restrict__ S,
                                         float *__restrict__ S32)
    {
      int64_t vi = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (vi >= n_vals)
        return;
      int lo = 0, hi = n_leaves - 1;
      while (lo < hi)
        {
          int mid = (lo + hi + 1) >> 1;
          if (val_ptr[mid] <= vi)
            lo = mid;
          else
            hi = mid - 1;
        }
      const int64_t nc  = col_ptr[lo + 1] - col_ptr[lo];
      const int64_t ld  = (nc + 3) / 4 * 4;
      const int64_t loc = vi - val_ptr[lo];
      if (loc % ld >= nc)
        {
          S[vi] = 0.0;
          if (S32)
            S32[vi] = 0.0f;
          return;
        }
      const int row = rows[row_ptr[lo] + loc / ld];
      const int col = cols[col_ptr[lo] + loc % ld];
      double        v   = dir[col] ? -Dv[vi] : Nv[vi];
      if (row == col && !dir[row])
        v += alpha[row];
      S[vi] = v;
      if (S32)
        S32[vi] = float(v);
    }

    // rhs = -(outN + alpha*(tmp.dir)) + outD  (BEMProblem::compute_rhs, bem_problem.cc:1240-1258)
    __global__ void rhs_combine_kernel(int64_t n, int R, const double *__restrict__ tmp,
                                       const uint8_t *__restrict__ dir,
                                       const double *__restrict__ alpha,
                                       const double *__restrict__ oN, const double *__restrict__ oD,
                                       double *__restrict__ rhs)
    {
      int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * R)
        return;
      int64_t t  = idx % n;
      double  sp = dir[t] ? tmp[idx] : 0.0;
      rhs[idx]   = -(oN[idx] + alpha[t] * sp) + oD[idx];
    }

    // split tmp_rhs into (tmp.dir, tmp.neu)
    __global__ void split_masks_kernel(int64_t n, int R, const double *__restrict__ tmp,
                                       const uint8_t *__restrict__ dir, double *__restrict__ a,
                                       double *__restrict__ b)
    {
      int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * R)
        return;
      int64_t t = idx % n;
      a[idx]    = dir[t] ? tmp[idx] : 0.0;
      b[idx]    = dir[t] ? 0.0 : tmp[idx];
    }

    // scatter: phi(i) = sol(i) on Neumann nodes, dphi_dn(i) = sol(i) on Dirichlet nodes
    __global__ void scatter_kernel(int64_t n, int R, const double *__restrict__ sol,
                                   const uint8_t *__restrict__ dir, double *__restrict__ phi,
                                   double *__restrict__ dphi)
    {
      int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * R)
        return;
      int64_t t = idx % n;
      if (dir[t])
        dphi[idx] = sol[idx];
      else
        phi[idx] = sol[idx];
    }

    __global__ void add_scalar_kernel(int64_t n, int R, const double *__restrict__ shift,
                                      double *__restrict__ x)
    {
      int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * R)
        return;
      x[idx] += shift[idx / n];
    }

    // x[r] += -sqrt(nrm2[r])  (the pure-Neumann shift v - ||v||)
    __global__ void sub_norm_kernel(int64_t n, int R, const double *__restrict__ nrm2,
                                    double *__restrict__ x)
    {
      int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * R)
        return;
      x[idx] += -sqrt(nrm2[idx / n]);
    }

    // Leaf-block Jacobi (right preconditioner), z[node] = sum_c Pinv[leaf][r][c]
    // v[rows_c], in the precision P of the stored inverses: FP32 for the mixed
    // path's inner solves (GB300's FP64 rate is 1/58 of its FP32 rate), FP64 for
    // the plain FP64 path (whose GMRES would otherwise see the FP32 rounding as a
    // nonlinearity near its 1e-8 target).  One warp per leaf: the leaf's v entries
    // of CB columns are in the warp's shared slice sv, lane i computes rows i,
    // i + 32, ... with c ascending (the same chain for every CB); the blocks are
    // stored column-major (entry (r, c) at c * nr + r), so a column is read across
    // the lanes, once for the CB columns.  put(column, row, value) takes the result.
    template <int CB, typename P, typename F>
    __device__ __forceinline__ void block_rows(int nr, const int32_t *rows, const P *B, const P *sv,
                                               int max_rows, F put)
    {
      const int lane = threadIdx.x & 31;
      for (int i = lane; i < nr; i += 32)
        {
          P s[CB];
#pragma unroll
          for (int q = 0; q < CB; ++q)
            s[q] = P(0);
          int c = 0;
          for (; c + 8 <= nr; c += 8)
            {
              P p[8];
#pragma unroll
              for (int u = 0; u < 8; ++u)
                p[u] = B[int64_t(c + u) * nr + i];
#pragma unroll
              for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int q = 0; q < CB; ++q)
                  s[q] = fma(p[u], sv[q * max_rows + c + u], s[q]);
            }
          for (; c < nr; ++c)
            {
              const P p = B[int64_t(c) * nr + i];
#pragma unroll
              for (int q = 0; q < CB; ++q)
                s[q] = fma(p, sv[q * max_rows + c], s[q]);
            }
          const int row = rows[i];
#pragma unroll
          for (int q = 0; q < CB; ++q)
            put(q, row, s[q]);
        }
    }

    template <typename P>
    __global__ void __launch_bounds__(256)
      block_apply_kernel(int n_leaves, int max_rows, int R, int64_t n, int64_t ldv,
                         const int64_t *__restrict__ row_ptr, const int64_t *__restrict__ blk_ptr,
                         const int32_t *__restrict__ rows, const P *__restrict__ Pinv,
                         const double *__restrict__ v, double *__restrict__ z,
                         const int *__restrict__ sel)
    {
      extern __shared__ __align__(8) unsigned char sv_raw[];
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      const int leaf = blockIdx.x * 8 + warp;
      if (leaf >= n_leaves)
        return;
      P            *sv = reinterpret_cast<P *>(sv_raw) + int64_t(warp) * max_rows;
      const int64_t r0 = row_ptr[leaf];
      const int     nr = int(row_ptr[leaf + 1] - r0);
      for (int rr = 0; rr < R; ++rr)
        {
          if (sel && !sel[rr])
            continue;
          for (int c = lane; c < nr; c += 32)
            sv[c] = P(v[int64_t(rr) * ldv + rows[r0 + c]]);
          __syncwarp();
          block_rows<1, P>(nr, rows + r0, Pinv + blk_ptr[leaf], sv, max_rows,
                           [&](int, int row, P s) { z[int64_t(rr) * n + row] = double(s); });
          __syncwarp();
        }
    }

    // The Givens step of the batch's columns (one block): the Hessenberg column
    // h1 + h2, the previous rotations, the new one and the stopping test (|g_{j+1}|
    // / bn <= tol, or a zero subdiagonal); then jvec and the iteration count
    // advance.  A column ends its cycle when it meets its tolerance, after m steps
    // or at its iteration limit (jvec = -2 - steps: no more steps); when the steps
    // stop (see ctl), ctl[0] = 0 and, in a graph, the loop's condition is cleared.
    // A warp per column: lane l holds rotation l of a group of 32, the chain a <-
    // -s_l a + c_l h_{l+1} runs in every lane (one FMA a rotation), and lane l
    // forms its entry from the a it saw.
    __device__ __forceinline__ void givens_step(const GivensArgs &a, int Ra, int S, const int *act,
                                                const int *sj, const double *snr)
    {
      __shared__ int alive;
      if (threadIdx.x == 0)
        alive = 0;
      __syncthreads();
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
      const int m = a.m, L = m + 1;
      for (int k = warp; k < Ra; k += nw)
        {
          const int j = sj[k];
          if (j < 0)
            continue;
          const int     r  = act[k];
          double       *Hc = a.H + int64_t(r) * L * m;
          const double *h1 = a.hb + int64_t(r) * L, *h2 = h1 + int64_t(S) * L;
          double       *c = a.cs + int64_t(r) * m, *sv = a.sn + int64_t(r) * m;
          double        x = h1[0] + h2[0];
          for (int i0 = 0; i0 < j; i0 += 32)
            {
              const int i = i0 + lane;
              double    ci = 0, si = 0, hn = 0, mine = 0;
              if (i < j)
                {
                  ci = c[i];
                  si = sv[i];
                  hn = h1[i + 1] + h2[i + 1];
                }
              const double ch = ci * hn;
              for (int l = 0; l < 32 && i0 + l < j; ++l)
                {
                  mine = lane == l ? x : mine;
                  x    = fma(-__shfl_sync(0xffffffffu, si, l), x, __shfl_sync(0xffffffffu, ch, l));
                }
              if (i < j)
                Hc[int64_t(i) * m + j] = fma(ci, mine, si * hn);
            }
          if (lane == 0)
            {
              const double bb = sqrt(snr[k]), d = hypot(x, bb);
              const double cj = d > 0 ? x / d : 1.0, sj2 = d > 0 ? bb / d : 0.0;
              double      *gg = a.g + int64_t(r) * L;
              c[j]            = cj;
              sv[j]           = sj2;
              Hc[int64_t(j) * m + j]       = d;
              Hc[int64_t(j + 1) * m + j]   = 0;
              const double gj = gg[j], g1 = -sj2 * gj;
              gg[j + 1]       = g1;
              gg[j]           = cj * gj;
              const int it    = a.its[r] + 1;
              a.its[r]        = it;
              int done        = a.kdone[r];
              if (fabs(g1) / a.bn[r] <= a.tol[r] || bb == 0.0)
                a.kdone[r] = done = j + 1;
              if (done >= 0 || j + 1 >= m || it >= a.maxit[r])
                a.jvec[r] = -2 - (j + 1);
              else
                {
                  a.jvec[r] = j + 1;
                  alive     = 1;
                }
            }
        }
      __syncthreads();
      if (threadIdx.x == 0)
        {
          const int steps = a.ctl[1] + 1; // steps run since the host set ctl
          // the steps go on while some column is in its cycle (every one ends it within
          // m steps), for at most ctl[2] steps
          const int stop = !alive || steps >= a.ctl[2];
          a.ctl[0]       = !stop;
          a.ctl[1]       = steps;
          if (a.use_cond && stop)
            cudaGraphSetConditional(a.cond, 0);
        }
    }

    // End of an Arnoldi step.  Every block adds the columns' squared norms; block 0
    // takes the Givens step, the others V_{j+1} = w / |w| and, into out (the
    // operator's next input: batch column k, or slot act[k] with SLOT), BJ: the
    // leaf-block Jacobi result z = P^-1 V_{j+1}, a warp per leaf and CB columns at
    // a time; otherwise V_{j+1} itself.  Columns with jcur < 0 are skipped.
    // Shared memory: |w|^2 and 1 / |w| [Ra], steps [Ra], sv[warps][CB][max_rows].
    template <typename P, typename OUT, bool BJ, int CB, bool SLOT>
    __global__ void __launch_bounds__(AR_THREADS)
      arnoldi_finish_kernel(int64_t n, int S, int G, int Ra, int64_t ldr, const int *__restrict__ act,
                            const int *__restrict__ jcur, const double *__restrict__ pn,
                            const double *__restrict__ w, double *__restrict__ V,
                            OUT *__restrict__ out, BlockPrec<P> bp, GivensArgs ga)
    {
      pdl_entry();
      extern __shared__ __align__(16) unsigned char fin_raw[];
      double   *snr = reinterpret_cast<double *>(fin_raw), *sinv = snr + Ra;
      int      *sj   = reinterpret_cast<int *>(sinv + Ra);
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
      for (int k = warp; k < Ra; k += nw)
        {
          const int r = act[k], j = r < S ? jcur[r] : -1;
          double    s = 0;
          if (j >= 0)
            for (int b = lane; b < G; b += 32)
              s += pn[int64_t(k) * G + b];
          for (int o = 16; o > 0; o >>= 1)
            s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == 0)
            {
              snr[k]  = s;
              sinv[k] = s > 0 ? 1.0 / sqrt(s) : 0.0;
              sj[k]   = j;
            }
        }
      __syncthreads();
      if (blockIdx.x == 0)
        {
          givens_step(ga, Ra, S, act, sj, snr);
          return;
        }
      auto col_of = [&](int k) { return int64_t(SLOT ? act[k] : k) * n; };
      if constexpr (!BJ)
        {
          for (int k = 0; k < Ra; ++k)
            {
              const int j = sj[k];
              if (j < 0)
                continue;
              const int64_t r = act[k];
              double       *v = V + r * ldr + int64_t(j + 1) * n;
              for (int64_t t = int64_t(blockIdx.x - 1) * blockDim.x + threadIdx.x; t < n;
                   t += int64_t(gridDim.x - 1) * blockDim.x)
                {
                  const double x      = w[r * n + t] * sinv[k];
                  v[t]                = x;
                  out[col_of(k) + t]  = OUT(x);
                }
            }
        }
      else
        {
          P *sv = reinterpret_cast<P *>(fin_raw + (size_t(Ra) * 20 + 15) / 16 * 16) +
                  int64_t(warp) * CB * bp.max_rows;
          for (int leaf = int(blockIdx.x - 1) * nw + warp; leaf < bp.n_leaves;
               leaf += int(gridDim.x - 1) * nw)
            {
              const int64_t  r0   = bp.row_ptr[leaf];
              const int      nr   = int(bp.row_ptr[leaf + 1] - r0);
              const int32_t *rows = bp.rows + r0;
              const P       *B    = bp.Pinv + bp.blk_ptr[leaf];
              for (int k0 = 0; k0 < Ra; k0 += CB)
                {
                  bool any = false;
#pragma unroll
                  for (int q = 0; q < CB; ++q)
                    {
                      const int k = k0 + q, j = k < Ra ? sj[k] : -1;
                      if (j < 0)
                        {
                          for (int c = lane; c < nr; c += 32)
                            sv[q * bp.max_rows + c] = P(0);
                          continue;
                        }
                      any             = true;
                      const int64_t r = act[k];
                      double       *v = V + r * ldr + int64_t(j + 1) * n;
                      for (int c = lane; c < nr; c += 32)
                        {
                          const int64_t row       = rows[c];
                          const double  x         = w[r * n + row] * sinv[k];
                          v[row]                  = x;
                          sv[q * bp.max_rows + c] = P(x);
                        }
                    }
                  __syncwarp();
                  if (any)
                    block_rows<CB, P>(nr, rows, B, sv, bp.max_rows, [&](int q, int row, P s) {
                      const int k = k0 + q;
                      if (k < Ra && sj[k] >= 0)
                        out[col_of(k) + row] = OUT(s);
                    });
                  __syncwarp();
                }
            }
        }
    }

    // ---- ILU(0) of the near-field system matrix (preconditioner 2) ----------
    // CSR in node order: ptr, col (ascending), val, diag (position of the
    // diagonal).  Level sets: the rows of a level depend only on rows of
    // earlier levels (lower part for the factorisation and the forward
    // substitution, upper part for the backward one).

    // one row of the near field (or a constraint line) into the CSR: warp per node
    __global__ void ilu_fill_kernel(int64_t n, const int64_t *__restrict__ ptr,
                                    const int32_t *__restrict__ pos, const int32_t *__restrict__ row_leaf,
                                    const int64_t *__restrict__ nrow_ptr, const int64_t *__restrict__ ncol_ptr,
                                    const int64_t *__restrict__ nval_ptr, const int32_t *__restrict__ ncols,
                                    const double *__restrict__ S, const int32_t *__restrict__ con,
                                    int32_t *__restrict__ col, double *__restrict__ val)
    {
      const int64_t i    = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
      const int     lane = threadIdx.x & 31;
      if (i >= n)
        return;
      const int64_t o = ptr[i];
      if (con[i] != -2)
        {
          // a constrained row: 1 on the diagonal and +1 at the line's column
          // (bem_fma.cc:3190-3201 stores the constraint entries as they are)
          if (lane == 0)
            {
              const int c = con[i];
              if (c >= 0 && c != int(i))
                {
                  const bool lo = c < int(i);
                  col[o]        = lo ? c : int32_t(i);
                  col[o + 1]    = lo ? int32_t(i) : c;
                  val[o]        = 1.0;
                  val[o + 1]    = 1.0;
                }
              else
                {
                  col[o] = int32_t(i);
                  val[o] = 1.0;
                }
            }
          return;
        }
      const int     r  = pos[i];
      const int     lf = row_leaf[r];
      const int64_t c0 = ncol_ptr[lf], nc = ncol_ptr[lf + 1] - c0;
      const int64_t ld = (nc + 3) / 4 * 4;
      const double *v  = S + nval_ptr[lf] + (r - nrow_ptr[lf]) * ld;
      for (int64_t k = lane; k < nc; k += 32)
        {
          col[o + k] = ncols[c0 + k];
          val[o + k] = v[k];
        }
    }

    // IKJ ILU(0) of the rows of one level, a block per row with the row in
    // shared memory: for the row's columns k < i in ascending order,
    // a_ik /= a_kk, then a_ij -= a_ik a_kj for the columns j > k of row k that
    // row i holds (threads take row k's entries, a binary search finds j in
    // the row's sorted columns); row k is final (an earlier level)
    __global__ void ilu_factor_kernel(const int32_t *__restrict__ rows, const int64_t *__restrict__ ptr,
                                      const int32_t *__restrict__ col, double *__restrict__ val,
                                      const int64_t *__restrict__ diag)
    {
      extern __shared__ __align__(16) unsigned char ilu_smem[];
      const int     i  = rows[blockIdx.x];
      const int64_t a0 = ptr[i], n = ptr[i + 1] - a0, nd = diag[i] - a0;
      double       *sv = reinterpret_cast<double *>(ilu_smem);
      int32_t      *sc = reinterpret_cast<int32_t *>(sv + n);
      for (int64_t e = threadIdx.x; e < n; e += blockDim.x)
        {
          sv[e] = val[a0 + e];
          sc[e] = col[a0 + e];
        }
      __syncthreads();
      for (int64_t e = 0; e < nd; ++e)
        {
          const int     k   = sc[e];
          const int64_t dk  = diag[k], k1 = ptr[k + 1];
          const double  lik = sv[e] / val[dk];
          for (int64_t f = dk + 1 + threadIdx.x; f < k1; f += blockDim.x)
            {
              const int j  = col[f];
              int64_t   lo = e + 1, hi = n;
              while (lo < hi)
                {
                  const int64_t m = (lo + hi) >> 1;
                  if (sc[m] < j)
                    lo = m + 1;
                  else
                    hi = m;
                }
              if (lo < n && sc[lo] == j)
                sv[lo] -= lik * val[f];
            }
          __syncthreads();
          if (threadIdx.x == 0)
            sv[e] = lik;
        }
      __syncthreads();
      for (int64_t e = threadIdx.x; e < n; e += blockDim.x)
        val[a0 + e] = sv[e];
    }

    // z[r] = v[r] for the columns with sel[r] (v column stride ldv, z stride n)
    __global__ void copy_sel_kernel(int64_t n, int R, const double *__restrict__ v, int64_t ldv,
                                    double *__restrict__ z, const int *__restrict__ sel)
    {
      const int64_t idx = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (idx >= n * R)
        return;
      const int64_t r = idx / n, t = idx - r * n;
      if (sel && !sel[r])
        return;
      z[idx] = v[r * ldv + t];
    }

    // One level of a substitution (forward: lower triangle, unit diagonal; backward: upper),
    // in place on the selected columns of z: a warp per (row, column), lanes over the row's
    // entries, fixed butterfly.  For triangles of wide levels (launch_ilu_apply).
    template <bool FWD>
    __global__ void ilu_level_kernel(int nrows, const int32_t *__restrict__ rows, int R, int64_t n,
                                     const int64_t *__restrict__ ptr, const int32_t *__restrict__ col,
                                     const double *__restrict__ val, const int64_t *__restrict__ diag,
                                     double *__restrict__ z, const int *__restrict__ sel,
                                     const int *__restrict__ jvec)
    {
      const int64_t w    = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
      const int     lane = threadIdx.x & 31;
      if (w >= int64_t(nrows) * R)
        return;
      const int r = int(w / nrows), i = rows[w - int64_t(r) * nrows];
      if ((sel && !sel[r]) || (jvec && jvec[r] < 0))
        return;
      double       *zr = z + int64_t(r) * n;
      const int64_t a0 = FWD ? ptr[i] : diag[i] + 1, a1 = FWD ? diag[i] : ptr[i + 1];
      double        s  = 0;
      for (int64_t e = a0 + lane; e < a1; e += 32)
        s = fma(val[e], zr[col[e]], s);
      for (int o = 16; o > 0; o >>= 1)
        s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0)
        zr[i] = FWD ? zr[i] - s : (zr[i] - s) / val[diag[i]];
    }

    // z = U^-1 L^-1 z in place: one block per column (blockIdx.x) runs both
    // substitutions.  Its warps take the rows in level order, one after another in
    // turn; a warp waits for the solution values of its row's columns in the vector
    // itself, which starts as a NaN pattern that no arithmetic result is stored as,
    // so a value is its own flag.  A row only waits for rows before it in the list
    // and each warp takes its rows in order, so the first unfinished row can always
    // proceed; every wait is bounded.  A row's sum: lanes stride over its entries,
    // fixed butterfly, with the bits of ilu_level_kernel.
    //   What bounds it: the chain of dependent rows (some 650 levels of 4 rows at 2.4k
    // nodes, 17,000 of 6 at 98k): no parallelism for more than an SM, so the
    // hand-over between rows decides.  Inside one block it goes through shared memory
    // (SMEM: up to 25,600 nodes) or the L1 cache, 1.2-1.7 us a level (FP64 latency:
    // the last FMA, five shuffled additions, the division by the pivot, which takes 4 %
    // more than a product with its reciprocal but rounds once), where one launch per
    // level took 4.7 us.  The next row's indices are loaded a row ahead.  One application
    // (leaf 40): 2.4k nodes 13.4 -> 3.5 ms, 13.8k 29 -> 7.3, 31k 65 -> 21.
    constexpr int                ILU_THREADS = 512;
    constexpr int                ILU_E       = 16; // entries per lane loaded at once
    constexpr unsigned long long ILU_UNSET   = ~0ull;
    constexpr long               ILU_SPIN    = 1L << 22;

    template <bool SMEM>
    __device__ __forceinline__ double ilu_peek(const double *p)
    {
      double v;
      if constexpr (SMEM)
        v = *reinterpret_cast<const volatile double *>(p);
      else
        asm volatile("ld.relaxed.cta.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
      return v;
    }
    template <bool SMEM>
    __device__ __forceinline__ void ilu_put(double *p, double v)
    {
      if (__double_as_longlong(v) == (long long)ILU_UNSET)
        v = __longlong_as_double(0x7ff8000000000000ll); // another NaN
      if constexpr (SMEM)
        *reinterpret_cast<volatile double *>(p) = v;
      else
        asm volatile("st.relaxed.cta.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
    }

    template <bool FWD, bool SMEM>
    __device__ __forceinline__ void ilu_sweep(int n, const int32_t *__restrict__ rows,
                                              const int64_t *__restrict__ ptr,
                                              const int32_t *__restrict__ col,
                                              const double *__restrict__ val,
                                              const int64_t *__restrict__ diag, const double *rhs,
                                              double *out, int *err, volatile int *abort)
    {
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = ILU_THREADS / 32;
      auto row_at = [&](int k) { return k < n ? rows[k] : -1; };
      auto begin  = [&](int i) { return i < 0 ? int64_t(0) : (FWD ? ptr[i] : diag[i] + 1); };
      auto end    = [&](int i) { return i < 0 ? int64_t(0) : (FWD ? diag[i] : ptr[i + 1]); };
      auto right  = [&](int i) { return i < 0 ? 0.0 : rhs[i]; };
      auto pivot  = [&](int i) { return i < 0 || FWD ? 1.0 : val[diag[i]]; };
      int     i = row_at(warp), i1 = row_at(warp + nw);
      int64_t a0 = begin(i), a1 = end(i);
      double  b = right(i), d = pivot(i);
      for (int k = warp; k < n; k += nw)
        {
          const int     i2 = row_at(k + 2 * nw);
          const int64_t n0 = begin(i1), n1 = end(i1);
          const double  nb = right(i1), nd = pivot(i1);
          double        s = 0;
          for (int64_t e0 = a0; e0 < a1; e0 += 32 * ILU_E)
            {
              int    c[ILU_E];
              double v[ILU_E];
              int    cnt = 0, next = 0; // entries of this lane, entries already added
#pragma unroll
              for (int u = 0; u < ILU_E; ++u)
                {
                  const int64_t e = e0 + lane + 32 * u;
                  if (e < a1)
                    {
                      c[u] = col[e];
                      v[u] = val[e];
                      cnt  = u + 1;
                    }
                }
              // Add the entries in order, each once its value is there; the late ones are
              // the last columns, so little is left to add when they arrive.
              auto ready = [](double x) { return __double_as_longlong(x) != (long long)ILU_UNSET; };
              auto give_up = [&](long it) {
                if ((it & 255) != 255 || (!*abort && it < ILU_SPIN))
                  return;
                if (!*abort)
                  {
                    *abort = 1;
                    atomicOr(err, int(DEV_TIMEOUT_ILU));
                  }
                next = cnt;
              };
              if constexpr (SMEM)
                // shared memory: every pass looks at all entries that are due
                for (long it = 0; __any_sync(0xffffffffu, next < cnt); ++it)
                  {
#pragma unroll
                    for (int u = 0; u < ILU_E; ++u)
                      if (u == next && u < cnt)
                        {
                          const double x = ilu_peek<SMEM>(out + c[u]);
                          if (ready(x))
                            {
                              s = fma(v[u], x, s);
                              ++next;
                            }
                        }
                    give_up(it);
                  }
              else
                {
                  // L1: one look at all entries together, then at the first missing one
                  // only (24 -> 21 ms per application at 31k nodes; every pass over all
                  // entries 32 ms.  In shared memory this one is the slower, 4.5 against
                  // 3.3 ms at 2.4k nodes)
                  double x[ILU_E], vv = 0;
                  int    cc   = 0;
                  auto   take = [&] {
#pragma unroll
                    for (int u = 0; u < ILU_E; ++u)
                      if (u == next)
                        {
                          cc = c[u];
                          vv = v[u];
                        }
                  };
#pragma unroll
                  for (int u = 0; u < ILU_E; ++u)
                    if (u < cnt)
                      x[u] = ilu_peek<SMEM>(out + c[u]);
#pragma unroll
                  for (int u = 0; u < ILU_E; ++u)
                    if (u == next && u < cnt && ready(x[u]))
                      {
                        s = fma(v[u], x[u], s);
                        ++next;
                      }
                  take();
                  for (long it = 0; __any_sync(0xffffffffu, next < cnt); ++it)
                    {
                      if (next < cnt)
                        {
                          const double xc = ilu_peek<SMEM>(out + cc);
                          if (ready(xc))
                            {
                              s = fma(vv, xc, s);
                              ++next;
                              take();
                            }
                        }
                      give_up(it);
                    }
                }
            }
          for (int o = 16; o > 0; o >>= 1)
            s += __shfl_xor_sync(0xffffffffu, s, o);
          if (lane == 0)
            ilu_put<SMEM>(out + i, FWD ? b - s : (b - s) / d);
          i  = i1;
          i1 = i2;
          a0 = n0;
          a1 = n1;
          b  = nb;
          d  = nd;
        }
    }

    template <bool SMEM>
    __global__ void __launch_bounds__(ILU_THREADS, 1)
      ilu_apply_kernel(int n, const int32_t *__restrict__ rows_lo, const int32_t *__restrict__ rows_up,
                       const int64_t *__restrict__ ptr, const int32_t *__restrict__ col,
                       const double *__restrict__ val, const int64_t *__restrict__ diag, double *z,
                       double *y, const int *__restrict__ sel, const int *__restrict__ jvec, int *err)
    {
      extern __shared__ double ilu_zs[];
      __shared__ volatile int  abort;
      const int64_t r = blockIdx.x;
      if ((sel && !sel[r]) || (jvec && jvec[r] < 0))
        return;
      double *zr = z + r * n, *yr = y + r * n;
      double *f  = SMEM ? ilu_zs : yr; // forward solution
      const double unset = __longlong_as_double((long long)ILU_UNSET);
      for (int t = threadIdx.x; t < n; t += ILU_THREADS)
        f[t] = unset;
      if (threadIdx.x == 0)
        abort = 0;
      __syncthreads();
      ilu_sweep<true, SMEM>(n, rows_lo, ptr, col, val, diag, zr, f, err, &abort);
      __syncthreads();
      double *g = SMEM ? ilu_zs : zr; // backward solution
      for (int t = threadIdx.x; t < n; t += ILU_THREADS)
        {
          if (SMEM)
            yr[t] = f[t];
          g[t] = unset;
        }
      __syncthreads();
      ilu_sweep<false, SMEM>(n, rows_up, ptr, col, val, diag, yr, g, err, &abort);
      if constexpr (SMEM)
        {
          __syncthreads();
          for (int t = threadIdx.x; t < n; t += ILU_THREADS)
            zr[t] = g[t];
        }
    }

    template <typename T>
    __global__ void combine_p2m_kernel(int64_t n, int K4, const int32_t *__restrict__ prow_dof,
                                       const uint8_t *__restrict__ dir, const T *__restrict__ T1,
                                       const T *__restrict__ T2, T *__restrict__ Tc)
    {
      const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (i >= n)
        return;
      Tc[i] = dir[prow_dof[i / K4]] ? -T2[i] : T1[i];
    }

    inline unsigned nblocks(int64_t n, int t = 256) { return unsigned((n + t - 1) / t); }

    // Double-node constraint lines (deal.II ConstrainedOperator::vmult,
    // include/constrained_matrix.h:100-125): row rows[k] of y becomes
    // x[row] - x[cols[k]] (cols[k] < 0: x[row]).  One thread per (line, column).
    __global__ void constrain_rows_kernel(int n_con, int R, int64_t n, const int32_t *__restrict__ rows,
                                          const int32_t *__restrict__ cols,
                                          const double *__restrict__ x, double *__restrict__ y)
    {
      pdl_entry();
      const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (t >= int64_t(n_con) * R)
        return;
      const int64_t r = t / n_con, k = t - r * n_con;
      const double *xr = x + r * n;
      const int32_t c  = cols[k];
      y[r * n + rows[k]] = xr[rows[k]] - (c >= 0 ? xr[c] : 0.0);
    }

    // Right-hand side of the constraint lines (bem_problem.cc:1405-1579), per
    // (line, column): kind 0 -> 0 (x_row = x_col); kind 1 -> tmp[p] (the
    // potential given at the set's Dirichlet node); kind 2 -> the normal
    // derivative of a Dirichlet-Dirichlet pair (p, q) from the nodal normals
    // nrm (3 per node) and the surface gradients sg of tmp (3 per node, column
    // after column): c = n_p.n_q, (s_q.n_p + (s_p.n_q) c) / (1 - c^2).  Then
    // b[row] = that value (ConstrainedOperator::distribute_rhs).
    __global__ void constraint_rhs_kernel(int n_con, int R, int64_t n, const int32_t *__restrict__ rows,
                                          const uint8_t *__restrict__ kind,
                                          const int32_t *__restrict__ p, const int32_t *__restrict__ q,
                                          const double *__restrict__ tmp,
                                          const double *__restrict__ nrm,
                                          const double *__restrict__ sg, double *__restrict__ b)
    {
      const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (t >= int64_t(n_con) * R)
        return;
      const int64_t r = t / n_con, k = t - r * n_con;
      double        g = 0.0;
      if (kind[k] == 1)
        g = tmp[r * n + p[k]];
      else if (kind[k] == 2)
        {
          const double *np_ = nrm + 3 * int64_t(p[k]), *nq = nrm + 3 * int64_t(q[k]);
          const double *sp_ = sg + 3 * (r * n + p[k]), *sq = sg + 3 * (r * n + q[k]);
          const double  c   = np_[0] * nq[0] + np_[1] * nq[1] + np_[2] * nq[2];
          const double  sqnp = sq[0] * np_[0] + sq[1] * np_[1] + sq[2] * np_[2];
          const double  spnq = sp_[0] * nq[0] + sp_[1] * nq[1] + sp_[2] * nq[2];
          g = (1.0 / (1.0 - c * c)) * (sqnp + spnq * c);
        }
      b[r * n + rows[k]] = g;
    }

  } // namespace

  void launch_dots(int64_t n, int R, int ncols, int64_t ldv, int64_t ldr, const double *V,
                   const double *w, double *partial, int nblk, double *out, cudaStream_t s)
  {
    dim3 grid(nblk, R);
    dots_partial_kernel<<<grid, kDotBlock, 0, s>>>(n, ncols, ldv, ldr, V, w, nblk, partial);
    dots_final_kernel<<<nblocks(int64_t(R) * ncols * 32, 256), 256, 0, s>>>(R, ncols, nblk, partial, out);
    PIBEM_CUDA(cudaGetLastError());
    note_launch(2);
  }

  int arnoldi_blocks(int64_t n)
  {
    return std::max(1, std::min(AR_MAX_BLOCKS, int(std::ceil(0.5 * std::sqrt(double(n))))));
  }

  template <typename T>
  void launch_arnoldi_cgs(const ArnoldiArgs &a, const T *in, cudaStream_t s)
  {
    const int     G = arnoldi_blocks(a.n), L = a.m + 1;
    const dim3    grid(G, a.Ra);
    const size_t  smem = size_t(L) * sizeof(double);
    const int64_t ldr  = int64_t(L) * a.n;
    double       *pa = a.partial, *pb = pa + int64_t(a.S) * L * G, *pn = pb + int64_t(a.S) * L * G;
    if (smem > 16 * 1024)
      {
        raise_smem_limit(reinterpret_cast<const void *>(arnoldi_sub_kernel<false>), smem);
        raise_smem_limit(reinterpret_cast<const void *>(arnoldi_sub_kernel<true>), smem);
      }
    launch_pdl(arnoldi_dots_kernel<T>, grid, AR_THREADS, 0, s, a.n, a.S, G, L, ldr, a.act, in, a.V, a.w,
               a.g.jvec, a.jcur, pa);
    launch_pdl(arnoldi_sub_kernel<false>, grid, AR_THREADS, smem, s, a.n, a.S, G, L, ldr, a.act, a.V,
               a.w, a.jcur, pa, a.g.hb, pb);
    launch_pdl(arnoldi_sub_kernel<true>, grid, AR_THREADS, smem, s, a.n, a.S, G, L, ldr, a.act, a.V,
               a.w, a.jcur, pb, a.g.hb + int64_t(a.S) * L, pn);
    PIBEM_CUDA(cudaGetLastError());
    note_launch(3);
  }
  template void launch_arnoldi_cgs<float>(const ArnoldiArgs &, const float *, cudaStream_t);
  template void launch_arnoldi_cgs<double>(const ArnoldiArgs &, const double *, cudaStream_t);

  template <typename P, typename OUT>
  void launch_arnoldi_finish(const ArnoldiArgs &a, const BlockPrec<P> &bp, OUT *out, bool slot,
                             cudaStream_t s)
  {
    const int     G = arnoldi_blocks(a.n), L = a.m + 1;
    const int64_t ldr  = int64_t(L) * a.n;
    double       *pn   = a.partial + int64_t(2) * a.S * L * G;
    const size_t  head = (size_t(a.Ra) * 20 + 15) / 16 * 16;
    auto launch = [&](auto kern, int threads, int64_t blocks, size_t smem) {
      if (smem > 40 * 1024)
        raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
      launch_pdl(kern, unsigned(1 + std::max<int64_t>(1, blocks)), threads, smem, s, a.n, a.S, G, a.Ra,
                 ldr, a.act, a.jcur, pn, a.w, a.V, out, bp, a.g);
    };
    if (!bp.Pinv)
      {
        const int64_t nb = std::min<int64_t>(2 * AR_MAX_BLOCKS, (a.n + AR_THREADS - 1) / AR_THREADS);
        if (slot)
          launch(arnoldi_finish_kernel<P, OUT, false, 1, true>, AR_THREADS, nb, head);
        else
          launch(arnoldi_finish_kernel<P, OUT, false, 1, false>, AR_THREADS, nb, head);
      }
    else
      {
        // four columns at a time when several share the batch and their slices fit
        // beside two blocks per SM; else one, with fewer warps for very large leaves
        const size_t one = size_t(bp.max_rows) * sizeof(P);
        const bool   big = 16 * one + head > 200 * 1024;
        // 16 warps a block (a warp per column in the Givens step), fewer while SMs would
        // go without a block
        int nw = big ? 8 : 16;
        while (nw > 4 && bp.n_leaves < int64_t(nw) * AR_MAX_BLOCKS && nw / 2 >= a.Ra)
          nw /= 2;
        const int64_t nb = std::min<int64_t>(2 * AR_MAX_BLOCKS, (bp.n_leaves + nw - 1) / nw);
        if (a.Ra > 1 && 64 * one + head <= 100 * 1024)
          launch(arnoldi_finish_kernel<P, OUT, true, 4, false>, 32 * nw, nb, head + 4 * nw * one);
        else
          launch(arnoldi_finish_kernel<P, OUT, true, 1, false>, 32 * nw, nb, head + nw * one);
      }
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }
  template void launch_arnoldi_finish<float, float>(const ArnoldiArgs &, const BlockPrec<float> &, float *,
                                                    bool, cudaStream_t);
  template void launch_arnoldi_finish<float, double>(const ArnoldiArgs &, const BlockPrec<float> &,
                                                     double *, bool, cudaStream_t);
  template void launch_arnoldi_finish<double, double>(const ArnoldiArgs &, const BlockPrec<double> &,
                                                      double *, bool, cudaStream_t);

  void launch_gemv_sub(int64_t n, int R, int ncols, int64_t ldv, int64_t ldr, const double *V,
                       const double *h, int ldh, double *w, double sign, cudaStream_t s,
                       const int *jvec, const int *sel)
  {
    gemv_sub_kernel<<<nblocks(n * R), 256, 0, s>>>(n, R, ncols, ldv, ldr, V, h, ldh, w, sign, jvec,
                                                   sel);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_normalize(int64_t n, int R, const double *w, const double *nrm2, double *out,
                        int64_t ldr, cudaStream_t s, double *z, const int *sel)
  {
    normalize_kernel<<<nblocks(n * R), 256, 0, s>>>(n, R, w, nrm2, out, ldr, z, sel);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_gmres_cycle_init(int R, int m, const int *sel, const double *nrm2, double *g, int *kdone,
                               int *jvec, cudaStream_t s)
  {
    gmres_cycle_init_kernel<<<1, 256, 0, s>>>(R, m + 1, sel, nrm2, g, kdone, jvec);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_gmres_lsq(int R, int m, const int *sel, const double *H, const double *g,
                        const int *kdone, const int *jvec, double *y, cudaStream_t s)
  {
    gmres_lsq_kernel<<<1, 256, 0, s>>>(R, m, sel, H, g, kdone, jvec, y);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_gather_cols(int64_t n, int Rc, const int *cols, const double *src, int64_t lds,
                          double *dst, cudaStream_t s)
  {
    if (Rc == 0)
      return;
    launch_pdl(gather_cols_kernel, nblocks(n * Rc), 256, 0, s, n, Rc, cols, src, lds, dst);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_scatter_cols(int64_t n, int Rc, const int *cols, const double *src, double *dst,
                           int64_t ldd, cudaStream_t s)
  {
    if (Rc == 0)
      return;
    launch_pdl(scatter_cols_kernel, nblocks(n * Rc), 256, 0, s, n, Rc, cols, src, dst, ldd);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_gather_d2f(int64_t n, int Rc, const int *cols, const double *src, float *dst,
                         cudaStream_t s)
  {
    if (Rc == 0)
      return;
    launch_pdl(gather_d2f_kernel, nblocks(n * Rc), 256, 0, s, n, Rc, cols, src, dst);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_f2d_scatter(int64_t n, int Rc, const int *cols, const float *src, double *dst,
                          cudaStream_t s)
  {
    if (Rc == 0)
      return;
    f2d_scatter_kernel<<<nblocks(n * Rc), 256, 0, s>>>(n, Rc, cols, src, dst);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_axpby_sel(int64_t n, int R, const int *sel, double a, const double *x, double b,
                        double *y, cudaStream_t s)
  {
    axpby_sel_kernel<<<nblocks(n * R), 256, 0, s>>>(n, R, sel, a, x, b, y);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_axpby(int64_t n, double a, const double *x, double b, double *y, cudaStream_t s)
  {
    if (n == 0)
      return;
    axpby_kernel<<<nblocks(n), 256, 0, s>>>(n, a, x, b, y);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_convert_d2f(int64_t n, const double *a, float *b, cudaStream_t s)
  {
    if (n == 0)
      return;
    launch_pdl(d2f_kernel, nblocks(n), 256, 0, s, n, a, b);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }
  void launch_convert_f2d(int64_t n, const float *a, double *b, cudaStream_t s)
  {
    if (n == 0)
      return;
    launch_pdl(f2d_kernel, nblocks(n), 256, 0, s, n, a, b);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_build_system_matrix(int64_t n_vals, int n_leaves, const int64_t *val_ptr,
                                  const int64_t *col_ptr, const int64_t *row_ptr,
                                  const int32_t *rows, const int32_t *cols, const uint8_t *dir,
                                  const double *alpha, const double *Nval, const double *Dval,
                                  double *S, float *S32, cudaStream_t s)
  {
    if (n_vals == 0)
      return;
    system_matrix_kernel<<<nblocks(n_vals), 256, 0, s>>>(n_vals, n_leaves, val_ptr, col_ptr,
                                                         row_ptr, rows, cols, dir, alpha, Nval,
                                                         Dval, S, S32);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_rhs_combine(int64_t n, int R, const double *tmp, const uint8_t *dir,
                          const double *alpha, const double *oN, const double *oD, double *rhs,
                          cudaStream_t s)
  {
    rhs_combine_kernel<<<nblocks(n * R), 256, 0, s>>>(n, R, tmp, dir, alpha, oN, oD, rhs);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_split_masks(int64_t n, int R, const double *tmp, const uint8_t *dir, double *a,
                          double *b, cudaStream_t s)
  {
    split_masks_kernel<<<nblocks(n * R), 256, 0, s>>>(n, R, tmp, dir, a, b);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_scatter(int64_t n, int R, const double *sol, const uint8_t *dir, double *phi,
                      double *dphi, cudaStream_t s)
  {
    scatter_kernel<<<nblocks(n * R), 256, 0, s>>>(n, R, sol, dir, phi, dphi);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_constrain_rows(int n_con, int R, int64_t n, const int32_t *rows, const int32_t *cols,
                             const double *x, double *y, cudaStream_t s)
  {
    if (n_con == 0 || R == 0)
      return;
    launch_pdl(constrain_rows_kernel, nblocks(int64_t(n_con) * R), 256, 0, s, n_con, R, n, rows, cols, x, y);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_constraint_rhs(int n_con, int R, int64_t n, const int32_t *rows, const uint8_t *kind,
                             const int32_t *p, const int32_t *q, const double *tmp,
                             const double *nrm, const double *sg, double *b, cudaStream_t s)
  {
    if (n_con == 0 || R == 0)
      return;
    constraint_rhs_kernel<<<nblocks(int64_t(n_con) * R), 256, 0, s>>>(n_con, R, n, rows, kind, p, q,
                                                                      tmp, nrm, sg, b);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_sub_norm(int64_t n, int R, const double *nrm2, double *x, cudaStream_t s)
  {
    sub_norm_kernel<<<nblocks(n * R), 256, 0, s>>>(n, R, nrm2, x);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_add_scalar(int64_t n, int R, const double *shift, double *x, cudaStream_t s)
  {
    add_scalar_kernel<<<nblocks(n * R), 256, 0, s>>>(n, R, shift, x);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  template <typename P>
  void launch_block_apply(const BlockPrec<P> &bp, int R, int64_t n, const double *v, int64_t ldv,
                          double *z, const int *sel, cudaStream_t s)
  {
    if (bp.n_leaves == 0)
      return;
    const size_t smem = size_t(8) * bp.max_rows * sizeof(P);
    if (smem > 48 * 1024)
      raise_smem_limit(reinterpret_cast<const void *>(block_apply_kernel<P>), smem);
    block_apply_kernel<P><<<(bp.n_leaves + 7) / 8, 256, smem, s>>>(
      bp.n_leaves, bp.max_rows, R, n, ldv, bp.row_ptr, bp.blk_ptr, bp.rows, bp.Pinv, v, z, sel);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }
  template void launch_block_apply<float>(const BlockPrec<float> &, int, int64_t, const double *, int64_t,
                                          double *, const int *, cudaStream_t);
  template void launch_block_apply<double>(const BlockPrec<double> &, int, int64_t, const double *,
                                           int64_t, double *, const int *, cudaStream_t);

  void launch_ilu_fill(int64_t n, const int64_t *ptr, const int32_t *pos, const int32_t *row_leaf,
                       const int64_t *nrow_ptr, const int64_t *ncol_ptr, const int64_t *nval_ptr,
                       const int32_t *ncols, const double *S, const int32_t *con, int32_t *col,
                       double *val, cudaStream_t s)
  {
    if (n == 0)
      return;
    ilu_fill_kernel<<<nblocks(n * 32), 256, 0, s>>>(n, ptr, pos, row_leaf, nrow_ptr, ncol_ptr, nval_ptr,
                                                    ncols, S, con, col, val);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_ilu_factor(const std::vector<int64_t> &lptr, const int32_t *rows, const int64_t *ptr,
                         const int32_t *col, double *val, const int64_t *diag, int64_t max_row,
                         cudaStream_t s)
  {
    const size_t smem = size_t(max_row) * (sizeof(double) + sizeof(int32_t));
    if (smem > 48 * 1024)
      PIBEM_CUDA(cudaFuncSetAttribute(ilu_factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      int(smem)));
    for (size_t l = 0; l + 1 < lptr.size(); ++l)
      {
        const int64_t nr = lptr[l + 1] - lptr[l];
        if (nr == 0)
          continue;
        ilu_factor_kernel<<<unsigned(nr), 256, smem, s>>>(rows + lptr[l], ptr, col, val, diag);
        note_launch();
      }
    PIBEM_CUDA(cudaGetLastError());
  }

  void launch_copy_sel(int64_t n, int R, const double *v, int64_t ldv, double *z, const int *sel,
                       cudaStream_t s)
  {
    if (n * R == 0)
      return;
    copy_sel_kernel<<<nblocks(n * R), 256, 0, s>>>(n, R, v, ldv, z, sel);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  // Bytes of a column's solution up to which it is handed on in shared memory
  static constexpr size_t ILU_SMEM = 200 * 1024;

  // One block per column (ilu_apply_kernel) costs a latency per level while the levels hold
  // a few rows, and then a time per row that one SM sets: 0.13 - 0.17 us in shared memory,
  // 0.23 - 0.25 through L1.  A launch per level costs 6 us (200 entries a row) to 10 (500)
  // whatever its width.  So triangles of wide levels (few long chains: nodes numbered at
  // random or by colour; along a surface a level holds 2 - 10 rows) run level by level.
  // Measured, ms an application, block / level launches, by rows per level:
  //   shared memory (13.8k, 24.6k nodes)   21: 4.5 / 9.4   33: 8.2 / 13.0   47: 3.5 / 3.5   75: 5.9 / 4.2
  //   L1 (38k, 65k nodes)   18: 18.5 / 27.2   21: 30.7 / 37.3   25: 25 / 39   51: 18.7 / 14.8   73: 33.7 / 19.6
  //                        114: 17.3 / 4.8   231: 29.3 / 4.3
  bool ilu_by_level(int64_t n, int64_t levels)
  {
    const int64_t wide = size_t(n) * sizeof(double) <= ILU_SMEM ? 46 : 32; // rows per level
    return 2 * n > wide * levels;
  }

  void launch_ilu_levels(const std::vector<int64_t> &lptr_lo, const int32_t *rows_lo,
                         const std::vector<int64_t> &lptr_up, const int32_t *rows_up, int R, int64_t n,
                         const int64_t *ptr, const int32_t *col, const double *val,
                         const int64_t *diag, double *z, const int *sel, const int *jvec,
                         cudaStream_t s)
  {
    if (n == 0 || R == 0)
      return;
    auto sweep = [&](auto kern, const std::vector<int64_t> &lptr, const int32_t *rows) {
      for (size_t l = 0; l + 1 < lptr.size(); ++l)
        {
          const int nr = int(lptr[l + 1] - lptr[l]);
          if (nr == 0)
            continue;
          kern<<<nblocks(int64_t(nr) * R * 32), 256, 0, s>>>(nr, rows + lptr[l], R, n, ptr, col, val, diag, z,
                                                             sel, jvec);
          note_launch();
        }
    };
    sweep(ilu_level_kernel<true>, lptr_lo, rows_lo);
    sweep(ilu_level_kernel<false>, lptr_up, rows_up);
    PIBEM_CUDA(cudaGetLastError());
  }

  void launch_ilu_apply(int64_t n, int R, const int32_t *rows_lo, const int32_t *rows_up,
                        const int64_t *ptr, const int32_t *col, const double *val,
                        const int64_t *diag, double *z, double *y, const int *sel, const int *jvec,
                        int *err, cudaStream_t s)
  {
    if (n == 0 || R == 0)
      return;
    const size_t smem = size_t(n) * sizeof(double);
    if (smem <= ILU_SMEM)
      {
        if (smem > 40 * 1024)
          raise_smem_limit(reinterpret_cast<const void *>(ilu_apply_kernel<true>), smem);
        ilu_apply_kernel<true><<<R, ILU_THREADS, smem, s>>>(int(n), rows_lo, rows_up, ptr, col, val, diag,
                                                            z, y, sel, jvec, err);
      }
    else
      ilu_apply_kernel<false><<<R, ILU_THREADS, 0, s>>>(int(n), rows_lo, rows_up, ptr, col, val, diag, z,
                                                        y, sel, jvec, err);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  template <typename T>
  void launch_combine_p2m(int64_t n_rows, int K4, const int32_t *prow_dof, const uint8_t *dir,
                          const T *T1, const T *T2, T *Tc, cudaStream_t s)
  {
    const int64_t n = n_rows * K4;
    if (n == 0)
      return;
    combine_p2m_kernel<T><<<nblocks(n), 256, 0, s>>>(n, K4, prow_dof, dir, T1, T2, Tc);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }
  template void launch_combine_p2m<float>(int64_t, int, const int32_t *, const uint8_t *,
                                          const float *, const float *, float *, cudaStream_t);
  template void launch_combine_p2m<double>(int64_t, int, const int32_t *, const uint8_t *,
                                           const double *, const double *, double *, cudaStream_t);
} // namespace pibem
