// FMM operator kernels, one pass of BEMFMA::generate_multipole_expansions +
// multipole_matr_vect_products (source/bem_fma.cc:1971-3072) for R right-hand
// sides at once, in FP64 or FP32 (template parameter T):
//   near-field leaf-block SpMV          (prec_*_matrix.vmult, bem_fma.cc:2408-2409)
//   P2M apply from precomputed tables   (bem_fma.cc:2064-2114)
//   M2M, level by level upwards         (bem_fma.cc:2274-2376)
//   L2L + M2L, level by level downwards (bem_fma.cc:2582-2652)
//   M2P for deeper non-interaction boxes (bem_fma.cc:2664-2704)
//   L2P at the nodes of childless boxes (bem_fma.cc:2959-2986)
// Expansions are laid out [box][rhs][k] with K = (p+1)^2 scaled reals.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "devmath.cuh"
#include "ffmath.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace pibem
{
  namespace
  {
    template <typename T>
    __device__ inline T warp_sum(T v)
    {
      for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
      return v;
    }

    __device__ __forceinline__ float  shfl_xor(float v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
    __device__ __forceinline__ double shfl_xor(double v, int o) { return __shfl_xor_sync(0xffffffffu, v, o); }
    __device__ __forceinline__ float2 shfl_xor(float2 v, int o)
    {
      return make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
    }

    // a * b + c with one rounding (no dependence on the compiler's contraction)
    __device__ __forceinline__ float  fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
    __device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
    __device__ __forceinline__ float  mul_rn(float a, float b) { return __fmul_rn(a, b); }
    __device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

    // s + a . x for 4 values, with the rounding steps spelled out so that every
    // code path (one column or several) computes a column bit-for-bit alike.
    __device__ inline float dot4_acc(float s, const float (&a)[4], const float *x)
    {
      float d = __fmul_rn(a[0], x[0]);
      d       = __fmaf_rn(a[1], x[1], d);
      d       = __fmaf_rn(a[2], x[2], d);
      d       = __fmaf_rn(a[3], x[3], d);
      return __fadd_rn(s, d);
    }
    __device__ inline double dot4_acc(double s, const double (&a)[4], const double *x)
    {
      double d = __dmul_rn(a[0], x[0]);
      d        = __fma_rn(a[1], x[1], d);
      d        = __fma_rn(a[2], x[2], d);
      d        = __fma_rn(a[3], x[3], d);
      return __dadd_rn(s, d);
    }

    // 4-wide loads from 16-byte aligned rows.
    __device__ inline void load4(const float *p, float (&v)[4])
    {
      const float4 t = *reinterpret_cast<const float4 *>(p);
      v[0] = t.x;
      v[1] = t.y;
      v[2] = t.z;
      v[3] = t.w;
    }
    __device__ inline void load4(const double *p, double (&v)[4])
    {
      const double2 a = *reinterpret_cast<const double2 *>(p);
      const double2 b = *reinterpret_cast<const double2 *>(p + 2);
      v[0] = a.x;
      v[1] = a.y;
      v[2] = b.x;
      v[3] = b.y;
    }

    // Sums over the warp of M values per lane (M = 2, 4, 8 or 16) with the additions
    // of warp_sum's butterfly: after each of the first log2(M) steps a lane keeps half
    // of the values, so M + 4 - log2(M) shuffles instead of 5 M.  Lane l ends with the
    // sum of value l / (32 / M).
    template <int M, typename T, typename ADD>
    __device__ __forceinline__ T warp_sums(T (&v)[M], ADD add)
    {
      const int lane = threadIdx.x & 31;
      int       o    = 16;
#pragma unroll
      for (int n = M / 2; n > 0; n >>= 1, o >>= 1)
        {
          const bool up = (lane & o) != 0;
#pragma unroll
          for (int i = 0; i < n; ++i)
            v[i] = add(up ? v[i + n] : v[i], shfl_xor(up ? v[i] : v[i + n], o));
        }
      for (; o > 0; o >>= 1)
        v[0] = add(v[0], shfl_xor(v[0], o));
      return v[0];
    }

    // Near-field leaf-block SpMV for several columns: one block per childless box.
    // The x entries of the block's columns are gathered into shared memory (rb
    // right-hand sides at a time, zero in the paddings); a warp takes RR rows and RC
    // columns at a time, so that a row's 16-byte loads serve RC columns and an x
    // load RR rows.  A (row, column) sum has the chunks per lane, the order and the
    // butterfly of the one-column kernels.
    // What bounds it: the x gathers (4 bytes each) and shared-memory loads.
    template <typename T, int RC, int RR>
    __global__ void __launch_bounds__(128)
      near_leaf_multi_kernel(int R, int rb, int N, const int64_t *__restrict__ nrow_ptr,
                             const int64_t *__restrict__ ncol_ptr, const int64_t *__restrict__ nval_ptr,
                             const int32_t *__restrict__ nrows, const int32_t *__restrict__ ncols,
                             const T *__restrict__ vals, const T *__restrict__ x, T *__restrict__ y,
                             bool acc)
    {
      pdl_entry();
      extern __shared__ __align__(16) unsigned char smem_raw[];
      T            *sx   = reinterpret_cast<T *>(smem_raw); // [rb][ld]
      const int     leaf = blockIdx.x;
      const int64_t c0   = ncol_ptr[leaf];
      const int     nc = int(ncol_ptr[leaf + 1] - c0), ld = (nc + 3) / 4 * 4, n4 = ld / 4;
      const int64_t r0 = nrow_ptr[leaf];
      const int     nr = int(nrow_ptr[leaf + 1] - r0);
      const T      *V    = vals + nval_ptr[leaf];
      const int     warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      for (int ra = 0; ra < R; ra += rb)
        {
          const int rc = min(rb, R - ra), rcp = (rc + RC - 1) / RC * RC;
          __syncthreads();
          for (int c = threadIdx.x; c < ld; c += blockDim.x)
            {
              const T *xc = x + ra * int64_t(N) + (c < nc ? ncols[c0 + c] : 0);
#pragma unroll 8
              for (int r = 0; r < rcp; ++r)
                sx[r * ld + c] = c < nc && r < rc ? xc[r * int64_t(N)] : T(0);
            }
          __syncthreads();
          for (int row = warp * RR; row < nr; row += 4 * RR)
            for (int rq = 0; rq < rcp; rq += RC)
              {
                T s[RR * RC];
#pragma unroll
                for (int i = 0; i < RR * RC; ++i)
                  s[i] = T(0);
                const T *v[RR];
#pragma unroll
                for (int i = 0; i < RR; ++i) // a row beyond the leaf's repeats the last one
                  v[i] = V + int64_t(min(row + i, nr - 1)) * ld;
                for (int j = lane; j < n4; j += 32)
                  {
                    T a[RR][4], b[RC][4];
#pragma unroll
                    for (int i = 0; i < RR; ++i)
                      load4(v[i] + 4 * j, a[i]);
#pragma unroll
                    for (int r = 0; r < RC; ++r)
                      load4(sx + (rq + r) * ld + 4 * j, b[r]);
#pragma unroll
                    for (int i = 0; i < RR; ++i)
#pragma unroll
                      for (int r = 0; r < RC; ++r)
                        s[i * RC + r] = dot4_acc(s[i * RC + r], a[i], b[r]);
                  }
                const T t = warp_sums<RR * RC>(s, [](T p, T q) { return p + q; });
                constexpr int W = 32 / (RR * RC); // lanes per value
                const int     i = row + lane / (W * RC), r = rq + (lane / W) % RC;
                if (lane % W == 0 && i < nr && r < rc)
                  {
                    T &o = y[(ra + r) * int64_t(N) + nrows[r0 + i]];
                    o    = acc ? o + t : t;
                  }
              }
        }
    }

    // 4-byte asynchronous global -> shared copy (cp.async, L1-allocating)
    __device__ inline void cp_async4(void *dst, const void *src)
    {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                   "l"(src)
                   : "memory");
    }
    __device__ inline void cp_async8(void *dst, const void *src)
    {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                   "l"(src)
                   : "memory");
    }
    __device__ inline void cp_async_x(float *dst, const float *src) { cp_async4(dst, src); }
    __device__ inline void cp_async_x(double *dst, const double *src) { cp_async8(dst, src); }

    // Near-field SpMV for one column where near_leaf_sched_kernel's shared
    // memory would not fit (more than about 14,500 columns in a leaf in FP32,
    // 9,600 in FP64),
    // software-pipelined: persistent blocks
    // take leaves L, L + gridDim.x, ... (the grid works through the leaves in
    // ascending windows.  Measured on GB300, 98k spheroid: 80 us; contiguous
    // leaf ranges of equal bytes per block 125 us; an L2 prefetch of the leaves
    // ahead with cp.async.bulk.prefetch 89-92 us; a dynamic schedule drawing
    // leaves from an atomic counter 89 us); while the warps stream the rows of a
    // leaf, the x entries of the block's next leaf are gathered into the other
    // half of a double buffer with cp.async.  A row is computed exactly as in
    // near_leaf_multi_kernel (same chunks per lane, same order, same butterfly).
    // Shared memory: 2 x ld_max values.
    template <typename T>
    __global__ void __launch_bounds__(256)
      near_leaf_pipe_kernel(int n_leaves, int ld_max, const int64_t *__restrict__ nrow_ptr,
                            const int64_t *__restrict__ ncol_ptr,
                            const int64_t *__restrict__ nval_ptr, const int32_t *__restrict__ nrows,
                            const int32_t *__restrict__ ncols, const T *__restrict__ vals,
                            const T *__restrict__ x, T *__restrict__ y, bool acc)
    {
      pdl_entry();
      extern __shared__ __align__(16) unsigned char smem_raw[];
      T        *sxb  = reinterpret_cast<T *>(smem_raw); // [2][ld_max]
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
      // gather of leaf l into buffer b: cp.async for the columns, zeros in the padding
      auto gather = [&](int l, int b) {
        const int64_t c0 = ncol_ptr[l], nc = ncol_ptr[l + 1] - c0;
        const int64_t ld = (nc + 3) / 4 * 4;
        T            *sx = sxb + int64_t(b) * ld_max;
        for (int64_t c = threadIdx.x; c < ld; c += blockDim.x)
          if (c < nc)
            cp_async_x(sx + c, x + ncols[c0 + c]);
          else
            sx[c] = T(0);
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      int leaf = blockIdx.x, buf = 0;
      if (leaf >= n_leaves)
        return;
      gather(leaf, 0);
      for (; leaf < n_leaves; leaf += gridDim.x, buf ^= 1)
        {
          asm volatile("cp.async.wait_group 0;" ::: "memory");
          __syncthreads(); // this leaf's x is in place; the other buffer is free
          const int next = leaf + gridDim.x;
          if (next < n_leaves)
            gather(next, buf ^ 1);
          const T      *sx = sxb + int64_t(buf) * ld_max;
          const int64_t c0 = ncol_ptr[leaf], nc = ncol_ptr[leaf + 1] - c0;
          const int64_t ld = (nc + 3) / 4 * 4;
          const int     n4 = int(ld / 4);
          const int64_t r0 = nrow_ptr[leaf], nr = nrow_ptr[leaf + 1] - r0;
          const T      *V  = vals + nval_ptr[leaf];
          // two rows per warp at a time (rows row and row + nw), four 16-byte
          // loads of each in flight per lane
          for (int64_t row = warp; row < nr; row += 2 * nw)
            {
              const bool two = row + nw < nr;
              const T   *v0  = V + row * ld;
              const T   *v1  = V + (two ? row + nw : row) * ld;
              T          s0 = T(0), s1 = T(0);
#pragma unroll 4
              for (int j = lane; j < n4; j += 32)
                {
                  T a0[4], a1[4];
                  load4(v0 + 4 * j, a0);
                  load4(v1 + 4 * j, a1);
                  s0 = dot4_acc(s0, a0, sx + 4 * j);
                  s1 = dot4_acc(s1, a1, sx + 4 * j);
                }
              const T t0 = warp_sum(s0), t1 = warp_sum(s1);
              if (lane == 0)
                {
                  T &o0 = y[nrows[r0 + row]];
                  o0    = acc ? o0 + t0 : t0;
                  if (two)
                    {
                      T &o1 = y[nrows[r0 + row + nw]];
                      o1    = acc ? o1 + t1 : t1;
                    }
                }
            }
        }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }

    __device__ inline void cp_async16(void *dst, const void *src)
    {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                   "l"(src)
                   : "memory");
    }

    // Schedule position of the t-th leaf of block b: snake order over the G
    // blocks (b, 2G-1-b, 2G+b, ...), so that with the leaves sorted by bytes
    // every block streams about the same amount.
    __device__ __forceinline__ int64_t near_sched_pos(int b, int t, int G)
    {
      return int64_t(t) * G + ((t & 1) ? G - 1 - b : b);
    }

    // 16-byte streaming loads that do not allocate in L1
    __device__ inline void load4_na(const float *p, float (&v)[4])
    {
      asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
          : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
          : "l"(p));
    }
    __device__ inline void load4_na(const double *p, double (&v)[4])
    {
      asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(p));
      asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v[2]), "=d"(v[3]) : "l"(p + 2));
    }
    template <bool NA, typename T>
    __device__ __forceinline__ void load4v(const T *p, T (&v)[4])
    {
      if constexpr (NA)
        load4_na(p, v);
      else
        load4(p, v);
    }

    // Near-field SpMV for one column: persistent blocks over a schedule of the
    // leaves sorted by value bytes (record per leaf: value offset, column
    // offset, row offset, rows | columns << 32), three stages deep.  While the
    // warps stream the rows of the block's leaf t, the block has one cp.async
    // group in flight holding the x entries of its leaf t+1 (gathered through
    // the column ids already in shared memory), the column ids of leaf t+2 and
    // the schedule record of leaf t+3, so that inside a leaf only the row
    // values are waited for.  Rows: two per warp at a time, the 16-byte loads of NB
    // chunks per lane and row issued before any is used (NA: loads that do not
    // allocate in L1).  A row is computed exactly as in near_leaf_multi_kernel (same
    // chunks per lane, same order, same butterfly), so the leaf order and the
    // block shape do not change a bit of y.
    // Shared memory: 128 bytes of records, 2 x ld_max column ids, 2 x ld_max x.
    template <typename T, int NB, int BS, bool NA>
    __global__ void __launch_bounds__(BS)
      near_leaf_sched_kernel(int n_leaves, int ld_max, const int64_t *__restrict__ sched,
                             const int32_t *__restrict__ nrows, const int32_t *__restrict__ ncols,
                             const T *__restrict__ vals, const T *__restrict__ x,
                             T *__restrict__ y, bool acc)
    {
      pdl_entry();
      extern __shared__ __align__(16) unsigned char smem_raw[];
      int64_t  *srec = reinterpret_cast<int64_t *>(smem_raw);       // [4][4]
      int32_t  *sid  = reinterpret_cast<int32_t *>(smem_raw + 128); // [2][ld_max]
      T        *sxb  = reinterpret_cast<T *>(smem_raw + 128 + size_t(8) * ld_max); // [2][ld_max]
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
      const int G = gridDim.x, b = blockIdx.x;
      auto valid = [&](int t) { return near_sched_pos(b, t, G) < n_leaves; };
      auto rec   = [&](int t) { return srec + 4 * (t & 3); };
      // schedule record of leaf t (threads 0 and 1, 16 bytes each)
      auto fetch_rec = [&](int t) {
        if (threadIdx.x < 2 && valid(t))
          cp_async16(rec(t) + 2 * threadIdx.x, sched + 4 * near_sched_pos(b, t, G) + 2 * threadIdx.x);
      };
      // column ids of leaf t (its record in place)
      auto fetch_ids = [&](int t) {
        const int64_t c0 = rec(t)[1];
        const int     nc = int(uint64_t(rec(t)[3]) >> 32);
        int32_t      *d  = sid + (t & 1) * ld_max;
        for (int c = threadIdx.x; c < nc; c += blockDim.x)
          cp_async4(d + c, ncols + c0 + c);
      };
      // x entries of leaf t (its column ids in place), zeros in the padding
      auto gather_x = [&](int t) {
        const int      nc = int(uint64_t(rec(t)[3]) >> 32), ld = (nc + 3) & ~3;
        const int32_t *si = sid + (t & 1) * ld_max;
        T             *d  = sxb + (t & 1) * ld_max;
        for (int c = threadIdx.x; c < ld; c += blockDim.x)
          if (c < nc)
            cp_async_x(d + c, x + si[c]);
          else
            d[c] = T(0);
      };
      if (!valid(0))
        return;
      fetch_rec(0);
      fetch_rec(1);
      fetch_rec(2);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      fetch_ids(0);
      if (valid(1))
        fetch_ids(1);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      gather_x(0);
      asm volatile("cp.async.commit_group;" ::: "memory");
      for (int t = 0; valid(t); ++t)
        {
          asm volatile("cp.async.wait_group 0;" ::: "memory");
          __syncthreads(); // leaf t's x, leaf t+1's ids, records t..t+2 in place
          if (valid(t + 1))
            gather_x(t + 1);
          if (valid(t + 2))
            fetch_ids(t + 2);
          fetch_rec(t + 3);
          asm volatile("cp.async.commit_group;" ::: "memory");
          const int64_t *r  = rec(t);
          const T       *V  = vals + r[0];
          const int64_t  r0 = r[2];
          const int      nr = int(uint32_t(uint64_t(r[3]))), nc = int(uint64_t(r[3]) >> 32);
          const int      ld = (nc + 3) & ~3, n4 = ld >> 2;
          const T       *sx = sxb + (t & 1) * ld_max;
          for (int row = warp; row < nr; row += 2 * nw)
            {
              const bool two = row + nw < nr;
              int        o0 = 0, o1 = 0;
              if (lane == 0)
                {
                  o0 = nrows[r0 + row];
                  o1 = two ? nrows[r0 + row + nw] : o0;
                }
              const T *v0 = V + int64_t(row) * ld;
              const T *v1 = V + int64_t(two ? row + nw : row) * ld;
              T        s0 = T(0), s1 = T(0);
              for (int jb = lane; jb < n4; jb += 32 * NB)
                {
                  T a0[NB][4], a1[NB][4];
#pragma unroll
                  for (int k = 0; k < NB; ++k)
                    if (jb + 32 * k < n4)
                      {
                        load4v<NA>(v0 + 4 * (jb + 32 * k), a0[k]);
                        if (two)
                          load4v<NA>(v1 + 4 * (jb + 32 * k), a1[k]);
                      }
#pragma unroll
                  for (int k = 0; k < NB; ++k)
                    if (jb + 32 * k < n4)
                      {
                        s0 = dot4_acc(s0, a0[k], sx + 4 * (jb + 32 * k));
                        if (two)
                          s1 = dot4_acc(s1, a1[k], sx + 4 * (jb + 32 * k));
                      }
                }
              const T t0 = warp_sum(s0), t1 = warp_sum(s1);
              if (lane == 0)
                {
                  T &y0 = y[o0];
                  y0    = acc ? y0 + t0 : t0;
                  if (two)
                    {
                      T &y1 = y[o1];
                      y1    = acc ? y1 + t1 : t1;
                    }
                }
            }
        }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }

    // FP64-accurate near-field SpMV for one column on the FP32 pipes: the
    // values and x as (hi, lo) FP32 pairs (8 bytes a value, as FP64), every
    // product split exactly (TwoProduct) with its cross terms, the row sums
    // carried with TwoSum; about 11 FP32 instructions per value, so the kernel
    // streams at HBM speed where FP64 FMA (1/58 of the FP32 rate) could not.
    // Same structure as near_leaf_pipe_kernel: persistent blocks, the next
    // leaf's x gathered with cp.async while the warps stream two rows each.
    // y[row] = hi + lo in FP64 (acc: added).
    __global__ void __launch_bounds__(256)
      near_leaf_ff_kernel(int n_leaves, int ld_max,
                          const int64_t *__restrict__ nrow_ptr,
                          const int64_t *__restrict__ ncol_ptr, const int64_t *__restrict__ nval_ptr,
                          const int32_t *__restrict__ nrows, const int32_t *__restrict__ ncols,
                          const float2 *__restrict__ vals, const float2 *__restrict__ x,
                          double *__restrict__ y, bool acc)
    {
      extern __shared__ __align__(16) unsigned char smem_raw[];
      float2   *sxb  = reinterpret_cast<float2 *>(smem_raw); // [2][ld_max]
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
      auto gather = [&](int l, int b) {
        const int64_t c0 = ncol_ptr[l], nc = ncol_ptr[l + 1] - c0;
        const int64_t ld = (nc + 3) / 4 * 4;
        float2       *sx = sxb + int64_t(b) * ld_max;
        for (int64_t c = threadIdx.x; c < ld; c += blockDim.x)
          if (c < nc)
            cp_async8(reinterpret_cast<double *>(sx + c), reinterpret_cast<const double *>(x + ncols[c0 + c]));
          else
            sx[c] = make_float2(0.f, 0.f);
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      int leaf = blockIdx.x, buf = 0;
      if (leaf >= n_leaves)
        return;
      gather(leaf, 0);
      for (; leaf < n_leaves; leaf += gridDim.x, buf ^= 1)
        {
          asm volatile("cp.async.wait_group 0;" ::: "memory");
          __syncthreads();
          const int next = leaf + gridDim.x;
          if (next < n_leaves)
            gather(next, buf ^ 1);
          const float2 *sx = sxb + int64_t(buf) * ld_max;
          const int64_t c0 = ncol_ptr[leaf], nc = ncol_ptr[leaf + 1] - c0;
          const int64_t ld = (nc + 3) / 4 * 4;
          const int     n4 = int(ld / 4);
          const int64_t r0 = nrow_ptr[leaf], nr = nrow_ptr[leaf + 1] - r0;
          const float2 *V  = vals + nval_ptr[leaf];
          for (int64_t row = warp; row < nr; row += 2 * nw)
            {
              const bool    two = row + nw < nr;
              const float2 *v0  = V + row * ld;
              const float2 *v1  = V + (two ? row + nw : row) * ld;
              float         h0 = 0.f, l0 = 0.f, h1 = 0.f, l1 = 0.f;
#pragma unroll 2
              for (int j = lane; j < n4; j += 32)
                {
                  const float4 a0 = *reinterpret_cast<const float4 *>(v0 + 4 * j);
                  const float4 b0 = *reinterpret_cast<const float4 *>(v0 + 4 * j + 2);
                  const float4 a1 = *reinterpret_cast<const float4 *>(v1 + 4 * j);
                  const float4 b1 = *reinterpret_cast<const float4 *>(v1 + 4 * j + 2);
                  const float2 x0 = sx[4 * j], x1 = sx[4 * j + 1], x2 = sx[4 * j + 2], x3 = sx[4 * j + 3];
                  ff_mac(h0, l0, make_float2(a0.x, a0.y), x0);
                  ff_mac(h0, l0, make_float2(a0.z, a0.w), x1);
                  ff_mac(h0, l0, make_float2(b0.x, b0.y), x2);
                  ff_mac(h0, l0, make_float2(b0.z, b0.w), x3);
                  ff_mac(h1, l1, make_float2(a1.x, a1.y), x0);
                  ff_mac(h1, l1, make_float2(a1.z, a1.w), x1);
                  ff_mac(h1, l1, make_float2(b1.x, b1.y), x2);
                  ff_mac(h1, l1, make_float2(b1.z, b1.w), x3);
                }
              float2 t0 = ff_norm(h0, l0), t1 = ff_norm(h1, l1);
              for (int o = 16; o > 0; o >>= 1)
                {
                  t0 = ff_add(t0, make_float2(__shfl_xor_sync(0xffffffffu, t0.x, o),
                                              __shfl_xor_sync(0xffffffffu, t0.y, o)));
                  t1 = ff_add(t1, make_float2(__shfl_xor_sync(0xffffffffu, t1.x, o),
                                              __shfl_xor_sync(0xffffffffu, t1.y, o)));
                }
              if (lane == 0)
                {
                  double &o0 = y[nrows[r0 + row]];
                  o0         = acc ? __dadd_rn(o0, ff_join(t0)) : ff_join(t0);
                  if (two)
                    {
                      double &o1 = y[nrows[r0 + row + nw]];
                      o1         = acc ? __dadd_rn(o1, ff_join(t1)) : ff_join(t1);
                    }
                }
            }
        }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }

    // near_leaf_ff_kernel for several columns: RC columns' x pairs in shared memory,
    // a warp takes RR rows and RC columns at a time, so that the values (8 bytes each)
    // are read once per RC columns.  Per (row, column) the chunks, order and butterfly
    // of the one-column kernel, whose sums it therefore repeats bit for bit.
    // What bounds it: the FP32 pipes (11 instructions per value and column).
    template <int RC, int RR>
    __global__ void __launch_bounds__(128)
      near_leaf_ff_multi_kernel(int R, int N, const int64_t *__restrict__ nrow_ptr,
                                const int64_t *__restrict__ ncol_ptr, const int64_t *__restrict__ nval_ptr,
                                const int32_t *__restrict__ nrows, const int32_t *__restrict__ ncols,
                                const float2 *__restrict__ vals, const float2 *__restrict__ x,
                                double *__restrict__ y, bool acc)
    {
      extern __shared__ __align__(16) unsigned char smem_raw[];
      float2       *sx   = reinterpret_cast<float2 *>(smem_raw); // [RC][ld]
      const int     leaf = blockIdx.x, ra = blockIdx.y * RC, rc = min(RC, R - ra);
      const int64_t c0   = ncol_ptr[leaf];
      const int     nc = int(ncol_ptr[leaf + 1] - c0), ld = (nc + 3) / 4 * 4, n4 = ld / 4;
      const int64_t r0 = nrow_ptr[leaf];
      const int     nr = int(nrow_ptr[leaf + 1] - r0);
      const float2 *V    = vals + nval_ptr[leaf];
      const int     warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      for (int c = threadIdx.x; c < ld; c += blockDim.x)
        {
          const float2 *xc = x + ra * int64_t(N) + (c < nc ? ncols[c0 + c] : 0);
#pragma unroll
          for (int r = 0; r < RC; ++r)
            sx[r * ld + c] = c < nc && r < rc ? xc[r * int64_t(N)] : make_float2(0.f, 0.f);
        }
      __syncthreads();
      for (int row = warp * RR; row < nr; row += 4 * RR)
        {
          float h[RR][RC], l[RR][RC];
#pragma unroll
          for (int i = 0; i < RR; ++i)
#pragma unroll
            for (int r = 0; r < RC; ++r)
              h[i][r] = l[i][r] = 0.f;
          const float4 *v[RR];
#pragma unroll
          for (int i = 0; i < RR; ++i) // a row beyond the leaf's repeats the last one
            v[i] = reinterpret_cast<const float4 *>(V + int64_t(min(row + i, nr - 1)) * ld);
          for (int j = lane; j < n4; j += 32)
            {
              float4 a[RR][2];
#pragma unroll
              for (int i = 0; i < RR; ++i)
                {
                  a[i][0] = v[i][2 * j];
                  a[i][1] = v[i][2 * j + 1];
                }
#pragma unroll
              for (int r = 0; r < RC; ++r)
                {
                  const float4 *xr = reinterpret_cast<const float4 *>(sx + r * ld) + 2 * j;
                  const float4  p = xr[0], q = xr[1];
#pragma unroll
                  for (int i = 0; i < RR; ++i)
                    {
                      ff_mac(h[i][r], l[i][r], make_float2(a[i][0].x, a[i][0].y), make_float2(p.x, p.y));
                      ff_mac(h[i][r], l[i][r], make_float2(a[i][0].z, a[i][0].w), make_float2(p.z, p.w));
                      ff_mac(h[i][r], l[i][r], make_float2(a[i][1].x, a[i][1].y), make_float2(q.x, q.y));
                      ff_mac(h[i][r], l[i][r], make_float2(a[i][1].z, a[i][1].w), make_float2(q.z, q.w));
                    }
                }
            }
          float2 t[RR * RC];
#pragma unroll
          for (int i = 0; i < RR; ++i)
#pragma unroll
            for (int r = 0; r < RC; ++r)
              t[i * RC + r] = ff_norm(h[i][r], l[i][r]);
          const float2  u = warp_sums<RR * RC>(t, [](float2 p, float2 q) { return ff_add(p, q); });
          constexpr int W = 32 / (RR * RC);
          const int     i = row + lane / (W * RC), r = (lane / W) % RC;
          if (lane % W == 0 && i < nr && r < rc)
            {
              double &o = y[(ra + r) * int64_t(N) + nrows[r0 + i]];
              o         = acc ? __dadd_rn(o, ff_join(u)) : ff_join(u);
            }
        }
    }

    // The P2M and L2P kernels give a leaf `split` warps, 1, 2 or LEAF_SPLIT: a leaf's rows
    // are a serial chain of loads and sums, and one warp for each of a few hundred leaves
    // leaves the SMs waiting for it.  L2P rows are dealt to the warps in groups; the P2M sums
    // are formed over `split` runs of rows and added in run order.
    constexpr int LEAF_SPLIT = 4;
    __device__ __forceinline__ void p2m_part(const int64_t r0, const int64_t r1, int q, int split, int64_t &rb,
                                             int64_t &re)
    {
      const int64_t per = ((r1 - r0 + split - 1) / split + 7) / 8 * 8; // whole load groups
      rb                = min(r1, r0 + q * per);
      re                = min(r1, rb + per);
    }
    template <int RC, typename T>
    __device__ __forceinline__ void p2m_store(const T (*part)[RC][128], int w0, int split, int k, int rc, T *M,
                                              int K)
    {
#pragma unroll
      for (int rr = 0; rr < RC; ++rr)
        if (rr < rc)
          {
            T t = part[w0][rr][k];
            for (int q = 1; q < split; ++q)
              t += part[w0 + q][rr][k];
            M[int64_t(rr) * K + k] = t;
          }
    }

    // P2M apply: M^[leaf][r][k] = sum_rows w(row, r) T[row][k] x_r[dof(row)],
    // w selecting the double layer (Ker1), the single layer (Ker2) or the
    // combined system strengths.  SPLIT: `split` > 1 warps per leaf, else one (without the
    // code for the sum of the parts, 64 registers instead of 78: at 98k nodes 21 us against
    // 25).  Lane l owns coefficients 4l..4l+3 (table rows padded to K4 values);
    // the rows' weights are gathered 32 at a time (lane j: row j) and broadcast by
    // shuffles; eight table rows in flight; a warp's rows are summed in order.
    // COMBINED: every column uses the combined strengths, read from the table
    // Tc = (Dirichlet dof ? -T2 : T1) made at set_bc (one table row per row
    // instead of two); T1 is then Tc and T2 is unused.
    // RC: columns per block (1 for one right-hand side, else 4; the groups of columns
    // over blockIdx.y: a few hundred leaves alone would leave most of the chip idle).
    template <bool COMBINED, int RC, bool SPLIT>
    __global__ void __launch_bounds__(256)
      p2m_apply_kernel(int n_leaves, int split, int R, int K, int N, const int64_t *__restrict__ prow_ptr,
                       const int32_t *__restrict__ pleaf_box, const int32_t *__restrict__ prow_dof,
                       const float *__restrict__ T1, const float *__restrict__ T2,
                       const uint8_t *__restrict__ dir, const uint8_t *__restrict__ modes,
                       const float *__restrict__ x, float *__restrict__ M)
    {
      using T = float;
      pdl_entry();
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      const int wi   = blockIdx.x * (blockDim.x >> 5) + warp;
      const int leaf = SPLIT ? wi / split : wi;
      const int K4   = (K + 3) / 4 * 4;
      if (!SPLIT && leaf >= n_leaves)
        return;
      int64_t rb = 0, re = 0;
      if (!SPLIT || leaf < n_leaves)
        {
          rb = prow_ptr[leaf];
          re = prow_ptr[leaf + 1];
          if constexpr (SPLIT)
            p2m_part(rb, re, warp & (split - 1), split, rb, re);
        }
      const int64_t box = !SPLIT || leaf < n_leaves ? pleaf_box[leaf] : 0;
      const bool    act = 4 * lane < K4;
      const int rq = blockIdx.y * RC;
        {
          const int rc = min(RC, R - rq);
          T         acc[RC][4];
#pragma unroll
          for (int a = 0; a < RC; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b)
              acc[a][b] = T(0);
          for (int64_t b0 = rb; b0 < re; b0 += 32)
            {
              const int nb = re - b0 < 32 ? int(re - b0) : 32;
              T         w1[RC], w2[RC];
#pragma unroll
              for (int rr = 0; rr < RC; ++rr)
                w1[rr] = w2[rr] = T(0);
              if (lane < nb)
                {
                  const int  dof = prow_dof[b0 + lane];
                  const bool d   = dir[dof] != 0;
#pragma unroll
                  for (int rr = 0; rr < RC; ++rr)
                    if (rr < rc)
                      {
                        const T xv = x[int64_t(rq + rr) * N + dof];
                        if constexpr (COMBINED)
                          w1[rr] = xv;
                        else
                          {
                            const uint8_t mode = modes[rq + rr];
                            const bool    dd   = mode == MODE_SWAPPED ? !d : d;
                            w1[rr] = mode == MODE_KER2 ? T(0) : (mode == MODE_KER1 ? xv : (dd ? T(0) : xv));
                            w2[rr] = mode == MODE_KER1 ? T(0) : (mode == MODE_KER2 ? xv : (dd ? -xv : T(0)));
                          }
                      }
                }
              for (int j0 = 0; j0 < nb; j0 += 8)
                {
                  T t1[8][4], t2[8][4];
#pragma unroll
                  for (int u = 0; u < 8; ++u)
                    if (act && j0 + u < nb)
                      {
                        load4(T1 + (b0 + j0 + u) * K4 + 4 * lane, t1[u]);
                        if constexpr (!COMBINED)
                          load4(T2 + (b0 + j0 + u) * K4 + 4 * lane, t2[u]);
                      }
#pragma unroll
                  for (int u = 0; u < 8; ++u)
                    if (j0 + u < nb)
#pragma unroll
                      for (int rr = 0; rr < RC; ++rr)
                        if (rr < rc)
                          {
                            const T a1 = __shfl_sync(0xffffffffu, w1[rr], j0 + u);
                            if constexpr (COMBINED)
                              {
#pragma unroll
                                for (int c = 0; c < 4; ++c)
                                  acc[rr][c] += a1 * t1[u][c];
                              }
                            else
                              {
                                const T a2 = __shfl_sync(0xffffffffu, w2[rr], j0 + u);
#pragma unroll
                                for (int c = 0; c < 4; ++c)
                                  acc[rr][c] += a1 * t1[u][c] + a2 * t2[u][c];
                              }
                          }
                }
            }
          if constexpr (!SPLIT)
            {
              if (act)
#pragma unroll
                for (int rr = 0; rr < RC; ++rr)
                  if (rr < rc)
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                      if (4 * lane + c < K)
                        M[(box * R + rq + rr) * K + 4 * lane + c] = acc[rr][c];
            }
          else
            {
              __shared__ __align__(16) float part[2 * LEAF_SPLIT][RC][128];
              if (act)
#pragma unroll
                for (int rr = 0; rr < RC; ++rr)
                  *reinterpret_cast<float4 *>(&part[warp][rr][4 * lane]) =
                    make_float4(acc[rr][0], acc[rr][1], acc[rr][2], acc[rr][3]);
              __syncthreads();
              if (leaf < n_leaves)
                for (int k = threadIdx.x & (32 * split - 1); k < K; k += 32 * split)
                  p2m_store<RC>(part, warp & -split, split, k, rc, M + (box * R + rq) * K, K);
            }
        }
    }

    // P2M apply in FP64: the same sums, but lane l owns coefficients l,
    // l + 32, ... (NPL of them): the FP64 pipe takes a warp's FMA in the same time however
    // many lanes have work, and ceil(K / 32) FMA a row replace 4.  A column of one layer
    // only (KER1 / KER2) skips the other layer's table and products.  Bounded by those FMA and,
    // on small meshes, by the rows' serial chain.  GB300, two columns at 386 nodes: 36 us with
    // four coefficients a lane and eight warps a block -> 11.8, with four warps a leaf 7.5.
    template <bool COMBINED, int RC, int NPL>
    __global__ void __launch_bounds__(256)
      p2m_apply64_kernel(int n_leaves, int split, int R, int K, int N, const int64_t *__restrict__ prow_ptr,
                         const int32_t *__restrict__ pleaf_box, const int32_t *__restrict__ prow_dof,
                         const double *__restrict__ T1, const double *__restrict__ T2,
                         const uint8_t *__restrict__ dir, const uint8_t *__restrict__ modes,
                         const double *__restrict__ x, double *__restrict__ M)
    {
      pdl_entry();
      __shared__ double part[2 * LEAF_SPLIT][RC][128];
      const int         warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      const int         leaf = (blockIdx.x * (blockDim.x >> 5) + warp) / split;
      const int         K4   = (K + 3) / 4 * 4;
      int64_t           rb = 0, re = 0;
      if (leaf < n_leaves)
        p2m_part(prow_ptr[leaf], prow_ptr[leaf + 1], warp & (split - 1), split, rb, re);
      const int     rq = blockIdx.y * RC, rc = min(RC, R - rq);
      int           mode[RC];
      bool          one = COMBINED, two = false; // layers that some column takes
#pragma unroll
      for (int rr = 0; rr < RC; ++rr)
        {
          mode[rr] = COMBINED ? int(MODE_KER1) : (rr < rc ? int(modes[rq + rr]) : int(MODE_KER1));
          if (!COMBINED && rr < rc)
            {
              one = one || mode[rr] != MODE_KER2;
              two = two || mode[rr] != MODE_KER1;
            }
        }
      double acc[RC][NPL];
#pragma unroll
      for (int rr = 0; rr < RC; ++rr)
#pragma unroll
        for (int c = 0; c < NPL; ++c)
          acc[rr][c] = 0.0;
      for (int64_t b0 = rb; b0 < re; b0 += 32)
        {
          const int nb = re - b0 < 32 ? int(re - b0) : 32;
          double    w1[RC], w2[RC];
#pragma unroll
          for (int rr = 0; rr < RC; ++rr)
            w1[rr] = w2[rr] = 0.0;
          if (lane < nb)
            {
              const int  dof = prow_dof[b0 + lane];
              const bool d   = !COMBINED && dir[dof] != 0;
#pragma unroll
              for (int rr = 0; rr < RC; ++rr)
                if (rr < rc)
                  {
                    const double xv = x[int64_t(rq + rr) * N + dof];
                    if constexpr (COMBINED)
                      w1[rr] = xv;
                    else
                      {
                        const bool dd = mode[rr] == MODE_SWAPPED ? !d : d;
                        w1[rr] = mode[rr] == MODE_KER2 ? 0.0 : (mode[rr] == MODE_KER1 ? xv : (dd ? 0.0 : xv));
                        w2[rr] = mode[rr] == MODE_KER1 ? 0.0 : (mode[rr] == MODE_KER2 ? xv : (dd ? -xv : 0.0));
                      }
                  }
            }
          for (int j0 = 0; j0 < nb; j0 += 8)
            {
              double t1[8][NPL], t2[COMBINED ? 1 : 8][NPL];
#pragma unroll
              for (int u = 0; u < 8; ++u)
#pragma unroll
                for (int c = 0; c < NPL; ++c)
                  {
                    const bool   in = j0 + u < nb && lane + 32 * c < K4;
                    const int64_t o = (b0 + j0 + u) * K4 + lane + 32 * c;
                    t1[u][c]        = in && one ? T1[o] : 0.0;
                    if constexpr (!COMBINED)
                      t2[u][c] = in && two ? T2[o] : 0.0;
                  }
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (j0 + u < nb)
#pragma unroll
                  for (int rr = 0; rr < RC; ++rr)
                    if (rr < rc)
                      {
                        const double a1 = __shfl_sync(0xffffffffu, w1[rr], j0 + u);
                        if (COMBINED || mode[rr] != MODE_KER2)
#pragma unroll
                          for (int c = 0; c < NPL; ++c)
                            acc[rr][c] = fma_rn(a1, t1[u][c], acc[rr][c]);
                        if constexpr (!COMBINED)
                          {
                            const double a2 = __shfl_sync(0xffffffffu, w2[rr], j0 + u);
                            if (mode[rr] != MODE_KER1)
#pragma unroll
                              for (int c = 0; c < NPL; ++c)
                                acc[rr][c] = fma_rn(a2, t2[u][c], acc[rr][c]);
                          }
                      }
            }
        }
      if (split == 1)
        {
          if (leaf < n_leaves)
#pragma unroll
            for (int rr = 0; rr < RC; ++rr)
              if (rr < rc)
#pragma unroll
                for (int c = 0; c < NPL; ++c)
                  if (lane + 32 * c < K)
                    M[(int64_t(pleaf_box[leaf]) * R + rq + rr) * K + lane + 32 * c] = acc[rr][c];
          return;
        }
#pragma unroll
      for (int rr = 0; rr < RC; ++rr)
#pragma unroll
        for (int c = 0; c < NPL; ++c)
          part[warp][rr][lane + 32 * c] = acc[rr][c];
      __syncthreads();
      if (leaf < n_leaves)
        for (int k = threadIdx.x & (32 * split - 1); k < K; k += 32 * split)
          p2m_store<RC>(part, warp & -split, split, k, rc, M + (int64_t(pleaf_box[leaf]) * R + rq) * K, K);
    }

    // L2P in FP64: lane l multiplies coefficients l, l + 32, ...; RR rows x RC columns are
    // summed together by the butterfly's reduce-scatter (RR RC + 4 - log2(RR RC) additions
    // instead of 5 RR RC, on a pipe where each takes as long as an FMA).  GB300, two columns
    // at 386 nodes: 23 us as in FP32 -> 8.4, with four warps a leaf 4.1.
    template <int RC, int RR, int NPL>
    __global__ void __launch_bounds__(256)
      l2p64_kernel(int n_leaves, int split, int R, int K, int N, const int64_t *__restrict__ row_ptr,
                   const int32_t *__restrict__ lleaf_box, const int32_t *__restrict__ nrows,
                   const double *__restrict__ W, const double *__restrict__ Lx, double *__restrict__ y)
    {
      pdl_entry();
      const int wi   = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
      const int leaf = wi / split, part = wi & (split - 1);
      if (leaf >= n_leaves)
        return;
      const int     K4  = (K + 3) / 4 * 4;
      const int64_t box = lleaf_box[leaf];
      const int64_t i0 = row_ptr[leaf], i1 = row_ptr[leaf + 1];
      const int     ra = blockIdx.y * RC, rc = min(RC, R - ra);
      double        l[RC][NPL];
#pragma unroll
      for (int r = 0; r < RC; ++r)
#pragma unroll
        for (int c = 0; c < NPL; ++c)
          l[r][c] = r < rc && lane + 32 * c < K ? Lx[(box * R + ra + r) * K + lane + 32 * c] : 0.0;
      for (int64_t i = i0 + part * RR; i < i1; i += split * RR)
        {
          double w[RR][NPL], v[RR * RC];
#pragma unroll
          for (int u = 0; u < RR; ++u)
#pragma unroll
            for (int c = 0; c < NPL; ++c)
              w[u][c] = i + u < i1 && lane + 32 * c < K ? W[(i + u) * K4 + lane + 32 * c] : 0.0;
#pragma unroll
          for (int u = 0; u < RR; ++u)
#pragma unroll
            for (int r = 0; r < RC; ++r)
              {
                double s = mul_rn(w[u][0], l[r][0]);
#pragma unroll
                for (int c = 1; c < NPL; ++c)
                  s = fma_rn(w[u][c], l[r][c], s);
                v[u * RC + r] = s;
              }
          const double  t  = warp_sums<RR * RC>(v, [](double p, double q) { return p + q; });
          constexpr int Wn = 32 / (RR * RC); // lanes per value
          const int     u = lane / (Wn * RC), r = (lane / Wn) % RC;
          if (lane % Wn == 0 && i + u < i1 && r < rc)
            y[int64_t(ra + r) * N + nrows[i + u]] += t;
        }
    }

    // Batched translation GEMM.  Scaled operators do not depend on the level:
    // M2L depends only on the integer source-target offset, M2M / L2L only on
    // the child octant.  Pairs sharing an operator are cut into chunks of <= 128;
    // block (c, t, z) computes  Y[q] = T_op(c) E[src(q)]  for TY CJ columns of chunk c
    // (column = (pair, rhs)) from the t-th group on and rows z TX RI ... + TX RI - 1,
    // the operator's rows and the columns staged in shared memory.  Thread (tx, ty) of
    // TX x TY computes rows tx + TX i (i < RI) and columns ty + TY j (j < CJ), k ascending.
    // Arithmetic: the type's FMA, or float-float on the FP32 pipes (OP = float2, the
    // operator pre-split into (hi, lo) pairs; the expansions in that form too or, IO =
    // double, split on load and joined on store).
    //   What bounds it: the arithmetic, above all FP64's two FMA per clock and SM.  So
    // no thread computes rows beyond the block's (TX = ceil(K / RI)), and the columns a
    // chunk does not have are left out (most chunks of small meshes and of the small
    // levels hold a few pairs): the columns per thread are rounded up to 1, 2, 4 or 8,
    // and threads without a column leave.  Measured (GB300, one column,
    // against 64-column tiles computed whole): FP64 M2L at 13,826 nodes 749 -> 570 us and
    // M2M / L2L levels 38 -> 13; float-float levels at 198k nodes 77 -> 30, at 98k 28 -> 18;
    // FP64 M2L at 386 nodes 155 -> 78.
    __device__ __forceinline__ float2 ff_load(const double *p) { return ff_split(*p); }
    __device__ __forceinline__ float2 ff_load(const float2 *p) { return *p; }
    __device__ __forceinline__ void   ff_store(double *p, float h, float l) { *p = __dadd_rn(double(h), double(l)); }
    __device__ __forceinline__ void   ff_store(float2 *p, float h, float l) { *p = ff_norm(h, l); }

    // one running sum: plain (OP = IO) or float-float
    template <typename OP>
    struct GemmSum
    {
      OP s = OP(0);
      __device__ __forceinline__ void mac(OP a, OP b) { s = fma_rn(a, b, s); }
      __device__ __forceinline__ void store(OP *p) const { *p = s; }
      __device__ static OP            load(const OP *p) { return *p; }
      __device__ static OP            zero() { return OP(0); }
    };
    template <>
    struct GemmSum<float2>
    {
      float h = 0.0f, l = 0.0f;
      __device__ __forceinline__ void mac(float2 a, float2 b) { ff_mac(h, l, a, b); }
      template <typename IO>
      __device__ __forceinline__ void store(IO *p) const
      {
        ff_store(p, h, l);
      }
      template <typename IO>
      __device__ static float2 load(const IO *p)
      {
        return ff_load(p);
      }
      __device__ static float2 zero() { return make_float2(0.0f, 0.0f); }
    };

    template <typename IO, typename OP, int RI, int CJ, int TY>
    __global__ void __launch_bounds__(256, 2)
      trans_gemm_kernel(int R, int K, int TX, int chunk0, const int32_t *__restrict__ chunk_start,
                        const int32_t *__restrict__ chunk_cnt, const int32_t *__restrict__ chunk_off,
                        const int32_t *__restrict__ q_src, const OP *__restrict__ ops,
                        const IO *__restrict__ M, IO *__restrict__ Y,
                        const int32_t *__restrict__ yslot, int ldy)
    {
      using Sum = GemmSum<OP>;
      constexpr int COLS = TY * CJ, LDB = COLS + 1;
      extern __shared__ __align__(16) unsigned char smem_raw[];
      const int W     = TX * RI;                        // rows of this block
      OP       *sT    = reinterpret_cast<OP *>(smem_raw); // [K][W] in-major
      OP       *sB    = sT + K * W;                       // [K][LDB]
      const int ch    = chunk0 + blockIdx.x;
      const int start = chunk_start[ch], ncols = chunk_cnt[ch] * R;
      const int c0    = blockIdx.y * COLS;
      if (c0 >= ncols)
        return;
      const int nc = min(COLS, ncols - c0), row0 = blockIdx.z * W;
      const OP *op = ops + int64_t(chunk_off[ch]) * K * K;
      for (int i0 = threadIdx.x; i0 < K * W; i0 += 8 * blockDim.x)
        {
          OP v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u)
            {
              const int i = i0 + u * blockDim.x, ki = i / W, ko = row0 + i - ki * W;
              v[u]        = i < K * W && ko < K ? op[ki * K + ko] : Sum::zero();
            }
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (i0 + u * blockDim.x < K * W)
              sT[i0 + u * blockDim.x] = v[u];
        }
      for (int i0 = threadIdx.x; i0 < nc * K; i0 += 4 * blockDim.x)
        {
          OP v[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            {
              const int i = i0 + u * blockDim.x, c = i / K, cg = c0 + c;
              if (i < nc * K)
                v[u] = Sum::load(M + (int64_t(q_src[start + cg / R]) * R + cg % R) * K + (i - c * K));
            }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            {
              const int i = i0 + u * blockDim.x, c = i / K;
              if (i < nc * K)
                sB[(i - c * K) * LDB + c] = v[u];
            }
        }
      __syncthreads();
      const int     tx = threadIdx.x % TX, ty = threadIdx.x / TX;
      if (ty >= TY || ty >= nc)
        return;
      auto run = [&](auto nj) {
        constexpr int NJ = decltype(nj)::value;
        Sum           acc[RI][NJ];
        for (int ki = 0; ki < K; ++ki)
          {
            OP a[RI], b[NJ];
#pragma unroll
            for (int i = 0; i < RI; ++i)
              a[i] = sT[ki * W + tx + TX * i];
#pragma unroll
            for (int j = 0; j < NJ; ++j)
              b[j] = sB[ki * LDB + ty + TY * j];
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
              for (int j = 0; j < NJ; ++j)
                acc[i][j].mac(a[i], b[j]);
          }
#pragma unroll
        for (int j = 0; j < NJ; ++j)
          {
            const int c = ty + TY * j;
            if (c >= nc)
              continue;
            const int     cg = c0 + c;
            const int64_t q  = start + cg / R;
            const int64_t yr = (yslot ? int64_t(yslot[q]) : q) * R + cg % R; // row of (pair, rhs)
#pragma unroll
            for (int i = 0; i < RI; ++i)
              {
                const int ko = row0 + tx + TX * i;
                if (ko < K)
                  acc[i][j].store(Y + yr * ldy + ko);
              }
          }
      };
      const int nj = (nc + TY - 1) / TY; // columns per thread, the block's most
      if (CJ == 1 || nj <= 1)
        run(std::integral_constant<int, 1>());
      else if (CJ == 2 || nj <= 2)
        run(std::integral_constant<int, CJ < 2 ? CJ : 2>());
      else if (CJ == 4 || nj <= 4)
        run(std::integral_constant<int, CJ < 4 ? CJ : 4>());
      else
        run(std::integral_constant<int, CJ>());
    }

    // out[box] = sum of the box's (hi, lo) translation products, in list order,
    // in float-float arithmetic; 8 loads in flight.
    __global__ void gather_ff_kernel(int R, int K, const int32_t *__restrict__ boxes,
                                     const int64_t *__restrict__ q_ptr,
                                     const int32_t *__restrict__ q, const float2 *__restrict__ Y,
                                     float2 *__restrict__ out)
    {
      const int64_t b  = boxes[blockIdx.x];
      const int64_t e0 = q_ptr[blockIdx.x], e1 = q_ptr[blockIdx.x + 1];
      const int64_t RK = int64_t(R) * K;
      for (int i = threadIdx.x; i < R * K; i += blockDim.x)
        {
          float2 acc = make_float2(0.0f, 0.0f);
          for (int64_t e = e0; e < e1; e += 8)
            {
              float2 v[8];
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (e + u < e1)
                  v[u] = Y[int64_t(q[e + u]) * RK + i];
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (e + u < e1)
                  acc = ff_add(acc, v[u]);
            }
          out[b * RK + i] = acc;
        }
    }

    __global__ void d2ff_kernel(int64_t n, const double *__restrict__ a, float2 *__restrict__ b)
    {
      const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (i < n)
        b[i] = ff_split(a[i]);
    }
    __global__ void ff2d_kernel(int64_t n, const float2 *__restrict__ a, double *__restrict__ b)
    {
      const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (i < n)
        b[i] = ff_join(a[i]);
    }

    // out[box] = sum of the box's translation products Y[q], in list order.  The
    // loads of 8 consecutive products are issued before they are added (same
    // order of additions), so a thread has 8 L2 reads in flight.
    template <typename T>
    __global__ void gather_kernel(int R, int K, const int32_t *__restrict__ boxes,
                                  const int64_t *__restrict__ q_ptr, const int32_t *__restrict__ q,
                                  const T *__restrict__ Y, T *__restrict__ out)
    {
      const int64_t b  = boxes[blockIdx.x];
      const int64_t e0 = q_ptr[blockIdx.x], e1 = q_ptr[blockIdx.x + 1];
      const int64_t RK = int64_t(R) * K;
      for (int i = threadIdx.x; i < R * K; i += blockDim.x)
        {
          T acc = T(0);
          for (int64_t e = e0; e < e1; e += 8)
            {
              T v[8];
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (e + u < e1)
                  v[u] = Y[int64_t(q[e + u]) * RK + i];
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (e + u < e1)
                  acc += v[u];
            }
          out[b * RK + i] = acc;
        }
    }

    // Multipole values of nc <= NC columns (K apart) at the offset r in box units:
    // sum_k coef[k] basis_k(r) with the table-driven recurrences, m-major.  The basis
    // is formed once for the columns, two FMA per term and column; the order of the
    // additions and the roundings of a column do not depend on NC.
    template <int NC, typename T>
    __device__ __forceinline__ void eval_multipole_cols(const T *__restrict__ coef, int K, int nc, int p,
                                                        T rx, T ry, T rz, T (&acc)[NC])
    {
      using LT    = LegT<T>;
      const T r2  = rx * rx + ry * ry + rz * rz;
      const T rho = sqrt(r2);
      const T inv = T(1) / rho;
      const T x   = rz * inv;
      const T s   = sqrt(fmax(T(0), T(1) - x * x));
      const T rxy = sqrt(rx * rx + ry * ry);
      T       cb = T(1), sb = T(0);
      if (rxy > T(0))
        {
          cb = rx / rxy;
          sb = ry / rxy;
        }
      T pmm = T(1), rpm = inv, cm = T(1), sm = T(0);
#pragma unroll
      for (int r = 0; r < NC; ++r)
        acc[r] = T(0);
      // term (n, m): the basis value q (Legendre times power of r) times (cos, sin) m
      auto term = [&](int n, int m, T q) {
        const int k0 = n * n + (m == 0 ? 0 : 2 * m - 1);
        const T   a  = m == 0 ? q : mul_rn(T(2) * cm, q);
        const T   b  = m == 0 ? T(0) : mul_rn(-T(2) * sm, q);
#pragma unroll
        for (int r = 0; r < NC; ++r)
          if (r < nc)
            {
              acc[r] = fma_rn(coef[r * K + k0], a, acc[r]);
              if (m > 0)
                acc[r] = fma_rn(coef[r * K + k0 + 1], b, acc[r]);
            }
      };
      for (int m = 0; m <= p; ++m)
        {
          if (m > 0)
            {
              pmm        = mul_rn(pmm, mul_rn(-LT::cmm(m), s));
              rpm        = mul_rn(rpm, inv);
              const T c2 = fma_rn(cm, cb, -mul_rn(sm, sb));
              sm         = fma_rn(sm, cb, mul_rn(cm, sb));
              cm         = c2;
            }
          T p0 = pmm, rp = rpm;
          term(m, m, mul_rn(p0, rp));
          if (m + 1 <= p)
            {
              T p1 = mul_rn(mul_rn(x, LT::cm1(m)), pmm);
              rp   = mul_rn(rp, inv);
              term(m + 1, m, mul_rn(p1, rp));
              for (int n = m + 2; n <= p; ++n)
                {
                  const T p2 = fma_rn(mul_rn(LT::ra(n, m), x), p1, -mul_rn(LT::rb(n, m), p0));
                  p0         = p1;
                  p1         = p2;
                  rp         = mul_rn(rp, inv);
                  term(n, m, mul_rn(p1, rp));
                }
            }
        }
    }

    // M2P phase 1: one thread per (pair, collocation node of the pair's target
    // box) and NC columns: scratch[r][item] = multipole of the source box evaluated
    // at the node.  tnodes lists each target box's collocation nodes (tnode_ptr).
    template <typename T, int NC>
    __global__ void m2p_eval_kernel(int64_t n_items, int R, int K, int p,
                                    const int64_t *__restrict__ item_ptr,
                                    const int32_t *__restrict__ item_pair,
                                    const int32_t *__restrict__ pair_tgt,
                                    const int32_t *__restrict__ src,
                                    const int64_t *__restrict__ tnode_ptr,
                                    const int32_t *__restrict__ tnodes,
                                    const double *__restrict__ xyz,
                                    const double *__restrict__ center,
                                    const double *__restrict__ delta, const T *__restrict__ M,
                                    T *__restrict__ scratch)
    {
      pdl_entry();
      const int64_t it = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (it >= n_items)
        return;
      const int64_t e    = item_pair[it];
      const int64_t s    = src[e];
      const int     node = tnodes[tnode_ptr[pair_tgt[e]] + (it - item_ptr[e])];
      const double  h    = delta[s];
      T             rx, ry, rz, ih;
      if constexpr (std::is_same<T, float>::value)
        {
          // FP32 operator: the offset from the centre in FP64 (no cancellation),
          // scaled in FP32 (GB300's FP64 divide would dominate this kernel)
          ih = __frcp_rn(float(h));
          rx = float(xyz[3 * int64_t(node)] - center[3 * s]) * ih;
          ry = float(xyz[3 * int64_t(node) + 1] - center[3 * s + 1]) * ih;
          rz = float(xyz[3 * int64_t(node) + 2] - center[3 * s + 2]) * ih;
        }
      else
        {
          rx = (xyz[3 * int64_t(node)] - center[3 * s]) / h;
          ry = (xyz[3 * int64_t(node) + 1] - center[3 * s + 1]) / h;
          rz = (xyz[3 * int64_t(node) + 2] - center[3 * s + 2]) / h;
          ih = 1.0 / h;
        }
      const int r0 = blockIdx.y * NC, nc = min(NC, R - r0);
      T         v[NC];
      eval_multipole_cols<NC>(M + (s * R + r0) * K, K, nc, p, rx, ry, rz, v);
#pragma unroll
      for (int r = 0; r < NC; ++r)
        if (r < nc)
          scratch[int64_t(r0 + r) * n_items + it] = v[r] * ih;
    }

    // eval_multipole_cols in float-float arithmetic for the FP64-accurate operator: r
    // is the offset from the box centre in box units (pairs), coef the expansions as
    // pairs (K apart), the sums carried with TwoProduct / TwoSum (ff_mac): 22 FP32
    // instructions per term and column and about 40 shared by the columns, against
    // the FP64 pipe's 1/58 rate.
    template <int NC>
    __device__ __forceinline__ void eval_multipole_ff(const float2 *__restrict__ coef, int K, int nc, int p,
                                                      float2 rx, float2 ry, float2 rz, float2 (&out)[NC])
    {
      const float2 rxy2 = ff_add(ff_mul(rx, rx), ff_mul(ry, ry));
      const float2 rho  = ff_sqrt(ff_add(rxy2, ff_mul(rz, rz)));
      const float2 inv  = ff_recip(rho);
      const float2 x    = ff_mul(rz, inv);
      const float2 s    = ff_sqrt(ff_sub(make_float2(1.f, 0.f), ff_mul(x, x)));
      const float2 rxy  = ff_sqrt(rxy2);
      float2       cb = make_float2(1.f, 0.f), sb = make_float2(0.f, 0.f);
      if (rxy.x > 0.f)
        {
          const float2 ir = ff_recip(rxy);
          cb              = ff_mul(rx, ir);
          sb              = ff_mul(ry, ir);
        }
      float  h[NC], l[NC];
      float2 pmm = make_float2(1.f, 0.f), rpm = inv;
      float2 cm = make_float2(1.f, 0.f), sm = make_float2(0.f, 0.f);
#pragma unroll
      for (int r = 0; r < NC; ++r)
        h[r] = l[r] = 0.f;
      // term (n, m): the basis value q (Legendre times power of r) times (cos, sin) m
      auto term = [&](int n, int m, float2 q) {
        const int k0 = n * n + (m == 0 ? 0 : 2 * m - 1);
        // 2 cm and -2 sm: exact scalings
        const float2 a = m == 0 ? q : ff_mul(make_float2(2.f * cm.x, 2.f * cm.y), q);
        const float2 b = m == 0 ? q : ff_mul(make_float2(-2.f * sm.x, -2.f * sm.y), q);
#pragma unroll
        for (int r = 0; r < NC; ++r)
          if (r < nc)
            {
              ff_mac(h[r], l[r], coef[r * K + k0], a);
              if (m > 0)
                ff_mac(h[r], l[r], coef[r * K + k0 + 1], b);
            }
      };
      for (int m = 0; m <= p; ++m)
        {
          if (m > 0)
            {
              pmm             = ff_mul(pmm, ff_mul(ff_neg(c_leg.ffcmm[m]), s));
              rpm             = ff_mul(rpm, inv);
              const float2 c2 = ff_sub(ff_mul(cm, cb), ff_mul(sm, sb));
              sm              = ff_add(ff_mul(sm, cb), ff_mul(cm, sb));
              cm              = c2;
            }
          float2 p0 = pmm, rp = rpm;
          term(m, m, ff_mul(p0, rp));
          if (m + 1 <= p)
            {
              float2 p1 = ff_mul(ff_mul(x, c_leg.ffcm1[m]), pmm);
              rp        = ff_mul(rp, inv);
              term(m + 1, m, ff_mul(p1, rp));
              for (int n = m + 2; n <= p; ++n)
                {
                  const float2 p2 = ff_sub(ff_mul(ff_mul(c_leg.ffra[n][m], x), p1),
                                           ff_mul(c_leg.ffrb[n][m], p0));
                  p0 = p1;
                  p1 = p2;
                  rp = ff_mul(rp, inv);
                  term(n, m, ff_mul(p1, rp));
                }
            }
        }
#pragma unroll
      for (int r = 0; r < NC; ++r)
        out[r] = ff_norm(h[r], l[r]);
    }

    // M2P phase 1 of the FP64-accurate operator: as m2p_eval_kernel, from the
    // (hi, lo) multipoles; the offset from the centre is formed in FP64 and
    // split, the scaling by 1 / h in float-float; the value stored in FP64.
    template <int NC>
    __global__ void m2p_eval_ff_kernel(int64_t n_items, int R, int K, int p,
                                       const int64_t *__restrict__ item_ptr,
                                       const int32_t *__restrict__ item_pair,
                                       const int32_t *__restrict__ pair_tgt,
                                       const int32_t *__restrict__ src,
                                       const int64_t *__restrict__ tnode_ptr,
                                       const int32_t *__restrict__ tnodes,
                                       const double *__restrict__ xyz,
                                       const double *__restrict__ center,
                                       const double *__restrict__ delta,
                                       const float2 *__restrict__ M, double *__restrict__ scratch)
    {
      const int64_t it = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
      if (it >= n_items)
        return;
      const int64_t e    = item_pair[it];
      const int64_t s    = src[e];
      const int     node = tnodes[tnode_ptr[pair_tgt[e]] + (it - item_ptr[e])];
      const float2  ih   = ff_recip(ff_split(delta[s]));
      const float2  rx   = ff_mul(ff_split(__dsub_rn(xyz[3 * int64_t(node)], center[3 * s])), ih);
      const float2  ry   = ff_mul(ff_split(__dsub_rn(xyz[3 * int64_t(node) + 1], center[3 * s + 1])), ih);
      const float2  rz   = ff_mul(ff_split(__dsub_rn(xyz[3 * int64_t(node) + 2], center[3 * s + 2])), ih);
      const int     r0 = blockIdx.y * NC, nc = min(NC, R - r0);
      float2        v[NC];
      eval_multipole_ff<NC>(M + (s * R + r0) * K, K, nc, p, rx, ry, rz, v);
#pragma unroll
      for (int r = 0; r < NC; ++r)
        if (r < nc)
          scratch[int64_t(r0 + r) * n_items + it] = ff_join(ff_mul(v[r], ih));
    }

    // M2P phase 2: one warp per target box and column (blockIdx.y), one lane per node
    // of the box: the node's values over the box's sources, added in list order to y.  The
    // items of a target box are contiguous, source-major (item_ptr[e] =
    // item_ptr[e0] + (e - e0) nn), so a node's values sit nn apart; 16 loads
    // in flight, the last group's too.
    template <typename T>
    __global__ void __launch_bounds__(256)
      m2p_sum_kernel(int n_tgt, int N, int64_t n_items, const int64_t *__restrict__ tnode_ptr,
                     const int64_t *__restrict__ src_ptr,
                     const int64_t *__restrict__ item_ptr, const int32_t *__restrict__ tnodes,
                     const T *__restrict__ scratch, T *__restrict__ y)
    {
      pdl_entry();
      const int ti = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
      if (ti >= n_tgt)
        return;
      const int64_t  nn = tnode_ptr[ti + 1] - tnode_ptr[ti];
      const int64_t  e0 = src_ptr[ti], ns = src_ptr[ti + 1] - e0;
      const int64_t  base = e0 < src_ptr[n_tgt] ? item_ptr[e0] : 0;
      const int32_t *nodes = tnodes + tnode_ptr[ti];
      const int64_t  r     = blockIdx.y;
      for (int64_t i = lane; i < nn; i += 32)
        {
          const int node = nodes[i];
          const T  *sc   = scratch + r * n_items + base + i;
          T         acc  = T(0), v[16];
          int64_t   j    = 0;
          for (; j + 16 <= ns; j += 16)
            {
#pragma unroll
              for (int u = 0; u < 16; ++u)
                v[u] = sc[(j + u) * nn];
#pragma unroll
              for (int u = 0; u < 16; ++u)
                acc += v[u];
            }
#pragma unroll
          for (int u = 0; u < 15; ++u)
            if (j + u < ns)
              v[u] = sc[(j + u) * nn];
#pragma unroll
          for (int u = 0; u < 15; ++u)
            if (j + u < ns)
              acc += v[u];
          y[r * N + node] += acc;
        }
    }

    // L2P: y[r][node] += W[row] . L^[leaf][r] for every row (node of a
    // childless box).  `split` warps per leaf and RC columns (blockIdx.y): lane l
    // multiplies coefficients 4l..4l+3 (W rows padded to K4 values) of RR rows and
    // the columns; the lanes' products are added by warp_sum's butterfly.  A (row,
    // column) value has the same roundings for every RC and RR.
    // One column: 8 rows (16-byte loads) in flight.  Several: a row of W is read once
    // for RC columns.
    template <int RC, int RR>
    __global__ void __launch_bounds__(256)
      l2p_kernel(int n_leaves, int split, int R, int K, int N, const int64_t *__restrict__ row_ptr,
                 const int32_t *__restrict__ lleaf_box, const int32_t *__restrict__ nrows,
                 const float *__restrict__ W, const float *__restrict__ Lx, float *__restrict__ y)
    {
      using T = float;
      pdl_entry();
      const int wi   = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
      const int leaf = wi / split, part = wi & (split - 1);
      if (leaf >= n_leaves)
        return;
      const int     K4  = (K + 3) / 4 * 4;
      const int64_t box = lleaf_box[leaf];
      const int64_t i0 = row_ptr[leaf], i1 = row_ptr[leaf + 1];
      const int     ra = blockIdx.y * RC, rc = min(RC, R - ra);
      const bool    act = 4 * lane < K4;
      T             l[RC][4];
#pragma unroll
      for (int r = 0; r < RC; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          l[r][c] = r < rc && 4 * lane + c < K ? Lx[(box * R + ra + r) * K + 4 * lane + c] : T(0);
      for (int64_t i = i0 + part * RR; i < i1; i += split * RR)
        {
          T w[RR][4];
#pragma unroll
          for (int u = 0; u < RR; ++u)
            if (act && i + u < i1)
              load4(W + (i + u) * K4 + 4 * lane, w[u]);
            else
              w[u][0] = w[u][1] = w[u][2] = w[u][3] = T(0);
          auto dot = [&](int u, int r) {
            return fma_rn(w[u][0], l[r][0], mul_rn(w[u][1], l[r][1])) +
                   fma_rn(w[u][2], l[r][2], mul_rn(w[u][3], l[r][3]));
          };
          if constexpr (RC == 1)
            {
              T mine = T(0);
#pragma unroll
              for (int u = 0; u < RR; ++u)
                {
                  const T t = warp_sum(dot(u, 0));
                  if (lane == u)
                    mine = t;
                }
              if (lane < RR && i + lane < i1)
                y[int64_t(ra) * N + nrows[i + lane]] += mine;
            }
          else
            {
              T v[RR * RC];
#pragma unroll
              for (int u = 0; u < RR; ++u)
#pragma unroll
                for (int r = 0; r < RC; ++r)
                  v[u * RC + r] = dot(u, r);
              const T       t  = warp_sums<RR * RC>(v, [](T p, T q) { return p + q; });
              constexpr int Wn = 32 / (RR * RC); // lanes per value
              const int     u = lane / (Wn * RC), r = (lane / Wn) % RC;
              if (lane % Wn == 0 && i + u < i1 && r < rc)
                y[int64_t(ra + r) * N + nrows[i + u]] += t;
            }
        }
    }

    // L2P of the FP64-accurate operator in float-float: as l2p_kernel, from
    // the (hi, lo) locals and (hi, lo) rows of W, products by TwoProduct, the
    // row sums carried with TwoSum and reduced by the same butterfly; y += the
    // sum in FP64.
    __global__ void __launch_bounds__(256)
      l2p_ff_kernel(int n_leaves, int split, int R, int K, int N, const int64_t *__restrict__ row_ptr,
                    const int32_t *__restrict__ lleaf_box, const int32_t *__restrict__ nrows,
                    const float2 *__restrict__ W, const float2 *__restrict__ Lx,
                    double *__restrict__ y)
    {
      const int wi   = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
      const int leaf = wi / split, part = wi & (split - 1);
      if (leaf >= n_leaves)
        return;
      const int     K4  = (K + 3) / 4 * 4;
      const int64_t box = lleaf_box[leaf];
      const int64_t r0 = row_ptr[leaf], r1 = row_ptr[leaf + 1];
      const bool    act = 4 * lane < K4;
      const int r = blockIdx.y;
        {
          float2 l[4];
#pragma unroll
          for (int c = 0; c < 4; ++c)
            l[c] = make_float2(0.f, 0.f);
          if (act)
            {
              const float2 *lp = Lx + (box * R + r) * K;
#pragma unroll
              for (int c = 0; c < 4; ++c)
                if (4 * lane + c < K)
                  l[c] = lp[4 * lane + c];
            }
          for (int64_t i0 = r0 + part * 8; i0 < r1; i0 += split * 8)
            {
              float2 w[8][4];
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (act && i0 + u < r1)
                  {
                    const float4 a = *reinterpret_cast<const float4 *>(W + (i0 + u) * K4 + 4 * lane);
                    const float4 b = *reinterpret_cast<const float4 *>(W + (i0 + u) * K4 + 4 * lane + 2);
                    w[u][0] = make_float2(a.x, a.y);
                    w[u][1] = make_float2(a.z, a.w);
                    w[u][2] = make_float2(b.x, b.y);
                    w[u][3] = make_float2(b.z, b.w);
                  }
                else
                  w[u][0] = w[u][1] = w[u][2] = w[u][3] = make_float2(0.f, 0.f);
              double mine = 0.0;
#pragma unroll
              for (int u = 0; u < 8; ++u)
                {
                  float h = 0.f, lo = 0.f;
#pragma unroll
                  for (int c = 0; c < 4; ++c)
                    ff_mac(h, lo, w[u][c], l[c]);
                  float2 t = ff_norm(h, lo);
                  for (int o = 16; o > 0; o >>= 1)
                    t = ff_add(t, make_float2(__shfl_xor_sync(0xffffffffu, t.x, o),
                                              __shfl_xor_sync(0xffffffffu, t.y, o)));
                  if (lane == u)
                    mine = ff_join(t);
                }
              if (lane < 8 && i0 + lane < r1)
                {
                  double &o = y[int64_t(r) * N + nrows[i0 + lane]];
                  o         = __dadd_rn(o, mine);
                }
            }
        }
    }

    int near_sm_count()
    {
      int dev = 0, n_sm = 1;
      PIBEM_CUDA(cudaGetDevice(&dev));
      PIBEM_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
      return n_sm;
    }

  } // namespace

  // Warps per block of the kernels that give a warp to each leaf or target box: at
  // most 8, fewer while that leaves SMs without a block (a mesh of 1.5k nodes has some
  // hundred leaves).  FMM product at 386 nodes with eight 218 us, so 178 (with the FP64
  // P2M and L2P kernels)
  static int leaf_warps(int64_t warps)
  {
    int w = 8;
    while (w > 1 && warps < int64_t(w) * 2 * near_sm_count())
      w /= 2;
    return w;
  }

  // Warps per leaf: as many as keep the warps of the launch (leaves x column groups) within
  // what the SMs hold at once.  One warp -> four (GB300, us): P2M / L2P of a 1.5k-node mesh
  // 6.5 / 5.8 -> 4.1 / 3.6, four columns at 6.1k nodes 13.5 / 11.8 -> 6.6 / 4.8; at 98k nodes
  // (6,710 leaves) it would be 21 / 17 -> 27 / 23, every warp loading its leaf's expansion.
  // The line in between is flat: FP32 products of one and four columns at 1.5k to 55k nodes
  // (128 to 14,900 leaves) with 64 warps per SM within 4 % of 32 either way, with 16 up to 5 %
  // slower (four columns, 1,616 leaves 241 -> 254 us).
  static int leaf_split(int64_t warps)
  {
    int w = LEAF_SPLIT;
    while (w > 1 && warps * w > int64_t(32) * near_sm_count())
      w /= 2;
    return w;
  }

  void launch_l2p_ff(const OperatorDev<double> &op, int R, int N, const float2 *Lff, double *y,
                     cudaStream_t s)
  {
    if (op.n_rows == 0 || op.n_near_leaves == 0)
      return;
    const int     split = leaf_split(int64_t(op.n_near_leaves) * R);
    const int64_t nw    = int64_t(op.n_near_leaves) * split;
    const int     w     = leaf_warps(nw * R);
    l2p_ff_kernel<<<dim3(unsigned((nw + w - 1) / w), unsigned(R)), 32 * w, 0, s>>>(
      op.n_near_leaves, split, R, op.K, N, op.nrow_ptr, op.lleaf_box, op.nrows, op.Wff, Lff, y);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  template <typename T>
  void launch_near_spmv(const OperatorDev<T> &op, int R, int N, const T *vals, const T *x, T *y,
                        bool accumulate, cudaStream_t s)
  {
    if (op.n_near_leaves == 0)
      return;
    const int64_t maxnc = (std::max<int64_t>(op.max_near_cols, 1) + 3) / 4 * 4;
    const size_t smem_s = 128 + size_t(2) * maxnc * (4 + sizeof(T));
    if (R == 1 && op.near_sched && smem_s <= 227 * 1024)
      {
        // one column: the scheduled three-stage kernel, 4 warps a block, three
        // 4-value chunks per lane and row in flight, loads that do not
        // allocate in L1.  Measured on GB300 (98k spheroid, CUDA events)
        // against near_leaf_pipe_kernel: FP32 79.5 -> 55.6 us (8 warps with two
        // chunks 62 us; 4 warps with two / four / five chunks 67 / 58 / 64 us;
        // one row per warp with six chunks 62 us; a shared-memory carveout of
        // 100 % 66 us), FP64 328 -> 229 us (8 warps with two chunks 265 us; 4
        // warps with one / two chunks 269 / 233 us).
        constexpr int bs   = 128;
        auto          kern = near_leaf_sched_kernel<T, 3, 128, true>;
        if (smem_s > 48 * 1024)
          raise_smem_limit(reinterpret_cast<const void *>(kern), smem_s);
        int per_sm = 0;
        PIBEM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, bs, smem_s));
        const int grid = std::min(op.n_near_leaves, std::max(per_sm, 1) * near_sm_count());
        launch_pdl(kern, grid, bs, smem_s, s, op.n_near_leaves, int(maxnc), op.near_sched,
                   op.nrows, op.ncols, vals, x, y, accumulate);
        PIBEM_CUDA(cudaGetLastError());
        note_launch();
        return;
      }
    if (R == 1)
      {
        // one column: the software-pipelined persistent kernel (a row is
        // computed with the same rounding steps in the same order as below)
        // resident blocks per SM: FP32 6 (40 registers), FP64 4 (64 registers)
        constexpr int MINB  = sizeof(T) == 4 ? NEAR_BLOCKS_PER_SM_F32 : NEAR_BLOCKS_PER_SM_WIDE;
        auto          kern  = near_leaf_pipe_kernel<T>;
        const size_t  smem1 = size_t(2) * maxnc * sizeof(T);
        if (smem1 > 48 * 1024)
          raise_smem_limit(reinterpret_cast<const void *>(kern), smem1);
        const int grid = std::min(op.n_near_leaves, MINB * near_sm_count());
        launch_pdl(kern, grid, 256, smem1, s, op.n_near_leaves, int(maxnc), op.nrow_ptr, op.ncol_ptr,
                                      op.nval_ptr, op.nrows, op.ncols, vals, x, y, accumulate);
        PIBEM_CUDA(cudaGetLastError());
        note_launch();
        return;
      }
    // several columns: up to 96 KB of x at a time, a multiple of the columns a warp
    // takes (two for two right-hand sides, else four)
    auto launch = [&](auto kern, int rcw) {
      const int64_t fit = (96 * 1024) / (maxnc * int64_t(sizeof(T)) * rcw) * rcw;
      const int     rb  = int(std::min<int64_t>(std::max<int64_t>(fit, rcw), (R + rcw - 1) / rcw * rcw));
      const size_t  smem = size_t(rb) * maxnc * sizeof(T);
      if (smem > 48 * 1024)
        raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
      launch_pdl(kern, op.n_near_leaves, 128, smem, s, R, rb, N, op.nrow_ptr, op.ncol_ptr, op.nval_ptr,
                 op.nrows, op.ncols, vals, x, y, accumulate);
    };
    constexpr int RR4 = sizeof(T) == 4 ? 4 : 2;
    if (R == 2 || 4 * maxnc * int64_t(sizeof(T)) > 200 * 1024)
      {
        if (2 * maxnc * int64_t(sizeof(T)) > 200 * 1024) // one column's x for very wide leaves
          launch(near_leaf_multi_kernel<T, 1, 4>, 1);
        else
          launch(near_leaf_multi_kernel<T, 2, 4>, 2);
      }
    else
      launch(near_leaf_multi_kernel<T, 4, RR4>, 4);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  bool near_ff_fits(const OperatorDev<double> &op)
  {
    const int64_t maxnc = (std::max<int64_t>(op.max_near_cols, 1) + 3) / 4 * 4;
    return size_t(2) * maxnc * sizeof(float2) <= 227 * 1024;
  }

  void launch_near_spmv_ff(const OperatorDev<double> &op, int R, int N, const float2 *vals,
                           const float2 *xff, double *y, bool accumulate, cudaStream_t s)
  {
    if (op.n_near_leaves == 0)
      return;
    const int64_t maxnc = (std::max<int64_t>(op.max_near_cols, 1) + 3) / 4 * 4;
    const size_t smem1 = size_t(2) * maxnc * sizeof(float2);
    if (smem1 > 48 * 1024)
      raise_smem_limit(reinterpret_cast<const void *>(near_leaf_ff_kernel), smem1);
    if (R == 1)
      near_leaf_ff_kernel<<<std::min(op.n_near_leaves, NEAR_BLOCKS_PER_SM_WIDE * near_sm_count()), 256,
                            smem1, s>>>(op.n_near_leaves, int(maxnc), op.nrow_ptr, op.ncol_ptr,
                                        op.nval_ptr, op.nrows, op.ncols, vals, xff, y, accumulate);
    else
      {
        // two columns at a time for two and for leaves whose four columns would not
        // leave two blocks per SM, else four
        auto launch = [&](auto kern, int rc) {
          const size_t smem = size_t(rc) * maxnc * sizeof(float2);
          if (smem > 48 * 1024)
            raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
          kern<<<dim3(op.n_near_leaves, (R + rc - 1) / rc), 128, smem, s>>>(
            R, N, op.nrow_ptr, op.ncol_ptr, op.nval_ptr, op.nrows, op.ncols, vals, xff, y, accumulate);
        };
        if (R == 2 || 4 * maxnc * sizeof(float2) > 100 * 1024)
          launch(near_leaf_ff_multi_kernel<2, 2>, 2);
        else
          launch(near_leaf_ff_multi_kernel<4, 2>, 4);
      }
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  template <typename T>
  void launch_p2m_apply(const OperatorDev<T> &op, int R, int N, const uint8_t *dir,
                        const uint8_t *modes, const T *x, T *M, bool combined, cudaStream_t s)
  {
    if (op.n_p2m_leaves == 0)
      return;
    const bool comb = combined && op.Tc;
    auto launch = [&](auto kern, int rc) {
      const int groups = (R + rc - 1) / rc;
      const int split  = leaf_split(op.n_p2m_leaves); // the same for every R: it orders the sums
      const int w      = std::max(split, leaf_warps(int64_t(op.n_p2m_leaves) * split * groups));
      const int per    = w / split; // leaves per block
      launch_pdl(kern, dim3(unsigned((op.n_p2m_leaves + per - 1) / per), unsigned(groups)), 32 * w, 0, s,
                 op.n_p2m_leaves, split, R, op.K, N, op.prow_ptr, op.pleaf_box, op.prow_dof,
                 comb ? op.Tc : op.T1, op.T2, dir, modes, x, M);
    };
    if constexpr (std::is_same<T, double>::value)
      {
        auto by_k = [&](auto npl) {
          constexpr int NPL = decltype(npl)::value;
          if (comb)
            R == 1 ? launch(p2m_apply64_kernel<true, 1, NPL>, 1) : launch(p2m_apply64_kernel<true, 4, NPL>, 4);
          else
            R == 1 ? launch(p2m_apply64_kernel<false, 1, NPL>, 1) : launch(p2m_apply64_kernel<false, 2, NPL>, 2);
        };
        switch ((op.K + 31) / 32)
          {
            case 1: by_k(std::integral_constant<int, 1>()); break;
            case 2: by_k(std::integral_constant<int, 2>()); break;
            case 3: by_k(std::integral_constant<int, 3>()); break;
            default: by_k(std::integral_constant<int, 4>()); break;
          }
      }
    else
      {
        auto by_split = [&](auto sp) {
          constexpr bool SP = decltype(sp)::value;
          if (comb)
            R == 1 ? launch(p2m_apply_kernel<true, 1, SP>, 1) : launch(p2m_apply_kernel<true, 4, SP>, 4);
          else
            R == 1 ? launch(p2m_apply_kernel<false, 1, SP>, 1) : launch(p2m_apply_kernel<false, 4, SP>, 4);
        };
        leaf_split(op.n_p2m_leaves) > 1 ? by_split(std::true_type()) : by_split(std::false_type());
      }
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  // The downward pass of the FP32 operator as fused level passes: target-major
  // M2L products, their sums per box, then L2L level by level.
  static bool fused_down(const OperatorDev<float> &op, int R)
  {
    return op.down_par && op.down_m2l_beg && fused_levels_ok(op.K, R);
  }

  // Threads of a gather block: a box's R K values in one pass where they fit (121 values with
  // 96 threads took two: at 198k nodes, p = 10, the deepest level 87 us, now 74)
  static int gather_threads(int values) { return values > 96 ? 128 : 96; }

  // The CUDA-core translation GEMM for chunks [c0, c1): K / 32 rows per thread, at most
  // 4, and eight threads across 64 columns (32 in FP64, whose blocks take so long that
  // the last wave of 64-column ones left a third of the chip idle).  A launch with fewer
  // than 256 blocks of 64 columns (the tree's small levels) splits the rows over
  // blockIdx.z, 16 per block, and takes 16 (FP64) or 32 columns per block.  Whole products,
  // us, with the line at 64 / 256 / 1,024 blocks: float-float, four columns, p = 8 at 6.1k
  // nodes 701 / 528 / 530, p = 10 at 24.6k 1,987 / 1,622 / 1,622; FP64, four columns, p = 8 at
  // 6.1k 1,957 / 1,744 / 1,745; FP64, one column, p = 8 at 1.5k 309 / 307 / 236, at 6.1k 628 / 625 /
  // 612, at 13.8k alike: only one-column FP64 products of small meshes would want it higher.
  template <typename IO, typename OP>
  static void launch_cuda_core_gemm(int K, int max_chunk_pairs, int R, int c0,
                                    int c1, const int32_t *ch_start, const int32_t *ch_cnt,
                                    const int32_t *ch_op, const int32_t *q_src, const OP *ops, const IO *E,
                                    IO *Y, const int32_t *yslot, int ldy, cudaStream_t s)
  {
    if (c1 <= c0)
      return;
    if (K > 128)
      throw Error(PIBEM_EINVAL, "translations: K = (p+1)^2 above 128");
    constexpr bool fp64  = std::is_same<OP, double>::value;
    const unsigned gx    = unsigned(c1 - c0);
    const int      most  = max_chunk_pairs * R; // columns of a chunk
    const bool     split = int64_t(gx) * ((most + 63) / 64) < 256;
    const int      RI    = split ? 1 : std::min(4, (K + 31) / 32);
    const int      TX    = split ? 16 : (K + RI - 1) / RI;
    auto launch = [&](auto kern, int CJ, int TY) {
      const int    cols = CJ * TY;
      const size_t smem = (size_t(K) * TX * RI + size_t(K) * (cols + 1)) * sizeof(OP);
      const dim3   grid(gx, unsigned((most + cols - 1) / cols), split ? unsigned((K + 15) / 16) : 1u);
      if (smem > 48 * 1024)
        raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
      kern<<<grid, TY * TX, smem, s>>>(R, K, TX, c0, ch_start, ch_cnt, ch_op, q_src, ops, E, Y, yslot, ldy);
    };
    constexpr int CJ = fp64 ? 4 : 8, CJS = fp64 ? 1 : 2;
    if (split)
      launch(trans_gemm_kernel<IO, OP, 1, CJS, 16>, CJS, 16);
    else
      switch (RI)
        {
          case 1: launch(trans_gemm_kernel<IO, OP, 1, CJ, 8>, CJ, 8); break;
          case 2: launch(trans_gemm_kernel<IO, OP, 2, CJ, 8>, CJ, 8); break;
          case 3: launch(trans_gemm_kernel<IO, OP, 3, CJ, 8>, CJ, 8); break;
          default: launch(trans_gemm_kernel<IO, OP, 4, CJ, 8>, CJ, 8); break;
        }
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  // in float-float: IO = double (FP64 expansions) or float2 ((hi, lo) expansions)
  template <typename IO>
  void launch_ff_gemm(const OperatorDev<double> &op, int R, int c0, int c1, const IO *E, IO *Y,
                      cudaStream_t s)
  {
    launch_cuda_core_gemm<IO, float2>(op.K, op.max_chunk_pairs, R, c0, c1, op.ch_start, op.ch_cnt,
                                      op.ch_op, op.q_src, op.ops_ff, E, Y, nullptr, op.K, s);
  }
  template void launch_ff_gemm<double>(const OperatorDev<double> &, int, int, int, const double *,
                                       double *, cudaStream_t);
  template void launch_ff_gemm<float2>(const OperatorDev<double> &, int, int, int, const float2 *,
                                       float2 *, cudaStream_t);

  // the FP64-accurate tree passes on (hi, lo) expansions
  void launch_upward_level_ff(const OperatorDev<double> &op, int R, int level, float2 *M, float2 *Y,
                              cudaStream_t s)
  {
    launch_ff_gemm<float2>(op, R, op.up_chunk_ptr[level], op.up_chunk_ptr[level + 1], M, Y, s);
    const int a = op.up_box_ptr[level], b = op.up_box_ptr[level + 1];
    if (b > a)
      {
        gather_ff_kernel<<<b - a, gather_threads(R * op.K), 0, s>>>(
          R, op.K, op.up_box + a, op.up_q_ptr + a, op.up_q, Y, M);
        PIBEM_CUDA(cudaGetLastError());
        note_launch();
      }
  }
  void launch_m2l_ff(const OperatorDev<double> &op, int R, const float2 *M, float2 *Y, cudaStream_t s)
  {
    launch_ff_gemm<float2>(op, R, 0, op.m2l_chunk_end, M, Y, s);
  }
  void launch_downward_level_ff(const OperatorDev<double> &op, int R, int level, float2 *Lx,
                                float2 *Y, cudaStream_t s)
  {
    launch_ff_gemm<float2>(op, R, op.down_chunk_ptr[level], op.down_chunk_ptr[level + 1], Lx, Y, s);
    const int a = op.down_box_ptr[level], b = op.down_box_ptr[level + 1];
    if (b > a)
      {
        gather_ff_kernel<<<b - a, gather_threads(R * op.K), 0, s>>>(
          R, op.K, op.down_box + a, op.down_q_ptr + a, op.down_q, Y, Lx);
        PIBEM_CUDA(cudaGetLastError());
        note_launch();
      }
  }
  void launch_convert_d2ff(int64_t n, const double *a, float2 *b, cudaStream_t s)
  {
    if (n == 0)
      return;
    d2ff_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(n, a, b);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }
  void launch_convert_ff2d(int64_t n, const float2 *a, double *b, cudaStream_t s)
  {
    if (n == 0)
      return;
    ff2d_kernel<<<unsigned((n + 255) / 256), 256, 0, s>>>(n, a, b);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  // Y row of (pair q, rhs r): (yslot ? yslot[q] : q) * R + r, rows of ldy values
  template <typename T>
  static void launch_trans_gemm(const OperatorDev<T> &op, int R, int c0, int c1, const T *E, T *Y,
                                cudaStream_t s, const int32_t *yslot = nullptr, int ldy = 0)
  {
    if (c1 <= c0)
      return;
    if (ldy == 0)
      ldy = op.K;
    if constexpr (std::is_same<T, float>::value)
      if (op.tc_images)
        {
          launch_tc_gemm(op, R, c0, c1, E, Y, yslot, ldy, op.tc_err, s);
          return;
        }
    if constexpr (std::is_same<T, double>::value)
      if (op.ops_ff)
        {
          launch_ff_gemm<double>(op, R, c0, c1, E, Y, s);
          return;
        }
    launch_cuda_core_gemm<T, T>(op.K, op.max_chunk_pairs, R, c0, c1, op.ch_start, op.ch_cnt, op.ch_op,
                                op.q_src, op.ops, E, Y, yslot, ldy, s);
  }

  template <typename T>
  static void launch_gather(int R, int K, int nbox, const int32_t *boxes, const int64_t *q_ptr,
                            const int32_t *q, const T *Y, T *out, cudaStream_t s)
  {
    if (nbox <= 0)
      return;
    gather_kernel<T><<<nbox, gather_threads(R * K), 0, s>>>(R, K, boxes, q_ptr, q, Y, out);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  template <typename T>
  void launch_upward_level(const OperatorDev<T> &op, int R, int level, T *M, T *Y, cudaStream_t s)
  {
    if constexpr (std::is_same<T, float>::value)
      if (op.up_child8 && fused_levels_ok(op.K, R))
        {
          launch_m2m_level_fused(op, R, level, M, s);
          return;
        }
    launch_trans_gemm<T>(op, R, op.up_chunk_ptr[level], op.up_chunk_ptr[level + 1], M, Y, s);
    const int a = op.up_box_ptr[level], b = op.up_box_ptr[level + 1];
    launch_gather<T>(R, op.K, b - a, op.up_box + a, op.up_q_ptr + a, op.up_q, Y, M, s);
  }

  // the M2L products of all levels; for the fused level passes in the
  // target-major order with 16-byte aligned rows (what the M2L sums read)
  template <typename T>
  void launch_m2l_gemm(const OperatorDev<T> &op, int R, const T *M, T *Y, cudaStream_t s)
  {
    if constexpr (std::is_same<T, float>::value)
      if (fused_down(op, R))
        {
          launch_trans_gemm<T>(op, R, 0, op.m2l_chunk_end, M, Y, s, op.m2l_yslot,
                               (op.K + 3) / 4 * 4);
          return;
        }
    launch_trans_gemm<T>(op, R, 0, op.m2l_chunk_end, M, Y, s);
  }

  template <typename T>
  void launch_m2l_sums(const OperatorDev<T> &op, int R, T *Lx, const T *Y, cudaStream_t s)
  {
    if constexpr (std::is_same<T, float>::value)
      if (fused_down(op, R))
        launch_m2l_sums_fused(op, R, Lx, Y, s);
  }

  template <typename T>
  void launch_downward_level(const OperatorDev<T> &op, int R, int level, T *Lx, T *Y,
                             cudaStream_t s)
  {
    if constexpr (std::is_same<T, float>::value)
      if (fused_down(op, R))
        {
          launch_l2l_level_fused(op, R, level, Lx, s);
          return;
        }
    launch_trans_gemm<T>(op, R, op.down_chunk_ptr[level], op.down_chunk_ptr[level + 1], Lx, Y, s);
    const int a = op.down_box_ptr[level], b = op.down_box_ptr[level + 1];
    launch_gather<T>(R, op.K, b - a, op.down_box + a, op.down_q_ptr + a, op.down_q, Y, Lx, s);
  }

  template <typename T>
  void launch_m2p(const OperatorDev<T> &op, const TreeDev &td, int R, int N, const T *M, T *y,
                  cudaStream_t s)
  {
    if (op.n_m2p_tgt == 0)
      return;
    auto eval = [&](auto kern, int nc) {
      launch_pdl(kern, dim3(unsigned((op.n_m2p_items + 127) / 128), unsigned((R + nc - 1) / nc)), 128, 0, s,
                 op.n_m2p_items, R, op.K, op.p, op.m2p_item_ptr, op.m2p_item_pair, op.m2p_pair_tgt,
                 op.m2p_src, op.m2p_tnode_ptr, op.m2p_tnodes, td.xyz, td.center, td.delta, M,
                 op.m2p_scratch);
    };
    if (R == 1)
      eval(m2p_eval_kernel<T, 1>, 1);
    else if (R <= 4)
      eval(m2p_eval_kernel<T, 4>, 4);
    else
      eval(m2p_eval_kernel<T, 8>, 8);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
    const int w = leaf_warps(int64_t(op.n_m2p_tgt) * R);
    launch_pdl(m2p_sum_kernel<T>, dim3(unsigned((op.n_m2p_tgt + w - 1) / w), unsigned(R)), 32 * w, 0, s,
      op.n_m2p_tgt, N, op.n_m2p_items, op.m2p_tnode_ptr, op.m2p_src_ptr, op.m2p_item_ptr,
      op.m2p_tnodes, op.m2p_scratch, y);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_m2p_ff(const OperatorDev<double> &op, const TreeDev &td, int R, int N, const float2 *Mff,
                     double *y, cudaStream_t s)
  {
    if (op.n_m2p_tgt == 0)
      return;
    auto eval = [&](auto kern, int nc) {
      kern<<<dim3(unsigned((op.n_m2p_items + 127) / 128), unsigned((R + nc - 1) / nc)), 128, 0, s>>>(
        op.n_m2p_items, R, op.K, op.p, op.m2p_item_ptr, op.m2p_item_pair, op.m2p_pair_tgt, op.m2p_src,
        op.m2p_tnode_ptr, op.m2p_tnodes, td.xyz, td.center, td.delta, Mff, op.m2p_scratch);
    };
    if (R == 1)
      eval(m2p_eval_ff_kernel<1>, 1);
    else
      eval(m2p_eval_ff_kernel<4>, 4);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
    const int w = leaf_warps(int64_t(op.n_m2p_tgt) * R);
    m2p_sum_kernel<double><<<dim3(unsigned((op.n_m2p_tgt + w - 1) / w), unsigned(R)), 32 * w, 0, s>>>(
      op.n_m2p_tgt, N, op.n_m2p_items, op.m2p_tnode_ptr, op.m2p_src_ptr, op.m2p_item_ptr,
      op.m2p_tnodes, op.m2p_scratch, y);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void ensure_fmm_tables(int device, cudaStream_t s)
  {
    static bool       done[64] = {};
    static std::mutex mu; // handles may be set up from several host threads
    std::lock_guard<std::mutex> lock(mu);
    if (device < 0 || device >= 64 || done[device])
      return;
    LegendreTables t;
    fill_legendre_tables(t);
    PIBEM_CUDA(cudaMemcpyToSymbolAsync(c_leg, &t, sizeof(t), 0, cudaMemcpyHostToDevice, s));
    PIBEM_CUDA(cudaStreamSynchronize(s));
    done[device] = true;
  }

  template <typename T>
  void launch_l2p(const OperatorDev<T> &op, int R, int N, const T *Lx, T *y, cudaStream_t s)
  {
    if (op.n_rows == 0 || op.n_near_leaves == 0)
      return;
    auto launch = [&](auto kern, int rc) {
      const int     groups = (R + rc - 1) / rc, split = leaf_split(int64_t(op.n_near_leaves) * groups);
      const int64_t nw = int64_t(op.n_near_leaves) * split;
      const int     w  = leaf_warps(nw * groups);
      launch_pdl(kern, dim3(unsigned((nw + w - 1) / w), unsigned(groups)), 32 * w, 0, s,
                 op.n_near_leaves, split, R, op.K, N, op.nrow_ptr, op.lleaf_box, op.nrows, op.W, Lx, y);
    };
    if constexpr (std::is_same<T, double>::value)
      {
        auto by_k = [&](auto npl) {
          constexpr int NPL = decltype(npl)::value;
          if (R == 1)
            launch(l2p64_kernel<1, 8, NPL>, 1);
          else if (R <= 3)
            launch(l2p64_kernel<2, 4, NPL>, 2);
          else
            launch(l2p64_kernel<4, 4, NPL>, 4);
        };
        switch ((op.K + 31) / 32)
          {
            case 1: by_k(std::integral_constant<int, 1>()); break;
            case 2: by_k(std::integral_constant<int, 2>()); break;
            case 3: by_k(std::integral_constant<int, 3>()); break;
            default: by_k(std::integral_constant<int, 4>()); break;
          }
      }
    else if (R == 1)
      launch(l2p_kernel<1, 8>, 1);
    else
      launch(l2p_kernel<4, 4>, 4);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

#define PIBEM_INSTANTIATE(T)                                                                      \
  template void launch_near_spmv<T>(const OperatorDev<T> &, int, int, const T *, const T *, T *, \
                                    bool, cudaStream_t);                                         \
  template void launch_p2m_apply<T>(const OperatorDev<T> &, int, int, const uint8_t *,           \
                                    const uint8_t *, const T *, T *, bool, cudaStream_t);        \
  template void launch_upward_level<T>(const OperatorDev<T> &, int, int, T *, T *, cudaStream_t); \
  template void launch_m2l_gemm<T>(const OperatorDev<T> &, int, const T *, T *, cudaStream_t);    \
  template void launch_m2l_sums<T>(const OperatorDev<T> &, int, T *, const T *, cudaStream_t);    \
  template void launch_downward_level<T>(const OperatorDev<T> &, int, int, T *, T *,             \
                                         cudaStream_t);                                          \
  template void launch_m2p<T>(const OperatorDev<T> &, const TreeDev &, int, int, const T *, T *, \
                              cudaStream_t);                                                     \
  template void launch_l2p<T>(const OperatorDev<T> &, int, int, const T *, T *, cudaStream_t);
  PIBEM_INSTANTIATE(double)
  PIBEM_INSTANTIATE(float)
} // namespace pibem
