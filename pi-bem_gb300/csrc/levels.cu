// Fused level passes of the FP32 operator, on the CUDA cores:
//
//   M2L sums  L[b]  = sum_{M2L pairs q of b} Y[q]             all levels, one launch
//   L2L       L[b] += T_{oct(b)} L[parent(b)]                  one launch per level
//   M2M       M[P]  = sum_{octant o} T_o M[child_o(P)]          one launch per level
//
// (the reference's ascending pass, bem_fma.cc:2274-2376, and the L2L / M2L part
// of its descending pass, bem_fma.cc:2582-2652.)  The translations of one tree
// level are small (a few thousand K x K matrix-vector products); as batched
// GEMMs followed by a gather they cost two dependent launches per level and a
// round trip of the products through HBM.  Here a block computes complete
// expansions of a batch of columns (column = (box, right-hand side)).
//
// Threads: LV_G groups of KT = 32 ceil(K/32) (at most 128) threads; thread t of a
// group owns output coefficient t of the group's columns g, g + LV_G, ...  Every
// column's result is computed by a fixed sequence of operations that depends on
// the column's own data only (a K-term chain with k ascending per operator, in L2L
// beyond K = 81 four chains of a quarter each, added pairwise; M2M: the eight
// octants' products added in a fixed order; M2L sums: one warp per 32
// coefficients, pairs in list order): the same bits whatever the number of
// columns, their grouping into blocks or the other columns of the batch.
//
// A block holds one operator (26 KB at p = 8, 59 KB at p = 10) in shared memory.
// The passes are short chains of small launches, so what bounds them is latency:
// the operator's copy is started before the block waits for the launch ahead of
// it (the operators are constants of the mesh), and one operator per block
// leaves room for the next level's blocks beside the running ones.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "async_copy.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace pibem
{
  namespace
  {
    __host__ __device__ inline int lv_kx(int K) { return (K + 3) / 4 * 4; }

    constexpr int  LV_G          = 4; // column groups per block
    constexpr int  LV_ONE_CHAIN  = 81; // L2L: most terms in one chain (rounding grows with its length)
    constexpr long LV_SPIN_LIMIT = 1L << 24;

    __host__ __device__ inline int lv_kk(int K) { return (K * K + 3) / 4 * 4; } // padded operator

    // acc[i] = sum_k T[k][ko] X[g + LV_G i][k], k ascending; T one operator stored
    // [in][out], both in shared memory
    template <int C>
    __device__ __forceinline__ void lv_dot(float (&acc)[C], const float *T, const float *X, int K,
                                           int Kx, int ko)
    {
#pragma unroll
      for (int i = 0; i < C; ++i)
        acc[i] = 0.0f;
      int k = 0;
#pragma unroll 4
      for (; k + 4 <= K; k += 4)
        {
          float tv[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            tv[u] = T[(k + u) * K + ko];
#pragma unroll
          for (int i = 0; i < C; ++i)
            {
              const float4 xv = *reinterpret_cast<const float4 *>(X + i * LV_G * Kx + k);
              acc[i]          = fmaf(tv[0], xv.x, acc[i]);
              acc[i]          = fmaf(tv[1], xv.y, acc[i]);
              acc[i]          = fmaf(tv[2], xv.z, acc[i]);
              acc[i]          = fmaf(tv[3], xv.w, acc[i]);
            }
        }
      for (; k < K; ++k)
        {
          const float tv = T[k * K + ko];
#pragma unroll
          for (int i = 0; i < C; ++i)
            acc[i] = fmaf(tv, X[i * LV_G * Kx + k], acc[i]);
        }
    }

    // L2L: the chains CH of a sum (chain c: the terms [K c / CH, K (c + 1) / CH)), the row
    // stride of X (each chain's terms from a 16-byte boundary on) and the place of term k
    __host__ __device__ inline int lv_chains(int K) { return K <= LV_ONE_CHAIN ? 1 : 4; }
    __host__ __device__ inline int lv_chain_stride(int K, int CH) { return lv_kx((K + CH - 1) / CH); }
    __device__ inline int lv_chain_place(int K, int CH, int k)
    {
      const int c = CH == 1 ? 0 : (CH * k + CH - 1) / K;
      return c * lv_chain_stride(K, CH) + k - K * c / CH;
    }

    // As lv_dot in four chains side by side, added pairwise; X rows of four chains
    template <int C>
    __device__ __forceinline__ void lv_dot4(float (&acc)[C], const float *T, const float *X, int K, int ko)
    {
      const int cs = lv_chain_stride(K, 4), stride = 4 * cs, n = K / 4; // n: the shortest chain
      float     s[4][C];
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < C; ++i)
          s[c][i] = 0.0f;
      int k = 0;
      for (; k + 4 <= n; k += 4)
#pragma unroll
        for (int c = 0; c < 4; ++c)
          {
            float        tv[4];
            const float *Tc = T + (K * c / 4 + k) * K + ko;
#pragma unroll
            for (int u = 0; u < 4; ++u)
              tv[u] = Tc[u * K];
#pragma unroll
            for (int i = 0; i < C; ++i)
              {
                const float4 xv = *reinterpret_cast<const float4 *>(X + i * LV_G * stride + c * cs + k);
                s[c][i]         = fmaf(tv[0], xv.x, s[c][i]);
                s[c][i]         = fmaf(tv[1], xv.y, s[c][i]);
                s[c][i]         = fmaf(tv[2], xv.z, s[c][i]);
                s[c][i]         = fmaf(tv[3], xv.w, s[c][i]);
              }
          }
      for (; k < (K + 3) / 4; ++k) // at most four more terms, one more in some chains
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (K * c / 4 + k < K * (c + 1) / 4)
            {
              const float tv = T[(K * c / 4 + k) * K + ko];
#pragma unroll
              for (int i = 0; i < C; ++i)
                s[c][i] = fmaf(tv, X[i * LV_G * stride + c * cs + k], s[c][i]);
            }
#pragma unroll
      for (int i = 0; i < C; ++i)
        acc[i] = __fadd_rn(__fadd_rn(s[0][i], s[1][i]), __fadd_rn(s[2][i], s[3][i]));
    }

    // Thread 0 starts the bulk copy of one operator (lv_kk(K) floats, 16-byte
    // aligned) into shared memory, completing on the barrier.
    __device__ inline void lv_start_op(float *dst, const float *src, int K, uint32_t bar)
    {
      const uint32_t bytes = uint32_t(lv_kk(K)) * 4u;
      mbar_arrive_expect_tx(bar, bytes);
      bulk_copy(smem_u32(dst), src, bytes, bar);
    }

    // Every thread waits (bounded) for the operator; false after a timeout,
    // which is recorded in *err.
    __device__ inline bool lv_wait_op(uint32_t bar, uint32_t parity, int *err)
    {
      if (mbar_wait_bounded(bar, parity, LV_SPIN_LIMIT))
        return true;
      atomicOr(err, int(DEV_TIMEOUT_TRANSLATIONS));
      return false;
    }

    __device__ inline void prefetch_l1(const void *p)
    {
      asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
    }

    __device__ inline uint32_t cluster_rank()
    {
      uint32_t r;
      asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
      return r;
    }
    __device__ inline void cluster_barrier()
    {
      asm volatile("barrier.cluster.arrive.release;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    }
    // 16 bytes at shared-memory address addr of the block with the given rank
    __device__ inline float4 ld_cluster(uint32_t addr, uint32_t rank)
    {
      uint32_t a;
      float4   v;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                   : "r"(a)
                   : "memory");
      return v;
    }

    // One level of the upward pass.  Columns c = i * R + r over the level's
    // parents i (par[i], children child8[8 i + o], -1: none).  A cluster of
    // eight blocks takes batches of LV_G C columns: the block of rank o applies
    // the octant-o operator to the batch's octant-o children (zero where there
    // is none) and leaves its products in its shared memory; after a cluster
    // barrier each block adds the eight blocks' products of an eighth of the
    // batch, read through distributed shared memory.  The products are double
    // buffered, so a batch has one cluster barrier.
    // Shared memory: T[lv_kk], X[LV_G C][Kx], P[2][LV_G C][Kx].
    // What bounds it: latency (a level's arithmetic is below a microsecond).  Measured
    // (kernel times, warm caches, GB300), against one block per SM holding all
    // eight operators: 98k spheroid, p = 8, five levels 50 -> 43 us, and less in the
    // step, where the copies overlap the launch ahead; 55k hull, p = 10, seven
    // levels 85 -> 65 us (the operators read through L1 before).
    template <int C>
    __global__ void __launch_bounds__(LV_G * 128)
      m2m_level_kernel(int R, int K, int ncols, const int32_t *__restrict__ par,
                       const int32_t *__restrict__ child8, const float *__restrict__ lvops,
                       float *__restrict__ M, int *__restrict__ err)
    {
      extern __shared__ __align__(16) float lv_sm[];
      __shared__ uint64_t op_bar;
      constexpr int NB = LV_G * C; // columns of a batch
      const int Kx = lv_kx(K), n4 = Kx / 4;
      float    *T = lv_sm, *X = T + lv_kk(K), *P = X + NB * Kx;
      const int KT = blockDim.x / LV_G;
      const int g = threadIdx.x / KT, ko = threadIdx.x - g * KT; // KT >= Kx: one coefficient
      const int o = int(cluster_rank());
      const uint32_t bar = smem_u32(&op_bar);
      if (threadIdx.x == 0)
        {
          mbar_init(bar, 1);
          mbar_init_fence();
          lv_start_op(T, lvops + size_t(o) * lv_kk(K), K, bar);
        }
      const int cl = blockIdx.x >> 3, ncl = gridDim.x >> 3;
      if (threadIdx.x < NB && cl * NB + int(threadIdx.x) < ncols)
        {
          const int pi = (cl * NB + threadIdx.x) / R;
          prefetch_l1(child8 + 8 * pi + o);
          prefetch_l1(par + pi);
        }
      pdl_entry();
      bool      ops_ok = true, waited = false;
      int       buf = 0;
      for (int c0 = cl * NB; c0 < ncols; c0 += ncl * NB, buf ^= 1)
        {
          const int nc = min(NB, ncols - c0);
          // thread (g, ko) brings coefficient ko of the columns it computes
          float v[C];
#pragma unroll
          for (int i = 0; i < C; ++i)
            {
              const int c = g + LV_G * i, col = c0 + c, pi = col / R;
              const int ch = c < nc && ko < K ? child8[8 * pi + o] : -1;
              v[i]         = ch >= 0 ? M[(int64_t(ch) * R + (col - pi * R)) * K + ko] : 0.0f;
            }
          if (ko < Kx)
#pragma unroll
            for (int i = 0; i < C; ++i)
              X[(g + LV_G * i) * Kx + ko] = v[i];
          __syncthreads();
          if (!waited)
            {
              ops_ok = lv_wait_op(bar, 0, err);
              waited = true;
            }
          float *Pb = P + buf * NB * Kx;
          if (ko < Kx)
            {
              float acc[C];
              if (ko < K && ops_ok)
                lv_dot<C>(acc, T, X + g * Kx, K, Kx, ko);
              else
#pragma unroll
                for (int i = 0; i < C; ++i)
                  acc[i] = 0.0f;
#pragma unroll
              for (int i = 0; i < C; ++i)
                Pb[(g + LV_G * i) * Kx + ko] = acc[i];
            }
          cluster_barrier(); // the eight blocks' products are in place; X is no longer read
          for (int i = o * blockDim.x + threadIdx.x; i < nc * n4; i += 8 * blockDim.x)
            {
              const int c = i / n4, q = i - c * n4;
              float4    v[8];
#pragma unroll
              for (int b = 0; b < 8; ++b)
                v[b] = ld_cluster(smem_u32(Pb) + uint32_t(c * Kx + 4 * q) * 4u, uint32_t(b));
              const int   col = c0 + c, pi = col / R, r = col - pi * R;
              float      *m = M + (int64_t(par[pi]) * R + r) * K + 4 * q;
              const float s[4] = {
                ((v[0].x + v[1].x) + (v[2].x + v[3].x)) + ((v[4].x + v[5].x) + (v[6].x + v[7].x)),
                ((v[0].y + v[1].y) + (v[2].y + v[3].y)) + ((v[4].y + v[5].y) + (v[6].y + v[7].y)),
                ((v[0].z + v[1].z) + (v[2].z + v[3].z)) + ((v[4].z + v[5].z) + (v[6].z + v[7].z)),
                ((v[0].w + v[1].w) + (v[2].w + v[3].w)) + ((v[4].w + v[5].w) + (v[6].w + v[7].w))};
#pragma unroll
              for (int u = 0; u < 4; ++u)
                if (4 * q + u < K)
                  m[u] = s[u];
            }
        }
      if (!waited) // never leave with the copy in flight
        {
          __syncthreads();
          lv_wait_op(bar, 0, err);
        }
      cluster_barrier(); // no block leaves while another reads its products
    }

    // M2L sums of the boxes of the downward lists, all levels.  The M2L
    // products are target-major: the rows (slot, rhs) of a box's pairs are the
    // slots [beg, end) in list order, rows of Kx = round_up(K, 4) values.  One
    // warp per column c = i * R + r; lane l adds coefficients 4l..4l+3 over
    // the box's rows in order, 16 rows in flight.
    __global__ void __launch_bounds__(256)
      m2l_sum_kernel(int R, int K, int64_t ncols, const int32_t *__restrict__ box,
                     const int32_t *__restrict__ beg, const int32_t *__restrict__ end,
                     const float *__restrict__ Y, float *__restrict__ Lx)
    {
      pdl_entry();
      const int64_t col = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
      if (col >= ncols)
        return;
      const int     lane = threadIdx.x & 31;
      const int     bi = int(col / R), r = int(col - int64_t(bi) * R);
      const int     n4 = lv_kx(K) / 4;
      const int     e0 = beg[bi], e1 = end[bi];
      float4        s  = make_float4(0.f, 0.f, 0.f, 0.f);
      if (lane < n4)
        {
          const float4 *y      = reinterpret_cast<const float4 *>(Y) + (int64_t(e0) * R + r) * n4 + lane;
          const int64_t stride = int64_t(R) * n4;
          for (int e = e0; e < e1; e += 16, y += 16 * stride)
            {
              float4 v[16];
#pragma unroll
              for (int u = 0; u < 16; ++u)
                if (e + u < e1)
                  v[u] = __ldg(y + u * stride);
#pragma unroll
              for (int u = 0; u < 16; ++u)
                if (e + u < e1)
                  {
                    s.x += v[u].x;
                    s.y += v[u].y;
                    s.z += v[u].z;
                    s.w += v[u].w;
                  }
            }
          float *o = Lx + (int64_t(box[bi]) * R + r) * K + 4 * lane;
          const float sv[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (4 * lane + c < K)
              o[c] = sv[c];
        }
    }

    // One level of the downward pass after the M2L sums: L[b] += T_oct L[parent]
    // for the level's boxes with an L2L parent.  They are listed by octant (oct:
    // the bounds of the octants in the list); the columns c = i * R + r of an
    // octant are cut into batches of LV_G C, numbered octant after octant, and a
    // block takes a contiguous range of batches, so that a batch has one operator
    // and most blocks copy one only.  What does not depend on the launch ahead
    // (the operator, the box ids) is fetched before waiting for it.  Measured (as
    // above; one block per SM with up to eight operators before): 98k spheroid
    // 43 -> 33 us over five levels; 55k hull, p = 10, 76 -> 52 us over seven.  A
    // mixed solve to 1e-12: 50.8 -> 47.2 ms (98k), 67.9 -> 58.6 ms (hull).
    //   CH: the chains of a sum.  One chain of 121 terms would take 49 us on the hull but
    // double the rounding error of the four it had before; 64 registers keep two blocks
    // per SM with four (82 registers, one block: 54 us).
    // Shared memory: T[lv_kk], X[LV_G C][CH lv_chain_stride].
    template <int C, int CH>
    __global__ void __launch_bounds__(LV_G * 128, CH == 1 ? 0 : (C <= 4 ? 2 : 1))
      l2l_level_kernel(int R, int K, LevelOctants oct, int n_batches, const int32_t *__restrict__ box,
                       const int32_t *__restrict__ par, const float *__restrict__ lvops,
                       float *__restrict__ Lx, int *__restrict__ err)
    {
      extern __shared__ __align__(16) float lv_sm[];
      __shared__ uint64_t op_bar;
      constexpr int NB = LV_G * C; // columns of a batch
      const int Xs = CH * lv_chain_stride(K, CH); // row stride of X
      float    *T = lv_sm, *X = T + lv_kk(K);
      const int KT = blockDim.x / LV_G;
      const int g = threadIdx.x / KT, ko = threadIdx.x - g * KT, place = lv_chain_place(K, CH, ko);
      int       b_lo = int(int64_t(n_batches) * blockIdx.x / gridDim.x);
      const int b_hi = int(int64_t(n_batches) * (blockIdx.x + 1) / gridDim.x);
      if (b_lo >= b_hi)
        return;
      // octant of batch b_lo, its first column in the octant
      int o = 0, c0 = b_lo;
      for (; o < 7; ++o)
        {
          const int nb = ((oct.p[o + 1] - oct.p[o]) * R + NB - 1) / NB;
          if (c0 < nb)
            break;
          c0 -= nb;
        }
      c0 *= NB;
      const uint32_t bar = smem_u32(&op_bar);
      int            held = o, loads = 1, waited = 0; // operator held, copies started and waited for
      if (threadIdx.x == 0)
        {
          mbar_init(bar, 1);
          mbar_init_fence();
          lv_start_op(T, lvops + size_t(o) * lv_kk(K), K, bar);
        }
      if (threadIdx.x < NB && c0 + int(threadIdx.x) < (oct.p[o + 1] - oct.p[o]) * R)
        {
          prefetch_l1(par + oct.p[o] + (c0 + threadIdx.x) / R);
          prefetch_l1(box + oct.p[o] + (c0 + threadIdx.x) / R);
        }
      pdl_entry();
      bool ops_ok = true;
      for (; b_lo < b_hi; ++b_lo)
        {
          const int32_t *pb = par + oct.p[o], *bb = box + oct.p[o];
          const int      n = (oct.p[o + 1] - oct.p[o]) * R, nc = min(NB, n - c0);
          if (o != held)
            {
              if (threadIdx.x == 0 && ops_ok)
                {
                  // the reads of T by the last batch ended before the barrier below
                  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                  lv_start_op(T, lvops + size_t(o) * lv_kk(K), K, bar);
                }
              held = o;
              ++loads;
            }
          // thread (g, ko) brings coefficient ko of the parents' expansions and of the
          // boxes' M2L sums (needed last) of the columns it computes
          float *l[C], sum[C], v[C];
#pragma unroll
          for (int i = 0; i < C; ++i)
            {
              const int c = g + LV_G * i, col = c0 + c, bi = col / R, r = col - bi * R;
              l[i]        = nullptr;
              sum[i] = v[i] = 0.0f;
              if (c < nc && ko < K)
                {
                  v[i]   = Lx[(int64_t(pb[bi]) * R + r) * K + ko];
                  l[i]   = Lx + (int64_t(bb[bi]) * R + r) * K + ko;
                  sum[i] = *l[i];
                }
            }
          if (ko < (CH == 1 ? Xs : K))
#pragma unroll
            for (int i = 0; i < C; ++i)
              X[(g + LV_G * i) * Xs + place] = v[i];
          __syncthreads();
          if (waited < loads)
            {
              if (ops_ok)
                ops_ok = lv_wait_op(bar, uint32_t(loads - 1) & 1u, err);
              ops_ok = __syncthreads_and(ops_ok);
              waited = loads;
            }
          if (ko < K && ops_ok)
            {
              float acc[C];
              if constexpr (CH == 1)
                lv_dot<C>(acc, T, X + g * Xs, K, Xs, ko);
              else
                lv_dot4<C>(acc, T, X + g * Xs, K, ko);
#pragma unroll
              for (int i = 0; i < C; ++i)
                if (l[i])
                  *l[i] = sum[i] + acc[i];
            }
          __syncthreads(); // X and T no longer read
          c0 += NB;
          while (o < 7 && c0 >= (oct.p[o + 1] - oct.p[o]) * R) // on to the next octant with boxes
            {
              ++o;
              c0 = 0;
            }
        }
    }

    int lv_kt(int K) { return std::min(128, (K + 31) / 32 * 32); }

    int lv_n_sm()
    {
      int dev = 0, n_sm = 1;
      PIBEM_CUDA(cudaGetDevice(&dev));
      PIBEM_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
      return n_sm;
    }

    // Columns per thread (1, 2, 4 or 8): the fewest with which `blocks` blocks
    // (clusters) take the level in one batch each, so that a small level spreads
    // over the chip and a large one reads its operators fewest times.
    int lv_cols(int64_t ncols, int64_t blocks)
    {
      int c = 1;
      while (c < 8 && int64_t(LV_G) * c * blocks < ncols)
        c *= 2;
      return c;
    }
  } // namespace

  bool fused_levels_ok(int K, int R)
  {
    return R >= 1 && size_t(16) * lv_kx(K) * sizeof(float) <= 48 * 1024;
  }

  size_t fused_level_ops_floats(int K) { return size_t(16) * lv_kk(K); }

  void launch_m2m_level_fused(const OperatorDev<float> &op, int R, int level, float *M,
                              cudaStream_t s)
  {
    const int a = op.up_box_ptr[level], b = op.up_box_ptr[level + 1];
    if (b <= a)
      return;
    const int K     = op.K;
    const int ncols = (b - a) * R;
    // three blocks per SM where they fit (220 KB of the SM's 228 for them with 2 KB each
    // for static and reserved shared memory), else two, in clusters of eight (the deepest
    // level of a 98k-node mesh, 1,700 parents, with two: 14.7 us, with three 11.5)
    int    max_cl, C;
    size_t smem;
    for (int per_sm = 3;; --per_sm)
      {
        max_cl = std::max(1, per_sm * lv_n_sm() / 8);
        C      = lv_cols(ncols, max_cl);
        smem   = (size_t(lv_kk(K)) + size_t(3) * LV_G * C * lv_kx(K)) * sizeof(float);
        if (per_sm == 2 || size_t(per_sm) * (smem + 2048) <= 220 * 1024)
          break;
      }
    const int ncl = std::min(max_cl, (ncols + LV_G * C - 1) / (LV_G * C));
    auto launch = [&](auto kern) {
      if (smem > 48 * 1024)
        raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
      launch_pdl_cluster(kern, unsigned(8 * ncl), LV_G * lv_kt(K), 8, smem, s, R, K, ncols,
                         op.up_box + a, op.up_child8 + size_t(8) * a, op.lv_ops, M, op.dev_err);
    };
    switch (C)
      {
        case 8: launch(m2m_level_kernel<8>); break;
        case 4: launch(m2m_level_kernel<4>); break;
        case 2: launch(m2m_level_kernel<2>); break;
        default: launch(m2m_level_kernel<1>); break;
      }
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_m2l_sums_fused(const OperatorDev<float> &op, int R, float *Lx, const float *Y,
                             cudaStream_t s)
  {
    const int a = op.down_box_ptr.empty() ? 0 : op.down_box_ptr[1];
    const int b = op.down_box_ptr.empty() ? 0 : op.down_box_ptr.back();
    if (b <= a)
      return;
    const int64_t ncols = int64_t(b - a) * R;
    int w = 8; // a warp per column, fewer per block while SMs would go without one
    while (w > 1 && ncols < int64_t(w) * 2 * lv_n_sm())
      w /= 2;
    launch_pdl(m2l_sum_kernel, unsigned((ncols + w - 1) / w), 32 * w, 0, s,
      R, op.K, ncols, op.down_box + a, op.down_m2l_beg + a, op.down_m2l_end + a, Y, Lx);
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_l2l_level_fused(const OperatorDev<float> &op, int R, int level, float *Lx,
                              cudaStream_t s)
  {
    if (level >= int(op.down_oct_ptr.size()))
      return;
    const LevelOctants &oct   = op.down_oct_ptr[level];
    const int           ncols = (oct.p[8] - oct.p[0]) * R;
    if (ncols <= 0)
      return;
    const int K     = op.K;
    const int max_b = 2 * lv_n_sm();
    const int C     = lv_cols(ncols, max_b), CH = lv_chains(K);
    int       nb    = 0;
    for (int o = 0; o < 8; ++o)
      nb += ((oct.p[o + 1] - oct.p[o]) * R + LV_G * C - 1) / (LV_G * C);
    const size_t smem = (size_t(lv_kk(K)) + size_t(LV_G) * C * CH * lv_chain_stride(K, CH)) * sizeof(float);
    auto launch = [&](auto kern) {
      if (smem > 48 * 1024)
        raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
      launch_pdl(kern, unsigned(std::min(nb, max_b)), LV_G * lv_kt(K), smem, s, R, K, oct, nb,
                 op.down_box, op.down_par, op.lv_ops + size_t(8) * lv_kk(K), Lx, op.dev_err);
    };
    auto by_chains = [&](auto c) {
      constexpr int Cc = decltype(c)::value;
      CH == 1 ? launch(l2l_level_kernel<Cc, 1>) : launch(l2l_level_kernel<Cc, 4>);
    };
    switch (C)
      {
        case 8: by_chains(std::integral_constant<int, 8>()); break;
        case 4: by_chains(std::integral_constant<int, 4>()); break;
        case 2: by_chains(std::integral_constant<int, 2>()); break;
        default: by_chains(std::integral_constant<int, 1>()); break;
      }
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }
} // namespace pibem
