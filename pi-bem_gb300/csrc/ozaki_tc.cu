// FP64-accurate translation GEMM on the tensor cores: the product Y = T E of
// the FP64-accurate operator computed from exact BF16 products, an Ozaki-type
// splitting, with tcgen05.mma kind::f16.
//
// Every expansion row (box, rhs) is scaled by a power of two 2^-e_r so that
// its largest entry is below 1 in magnitude, and written as S signed digits
//     x 2^-e_r = sum_{i<S} d_i 2^-(7 + 8 i) + rest,   |d_i| <= 128, |rest| <= 2^-8S,
// each digit times its weight being exact in BF16 (8 significant bits); every
// operator row (output coefficient n) likewise, with its own exponent e_n.
// A product of two slices is exact in FP32 (at most 16 significant bits), and
// the sum over K <= 128 terms of the products of all slice pairs (i, j) with
// the same i + j = g is exact for g <= 6 (at most 7 x 128 x 2^14 < 2^24 units
// of its weight) in a tensor-memory accumulator of its own.  Pairs with
// i + j >= S are dropped.  The epilogue adds the accumulators in float-float
// arithmetic and scales the (hi, lo) pair by 2^(e_r + e_n).
//
// The error is relative to the largest entry of the expansion row times the
// largest of the operator row, not to the terms that occur: expansions are
// largest at degree 0, operator rows at the highest input degree, and the more
// so the higher the order.  So the orders have different digits:
//   K <= 96 (p <= 8)   S = 6, parts of 48 rows, five accumulators: g = 0 .. 3, and
//                      g = 4, 5 together (rounding below 2^-42 of the largest product);
//   K <= 128 (p <= 10) S = 7, parts of 32 rows, an accumulator for each g = 0 .. 6, and
//                      the exact factor 2^(n / 2) of input degree n (n / 2 rounded down)
//                      moved from the operator's entries to the expansion's.
// 2-norm error of the M2L product at p = 10, output degree 0 / 10, for sources on
// planes through the box, in its corners and at its centre (the float-float GEMM
// 1.4e-14 .. 5e-14 at every degree): six digits 5e-14 / 9.7e-12, 5e-14 / 2.4e-12, 2.5e-14 /
// 7.8e-12; seven 6e-16 / 3.4e-14, 6e-16 / 1.1e-14, 6e-16 / 3.2e-14; seven with the factor
// 6e-16 / 5.2e-15, 8e-16 / 3.7e-15, 6e-16 / 5.0e-15.  (A factor 2^n would suit planes and
// centre, 1.1e-15, but not corners, whose expansions hardly fall: 1.6e-14 / 2.1e-14.)
//
// A unit of work is 128 rows (pairs of one operator) times one part of the operator's
// rows, with two units' accumulators in tensor memory, so that a unit's epilogue runs
// beside the next one's MMAs.  Per 16 K values 11 MMAs (N = 48 to 240) take the 21 slice
// pairs of six digits, 7 MMAs (N = 32 to 224) the 28 of seven; K steps beyond K are neither
// loaded nor issued.
//
// Block (416 threads, one per SM, persistent over a contiguous range of chunks, part
// after part within a run of chunks of one operator):
//   warps 0-3  producers: a 6-deep ring of A stages (one K chunk of 64 values of one
//              slice for the unit's 128 rows, 128-byte-swizzled K-major), filled with
//              16-byte cp.async, eight lanes to a row's 128-byte line;
//   warps 4-11 epilogue: tensor-memory loads, float-float sums, staging in shared
//              memory and coalesced row segments;
//   warp 12    copies the part's 2 S operator slice tiles (pre-swizzled at set-up) with
//              one bulk copy when operator or part change, and issues the MMAs.
// What bounds it: the tensor unit's operand reads (sm__pipe_tc 34 - 35 % active, the
// products themselves 18 % with six digits, 21 % with seven), the epilogue's FP32
// instructions and the hand-overs between the roles.  Measured (GB300; before: one
// accumulator set of 96 columns, the epilogue after the MMAs, a row loaded and stored by
// one thread, and the CUDA-core float-float GEMM beyond K = 96): 98k spheroid (p = 8,
// 272,776 pairs) 441 -> 281 us, 198k hull (p = 10) 5,920 -> 1,095 us, 16 columns at 23,816
// nodes 1,754 -> 814 us.  (One MMA per slice pair 426 us for the first, four epilogue
// warps 318; six digits for the second 840.)
// All waits are bounded; a timeout is recorded in *err and the host reports
// PIBEM_ETIMEDOUT.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <type_traits>

#include "async_copy.cuh"
#include "ffmath.cuh"
#include "kernels.h"
#include "tcgen05.cuh"

namespace pibem
{
  namespace
  {
    constexpr int      OZ_K6       = 96;  // most coefficients with six digits
    constexpr int      OZ_KC       = 64;  // K values per chunk: one 128-byte line of BF16
    constexpr int      OZ_NKC      = 2;   // K chunks (K <= 128)
    constexpr int      OZ_ROWS     = 128; // unit rows (M of the MMA)
    constexpr int      OZ_RING     = 6;   // A stages
    constexpr int      OZ_LAG      = 3;   // stages a producer has in flight
    constexpr int      OZ_THREADS  = 416; // warps 0-3 producers, 4-11 epilogue, 12 MMA
    constexpr int      OZ_MMA_WARP = 12;
    constexpr uint32_t OZ_A_BYTES  = OZ_ROWS * 128;         // 16 KB
    constexpr uint32_t OZ_TMEM_COLS = 512;                  // two units (480, 448), a power of two
    constexpr long     OZ_SPIN      = 1L << 22;
    constexpr int      OZ_NBAR      = 2 * OZ_RING + 7;

    // sizes for S digits (slices) per operand.  Shared memory: B (72, 56 KB) | A ring (96 KB)
    // | staging (50, 34 KB) | barriers
    template <int S>
    struct OzShape
    {
      static_assert(S == 6 || S == 7, "digits per operand");
      static constexpr int      G  = S == 6 ? 5 : 7;   // accumulators
      static constexpr int      NP = S == 6 ? 48 : 32; // operator rows per part (N of the MMA)
      static constexpr int      EC = NP / 2;           // columns per epilogue warp
      static constexpr uint32_t BT_BYTES  = NP * 128;  // per (K chunk, slice)
      static constexpr uint32_t B_BYTES   = OZ_NKC * S * BT_BYTES; // per (operator, part)
      static constexpr uint32_t ACC_COLS  = G * NP;    // one unit's accumulators
      static constexpr int      STG_LD    = EC + 1;    // staging row stride (float2)
      static constexpr uint32_t STG_BYTES = 32 * STG_LD * 8; // per epilogue warp
      static constexpr uint32_t OFF_A     = B_BYTES;
      static constexpr uint32_t OFF_STG   = OFF_A + OZ_RING * OZ_A_BYTES;
      static constexpr uint32_t OFF_BAR   = OFF_STG + 8 * STG_BYTES;
      static constexpr uint32_t SMEM      = OFF_BAR + 8 * OZ_NBAR + 1024; // + alignment slack
      static_assert(2 * ACC_COLS <= OZ_TMEM_COLS && SMEM <= 227 * 1024 && B_BYTES % 1024 == 0, "");
      __host__ __device__ static int parts(int K) { return (K + NP - 1) / NP; }
      // power of two moved from the operator to the expansion at coefficient k (degree
      // floor(sqrt(k)))
      __device__ static int shift(int k) { return S == 6 ? 0 : int(sqrtf(float(k) + 0.5f)) / 2; }
    };

    // Bounded wait; after a timeout anywhere in the block (abort raised) no
    // further waiting, so a broken pipeline ends quickly (results then wrong,
    // reported through *err).
    __device__ inline bool oz_wait(uint32_t addr, uint32_t parity, int *err, volatile int *abort)
    {
      for (long it = 0; it < OZ_SPIN; ++it)
        {
          if (mbar_try(addr, parity))
            return true;
          if ((it & 255) == 255 && *abort)
            return false;
        }
      *abort = 1;
      atomicOr(err, int(DEV_TIMEOUT_TRANSLATIONS));
      return false;
    }

    __device__ inline void mma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                    uint32_t accumulate)
    {
      asm volatile("{\n\t.reg .pred p;\n\t"
                   "setp.ne.b32 p, %4, 0;\n\t"
                   "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                   :
                   : "r"(dtmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
                   : "memory");
    }

    // BF16 bits of a float that BF16 represents exactly (low 16 bits zero)
    __host__ __device__ inline uint16_t bf16_bits(float f)
    {
      uint32_t u;
      memcpy(&u, &f, 4);
      return uint16_t(u >> 16);
    }

    // Digits of the rows of the (hi, lo) expansions E (rows of K values): one
    // warp per row; slices[i][row][128] BF16 (zero beyond K), e_row[row].  Entries that are
    // not finite leave digits that are not, and so NaN in every product of the row.
    template <int S>
    __global__ void oz_slice_rows_kernel(int64_t nrows, int K, const float2 *__restrict__ E,
                                         uint16_t *__restrict__ slices, int *__restrict__ e_row)
    {
      const int64_t row = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
      if (row >= nrows)
        return;
      const int lane = threadIdx.x & 31;
      float2    x[4];
      int       e = INT_MIN; // every scaled entry is below 2^e
#pragma unroll
      for (int u = 0; u < 4; ++u)
        {
          const int k    = lane + 32 * u;
          x[u]           = k < K ? E[row * K + k] : make_float2(0.0f, 0.0f);
          const float mx = fabsf(x[u].x) + fabsf(x[u].y);
          if (mx > 0.0f && mx <= FLT_MAX)
            {
              int ex;
              frexpf(mx, &ex);
              e = max(e, ex + OzShape<S>::shift(k));
            }
        }
      e = __reduce_max_sync(0xffffffffu, e);
      if (e == INT_MIN)
        e = 0;
      if (lane == 0)
        e_row[row] = e;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        {
          const int k  = lane + 32 * u;
          const int sh = OzShape<S>::shift(k) - e;
          float     vh = ldexpf(x[u].x, sh), vl = ldexpf(x[u].y, sh);
#pragma unroll
          for (int i = 0; i < S; ++i)
            {
              const float sc = i == 0 ? 128.0f : 256.0f;
              vh *= sc;
              vl *= sc;
              const float d = rintf(vh);
              const float t = vh - d; // exact
              const float2 r = ff_add(make_float2(t, 0.0f), make_float2(vl, 0.0f));
              vh = r.x;
              vl = r.y;
              slices[(int64_t(i) * nrows + row) * 128 + k] = bf16_bits(ldexpf(d, -(7 + 8 * i)));
            }
        }
    }

    struct OzArgs
    {
      int            R, K, chunk0, n_chunks;
      const int32_t *ch_start, *ch_cnt, *ch_op, *q_src;
      const uint16_t *bimg;   // [op][part][kc][slice][NP x 64 swizzled]
      const int16_t  *e_col;  // [op][NP parts]
      const uint16_t *aslc;   // [slice][box row][128]
      const int      *e_row;  // [box row]
      int64_t         a_rows; // box rows (n_boxes * R)
      float2         *Y;
      int            *err;
    };

    // The block's units in order, f(operator, part, first pair, rows of the chunk,
    // first row): every role walks the same list.
    template <typename F>
    __device__ __forceinline__ void oz_units(const OzArgs &a, int parts, const TileRange &tr, F f)
    {
      for (int ch = tr.c_lo, end; ch <= tr.c_hi; ch = end)
        {
          const int op = a.ch_op[ch];
          for (end = ch + 1; end <= tr.c_hi && a.ch_op[end] == op;)
            ++end;
          for (int part = 0; part < parts; ++part)
            for (int c = ch; c < end; ++c)
              {
                const int start = a.ch_start[c], rows = a.ch_cnt[c] * a.R;
                const int first = c == tr.c_lo ? tr.t_lo * OZ_ROWS : 0;
                const int last  = c == tr.c_hi ? min(rows, tr.t_hi * OZ_ROWS) : rows;
                for (int t0 = first; t0 < last; t0 += OZ_ROWS)
                  f(op, part, start, rows, t0);
              }
        }
    }

    // 16 bytes global -> shared, asynchronous; zeros when !ok
    __device__ __forceinline__ void oz_cp16(uint32_t dst, const void *src, bool ok)
    {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0)
                   : "memory");
    }
    template <int N>
    __device__ __forceinline__ void oz_cp_wait()
    {
      asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
    }

    template <int S>
    __global__ void __launch_bounds__(OZ_THREADS, 1) oz_gemm_kernel(OzArgs a)
    {
      using Z = OzShape<S>;
      extern __shared__ uint8_t smem_raw[];
      __shared__ uint32_t     tmem_slot;
      __shared__ volatile int abort_flag;
      __shared__ int          rows_src[2][OZ_ROWS]; // a unit's source rows (-1: padding)
      const uint32_t raw  = smem_u32(smem_raw);
      const uint32_t base = (raw + 1023u) & ~1023u;
      const int      tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
      const uint32_t bar0   = base + Z::OFF_BAR;
      auto a_full  = [&](int s) { return bar0 + 8u * uint32_t(s); };
      auto a_empty = [&](int s) { return bar0 + 8u * uint32_t(OZ_RING + s); };
      auto t_full  = [&](int b) { return bar0 + 8u * uint32_t(2 * OZ_RING + b); };
      auto t_empty = [&](int b) { return bar0 + 8u * uint32_t(2 * OZ_RING + 2 + b); };
      const uint32_t b_full = bar0 + 8u * uint32_t(2 * OZ_RING + 4);
      const uint32_t b_free = b_full + 8u, drain = b_full + 16u;
      const int R = a.R, K = a.K;
      const int nkc = K > OZ_KC ? 2 : 1, parts = Z::parts(K);
      auto      steps = [&](int kc) { return min(OZ_KC / 16, (K - kc * OZ_KC + 15) / 16); };
      if (tid == 0)
        {
          abort_flag = 0;
          for (int s = 0; s < OZ_RING; ++s)
            {
              mbar_init(a_full(s), 128);
              mbar_init(a_empty(s), 1);
            }
          for (int b = 0; b < 2; ++b)
            {
              mbar_init(t_full(b), 1);
              mbar_init(t_empty(b), 256);
            }
          mbar_init(b_full, 1);
          mbar_init(b_free, 1);
          mbar_init(drain, 1);
          mbar_init_fence();
        }
      if (warp == OZ_MMA_WARP)
        {
          asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                       :
                       : "r"(smem_u32(&tmem_slot)), "r"(OZ_TMEM_COLS)
                       : "memory");
          asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
      TileRange range = tile_range(a.ch_cnt + a.chunk0, a.n_chunks, R);
      range.c_lo += a.chunk0;
      range.c_hi += a.chunk0;
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncthreads();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem = tmem_slot;

      if (warp < 4)
        {
          // ---------------- producers ----------------
          long g = 0; // A stages started
          int  unit = 0;
          auto done = [&](long st) { // this thread's copies of stage st have landed
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(a_full(int(st % OZ_RING)));
          };
          oz_units(a, parts, range, [&](int, int, int start, int rows, int t0) {
            int *src = rows_src[unit & 1];
            {
              const int row = t0 + tid;
              src[tid]      = row < rows ? a.q_src[start + row / R] * R + row % R : -1;
            }
            asm volatile("bar.sync 1, 128;" ::: "memory"); // the producers' table
            for (int kc = 0; kc < nkc; ++kc)
              {
                const int nch = 2 * steps(kc); // 16-byte pieces of a row that are used
                for (int i = 0; i < S; ++i, ++g)
                  {
                    const int slot = int(g % OZ_RING);
                    if (g >= OZ_RING)
                      oz_wait(a_empty(slot), uint32_t(g / OZ_RING - 1) & 1u, a.err, &abort_flag);
                    const uint32_t  at = base + Z::OFF_A + uint32_t(slot) * OZ_A_BYTES;
                    const uint16_t *E  = a.aslc + int64_t(i) * a.a_rows * 128 + kc * OZ_KC;
                    const int       ch = tid & 7;
                    if (ch < nch)
#pragma unroll
                      for (int u = 0; u < 8; ++u)
                        {
                          const int row = 16 * u + (tid >> 3), sr = src[row];
                          oz_cp16(at + sw128_off_b16(row, 8 * ch), E + int64_t(max(sr, 0)) * 128 + 8 * ch,
                                  sr >= 0);
                        }
                    asm volatile("cp.async.commit_group;" ::: "memory");
                    if (g >= OZ_LAG)
                      {
                        oz_cp_wait<OZ_LAG>();
                        done(g - OZ_LAG);
                      }
                  }
              }
            ++unit;
          });
          oz_cp_wait<0>();
          for (long st = g > OZ_LAG ? g - OZ_LAG : 0; st < g; ++st)
            done(st);
        }
      else if (warp == OZ_MMA_WARP)
        {
          // ---------------- operator copies and MMAs ----------------
          if (lane == 0)
            {
              // D f32, A and B bf16, both K-major, M = 128; idesc1: N = NP
              const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(OZ_ROWS >> 4) << 24);
              const uint32_t idesc1 = idesc | (uint32_t(Z::NP >> 3) << 17);
              int  held_op = -1, held_part = -1, b_loads = 0, unit = 0;
              long g      = 0;
              bool issued = false, b_pending = false;
              oz_units(a, parts, range, [&](int op, int part, int, int, int) {
                if (op != held_op || part != held_part)
                  {
                    if (issued) // the MMAs that read the held tiles
                      {
                        mma_commit(b_free);
                        oz_wait(b_free, uint32_t(b_loads - 1) & 1u, a.err, &abort_flag);
                      }
                    mbar_arrive_expect_tx(b_full, Z::B_BYTES);
                    bulk_copy(base, a.bimg + (size_t(op) * parts + part) * (Z::B_BYTES / 2),
                              Z::B_BYTES, b_full);
                    b_pending = !oz_wait(b_full, uint32_t(b_loads) & 1u, a.err, &abort_flag);
                    ++b_loads;
                    held_op   = op;
                    held_part = part;
                  }
                const int buf = unit & 1;
                if (unit >= 2)
                  oz_wait(t_empty(buf), uint32_t((unit >> 1) - 1) & 1u, a.err, &abort_flag);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d       = tmem + uint32_t(buf) * Z::ACC_COLS;
                for (int kc = 0; kc < nkc; ++kc)
                  {
                    const int      nks = steps(kc);
                    const uint64_t db  = smem_desc_sw128(base + uint32_t(kc * S) * Z::BT_BYTES);
                    for (int i = 0; i < S; ++i, ++g)
                      {
                        const int slot = int(g % OZ_RING);
                        oz_wait(a_full(slot), uint32_t(g / OZ_RING) & 1u, a.err, &abort_flag);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t at = base + Z::OFF_A + uint32_t(slot) * OZ_A_BYTES;
                        // Slice i with the operator slices j = 0 .. G - 1 - i: the groups i + j
                        // and the slices' tiles follow one another, so that one MMA of N =
                        // NP (G - i) reads A once for all of them; with six digits then j =
                        // 5 - i, also into the last accumulator.
                        // (Descriptors differ in their start address, 16-byte units, only.)
                        const uint64_t da = smem_desc_sw128(at);
                        const uint64_t dl = db + uint64_t((S - 1 - i) * (Z::BT_BYTES >> 4));
                        const int      nj = Z::G - i; // G .. G - S + 1
                        const uint32_t di = idesc + (uint32_t(nj * Z::NP >> 3) << 17);
                        const uint32_t first = kc == 0 && i == 0 ? 1u : 0u;
#pragma unroll
                        for (int ks = 0; ks < OZ_KC / 16; ++ks)
                          if (ks < nks)
                            {
                              if (S > 6 || nj > 0)
                                mma_bf16(d + uint32_t(i * Z::NP), da + uint64_t(2 * ks), db + uint64_t(2 * ks),
                                         di, ks > 0 ? 1u : 1u - first);
                              if constexpr (S == 6)
                                mma_bf16(d + uint32_t((Z::G - 1) * Z::NP), da + uint64_t(2 * ks),
                                         dl + uint64_t(2 * ks), idesc1, 1u);
                            }
                        mma_commit(a_empty(slot)); // frees the stage once these MMAs are done
                        issued = true;
                      }
                  }
                mma_commit(t_full(buf)); // the unit's accumulators are complete
                ++unit;
              });
              if (b_pending) // a copy whose wait gave up: let it land before the block ends
                mbar_wait_bounded(b_full, uint32_t(b_loads - 1) & 1u, OZ_SPIN);
              if (issued)
                {
                  mma_commit(drain); // every MMA issued above has completed
                  mbar_wait_bounded(drain, 0, OZ_SPIN);
                }
            }
          __syncwarp();
        }
      else
        {
          // -------- epilogue: rows 32 q .. 32 q + 31, half the columns of the unit --------
          const int q = warp & 3, c_lo = (warp - 4) / 4 * Z::EC;
          float2   *stg  = reinterpret_cast<float2 *>(smem_raw + (base - raw) + Z::OFF_STG +
                                                   size_t(warp - 4) * Z::STG_BYTES);
          const int n_ec = parts * Z::NP;
          int       unit = 0;
          oz_units(a, parts, range, [&](int op, int part, int start, int rows, int t0) {
            const int buf = unit & 1, row0 = t0 + 32 * q, nvalid = min(32, rows - row0);
            int       er = 0;
            if (lane < nvalid)
              er = a.e_row[int64_t(a.q_src[start + (row0 + lane) / R]) * R + (row0 + lane) % R];
            const int16_t *ec = a.e_col + size_t(op) * n_ec + part * Z::NP + c_lo;
            oz_wait(t_full(buf), uint32_t(unit >> 1) & 1u, a.err, &abort_flag);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d = tmem + (uint32_t(32 * q) << 16) + uint32_t(buf) * Z::ACC_COLS + uint32_t(c_lo);
#pragma unroll 1
            for (int c0 = 0; c0 < Z::EC; c0 += 8)
              {
                // the group sums of 8 columns (all loads, one wait): g0, g1 and g2, g3
                // (and g4, g5) pairwise by TwoSum, the pairs by TwoSum, the errors and the
                // last group added last (each below 2^-40 of the result with six digits),
                // one renormalisation
                uint32_t v[Z::G][8];
#pragma unroll
                for (int b = 0; b < Z::G; ++b)
                  tmem_ld8_nowait(d + uint32_t(b * Z::NP + c0), v[b]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int jj = 0; jj < 8; ++jj)
                  {
                    auto grp = [&](int b) { return __uint_as_float(v[b][jj]); };
                    // a + b = s + e
                    auto two_sum = [](float a, float b, float &e) {
                      const float s = __fadd_rn(a, b), z = __fsub_rn(s, a);
                      e             = __fadd_rn(__fsub_rn(a, __fsub_rn(s, z)), __fsub_rn(b, z));
                      return s;
                    };
                    float       e1, e2, dd;
                    const float t1 = two_sum(grp(0), grp(1), e1), t2 = two_sum(grp(2), grp(3), e2);
                    float       t  = two_sum(t1, t2, dd), lo;
                    if constexpr (S == 6)
                      lo = __fadd_rn(__fadd_rn(e1, __fadd_rn(e2, dd)), grp(4));
                    else
                      {
                        float       e3, d3;
                        const float t3 = two_sum(grp(4), grp(5), e3);
                        t              = two_sum(t, t3, d3);
                        lo = __fadd_rn(__fadd_rn(e1, __fadd_rn(e2, dd)), __fadd_rn(d3, __fadd_rn(e3, grp(6))));
                      }
                    const float2 r = ff_norm(t, lo);
                    // times 2^(e_r + e_n): a power of two built from its bits
                    // when it is a normal float, else ldexpf
                    const int e = er + ec[c0 + jj];
                    float2    y;
                    if (e > -127 && e < 128)
                      {
                        const float sc = __int_as_float((e + 127) << 23);
                        y              = make_float2(__fmul_rn(r.x, sc), __fmul_rn(r.y, sc));
                      }
                    else
                      y = make_float2(ldexpf(r.x, e), ldexpf(r.y, e));
                    stg[lane * Z::STG_LD + c0 + jj] = y;
                  }
              }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(t_empty(buf)); // the accumulators may be overwritten
            __syncwarp();
            // a row at a time, or two of 16 columns
            constexpr int RP = 32 / Z::EC;
            const int     n0 = part * Z::NP + c_lo, nc = min(Z::EC, K - n0);
            const int     rl = RP > 1 ? lane / Z::EC : 0, cl = RP > 1 ? lane % Z::EC : lane;
            float2       *y  = a.Y + (int64_t(start) * R + row0) * K + n0;
            for (int r = rl; r < nvalid; r += RP)
              if (cl < nc)
                y[int64_t(r) * K + cl] = stg[r * Z::STG_LD + cl];
            __syncwarp(); // the staging rows are read
            ++unit;
          });
        }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncthreads();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (warp == OZ_MMA_WARP)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     :
                     : "r"(tmem), "r"(OZ_TMEM_COLS)
                     : "memory");
    }

    // Digits of every operator row (output coefficient; operators [in][out] K x K): B images
    // and column exponents, zero beyond K.  One warp per row of a part's NP.
    template <int S>
    __global__ void __launch_bounds__(256)
      oz_image_kernel(int64_t rows, int K, const double *__restrict__ ops, uint16_t *__restrict__ img,
                      int16_t *__restrict__ e_col)
    {
      const int64_t r    = int64_t(blockIdx.x) * 8 + (threadIdx.x >> 5);
      const int     lane = threadIdx.x & 31;
      if (r >= rows)
        return;
      using Z            = OzShape<S>;
      const int64_t part = r / Z::NP; // of all operators
      const int     row = int(r % Z::NP), parts = Z::parts(K), n = int(part % parts) * Z::NP + row;
      const double *t   = ops + part / parts * K * K + n;
      constexpr int NV  = OZ_NKC * OZ_KC / 32;
      double        v[NV], mx = 0.0;
#pragma unroll
      for (int c = 0; c < NV; ++c)
        {
          const int k = lane + 32 * c;
          v[c]        = n < K && k < K ? ldexp(t[int64_t(k) * K], -Z::shift(k)) : 0.0;
          mx          = fmax(mx, fabs(v[c]));
        }
      for (int o = 16; o > 0; o >>= 1)
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      int e = 0;
      if (mx > 0.0)
        frexp(mx, &e); // mx < 2^e
      if (lane == 0)
        e_col[r] = int16_t(e);
      uint16_t *tile = img + part * (Z::B_BYTES / 2);
#pragma unroll
      for (int c = 0; c < NV; ++c)
        {
          const int k = lane + 32 * c;
          double    x = ldexp(v[c], -e);
          for (int i = 0; i < S; ++i)
            {
              x *= (i == 0 ? 128.0 : 256.0);
              const double d = rint(x);
              x -= d;
              tile[size_t(k / OZ_KC * S + i) * (Z::BT_BYTES / 2) + sw128_off_b16(row, k % OZ_KC) / 2] =
                bf16_bits(ldexpf(float(d), -(7 + 8 * i))); // exact
            }
        }
    }
  } // namespace

  bool ozaki_ok(int K) { return K >= 1 && K <= OZ_NKC * OZ_KC; }

  // f with the number of digits of K coefficients as a constant
  template <typename F>
  static auto oz_digits(int K, F f)
  {
    return K <= OZ_K6 ? f(std::integral_constant<int, 6>()) : f(std::integral_constant<int, 7>());
  }

  size_t ozaki_image_values(int nops, int K)
  {
    return oz_digits(K, [&](auto S) {
      using Z = OzShape<S()>;
      return size_t(nops) * Z::parts(K) * (Z::B_BYTES / 2);
    });
  }
  size_t ozaki_column_values(int nops, int K)
  {
    return oz_digits(K, [&](auto S) { return size_t(nops) * OzShape<S()>::parts(K) * OzShape<S()>::NP; });
  }
  size_t ozaki_slice_values(int64_t nrows, int K)
  {
    return oz_digits(K, [&](auto S) { return size_t(S()) * size_t(nrows) * 128; });
  }

  void launch_ozaki_images(const double *ops, int nops, int K, uint16_t *img, int16_t *e_col, cudaStream_t s)
  {
    const int64_t rows = int64_t(ozaki_column_values(nops, K));
    oz_digits(K, [&](auto S) {
      oz_image_kernel<S()><<<unsigned((rows + 7) / 8), 256, 0, s>>>(rows, K, ops, img, e_col);
    });
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_ozaki_slices(int64_t nrows, int K, const float2 *E, uint16_t *slices, int *e_row,
                           cudaStream_t s)
  {
    if (nrows == 0)
      return;
    oz_digits(K, [&](auto S) {
      oz_slice_rows_kernel<S()><<<unsigned((nrows * 32 + 255) / 256), 256, 0, s>>>(nrows, K, E, slices,
                                                                                 e_row);
    });
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }

  void launch_ozaki_gemm(const OperatorDev<double> &op, int R, int c0, int c1,
                         const uint16_t *aslc, const int *e_row, int64_t a_rows, float2 *Y,
                         cudaStream_t s)
  {
    if (c1 <= c0)
      return;
    int dev = 0, n_sm = 1;
    PIBEM_CUDA(cudaGetDevice(&dev));
    PIBEM_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    OzArgs a;
    a.R = R, a.K = op.K, a.chunk0 = c0, a.n_chunks = c1 - c0;
    a.ch_start = op.ch_start, a.ch_cnt = op.ch_cnt, a.ch_op = op.ch_op, a.q_src = op.q_src;
    a.bimg = op.oz_images, a.e_col = op.oz_ecol, a.aslc = aslc, a.e_row = e_row;
    a.a_rows = a_rows, a.Y = Y, a.err = op.dev_err;
    oz_digits(op.K, [&](auto S) {
      constexpr uint32_t smem = OzShape<S()>::SMEM;
      raise_smem_limit(reinterpret_cast<const void *>(oz_gemm_kernel<S()>), smem);
      oz_gemm_kernel<S()><<<std::min(c1 - c0, n_sm), OZ_THREADS, smem, s>>>(a);
    });
    PIBEM_CUDA(cudaGetLastError());
    note_launch();
  }
} // namespace pibem
