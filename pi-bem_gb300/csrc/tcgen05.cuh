// 5th-generation tensor-core helpers (inline PTX, sm_100-class): the
// 128-byte-swizzled K-major shared-memory layout and its matrix descriptor,
// MMA completion to an mbarrier, and 32-lane tensor-memory loads.
#pragma once

#include <cstdint>

namespace pibem
{
  // Byte offset of element (row, k) of a 128-byte-swizzled K-major tile of
  // 4-byte elements (0 <= k < 32): 8-row atoms of 1024 bytes, row r of an
  // atom at r * 128, 16-byte chunk c of the row at position c ^ (r & 7).
  __host__ __device__ inline uint32_t sw128_off(int row, int k)
  {
    return uint32_t((row >> 3) * 1024 + (row & 7) * 128 + ((((k >> 2) ^ row) & 7) << 4) +
                    (k & 3) * 4);
  }

  // Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
  // 1024 bytes apart (stride byte offset); the leading byte offset is unused
  // for swizzled K-major operands.  A K-step of 8 TF32 values inside the
  // 128-byte line advances the start address by 32 bytes.
  __device__ inline uint64_t smem_desc_sw128(uint32_t saddr)
  {
    uint64_t d = 0;
    d |= uint64_t((saddr >> 4) & 0x3FFFu);
    d |= uint64_t(1) << 16;         // leading byte offset (unused), 16 bytes
    d |= uint64_t(1024 >> 4) << 32; // stride byte offset
    d |= uint64_t(1) << 46;         // descriptor version of sm_100-class tensor cores
    d |= uint64_t(2) << 61;         // swizzle mode: 128 bytes
    return d;                       // base offset 0 (atoms are 1024-byte aligned)
  }

  __device__ inline void mma_commit(uint32_t mbar)
  {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :
                 : "r"(mbar)
                 : "memory");
  }

  __device__ inline void tmem_ld32(uint32_t taddr, float (&v)[32])
  {
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                   "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
                   "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
                   "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j)
      v[j] = __uint_as_float(r[j]);
  }

  // 8 columns of the warp's 32 lanes, without waiting (tcgen05.wait::ld
  // before the registers are used)
  __device__ inline void tmem_ld8_nowait(uint32_t taddr, uint32_t (&r)[8])
  {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
  }

  // A block's share of the 128-row tiles of the chunks [0, n) of a persistent
  // tensor-core launch: from tile t_lo of chunk c_lo up to, not including, tile t_hi of
  // chunk c_hi.  A chunk of cnt pairs has ceil(cnt R / 128) tiles and every tile
  // costs the same, so the blocks get equal numbers of tiles, not of chunks (16
  // columns: chunks of 1 to 16 tiles left the SMs idle for a quarter of the time;
  // 23,816 nodes: FP32 M2L 197 -> 154 us, FP64-accurate M2L 1,016 -> 814 us).
  // All threads of the block call it; cnt is constant data.
  struct TileRange
  {
    int c_lo, t_lo, c_hi, t_hi;
  };
  __device__ inline TileRange tile_range(const int32_t *__restrict__ cnt, int n, int R)
  {
    __shared__ TileRange out;
    __shared__ int       warp_sum[32];
    const int b = blockIdx.x, G = gridDim.x;
    if (R == 1) // one tile per chunk of at most 128 pairs
      {
        TileRange r;
        r.c_lo = int(int64_t(n) * b / G);
        r.c_hi = int(int64_t(n) * (b + 1) / G) - 1;
        r.t_lo = 0;
        r.t_hi = 1;
        return r;
      }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = int(blockDim.x + 31) >> 5;
    const int seg = (n + int(blockDim.x) - 1) / int(blockDim.x);
    const int a = min(n, tid * seg), e = min(n, a + seg);
    int       s = 0;
    for (int i = a; i < e; ++i)
      s += (cnt[i] * R + 127) / 128;
    int inc = s; // inclusive sum over the block
    for (int o = 1; o < 32; o <<= 1)
      {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        inc += lane >= o ? v : 0;
      }
    if (lane == 31)
      warp_sum[warp] = inc;
    if (tid == 0)
      out = {0, 0, -1, 0};
    __syncthreads();
    int total = 0;
    for (int w = 0; w < nw; ++w)
      {
        inc += w < warp ? warp_sum[w] : 0;
        total += warp_sum[w];
      }
    const int lo = int(int64_t(total) * b / G), hi = int(int64_t(total) * (b + 1) / G);
    int       at = inc - s; // tiles before chunk a
    if (lo < hi)
      for (int i = a; i < e; ++i)
        {
          const int t = (cnt[i] * R + 127) / 128;
          if (lo >= at && lo < at + t)
            {
              out.c_lo = i;
              out.t_lo = lo - at;
            }
          if (hi - 1 >= at && hi - 1 < at + t)
            {
              out.c_hi = i;
              out.t_hi = hi - at;
            }
          at += t;
        }
    __syncthreads();
    return out;
  }

  // The same layout for 2-byte elements (0 <= k < 64, 8 per 16-byte chunk).
  __host__ __device__ inline uint32_t sw128_off_b16(int row, int k)
  {
    return uint32_t((row >> 3) * 1024 + (row & 7) * 128 + ((((k >> 3) ^ row) & 7) << 4) +
                    (k & 7) * 2);
  }
} // namespace pibem
