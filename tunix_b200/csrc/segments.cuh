// Segment ids (packed rows, padding) of the flash-attention kernels.
//
// Ids decide for most blocks of 64 tokens as a whole. A tile of rows lists the blocks with any id between the smallest and the
// largest of its rows, and marks those where all ids are the one that all its rows have; the others are never loaded. Elements
// are compared in the rest only, by warp votes. Every tile of every head reads the ids of all blocks that it may see: with the square
// of a row's tokens, so rows of very many short segments are better cut into several calls (512 segments of 128 to 256 tokens, 32
// heads of 128: 4612 us in one call, 1507 in calls of 16384 tokens).
#pragma once
#include "common.cuh"

namespace tb {

constexpr int SEG_W = 64;                                   // tokens of a block
constexpr uint16_t SEG_SAME = 0x8000, SEG_ID = 0x7fff;

template <int CAP>
struct SegList {
  static_assert(CAP < SEG_ID, "block numbers share their 16 bits with a mark");
  uint16_t id[CAP];
  int lo[16], hi[16], n;
};

// All threads of the CTA (whole warps, at most 16): blocks jb0 .. jb0 + nblk - 1 (nblk <= CAP) of the T ids at `seg`, for rows with
// the ids rows[0 .. nrows) (null: all 0) -> the number of blocks listed. Each half-warp reads four consecutive ids a lane, four
// blocks in flight.
template <int CAP>
__device__ __forceinline__ int build_seg_list(SegList<CAP>& s, const int* rows, int nrows, const int* seg, int T, int jb0, int nblk) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  int lo = 0x7fffffff, hi = -0x7fffffff - 1;
  for (int i = tid; i < nrows; i += blockDim.x) {
    const int v = rows ? rows[i] : 0;
    lo = min(lo, v);
    hi = max(hi, v);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (lane == 0) {
    s.lo[warp] = lo;
    s.hi[warp] = hi;
  }
  __syncthreads();
  for (int w = 0; w < nwarp; ++w) {
    lo = min(lo, s.lo[w]);
    hi = max(hi, s.hi[w]);
  }
  for (int j0 = warp * 8; j0 < nblk; j0 += nwarp * 8) {
    int v[4][4];
    bool in[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int j = j0 + 2 * u + (lane >> 4), k = (jb0 + j) * SEG_W + (lane & 15) * 4 + e;
        in[u][e] = j < nblk && k < T;
        v[u][e] = in[u][e] ? __ldg(seg + k) : 0;
      }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      bool any = false, same = lo == hi;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        any = any || (in[u][e] && v[u][e] >= lo && v[u][e] <= hi);
        same = same && in[u][e] && v[u][e] == lo;
      }
      const uint32_t half = (lane & 16) ? 0xffff0000u : 0xffffu;
      const uint32_t anys = __ballot_sync(0xffffffffu, any) & half, sames = __ballot_sync(0xffffffffu, same) & half;
      const int j = j0 + 2 * u + (lane >> 4);
      if ((lane & 15) == 0 && j < nblk) s.id[j] = anys ? (uint16_t)(j | (sames == half ? SEG_SAME : 0)) : (uint16_t)SEG_ID;
    }
  }
  __syncthreads();
  if (warp == 0) {                                  // in place: entry n is written after entries up to n have been read
    int n = 0;
    for (int j = lane; j - lane < nblk; j += 32) {
      const uint16_t v = j < nblk ? s.id[j] : SEG_ID;
      const uint32_t take = __ballot_sync(0xffffffffu, v != SEG_ID);
      if (v != SEG_ID) s.id[n + __popc(take & ((1u << lane) - 1))] = v;
      n += __popc(take);
      __syncwarp();
    }
    if (lane == 0) s.n = n;
  }
  __syncthreads();
  return s.n;
}

__device__ __forceinline__ uint32_t bits_below(int n) { return n >= 32 ? ~0u : n <= 0 ? 0u : (1u << n) - 1; }

// Clears the bits of the 32 tokens from k0 whose id is not the row's: one vote per id among the rows of the warp.
__device__ __forceinline__ void seg_bits(const int* seg, int k0, int T, int mine, uint32_t& keep) {
  const int lane = threadIdx.x & 31;
  const int v = k0 + lane < T ? __ldg(seg + k0 + lane) : 0;
  uint32_t todo = ~0u;
  while (todo) {
    const int id = __shfl_sync(0xffffffffu, mine, __ffs(todo) - 1);
    const uint32_t bits = __ballot_sync(0xffffffffu, v == id);
    const bool now = mine == id;
    if (now) keep &= bits;
    todo &= ~__ballot_sync(0xffffffffu, now);
  }
}

}  // namespace tb
