// Fused token sampling for the rollout engine: temperature, top-k, top-p, categorical draw and the
// chosen token's log-probability, one cluster of 1 to 8 thread blocks per sequence, logits read straight from the lm_head
// output (fp32 [B, V]).
//
//  * top-k / top-p as probability thresholds found by bisection (count(p >= t) >= k, mass(p >= t) >= top_p):
//    no sort, no [B, V] scratch; a histogram of the row leaves a short list to bisect over;
//  * the draw is Gumbel-max over the kept tokens with a counter-based Philox stream keyed by
//    (seed, step, row, token), so a sequence's randomness does not depend on batch composition;
//  * the final logit soft-cap (cap * tanh(z / cap), Gemma-2/3) and a list of forbidden token ids
//    (tunix/generate/sampler.py:84-85,407) are applied to the row in place by the first pass, so the
//    engine needs no [B, V] element-wise kernel in front of this one and the returned log-probability
//    is the one of the distribution that was sampled from.
//
// Replaces lax.top_k + softmax + cumsum mask + categorical of the reference (tunix/generate/sampler.py:112-168).
#include "common.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

using namespace tb;

namespace {

__device__ __forceinline__ uint32_t mulhilo(uint32_t a, uint32_t b, uint32_t& hi) {
  const unsigned long long p = (unsigned long long)a * b;
  hi = (uint32_t)(p >> 32);
  return (uint32_t)p;
}
// Philox-4x32-10
__device__ __forceinline__ uint4 philox(uint4 ctr, uint2 key) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    uint32_t hi0, hi1;
    const uint32_t lo0 = mulhilo(0xD2511F53u, ctr.x, hi0);
    const uint32_t lo1 = mulhilo(0xCD9E8D57u, ctr.z, hi1);
    ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
    key.x += 0x9E3779B9u;
    key.y += 0xBB67AE85u;
  }
  return ctr;
}
__device__ __forceinline__ float u01(uint32_t x) { return ((x >> 8) + 0.5f) * (1.0f / 16777216.0f); }

struct ArgMax {
  float v;
  int i;
};
__device__ __forceinline__ ArgMax amax(ArgMax a, ArgMax b) { return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a; }

__device__ __forceinline__ ArgMax warp_amax(ArgMax b) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    b = amax(b, ArgMax{__shfl_xor_sync(0xffffffffu, b.v, o), __shfl_xor_sync(0xffffffffu, b.i, o)});
  return b;
}

// Block-wide best (valid in every thread); s_v / s_i: 33 entries each.
__device__ __forceinline__ ArgMax block_amax(ArgMax b, float* s_v, int* s_i) {
  const int tid = threadIdx.x, nw = (blockDim.x + 31) >> 5;
  b = warp_amax(b);
  if ((tid & 31) == 0) {
    s_v[tid >> 5] = b.v;
    s_i[tid >> 5] = b.i;
  }
  __syncthreads();
  if (tid < 32) {
    b = warp_amax(tid < nw ? ArgMax{s_v[tid], s_i[tid]} : ArgMax{-INFINITY, 0x7fffffff});
    __syncwarp();
    if (tid == 0) {
      s_v[32] = b.v;
      s_i[32] = b.i;
    }
  }
  __syncthreads();
  return ArgMax{s_v[32], s_i[32]};
}

// Inclusive sums over the lanes of a warp.
__device__ __forceinline__ void warp_scan(unsigned& n, float& f) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, n, o);
    const float v = __shfl_up_sync(0xffffffffu, f, o);
    if (lane >= o) {
      n += u;
      f += v;
    }
  }
}

constexpr int LT = 512;                // most threads that bisect over the list of candidates, of one block
constexpr int BINS = 1024;             // of the distance to the maximum, up to BIN_SPAN (e^-18.5 < 2^-26, the last bisection step)
constexpr float BIN_SPAN = 18.5f;
constexpr int CAND = 4 * LT;           // candidates of the list
constexpr int BISECT = 26;
constexpr int HOLD = 16;               // weights that a thread holds for halvings over the row

struct SampleShared {
  float red[33];
  float s_v[33];
  int s_i[33];
  float tot[2][32];                    // sums of the warps: two slots, used in turn
  float part[2][2];                    // what the other CTAs of the cluster read: two slots, used in turn
  float pv;
  int pi;
  int cut;                             // rank 0: last histogram bin of the candidates, or -1
  int ncand;                           // rank 0
  unsigned long long sums[2][LT / 32];
  unsigned hist[BINS];
  unsigned cum[BINS];                  // rank 0, for halvings over the row: tokens up to and with a bin,
  float low[BINS], high[BINS];         // and bounds of their mass
  float cz[CAND];                      // rank 0: logits of the candidates and their ids
  int ci[CAND];
};

// One row per cluster of 1, 4 or 8 CTAs, each with a contiguous share of the vocabulary.
//
// Top-k and top-p keep e = exp(z - max) >= t for a threshold t found by BISECT halvings of [0, 1]. Every halving needs
// count(e >= mid) or mass(e >= mid), which the few candidates above a histogram bin decide as well as the whole row: the bins
// of z's distance to the maximum are counted once, the bins that surely hold the kept tokens are gathered into one list, and
// one warp (or block) bisects over that list. Where the list would overflow (flat distributions under top-p alone) or the maximum is not
// finite, the halvings run over the row (all CTAs, one exchange each).
//
// Bound by the passes over the row (three, from L2: max, sum + histogram, gather) and five cluster barriers. B200, rows of
// 151,936 (before: one CTA a row, every halving over the row): top-k 50 and top-p 0.95, 1 / 64 / 256 rows 721 / 728 / 1478 -> 26 /
// 36 / 104 us; top-p 0.95 alone, N(0, 4) logits, 64 rows 387 -> 52 us; flat logits (every halving over the row) 397 -> 191 us;
// no filter, 1 / 64 / 256 rows 43 / 44 / 98 -> 13 / 28 / 98 us. Slower than before by up to a fifth: flat logits under top-p in rows
// that are neither aligned nor split (128 of 50,257: 108 -> 126 us).
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT)
sample_kernel(float* __restrict__ logits, long long ld, int V, float inv_temp, int top_k, float top_p,
              unsigned long long seed, const unsigned long long* __restrict__ seed_dev, int step_host, const int* __restrict__ step_dev, int greedy,
              long long* __restrict__ tokens, float* __restrict__ logprobs, float softcap,
              const int* __restrict__ forbidden, int n_forbidden) {
  pdl_trigger();
  pdl_wait();
  const int step = step_dev ? *step_dev : step_host;  // device-resident step and seed keep the launch graph-capturable, and a graph usable
  if (seed_dev) seed = *seed_dev;                     // for calls of other seeds
  __shared__ SampleShared sh;
  const cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  SampleShared& sh0 = *cluster.map_shared_rank(&sh, 0);
  auto csync = [&] {
    if (C > 1) cluster.sync();
    else __syncthreads();
  };
  const int row = blockIdx.x / C;
  float* z = logits + (long long)row * ld;
  const int tid = threadIdx.x;
  constexpr int nt = NT;
  const int share = (V + 4 * C - 1) / (4 * C) * 4;               // a multiple of 4: Philox draws four tokens at a time
  const int i0 = min(V, rank * share), i1 = min(V, i0 + share);
  const int skew = (int)((reinterpret_cast<uintptr_t>(z) >> 2) & 3);   // elements by which a row lies past a 16-byte boundary

  if (softcap > 0.f) {
    const float inv_cap = 1.f / softcap;
    for (int i = i0 + tid; i < i1; i += nt) z[i] = softcap * tanhf(z[i] * inv_cap);
  }
  if (n_forbidden > 0) {
    __syncthreads();                                    // the capped values are in place before they are overwritten
    for (int j = tid; j < n_forbidden; j += nt) {
      const int t = forbidden[j];
      if (t >= i0 && t < i1) z[t] = -INFINITY;
    }
  }
  if (softcap > 0.f || n_forbidden > 0) __syncthreads();

  auto load4 = [&](int i4, bool vec, float (&q)[4]) {   // outside of the share: -inf, which every pass passes over
    if (vec && i4 >= i0 && i4 + 4 <= i1) {
      const float4 t = *reinterpret_cast<const float4*>(z + i4);
      q[0] = t.x; q[1] = t.y; q[2] = t.z; q[3] = t.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) q[j] = (i4 + j >= i0 && i4 + j < i1) ? z[i4 + j] : -INFINITY;
    }
  };
  // f(i, z[i]) over the share, and -inf for what the first and last vectors have outside of it; vectors start at 16-byte boundaries,
  // and four loads of a thread are in flight together
  auto walk = [&](auto&& f) {
    for (int i4 = i0 - skew + tid * 4; i4 < i1; i4 += nt * 16) {
      float q[4][4];
#pragma unroll
      for (int k = 0; k < 4; ++k) load4(i4 + k * nt * 4, true, q[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) f(i4 + k * nt * 4 + j, q[k][j]);
    }
  };
  const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
  auto gumbel4 = [&](int i4) { return philox(make_uint4((uint32_t)(i4 >> 2), (uint32_t)row, (uint32_t)step, 0x5A17u), key); };
  // Sum / maximum over the cluster, the same value in every thread of it. Slots alternate: a CTA that is one exchange ahead
  // writes the other slot, and two ahead it has met everybody at the barrier between.
  int phase = 0;
  auto exchange = [&](float a, float b, float (&all)[8][2]) {
    if (C == 1) {                                       // sums of a block are in all of its threads
      all[0][0] = a;
      all[0][1] = b;
      return;
    }
    if (tid == 0) {
      sh.part[phase][0] = a;
      sh.part[phase][1] = b;
    }
    csync();
    for (int r = 0; r < C; ++r) {
      const SampleShared* o = cluster.map_shared_rank(&sh, r);
      all[r][0] = o->part[phase][0];
      all[r][1] = o->part[phase][1];
    }
    phase ^= 1;
  };
  float all[8][2];
  // Sum over the block, in every thread, behind one barrier: who is one sum ahead writes the other slot.
  int turn = 0;
  auto block_total = [&](float c) {
    c = warp_sum(c);
    if ((tid & 31) == 0) sh.tot[turn][tid >> 5] = c;
    __syncthreads();
    c = warp_sum((tid & 31) < NT / 32 ? sh.tot[turn][tid & 31] : 0.f);
    turn ^= 1;
    return c;
  };
  // Best candidate of every CTA (in its thread 0) -> the row's result, then the barrier before any CTA may leave.
  auto finish = [&](ArgMax best, auto&& log_prob) {
    if (tid == 0) {
      sh.pv = best.v;
      sh.pi = best.i;
    }
    if (C > 1) cluster.sync();
    if (rank == 0 && tid == 0) {
      for (int r = 1; r < C; ++r) {
        const SampleShared* o = cluster.map_shared_rank(&sh, r);
        best = amax(best, ArgMax{o->pv, o->pi});
      }
      const int tok = best.i < V ? best.i : 0;
      tokens[row] = tok;
      if (logprobs) logprobs[row] = log_prob(z[tok]);
    }
    if (C > 1) cluster.sync();
  };

  const bool by_k = top_k > 0 && top_k < V, by_p = top_p > 0.f && top_p < 1.f;
  if (greedy || !(by_k || by_p)) {
    // No top-k / top-p: one pass over the row. Every thread keeps a running (max, sum exp) pair and its best
    // Gumbel-perturbed score; the pairs are merged after the loop.
    float lm = -INFINITY, ls = 0.f;
    ArgMax best{-INFINITY, 0x7fffffff};
#pragma unroll 2
    for (int i4 = i0 + tid * 4; i4 < i1; i4 += nt * 4) {
      float zz[4];
      load4(i4, skew == 0, zz);
      uint4 r = make_uint4(0, 0, 0, 0);
      if (!greedy) r = gumbel4(i4);
      const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
      float cm = lm;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        zz[j] *= inv_temp;
        cm = fmaxf(cm, zz[j]);
      }
      if (cm > lm) {
        ls *= __expf(lm - cm);          // exp(-inf) = 0 on the first group
        lm = cm;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (i4 + j >= i1) break;
        if (zz[j] > -INFINITY) ls += __expf(zz[j] - lm);      // a forbidden token (-inf) adds nothing
        const float score = greedy ? zz[j] : zz[j] - __logf(-__logf(u01(rr[j])));
        best = amax(best, ArgMax{score, i4 + j});
      }
    }
    // warps, then the first warp over theirs
    auto merge = [&] {
      const float wm = warp_max(lm);
      ls = warp_sum(lm == -INFINITY ? 0.f : ls * __expf(lm - wm));
      lm = wm;
      best = warp_amax(best);
    };
    merge();
    if ((tid & 31) == 0) {
      sh.tot[0][tid >> 5] = lm;
      sh.tot[1][tid >> 5] = ls;
      sh.s_v[tid >> 5] = best.v;
      sh.s_i[tid >> 5] = best.i;
    }
    __syncthreads();
    if (tid < 32) {
      const bool in = tid < NT / 32;
      lm = in ? sh.tot[0][tid] : -INFINITY;
      ls = in ? sh.tot[1][tid] : 0.f;
      best = in ? ArgMax{sh.s_v[tid], sh.s_i[tid]} : ArgMax{-INFINITY, 0x7fffffff};
      merge();
    }
    if (tid == 0) {                                     // read by rank 0 when it has everybody's best
      sh.part[0][0] = lm;
      sh.part[0][1] = ls;
    }
    finish(best, [&](float v) {
      float m = -INFINITY, s = 0.f;
      for (int r = 0; r < C; ++r) m = fmaxf(m, cluster.map_shared_rank(&sh, r)->part[0][0]);
      for (int r = 0; r < C; ++r) {
        const float* o = cluster.map_shared_rank(&sh, r)->part[0];
        s += o[0] == -INFINITY ? 0.f : o[1] * __expf(o[0] - m);
      }
      return v * inv_temp - m - logf(s);
    });
    return;
  }

  float lm = -INFINITY;
  walk([&](int, float v) { lm = fmaxf(lm, v); });
  for (int b = tid; b < BINS; b += nt) sh.hist[b] = 0;
  if (tid == 0) sh.ncand = 0;
  lm = block_max(lm, sh.red);
  exchange(lm, 0.f, all);                               // and rank 0's histogram is clear
  float top = -INFINITY;
  for (int r = 0; r < C; ++r) top = fmaxf(top, all[r][0]);
  const bool finite = fabsf(top * inv_temp) < INFINITY;
  constexpr float PER = BINS / BIN_SPAN;
  // Log of a token's weight: the difference to the largest logit, then the scale. It is never positive, so that a bin is never
  // negative and no weight above 1; the product first would leave its rounding, half an ulp of the maximum: 105 bins at a temperature of 1e-6.
  // Bisection and draw compare this one value: a threshold ends within 2^-26 below the weight that it was found by.
  auto below = [&](float v) { return __fmul_rn(__fadd_rn(v, -top), inv_temp); };
  float ls = 0.f;
  walk([&](int, float v) {
    const float x = below(v);
    ls += __expf(x);
    if (finite && x > -BIN_SPAN) atomicAdd(&sh.hist[min((int)(-x * PER), BINS - 1)], 1u);
  });
  ls = block_sum(ls, sh.red);
  if (rank != 0 && finite)
    for (int b = tid; b < BINS; b += nt)
      if (sh.hist[b]) atomicAdd(&sh0.hist[b], sh.hist[b]);
  exchange(ls, 0.f, all);
  float s = 0.f;
  for (int r = 0; r < C; ++r) s += all[r][0];
  const float log_s = logf(s);

  // The bins that hold what is kept: top_k tokens, or (top-p alone) about a mass of top_p * s, which is checked below. Bins that
  // reach past the last halving are as good as all: there the threshold is 0.
  if (rank == 0 && tid < 32) {
    int cut = -1;
    unsigned seen = 0;
    float mass = 0.f;
    const float want = top_p * s * 1.002f;
    for (int b0 = 0; finite && cut < 0 && b0 < BINS; b0 += 32) {
      unsigned run = sh.hist[b0 + tid];
      float run_m = (float)run * __expf(-((float)(b0 + tid) + 0.5f) / PER);
      warp_scan(run, run_m);
      const unsigned hit = __ballot_sync(0xffffffffu, by_k ? seen + run >= (unsigned)top_k : mass + run_m >= want);
      if (hit) {
        const int at = __ffs(hit) - 1 + (by_k ? 0 : 2);
        cut = min(b0 + at, BINS - 1);
        for (int b = b0 + 32; b <= cut; ++b) seen += sh.hist[b];
        seen += __shfl_sync(0xffffffffu, run, min(at, 31));
      } else {
        seen += __shfl_sync(0xffffffffu, run, 31);
        mass += __shfl_sync(0xffffffffu, run_m, 31);
      }
    }
    if (cut < 0 && finite) cut = BINS - 1;
    if (seen > (unsigned)CAND) cut = -1;
    if (tid == 0) sh.cut = cut;
  }
  csync();
  const int cut = sh0.cut;
  float thr = 0.f;
  if (cut >= 0) {
    walk([&](int i, float v) {
      const float x = below(v);
      if (x > -BIN_SPAN && min((int)(-x * PER), BINS - 1) <= cut) {
        const int at = atomicAdd(&sh0.ncand, 1);
        if (at < CAND) {
          sh0.cz[at] = v;
          sh0.ci[at] = i;
        }
      }
    });
    csync();
    const int n = min(sh.ncand, CAND);
    const int stride = min(LT, max(32, (n + 127) / 128 * 32));        // four candidates a thread, of as many warps as that takes
    const bool one = stride == 32;
    if (rank == 0 && tid < stride) {
      auto lsync = [&] { asm volatile("bar.sync 1, %0;" ::"r"(stride) : "memory"); };
      float e[4], zc[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int j = tid + k * stride;
        zc[k] = j < n ? sh.cz[j] : -INFINITY;
        e[k] = j < n ? __expf(below(zc[k])) : -1.f;     // below every threshold
      }
      int turn = 0;
      auto total = [&](unsigned long long v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (one) return v;
        if ((tid & 31) == 0) sh.sums[turn][tid >> 5] = v;
        lsync();
        v = 0;
        for (int w = 0; w < stride / 32; ++w) v += sh.sums[turn][w];
        turn ^= 1;
        return v;
      };
      // masses in units of 2^-50: whole numbers, so the order in which the list was filled leaves no trace
      auto mass_from = [&](float t) {
        unsigned long long c = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (e[k] >= t) c += (unsigned long long)(e[k] * 1125899906842624.f);
        return (double)total(c);
      };
      double kept = (double)s * 1125899906842624.0;
      float lo = 0.f, hi = 1.f;
      if (by_k) {
        for (int it = 0; it < BISECT; ++it) {           // count(e >= lo) >= k always; find the largest such lo
          const float mid = 0.5f * (lo + hi);
          int c = 0;
#pragma unroll
          for (int k = 0; k < 4; ++k) c += e[k] >= mid;
          if (total(c) >= (unsigned long long)top_k) lo = mid; else hi = mid;
        }
        if (lo > 0.f) kept = mass_from(lo);             // else fewer than top_k above the last halving: all are kept
      }
      bool held = true;
      if (by_p) {
        const double target = (double)top_p * kept;
        if (lo <= 0.f) held = mass_from(0.f) >= target; // the list has to hold the mass
        hi = 1.f;
        for (int it = 0; held && it < BISECT; ++it) {   // mass(e >= lo) >= target; find the largest such lo
          const float mid = 0.5f * (lo + hi);
          if (mass_from(mid) >= target) lo = mid; else hi = mid;
        }
      }
      if (held && lo > 0.f) {
        ArgMax best{-INFINITY, 0x7fffffff};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (e[k] < lo) continue;                      // (and what is past the list)
          const float zi = __fmul_rn(zc[k], inv_temp);
          const int i = sh.ci[tid + k * stride];
          const uint4 r = gumbel4(i & ~3);
          const int c = i & 3;
          const uint32_t u = c == 0 ? r.x : c == 1 ? r.y : c == 2 ? r.z : r.w;
          best = amax(best, ArgMax{zi - __logf(-__logf(u01(u))), i});
        }
        best = warp_amax(best);
        if (!one) {
          if ((tid & 31) == 0) {
            sh.s_v[tid >> 5] = best.v;
            sh.s_i[tid >> 5] = best.i;
          }
          lsync();
          for (int w = 0; w < stride / 32; ++w) best = amax(best, ArgMax{sh.s_v[w], sh.s_i[w]});
        }
        if (tid == 0) {
          const int tok = best.i < V ? best.i : 0;
          tokens[row] = tok;
          if (logprobs) logprobs[row] = below(z[tok]) - log_s;
        }
      } else if (tid == 0) {
        sh.cut = by_p ? -1 : -2;                        // the list is too short; or the threshold is 0 and all are drawn from
      }
    }
    csync();
    if (sh0.cut >= 0) {
      csync();                                   // rank 0's answer has been read
      return;
    }
  }

  if (cut < 0 || sh0.cut == -1) {
    // The halvings over the row. The histogram decides those whose outcome no token of the threshold's own bin (or, for the
    // rounding of the bins, its neighbours) can change: the first few of a mass, most of a count.
    if (rank == 0) {
      constexpr int G = BINS / NT;                      // groups of 32 bins of a warp
      const int lane = tid & 31;
      unsigned n[G];
      float l[G], h[G];
#pragma unroll
      for (int k = 0; k < G; ++k) {
        const int b = tid + k * NT;
        unsigned again = n[k] = sh.hist[b];
        l[k] = (float)n[k] * __expf(-(float)(b + 1) / PER);
        h[k] = (float)n[k] * __expf(-(float)b / PER);
        warp_scan(n[k], l[k]);
        warp_scan(again, h[k]);
        if (lane == 31) {
          sh.cum[b] = n[k];
          sh.low[b] = l[k];
          sh.high[b] = h[k];
        }
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < G; ++k) {                     // and what the groups before sum up to: lane g reads group g
        const bool before = lane < (tid + k * NT) >> 5;
        n[k] += __reduce_add_sync(0xffffffffu, before ? sh.cum[lane * 32 + 31] : 0u);
        l[k] += warp_sum(before ? sh.low[lane * 32 + 31] : 0.f);
        h[k] += warp_sum(before ? sh.high[lane * 32 + 31] : 0.f);
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < G; ++k) {
        sh.cum[tid + k * NT] = n[k];
        sh.low[tid + k * NT] = l[k];
        sh.high[tid + k * NT] = h[k];
      }
    }
    csync();
    // the weights of a small share stay in registers (5000 tokens, top-p alone, flat: 45 -> 26 us with the sums
    // behind one barrier)
    float held[HOLD];
    const bool hold = i1 - i0 + skew <= NT * HOLD;
    if (hold)
#pragma unroll
      for (int k = 0; k < HOLD; k += 4) {
        float q[4];
        load4(i0 - skew + (tid + k / 4 * NT) * 4, true, q);
#pragma unroll
        for (int j = 0; j < 4; ++j) held[k + j] = __expf(below(q[j]));
      }
    auto row_sum = [&](auto&& f) {
      float c = 0.f;
      if (hold) {
#pragma unroll
        for (int k = 0; k < HOLD; ++k) c += f(held[k]);
      } else {
        walk([&](int, float v) { c += f(__expf(below(v))); });
      }
      exchange(block_total(c), 0.f, all);
      float t = 0.f;
      for (int r = 0; r < C; ++r) t += all[r][0];
      return t;
    };
    auto bin_of = [&](float mid) { return (int)(-__logf(mid) * PER); };
    float kept_mass = s;
    if (by_k) {
      float lo = 0.f, hi = 1.f;
      for (int it = 0; it < BISECT; ++it) {
        const float mid = 0.5f * (lo + hi);
        const int b = bin_of(mid);
        bool more;
        if (finite && b >= 2 && sh0.cum[min(b - 2, BINS - 1)] >= (unsigned)top_k) more = true;
        else if (finite && b + 1 < BINS && sh0.cum[b + 1] < (unsigned)top_k) more = false;
        else more = row_sum([&](float e) { return e >= mid ? 1.f : 0.f; }) >= (float)top_k;
        if (more) lo = mid; else hi = mid;
      }
      thr = lo;
      kept_mass = row_sum([&](float e) { return e >= thr ? e : 0.f; });
    }
    if (by_p) {
      const float target = top_p * kept_mass;
      float lo = thr, hi = 1.f;
      for (int it = 0; it < BISECT; ++it) {
        const float mid = 0.5f * (lo + hi);
        const int b = bin_of(mid);
        bool more;
        if (finite && b >= 2 && sh0.low[min(b - 2, BINS - 1)] >= target * 1.001f) more = true;
        else if (finite && b + 1 < BINS && sh0.high[b + 1] < target * 0.999f) more = false;
        else more = row_sum([&](float e) { return e >= mid ? e : 0.f; }) >= target;
        if (more) lo = mid; else hi = mid;
      }
      thr = lo;
    }
  }
  ArgMax best{-INFINITY, 0x7fffffff};
  for (int i4 = i0 + tid * 4; i4 < i1; i4 += nt * 4) {
    float zz[4];
    load4(i4, skew == 0, zz);
    const uint4 r = gumbel4(i4);
    const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (i4 + j >= i1) break;
      if (__expf(below(zz[j])) < thr) continue;
      const float zi = __fmul_rn(zz[j], inv_temp);
      best = amax(best, ArgMax{zi - __logf(-__logf(u01(rr[j]))), i4 + j});
    }
  }
  finish(block_amax(best, sh.s_v, sh.s_i), [&](float v) { return below(v) - log_s; });
}

template <int NT>
cudaError_t launch_clusters(int B, int C, float* logits, long long ld, int V, float inv_temp, int top_k, float top_p, unsigned long long seed,
                            const unsigned long long* seed_dev, int step, const int* step_dev, int greedy, long long* tokens, float* logprobs, float softcap,
                            const int* forbidden, int n_forbidden, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((long long)B * C));
  cfg.blockDim = dim3(NT);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = tb_pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = C;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = C > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, sample_kernel<NT>, logits, ld, V, inv_temp, top_k, top_p, seed, seed_dev, step, step_dev, greedy,
                            tokens, logprobs, softcap, forbidden, n_forbidden);
}

// CTAs per row: up to 8, as long as the grid is one wave of two CTAs an SM. More CTAs shorten every pass over the row; past
// one wave they only add exchanges. In the place of two, one CTA of twice the threads needs none: 128 rows of 151,936, no filter,
// 51 us as two and 46 as one, 128 of 10,000 under top-p alone, flat, 66 and 36.
int launch_sample(float* logits, long long ld, int B, int V, float temperature, int top_k, float top_p, unsigned long long seed,
                  const unsigned long long* seed_dev, int step, const int* step_dev, long long* tokens, float* logprobs, float softcap, const int* forbidden,
                  int n_forbidden, cudaStream_t stream) {
  const int greedy = temperature <= 0.f;
  const float inv_temp = greedy ? 1.f : 1.f / temperature;
  int C = 8;
  while (C > 1 && ((long long)B * C > 296 || V < C * 4096)) C >>= 1;
  const auto run = C == 2 ? launch_clusters<1024> : launch_clusters<512>;
  return run(B, C == 2 ? 1 : C, logits, ld, V, inv_temp, top_k, top_p, seed, seed_dev, step, step_dev, greedy, tokens, logprobs,
             softcap, forbidden, n_forbidden, stream) == cudaSuccess ? 0 : -5;
}

}  // namespace

// logits fp32 [B, V] (row stride ld). tokens int64 [B]; logprobs fp32 [B] or null.
// temperature <= 0 selects greedy decoding. top_k <= 0 and top_p >= 1 disable the filters.
TB_API int tb_sample(const float* logits, long long ld, int B, int V, float temperature, int top_k, float top_p,
                     unsigned long long seed, int step, const int* step_dev, long long* tokens, float* logprobs,
                     cudaStream_t stream) {
  if (B <= 0) return 0;
  return launch_sample(const_cast<float*>(logits), ld, B, V, temperature, top_k, top_p, seed, nullptr, step, step_dev, tokens, logprobs,
                       0.f, nullptr, 0, stream);
}

// The same with the final logit soft-cap and forbidden token ids applied inside the kernel. The logits row is
// MODIFIED in place (capped values, -inf at the forbidden ids): it is the caller's scratch.
// softcap <= 0 disables the cap; forbidden: device int32 [n_forbidden] or null.
TB_API int tb_sample_ex(float* logits, long long ld, int B, int V, float temperature, int top_k, float top_p,
                        unsigned long long seed, int step, const int* step_dev, long long* tokens, float* logprobs,
                        float softcap, const int* forbidden, int n_forbidden, cudaStream_t stream) {
  if (B <= 0) return 0;
  if (n_forbidden < 0 || (n_forbidden > 0 && !forbidden)) return -2;
  return launch_sample(logits, ld, B, V, temperature, top_k, top_p, seed, nullptr, step, step_dev, tokens, logprobs, softcap, forbidden,
                       n_forbidden, stream);
}

// The same with the seed read on the device.
TB_API int tb_sample_seed(float* logits, long long ld, int B, int V, float temperature, int top_k, float top_p,
                          const unsigned long long* seed_dev, int step, const int* step_dev, long long* tokens, float* logprobs,
                          float softcap, const int* forbidden, int n_forbidden, cudaStream_t stream) {
  if (B <= 0) return 0;
  if (!seed_dev || n_forbidden < 0 || (n_forbidden > 0 && !forbidden)) return -2;
  return launch_sample(logits, ld, B, V, temperature, top_k, top_p, 0, seed_dev, step, step_dev, tokens, logprobs, softcap, forbidden,
                       n_forbidden, stream);
}
