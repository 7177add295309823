// Per-head RMS norm and rotary embedding of queries and keys in one pass, forward and backward, both tensors in one launch.
//
//   y = rotate(x * rsqrt(mean(x^2) + eps) * (w + add_one), angle(position))        without weights: y = rotate(x)
//
// The norm's own kernel and the rotation's were a pass each over queries and over keys, and a projection output that was rotated in
// place through a view cost autograd four more copies of its gradient.
// (reference: per-head norms tunix/models/qwen3/model.py, rotation tunix/models/llama3/model.py:249-270)
//
// B200, us in a graph, four launches -> one: 16384 tokens of 32 / 8 heads of 128 126 -> 83, backward 207 -> 88; 4096 tokens 36 -> 19 and 61 -> 27; 2331 of
// 14 / 2 heads of 64 10.4 -> 4.7 and 13.6 -> 6.4; without norms (two launches) 55 -> 53, 11.1 -> 9.5, 4.4 -> 3.3.
// Bound by HBM: every row read and written once (the backward reads two). A thread holds 8 pairs (x[j], x[j + H / 2]) of QK_HEADS
// heads of one token, which share the angles; H / 16 lanes make a row.
#include "common.cuh"

using namespace tb;

namespace {

constexpr int QK_HEADS = 4;

struct QkRows {                   // queries or keys: [tokens, heads * H], the heads of a token contiguous
  const __nv_bfloat16* x;
  __nv_bfloat16* y;               // may be x
  long long ldx, ldy;
  const __nv_bfloat16* w;         // [H]; null: no norm
  float* rstd;                    // [tokens * heads]
  int heads;
  int vectors;                    // rotate as the tensor's own kernel by vectors does, else as the one by pairs
  // backward
  const __nv_bfloat16* dy;
  long long lddy;
  float* dw;                      // fp32 [H], added to; null: not wanted
};
struct QkArgs {
  QkRows q, k;
  const int* pos;
  const float *cos_t, *sin_t;     // [positions, H / 2]
  unsigned tokens;
  float eps, add_one, sign;
};

__device__ __forceinline__ void unpack8(const uint4& u, float (&v)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = bf16_lo(w[i]);
    v[2 * i + 1] = bf16_hi(w[i]);
  }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
__device__ __forceinline__ uint4 ld16(const __nv_bfloat16* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void angles(const QkArgs& a, unsigned tok, int half, int j, float (&c)[8], float (&s)[8]) {
  const long long at = (long long)max(a.pos[tok], 0) * half + j;           // idle rows carry position -1
#pragma unroll
  for (int i = 0; i < 8; i += 4) {
    const float4 cv = *reinterpret_cast<const float4*>(a.cos_t + at + i), sv = *reinterpret_cast<const float4*>(a.sin_t + at + i);
    c[i] = cv.x; c[i + 1] = cv.y; c[i + 2] = cv.z; c[i + 3] = cv.w;
    s[i] = sv.x * a.sign; s[i + 1] = sv.y * a.sign; s[i + 2] = sv.z * a.sign; s[i + 3] = sv.w * a.sign;
  }
}
template <int T>
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = T / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int T, bool NORM>       // T lanes a row: H = 16 T
__global__ void __launch_bounds__(256)
qk_rope_kernel(const QkArgs a) {
  constexpr int HALF = 8 * T, PER = 256 / T;
  const unsigned gq = (a.q.heads + QK_HEADS - 1) / QK_HEADS, per = gq + (a.k.heads + QK_HEADS - 1) / QK_HEADS, total = a.tokens * per;
  const int j = (threadIdx.x % T) * 8;
  // every lane of a warp makes the same number of turns: the shuffles below need all of them
  for (unsigned u0 = blockIdx.x * PER; u0 < total; u0 += gridDim.x * PER) {
    const unsigned u = u0 + threadIdx.x / T;
    const bool live = u < total;
    const unsigned tok = live ? u / per : 0, g = u - tok * per;
    const bool is_k = g >= gq;
    const QkRows& r = is_k ? a.k : a.q;
    const int h0 = (int)(is_k ? g - gq : g) * QK_HEADS, n = live ? min(QK_HEADS, r.heads - h0) : 0;
    const __nv_bfloat16* x = r.x + (long long)tok * r.ldx + (long long)h0 * (2 * HALF) + j;
    uint4 lo[QK_HEADS], hi[QK_HEADS];
#pragma unroll
    for (int h = 0; h < QK_HEADS; ++h) {
      lo[h] = hi[h] = make_uint4(0u, 0u, 0u, 0u);
      if (h < n) {
        lo[h] = ld16(x + h * 2 * HALF);
        hi[h] = ld16(x + h * 2 * HALF + HALF);
      }
    }
    float c[8], s[8], wl[8], wh[8];
    if (live) angles(a, tok, HALF, j, c, s);
    if (NORM && live) {
      unpack8(ld16(r.w + j), wl);
      unpack8(ld16(r.w + HALF + j), wh);
    }
    __nv_bfloat16* y = r.y + (long long)tok * r.ldy + (long long)h0 * (2 * HALF) + j;
#pragma unroll
    for (int h = 0; h < QK_HEADS; ++h) {
      float p[8], q[8];
      unpack8(lo[h], p);
      unpack8(hi[h], q);
      if (NORM) {
        // in the order of the norm's own kernels, where the two halves of a row belong to lanes that meet first
        float sl = 0.f, sh = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          sl += p[i] * p[i];
          sh += q[i] * q[i];
        }
        const float rstd = rsqrtf(row_sum<T>(sl + sh) / (float)(2 * HALF) + a.eps);
        if (h < n && j == 0 && r.rstd) r.rstd[(long long)tok * r.heads + h0 + h] = rstd;
#pragma unroll
        for (int i = 0; i < 8; ++i) {      // rounded as by the norm's own kernel and by the decode step's (decode.cu), so that all agree
          p[i] = __bfloat162float(__float2bfloat16(p[i] * rstd * (wl[i] + a.add_one)));
          q[i] = __bfloat162float(__float2bfloat16(q[i] * rstd * (wh[i] + a.add_one)));
        }
      }
      if (h < n) {
        float o[8], t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          o[i] = rope_lo(p[i], q[i], c[i], s[i]);
          t[i] = rope_hi(p[i], q[i], c[i], s[i], r.vectors);
        }
        *reinterpret_cast<uint4*>(y + h * 2 * HALF) = pack8(o);
        *reinterpret_cast<uint4*>(y + h * 2 * HALF + HALF) = pack8(t);
      }
    }
  }
}

// dx = the norm's gradient of dy rotated back, dw += its weight gradient (one atomic a block and column). The first q_blocks blocks take
// queries, the others keys, so that a thread's column sums belong to one weight. a.sign is that of the forward.
template <int T>
__global__ void __launch_bounds__(256)
qk_rope_bwd_kernel(const QkArgs a, unsigned q_blocks) {
  constexpr int HALF = 8 * T, PER = 256 / T, HEADS = QK_HEADS / 2;
  __shared__ float s_dw[2 * HALF];
  const bool is_k = blockIdx.x >= q_blocks;
  const QkRows& r = is_k ? a.k : a.q;
  const unsigned block = is_k ? blockIdx.x - q_blocks : blockIdx.x, blocks = is_k ? gridDim.x - q_blocks : q_blocks;
  const unsigned per = (r.heads + HEADS - 1) / HEADS, total = a.tokens * per;
  const int j = (threadIdx.x % T) * 8;
  for (int i = threadIdx.x; i < 2 * HALF; i += 256) s_dw[i] = 0.f;
  __syncthreads();
  const uint4 wlq = ld16(r.w + j), whq = ld16(r.w + HALF + j);
  float al[8], ah[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) al[i] = ah[i] = 0.f;
  for (unsigned u0 = block * PER; u0 < total; u0 += blocks * PER) {
    const unsigned u = u0 + threadIdx.x / T;
    const bool live = u < total;
    const unsigned tok = live ? u / per : 0;
    const int h0 = (int)(u - tok * per) * HEADS, n = live ? min(HEADS, r.heads - h0) : 0;
    const long long col = (long long)h0 * (2 * HALF) + j;
    uint4 xl[HEADS], xh[HEADS], dl[HEADS], dh[HEADS];
    float rs[HEADS];
#pragma unroll
    for (int h = 0; h < HEADS; ++h) {
      xl[h] = xh[h] = dl[h] = dh[h] = make_uint4(0u, 0u, 0u, 0u);
      rs[h] = 0.f;
      if (h < n) {
        const __nv_bfloat16 *x = r.x + (long long)tok * r.ldx + col + h * 2 * HALF, *d = r.dy + (long long)tok * r.lddy + col + h * 2 * HALF;
        xl[h] = ld16(x);
        xh[h] = ld16(x + HALF);
        dl[h] = ld16(d);
        dh[h] = ld16(d + HALF);
        rs[h] = r.rstd[(long long)tok * r.heads + h0 + h];
      }
    }
    float c[8], s[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) c[i] = s[i] = 0.f;
    if (live) angles(a, tok, HALF, j, c, s);
#pragma unroll
    for (int h = 0; h < HEADS; ++h) {
      float p[8], q[8], g[8], e[8], wl[8], wh[8], dot = 0.f;
      unpack8(xl[h], p);
      unpack8(xh[h], q);
      unpack8(dl[h], g);
      unpack8(dh[h], e);
      unpack8(wlq, wl);
      unpack8(whq, wh);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float lo = g[i] * c[i] + e[i] * s[i], hi = e[i] * c[i] - g[i] * s[i];       // rotated back
        p[i] *= rs[h];
        q[i] *= rs[h];
        al[i] += lo * p[i];
        ah[i] += hi * q[i];
        g[i] = lo * (wl[i] + a.add_one);
        e[i] = hi * (wh[i] + a.add_one);
        dot += g[i] * p[i] + e[i] * q[i];
      }
      dot = row_sum<T>(dot) * (1.f / (float)(2 * HALF));
      if (h < n) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          g[i] = rs[h] * (g[i] - p[i] * dot);
          e[i] = rs[h] * (e[i] - q[i] * dot);
        }
        __nv_bfloat16* y = r.y + (long long)tok * r.ldy + col + h * 2 * HALF;
        *reinterpret_cast<uint4*>(y) = pack8(g);
        *reinterpret_cast<uint4*>(y + HALF) = pack8(e);
      }
    }
  }
  if (!r.dw) return;
#pragma unroll
  for (int o = 16; o >= T; o >>= 1)                        // the lanes of a warp that have the same columns
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      al[i] += __shfl_xor_sync(0xffffffffu, al[i], o);
      ah[i] += __shfl_xor_sync(0xffffffffu, ah[i], o);
    }
  if ((threadIdx.x & 31) < T)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      atomicAdd(s_dw + j + i, al[i]);
      atomicAdd(s_dw + HALF + j + i, ah[i]);
    }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * HALF; i += 256) atomicAdd(r.dw + i, s_dw[i]);
}

bool off16(const void* p) { return reinterpret_cast<uintptr_t>(p) & 15; }
// what both launches need: whole 16-byte pieces, and units (with a turn's step beyond the last) that 32 bits count
bool fits(const QkArgs& a, int H) {
  return (H == 64 || H == 128 || H == 256) && !off16(a.cos_t) && !off16(a.sin_t) &&
         (long long)a.tokens * (a.q.heads + a.k.heads + 8) < (1LL << 30);
}
bool rows_ok(const QkRows& r) {
  return r.heads > 0 && !off16(r.x) && !off16(r.y) && !off16(r.w) && r.ldx % 8 == 0 && r.ldy % 8 == 0;
}
unsigned blocks_for(long long units, int T, unsigned cap) {
  const long long b = (units * T + 255) / 256;
  return b < 1 ? 1u : b > cap ? cap : (unsigned)b;
}

}  // namespace

// y_q / y_k [tokens, heads * H] (may be the inputs) = rotation of q / k, behind a norm over each head where wq and wk are given (both or
// neither; rstd_q / rstd_k then take 1 / rms of every row unless null). sign -1 rotates back (without weights). Heads of 64, 128 or 256,
// 16-byte aligned rows. Returns 0, or -2 for a call that is not covered (nothing is launched).
TB_API int tb_qk_rope(const void* q, long long ldq, void* yq, long long ldyq, const void* wq, float* rstd_q, int heads_q, const void* k,
                      long long ldk, void* yk, long long ldyk, const void* wk, float* rstd_k, int heads_k, const int* pos, const float* cos_t,
                      const float* sin_t, long long tokens, int H, float eps, float add_one, int backward, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (tokens >= (1LL << 30) || (wq == nullptr) != (wk == nullptr) || (wq && backward)) return -2;
  QkArgs a = {};
  a.q = {(const __nv_bfloat16*)q, (__nv_bfloat16*)yq, ldq, ldyq, (const __nv_bfloat16*)wq, rstd_q, heads_q,
         rope_by_vectors(rope_units(tokens, heads_q, H)), nullptr, 0, nullptr};
  a.k = {(const __nv_bfloat16*)k, (__nv_bfloat16*)yk, ldk, ldyk, (const __nv_bfloat16*)wk, rstd_k, heads_k,
         rope_by_vectors(rope_units(tokens, heads_k, H)), nullptr, 0, nullptr};
  a.pos = pos; a.cos_t = cos_t; a.sin_t = sin_t; a.tokens = (unsigned)tokens; a.eps = eps; a.add_one = add_one;
  a.sign = backward ? -1.f : 1.f;
  if (!rows_ok(a.q) || !rows_ok(a.k) || !fits(a, H)) return -2;
  const long long units = tokens * ((heads_q + QK_HEADS - 1) / QK_HEADS + (heads_k + QK_HEADS - 1) / QK_HEADS);
  auto run = [&](auto plain, auto norm, int T) {
    const unsigned grid = blocks_for(units, T, 148 * 16);
    if (wq) norm<<<grid, 256, 0, stream>>>(a);
    else plain<<<grid, 256, 0, stream>>>(a);
  };
  if (H == 64) run(qk_rope_kernel<4, false>, qk_rope_kernel<4, true>, 4);
  else if (H == 128) run(qk_rope_kernel<8, false>, qk_rope_kernel<8, true>, 8);
  else run(qk_rope_kernel<16, false>, qk_rope_kernel<16, true>, 16);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// The backward of the form with norms: dxq / dxk from the gradients of the rotated rows, the rows before the norm and what the forward left
// in rstd; dwq / dwk (fp32 [H]) are added to, or null.
TB_API int tb_qk_rope_bwd(const void* dyq, long long lddyq, const void* xq, long long ldxq, const void* wq, const float* rstd_q, void* dxq,
                          long long lddxq, float* dwq, int heads_q, const void* dyk, long long lddyk, const void* xk, long long ldxk,
                          const void* wk, const float* rstd_k, void* dxk, long long lddxk, float* dwk, int heads_k, const int* pos,
                          const float* cos_t, const float* sin_t, long long tokens, int H, float add_one, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (tokens >= (1LL << 30) || !wq || !wk || !rstd_q || !rstd_k) return -2;
  QkArgs a = {};
  a.q = {(const __nv_bfloat16*)xq, (__nv_bfloat16*)dxq, ldxq, lddxq, (const __nv_bfloat16*)wq, const_cast<float*>(rstd_q), heads_q, 0,
         (const __nv_bfloat16*)dyq, lddyq, dwq};
  a.k = {(const __nv_bfloat16*)xk, (__nv_bfloat16*)dxk, ldxk, lddxk, (const __nv_bfloat16*)wk, const_cast<float*>(rstd_k), heads_k, 0,
         (const __nv_bfloat16*)dyk, lddyk, dwk};
  a.pos = pos; a.cos_t = cos_t; a.sin_t = sin_t; a.tokens = (unsigned)tokens; a.add_one = add_one; a.sign = 1.f;
  if (!rows_ok(a.q) || !rows_ok(a.k) || !fits(a, H) || off16(dyq) || off16(dyk) || lddyq % 8 || lddyk % 8) return -2;
  const long long uq = tokens * ((heads_q + 1) / 2), uk = tokens * ((heads_k + 1) / 2);
  auto run = [&](auto kernel, int T) {
    // the SMs are filled once with blocks of several turns, so that the sums over columns meet in few atomics; keys get their share
    const unsigned most = 148 * 2;
    unsigned bk = blocks_for(uk, T, max(1u, (unsigned)(most * uk / (uq + uk)))), bq = blocks_for(uq, T, most - min(most - 1, bk));
    kernel<<<bq + bk, 256, 0, stream>>>(a, bq);
  };
  if (H == 64) run(qk_rope_bwd_kernel<4>, 4);
  else if (H == 128) run(qk_rope_bwd_kernel<8>, 8);
  else run(qk_rope_bwd_kernel<16>, 16);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
