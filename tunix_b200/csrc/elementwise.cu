// Memory-bound transformer ops for sm_100a: RMSNorm, RoPE, gated activations, embedding.
// All tensors bf16 with fp32 math; 16-byte vector accesses; one warp per row for the
// row-wise ops so a row's two passes stay in L1/L2.
//
// Replaces the XLA elementwise fusions of the reference models
// (RMSNorm: tunix/models/llama3/model.py:290-297, gemma (1+w): tunix/models/gemma/model.py:730-740,
//  RoPE: tunix/models/llama3/model.py:249-270, SwiGLU/GeGLU: llama3/model.py:489-496, gemma/model.py:592-601).
#include "activation.cuh"
#include "common.cuh"

using namespace tb;

namespace {

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&v)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[2 * j] = bf16_lo(w[j]);
    v[2 * j + 1] = bf16_hi(w[j]);
  }
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&v)[8]) {
  uint4 o;
  o.x = pack_bf16(v[0], v[1]);
  o.y = pack_bf16(v[2], v[3]);
  o.z = pack_bf16(v[4], v[5]);
  o.w = pack_bf16(v[6], v[7]);
  *reinterpret_cast<uint4*>(p) = o;
}

// ------------------------------------------------------------------ RMSNorm
// y = x * rsqrt(mean(x^2) + eps) * (w + add_one). D % 8 == 0. One warp per row.
__global__ void rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, long long ldx,
                                   const __nv_bfloat16* __restrict__ w,
                                   __nv_bfloat16* __restrict__ y, long long ldy,
                                   float* __restrict__ rstd_out, int rows, int D, float eps,
                                   float add_one) {
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (long long row = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5); row < rows;
       row += (long long)gridDim.x * warps_per_block) {
    const __nv_bfloat16* xr = x + row * ldx;
    float ss = 0.f;
    for (int c = lane * 8; c < D; c += 256) {
      float v[8];
      load8(xr + c, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
    }
    ss = warp_sum(ss);
    const float rstd = rsqrtf(ss / (float)D + eps);
    if (lane == 0 && rstd_out) rstd_out[row] = rstd;
    __nv_bfloat16* yr = y + row * ldy;
    for (int c = lane * 8; c < D; c += 256) {
      float v[8], g[8];
      load8(xr + c, v);
      load8(w + c, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = v[i] * rstd * (g[i] + add_one);
      store8(yr + c, v);
    }
  }
}

// Same for many rows of at most 128 columns (the norms of single heads), which leave half of a warp idle or more: T lanes a row,
// 8 columns a lane, a row read once. B200, a warp a row -> here: 524288 x 128 95 -> 62 us, 131072 x 64 21 -> 12, 8192 x 128 3.4 -> 3.0;
// fewer rows fit one round of warps (4096 x 128 2.4, here 2.7), and rows of more columns fill them (131072 x 256 29, here 35).
template <int T>
__global__ void __launch_bounds__(256)
rmsnorm_fwd_narrow_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ w,
                          __nv_bfloat16* __restrict__ y, long long ldy, float* __restrict__ rstd_out, int rows, int D, float eps,
                          float add_one) {
  const int sub = threadIdx.x % T, col = sub * 8;
  const bool in = col < D;
  float g[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) g[i] = 0.f;
  if (in) load8(w + col, g);
#pragma unroll
  for (int i = 0; i < 8; ++i) g[i] += add_one;
  constexpr int U = 4;                                     // rows in flight per lane
  const long long step = (long long)gridDim.x * (256 / T), first = (long long)blockIdx.x * (256 / T) + threadIdx.x / T;
  for (long long r0 = first; r0 - threadIdx.x / T < rows; r0 += U * step) {
    float v[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[u][i] = 0.f;
      if (r0 + u * step < rows && in) load8(x + (r0 + u * step) * ldx + col, v[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long r = r0 + u * step;
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += v[u][i] * v[u][i];
#pragma unroll
      for (int o = T / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float rstd = rsqrtf(ss / (float)D + eps);
      if (r < rows && in) {
        if (sub == 0 && rstd_out) rstd_out[r] = rstd;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[u][i] = v[u][i] * rstd * g[i];
        store8(y + r * ldy + col, v[u]);
      }
    }
  }
}

// Same, one CTA per row: with few rows (decode) the warp-per-row kernel is a handful of warps each walking a
// whole row twice, and latency, not bandwidth, sets its time. The row is held in registers between the passes.
template <int VPT>   // 8-element vectors per thread
__global__ void __launch_bounds__(128)
rmsnorm_fwd_row_kernel(const __nv_bfloat16* __restrict__ x, long long ldx, const __nv_bfloat16* __restrict__ w,
                       __nv_bfloat16* __restrict__ y, long long ldy, float* __restrict__ rstd_out, int D, float eps,
                       float add_one) {
  __shared__ float red[33];
  pdl_trigger();
  pdl_wait();
  const long long row = blockIdx.x;
  const __nv_bfloat16* xr = x + row * ldx;
  float v[VPT][8];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int c = (threadIdx.x + j * 128) * 8;
    if (c < D) {
      load8(xr + c, v[j]);
#pragma unroll
      for (int i = 0; i < 8; ++i) ss += v[j][i] * v[j][i];
    }
  }
  ss = block_sum(ss, red);
  const float rstd = rsqrtf(ss / (float)D + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
  __nv_bfloat16* yr = y + row * ldy;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int c = (threadIdx.x + j * 128) * 8;
    if (c < D) {
      float g[8];
      load8(w + c, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[j][i] = v[j][i] * rstd * (g[i] + add_one);
      store8(yr + c, v[j]);
    }
  }
}

// dx = rstd * (dy*w' - xhat * mean(dy*w'*xhat)) (+ add: the residual stream's gradient, or dx itself), xhat = x*rstd, w' = w + add_one, and
// dw[c] += sum_rows dy[r,c] * x[r,c] * rstd[r] (fp32 atomics into a zeroed buffer), in one pass over x and dy: a row is held in
// registers between its reduction and its dx, and a thread keeps the sums of its columns over all its rows.
//
// Bound by HBM: x, dy and dx once each. B200, dx and dw together, before (two kernels, three passes over x and dy) -> after:
// 524288 x 128 686 -> 120 us, 16384 x 4096 214 -> 99, 8192 x 4096 109 -> 54, 4096 x 4096 51 -> 30, 2048 x 896 10.5 -> 9.1,
// 4096 x 512 10.3 -> 8.8, 4096 x 64 7.5 -> 4.4 (8.4 without the sums over the lanes of a warp in front of the atomics).
__device__ __forceinline__ void add4(float* p, float a, float b, float c, float d) {     // p: 16-byte aligned
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// Rows of at most 256 columns (the norms of single heads): T lanes a row, 8 columns a lane.
template <int T>
__global__ void __launch_bounds__(256)
rmsnorm_bwd_narrow_kernel(const __nv_bfloat16* __restrict__ dy, long long lddy, const __nv_bfloat16* __restrict__ x, long long ldx,
                          const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx,
                          long long lddx, float* __restrict__ dw, int rows, int D, float add_one, const __nv_bfloat16* add, long long ldadd) {
  __shared__ float s_dw[T * 8];
  const int sub = threadIdx.x % T, col = sub * 8;
  const bool in = col < D;
  for (int i = threadIdx.x; i < T * 8; i += blockDim.x) s_dw[i] = 0.f;
  __syncthreads();
  float g[8], acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) g[i] = acc[i] = 0.f;
  if (in) load8(w + col, g);
#pragma unroll
  for (int i = 0; i < 8; ++i) g[i] += add_one;
  const float inv_d = 1.f / (float)D;
  constexpr int U = 2;                                     // rows in flight per lane
  const long long step = (long long)gridDim.x * (256 / T), first = (long long)blockIdx.x * (256 / T) + threadIdx.x / T;
  // every lane of a warp makes the same number of turns: the shuffles below need all of them
  for (long long r0 = first; r0 - threadIdx.x / T < rows; r0 += U * step) {
    float v[U][8], d[U][8], rs[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long r = r0 + u * step;
      rs[u] = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) v[u][i] = d[u][i] = 0.f;
      if (r < rows && in) {
        load8(x + r * ldx + col, v[u]);
        load8(dy + r * lddy + col, d[u]);
        rs[u] = rstd_in[r];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long r = r0 + u * step;
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[u][i] *= rs[u];
        acc[i] += d[u][i] * v[u][i];
        d[u][i] *= g[i];
        dot += d[u][i] * v[u][i];
      }
#pragma unroll
      for (int o = T / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      dot *= inv_d;
      if (r < rows && in) {
        float o[8];
        if (add) load8(add + r * ldadd + col, o);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float t = rs[u] * (d[u][i] - v[u][i] * dot);
          o[i] = add ? o[i] + t : t;
        }
        store8(dx + r * lddx + col, o);
      }
    }
  }
  if (!dw) return;
#pragma unroll
  for (int o = 16; o >= T; o >>= 1)                        // the lanes of a warp that have the same columns
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], o);
  if (in && (threadIdx.x & 31) < T)
#pragma unroll
    for (int i = 0; i < 8; ++i) atomicAdd(s_dw + col + i, acc[i]);
  __syncthreads();
  for (int i = threadIdx.x; i < D; i += blockDim.x) atomicAdd(dw + i, s_dw[i]);
}

// Wider rows: up to 512 threads a row, VPT vectors of 8 columns a thread; the next row is loaded before the sum of this one is
// formed. The groups of threads of a block (threadIdx.y) walk over rows of their own, and their column sums meet in shared memory
// before they leave as one atomic a block and column.
constexpr int RMS_GROUPS = 8;
template <int VPT>
__global__ void __launch_bounds__(VPT == 1 ? 1024 : 512, 1)
rmsnorm_bwd_row_kernel(const __nv_bfloat16* __restrict__ dy, long long lddy, const __nv_bfloat16* __restrict__ x, long long ldx,
                       const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd_in, __nv_bfloat16* __restrict__ dx,
                       long long lddx, float* __restrict__ dw, int rows, int D, float add_one, const __nv_bfloat16* add, long long ldadd) {
  __shared__ float red[RMS_GROUPS][2][16];
  extern __shared__ float s_dw[];                          // [D]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, grp = threadIdx.y;
  constexpr int AHEAD = VPT == 1 ? 2 : 1;                  // rows that are loaded before their turn
  float acc[VPT][8], ns[AHEAD];
  uint4 nx[AHEAD][VPT], nd[AHEAD][VPT], wq[VPT];
  auto col = [&](int j) { return (int)(threadIdx.x + j * blockDim.x) * 8; };
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[j][i] = 0.f;
    wq[j] = col(j) < D ? *reinterpret_cast<const uint4*>(w + col(j)) : make_uint4(0u, 0u, 0u, 0u);
  }
  auto fetch = [&](long long r, uint4 (&fx)[VPT], uint4 (&fd)[VPT], float& fs) {
    fs = r < rows ? rstd_in[r] : 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      fx[j] = fd[j] = make_uint4(0u, 0u, 0u, 0u);
      if (r < rows && col(j) < D) {
        fx[j] = *reinterpret_cast<const uint4*>(x + r * ldx + col(j));
        fd[j] = *reinterpret_cast<const uint4*>(dy + r * lddy + col(j));
      }
    }
  };
  auto unpack = [](const uint4& q, float (&v)[8]) {
    const uint32_t t[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = bf16_lo(t[i]);
      v[2 * i + 1] = bf16_hi(t[i]);
    }
  };
  const float inv_d = 1.f / (float)D;
  int turn = 0;
  const long long first = (long long)blockIdx.x * blockDim.y + grp, step = (long long)gridDim.x * blockDim.y;
#pragma unroll
  for (int q = 0; q < AHEAD; ++q) fetch(first + q * step, nx[q], nd[q], ns[q]);
  for (long long r = first; r < rows; r += step, turn ^= 1) {
    constexpr int EARLY = VPT <= 2 ? VPT : 1;              // of `add`: wider rows have no registers left for it
    uint4 cx[VPT], cd[VPT], ca[EARLY];
    const float rs = ns[0];
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      cx[j] = nx[0][j];
      cd[j] = nd[0][j];
      if (j < EARLY) ca[j] = add && col(j) < D ? *reinterpret_cast<const uint4*>(add + r * ldadd + col(j)) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int q = 0; q + 1 < AHEAD; ++q) {
      ns[q] = ns[q + 1];
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        nx[q][j] = nx[q + 1][j];
        nd[q][j] = nd[q + 1][j];
      }
    }
    fetch(r + AHEAD * step, nx[AHEAD - 1], nd[AHEAD - 1], ns[AHEAD - 1]);
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      if (col(j) >= D) continue;
      float v[8], d[8], g[8];
      unpack(cx[j], v);
      unpack(cd[j], d);
      unpack(wq[j], g);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float p = d[i] * (v[i] * rs);
        acc[j][i] += p;
        dot += p * (g[i] + add_one);
      }
    }
    dot = warp_sum(dot);
    if (lane == 0) red[grp][turn][warp] = dot;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"((int)blockDim.x) : "memory");   // of the group; the other buffer is next
    dot = 0.f;
    for (int i = 0; i < nw; ++i) dot += red[grp][turn][i];
    dot *= inv_d;
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      if (col(j) >= D) continue;
      float v[8], d[8], g[8], o[8];
      unpack(cx[j], v);
      unpack(cd[j], d);
      unpack(wq[j], g);
      if (j < EARLY) {
        unpack(ca[j], o);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = 0.f;
        if (add) load8(add + r * ldadd + col(j), o);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] += rs * (d[i] * (g[i] + add_one) - v[i] * rs * dot);
      store8(dx + r * lddx + col(j), o);
    }
  }
  if (!dw) return;
  for (int g = 0; g < (int)blockDim.y; ++g) {
    if (grp == g) {
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        if (col(j) >= D) continue;
        float4* d = reinterpret_cast<float4*>(s_dw + col(j));
        float4 lo = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
        float4 hi = make_float4(acc[j][4], acc[j][5], acc[j][6], acc[j][7]);
        if (g > 0) {
          lo.x += d[0].x; lo.y += d[0].y; lo.z += d[0].z; lo.w += d[0].w;
          hi.x += d[1].x; hi.y += d[1].y; hi.z += d[1].z; hi.w += d[1].w;
        }
        if (g + 1 < (int)blockDim.y) {
          d[0] = lo;
          d[1] = hi;
        } else {
          add4(dw + col(j), lo.x, lo.y, lo.z, lo.w);
          add4(dw + col(j) + 4, hi.x, hi.y, hi.z, hi.w);
        }
      }
    }
    __syncthreads();
  }
}

// The same in two kernels: for rows too wide for the registers of a block, for most calls without dw, and for dw alone (x and dy
// 4-byte aligned, no w).
__global__ void rmsnorm_bwd_dx_kernel(const __nv_bfloat16* __restrict__ dy, long long lddy,
                                      const __nv_bfloat16* __restrict__ x, long long ldx,
                                      const __nv_bfloat16* __restrict__ w,
                                      const float* __restrict__ rstd_in,
                                      __nv_bfloat16* __restrict__ dx, long long lddx, int rows,
                                      int D, float add_one, const __nv_bfloat16* add, long long ldadd) {
  const int warps_per_block = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (long long row = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5); row < rows;
       row += (long long)gridDim.x * warps_per_block) {
    const __nv_bfloat16* xr = x + row * ldx;
    const __nv_bfloat16* dyr = dy + row * lddy;
    const float rstd = rstd_in[row];
    float dot = 0.f;
    for (int c = lane * 8; c < D; c += 256) {
      float v[8], g[8], d[8];
      load8(xr + c, v);
      load8(w + c, g);
      load8(dyr + c, d);
#pragma unroll
      for (int i = 0; i < 8; ++i) dot += d[i] * (g[i] + add_one) * v[i] * rstd;
    }
    dot = warp_sum(dot) / (float)D;
    __nv_bfloat16* dxr = dx + row * lddx;
    for (int c = lane * 8; c < D; c += 256) {
      float v[8], g[8], d[8], o[8];
      load8(xr + c, v);
      load8(w + c, g);
      load8(dyr + c, d);
      if (add) load8(add + row * ldadd + c, o);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float r = rstd * (d[i] * (g[i] + add_one) - v[i] * rstd * dot);
        o[i] = add ? o[i] + r : r;
      }
      store8(dxr + c, o);
    }
  }
}

// dw[c] += sum_rows dy[r,c] * x[r,c] * rstd[r]   (fp32 atomics into a zeroed buffer)
__global__ void rmsnorm_bwd_dw_kernel(const __nv_bfloat16* __restrict__ dy, long long lddy,
                                      const __nv_bfloat16* __restrict__ x, long long ldx,
                                      const float* __restrict__ rstd_in, float* __restrict__ dw,
                                      int rows, int D) {
  __shared__ float red[4][128];
  const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;  // 64 x 4
  const int col = blockIdx.x * 128 + tx * 2;
  float a0 = 0.f, a1 = 0.f;
  if (col < D) {
    for (long long r = (long long)blockIdx.y * 4 + ty; r < rows; r += (long long)gridDim.y * 4) {
      uint32_t dv = *reinterpret_cast<const uint32_t*>(dy + r * lddy + col);
      uint32_t xv = *reinterpret_cast<const uint32_t*>(x + r * ldx + col);
      const float rs = rstd_in[r];
      a0 += bf16_lo(dv) * bf16_lo(xv) * rs;
      a1 += bf16_hi(dv) * bf16_hi(xv) * rs;
    }
  }
  red[ty][tx * 2] = a0;
  red[ty][tx * 2 + 1] = a1;
  __syncthreads();
  if (ty == 0 && col < D) {
    float s0 = red[0][tx * 2] + red[1][tx * 2] + red[2][tx * 2] + red[3][tx * 2];
    float s1 = red[0][tx * 2 + 1] + red[1][tx * 2 + 1] + red[2][tx * 2 + 1] + red[3][tx * 2 + 1];
    atomicAdd(dw + col, s0);
    atomicAdd(dw + col + 1, s1);
  }
}

// --------------------------------------------------------------------- RoPE
// In-place half-split rotation on x[tokens, heads, H] (row stride ld between tokens, heads
// contiguous). cos/sin tables are [max_pos, H/2] fp32; pos[token] selects the row.
// sign = +1 forward, -1 backward (the transpose of a rotation is the opposite rotation).
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, long long ld, const int* __restrict__ pos,
                            const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                            long long tokens, int heads, int H, float sign) {
  const int half = H >> 1;
  const int pairs_per_token = heads * (half >> 1);  // each thread rotates 2 adjacent pairs
  const long long total = tokens * pairs_per_token;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long tok = i / pairs_per_token;
    const int rem = (int)(i - tok * pairs_per_token);
    const int h = rem / (half >> 1);
    const int j = (rem - h * (half >> 1)) * 2;
    const int p = max(pos[tok], 0);                        // idle rows carry position -1
    const float2 c = *reinterpret_cast<const float2*>(cos_t + (long long)p * half + j);
    float2 s = *reinterpret_cast<const float2*>(sin_t + (long long)p * half + j);
    s.x *= sign;
    s.y *= sign;
    __nv_bfloat16* base = x + tok * ld + (long long)h * H;
    uint32_t lo = *reinterpret_cast<uint32_t*>(base + j);
    uint32_t hi = *reinterpret_cast<uint32_t*>(base + half + j);
    const float a0 = bf16_lo(lo), a1 = bf16_hi(lo), b0 = bf16_lo(hi), b1 = bf16_hi(hi);
    *reinterpret_cast<uint32_t*>(base + j) = pack_bf16(rope_lo(a0, b0, c.x, s.x), rope_lo(a1, b1, c.y, s.y));
    *reinterpret_cast<uint32_t*>(base + half + j) = pack_bf16(rope_hi(a0, b0, c.x, s.x, false), rope_hi(a1, b1, c.y, s.y, false));
  }
}

// The same with 16-byte accesses: a thread rotates 8 pairs of ROPE_HEADS heads of a token by the same angles. Bound by HBM: x read
// and written once. B200, before -> after: 16384 x 32 x 128 79 -> 46 us, 4096 x 32 x 128 22 -> 14, 4004 x 16 x 256 21 -> 14.
__global__ void __launch_bounds__(256)
rope_vec_kernel(__nv_bfloat16* __restrict__ x, long long ld, const int* __restrict__ pos, const float* __restrict__ cos_t,
                const float* __restrict__ sin_t, unsigned total, int heads, int H, float sign) {
  const int half = H >> 1;
  const unsigned vecs = half >> 3, per_token = vecs * ((heads + ROPE_HEADS - 1) / ROPE_HEADS);
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const unsigned tok = i / per_token, rem = i - tok * per_token, grp = rem / vecs;
    const int j = (int)(rem - grp * vecs) << 3, h0 = (int)grp * ROPE_HEADS;
    __nv_bfloat16* base = x + (long long)tok * ld + (long long)h0 * H + j;
    uint4 lo[ROPE_HEADS], hi[ROPE_HEADS];
#pragma unroll
    for (int h = 0; h < ROPE_HEADS; ++h)
      if (h0 + h < heads) {
        lo[h] = *reinterpret_cast<const uint4*>(base + h * H);
        hi[h] = *reinterpret_cast<const uint4*>(base + h * H + half);
      }
    float c[8], s[8];
    const long long at = (long long)max(pos[tok], 0) * half + j;    // idle rows carry position -1
#pragma unroll
    for (int k = 0; k < 8; k += 4) {
      const float4 cv = *reinterpret_cast<const float4*>(cos_t + at + k), sv = *reinterpret_cast<const float4*>(sin_t + at + k);
      c[k] = cv.x; c[k + 1] = cv.y; c[k + 2] = cv.z; c[k + 3] = cv.w;
      s[k] = sv.x * sign; s[k + 1] = sv.y * sign; s[k + 2] = sv.z * sign; s[k + 3] = sv.w * sign;
    }
#pragma unroll
    for (int h = 0; h < ROPE_HEADS; ++h) {
      if (h0 + h >= heads) break;
      uint32_t a[4] = {lo[h].x, lo[h].y, lo[h].z, lo[h].w}, b[4] = {hi[h].x, hi[h].y, hi[h].z, hi[h].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float a0 = bf16_lo(a[k]), a1 = bf16_hi(a[k]), b0 = bf16_lo(b[k]), b1 = bf16_hi(b[k]);
        a[k] = pack_bf16(rope_lo(a0, b0, c[2 * k], s[2 * k]), rope_lo(a1, b1, c[2 * k + 1], s[2 * k + 1]));
        b[k] = pack_bf16(rope_hi(a0, b0, c[2 * k], s[2 * k], true), rope_hi(a1, b1, c[2 * k + 1], s[2 * k + 1], true));
      }
      *reinterpret_cast<uint4*>(base + h * H) = make_uint4(a[0], a[1], a[2], a[3]);
      *reinterpret_cast<uint4*>(base + h * H + half) = make_uint4(b[0], b[1], b[2], b[3]);
    }
  }
}

// ------------------------------------------------------------- gated activation (act_fwd, act_bwd: activation.cuh)
// h = act(g) * u ; all [rows, F] with row strides. F % 8 == 0.
__global__ void glu_fwd_kernel(const __nv_bfloat16* __restrict__ g, long long ldg,
                               const __nv_bfloat16* __restrict__ u, long long ldu,
                               __nv_bfloat16* __restrict__ h, long long ldh, long long rows, int F,
                               int kind) {
  pdl_trigger();
  pdl_wait();
  const int vec_per_row = F >> 3;
  const long long total = rows * vec_per_row;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vec_per_row;
    const int c = (int)(i - r * vec_per_row) << 3;
    float a[8], b[8];
    load8(g + r * ldg + c, a);
    load8(u + r * ldu + c, b);
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = act_fwd(a[k], kind) * b[k];
    store8(h + r * ldh + c, a);
  }
}
// dg = dh * u * act'(g) ; du = dh * act(g). dg/du may alias g/u (in-place).
__global__ void glu_bwd_kernel(const __nv_bfloat16* __restrict__ dh, long long lddh,
                               const __nv_bfloat16* g, long long ldg, const __nv_bfloat16* u,
                               long long ldu, __nv_bfloat16* dg, long long lddg, __nv_bfloat16* du,
                               long long lddu, long long rows, int F, int kind) {
  const int vec_per_row = F >> 3;
  const long long total = rows * vec_per_row;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vec_per_row;
    const int c = (int)(i - r * vec_per_row) << 3;
    float a[8], b[8], d[8], og[8], ou[8];
    load8(g + r * ldg + c, a);
    load8(u + r * ldu + c, b);
    load8(dh + r * lddh + c, d);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      og[k] = d[k] * b[k] * act_bwd(a[k], kind);
      ou[k] = d[k] * act_fwd(a[k], kind);
    }
    store8(dg + r * lddg + c, og);
    store8(du + r * lddu + c, ou);
  }
}

// ---------------------------------------------------------------- embedding
// out[t, :] = table[ids[t], :] * scale
__global__ void embedding_fwd_kernel(const int* __restrict__ ids,
                                     const __nv_bfloat16* __restrict__ table, long long ldt,
                                     __nv_bfloat16* __restrict__ out, long long ldo,
                                     long long tokens, int D, int vocab, float scale) {
  pdl_trigger();
  pdl_wait();
  const int vec_per_row = D >> 3;
  const long long total = tokens * vec_per_row;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vec_per_row;
    const int c = (int)(i - t * vec_per_row) << 3;
    int id = ids[t];
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    float v[8];
    load8(table + (long long)id * ldt + c, v);
    if (scale != 1.f) {
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] *= scale;
    }
    store8(out + t * ldo + c, v);
  }
}
// dtable[ids[t], :] += dout[t, :] * scale: 16-byte reductions, the rows of a 32-bit table without a bf16 copy of it.
// Bound by HBM: dout once, and the reductions' rows, of which L2 holds a part. B200, bf16 table, 32-bit pairs before:
// 16384 x 4096 124 -> 60 us. A 32-bit table took a zeroed bf16 copy, a cast and a sum of the whole vocabulary (32768 x 4096: 0.74 ms)
// where it takes 28 us for 4096 tokens now.
template <typename T>
__global__ void embedding_bwd_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ dout, long long ldo,
                                     T* __restrict__ dtable, long long ldt, long long tokens, int D, int vocab, float scale) {
  const int vec_per_row = D >> 3;
  const long long total = tokens * vec_per_row;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vec_per_row;
    const int c = (int)(i - t * vec_per_row) << 3;
    const int id = ids[t];
    if (id < 0 || id >= vocab) continue;
    float v[8];
    load8(dout + t * ldo + c, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] *= scale;
    T* p = dtable + (long long)id * ldt + c;
    if constexpr (sizeof(T) == 4) {
      add4(p, v[0], v[1], v[2], v[3]);
      add4(p + 4, v[4], v[5], v[6], v[7]);
    } else {
      asm volatile("red.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(pack_bf16(v[0], v[1])),
                   "r"(pack_bf16(v[2], v[3])), "r"(pack_bf16(v[4], v[5])), "r"(pack_bf16(v[6], v[7])) : "memory");
    }
  }
}
// The same by pairs, for rows that are not whole 16-byte pieces.
template <typename T>
__global__ void embedding_bwd_pairs_kernel(const int* __restrict__ ids, const __nv_bfloat16* __restrict__ dout, long long ldo,
                                           T* __restrict__ dtable, long long ldt, long long tokens, int D, int vocab, float scale) {
  const int pairs = D >> 1;
  const long long total = tokens * pairs;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / pairs;
    const int c = (int)(i - t * pairs) << 1;
    const int id = ids[t];
    if (id < 0 || id >= vocab) continue;
    const uint32_t d = *reinterpret_cast<const uint32_t*>(dout + t * ldo + c);
    T* p = dtable + (long long)id * ldt + c;
    if constexpr (sizeof(T) == 4) {
      atomicAdd(p, bf16_lo(d) * scale);
      atomicAdd(p + 1, bf16_hi(d) * scale);
    } else {
      atomicAdd(reinterpret_cast<__nv_bfloat162*>(p), __floats2bfloat162_rn(bf16_lo(d) * scale, bf16_hi(d) * scale));
    }
  }
}

// y = a + b (bf16), n % 8 == 0
__global__ void add_kernel(const __nv_bfloat16* a, const __nv_bfloat16* b, __nv_bfloat16* y,
                           long long n) {
  for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8; i < n;
       i += (long long)gridDim.x * blockDim.x * 8) {
    float x[8], z[8];
    load8(a + i, x);
    load8(b + i, z);
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] += z[k];
    store8(y + i, x);
  }
}

inline int grid_for(long long work_items, int block, int cap = 148 * 16) {
  long long g = (work_items + block - 1) / block;
  if (g < 1) g = 1;
  return (int)(g > cap ? cap : g);
}

}  // namespace

TB_API int tb_rmsnorm_fwd(const void* x, long long ldx, const void* w, void* y, long long ldy,
                          float* rstd, int rows, int D, float eps, float add_one,
                          cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D % 8) return -2;
  if (rows <= 2048 && D >= 1024 && D <= 8192) {
    auto xx = (const __nv_bfloat16*)x;
    auto ww = (const __nv_bfloat16*)w;
    auto yy = (__nv_bfloat16*)y;
    cudaError_t e;
    if (D <= 2048) e = launch_pdl(rmsnorm_fwd_row_kernel<2>, dim3(rows), dim3(128), 0, stream, xx, ldx, ww, yy, ldy, rstd, D, eps, add_one);
    else if (D <= 4096) e = launch_pdl(rmsnorm_fwd_row_kernel<4>, dim3(rows), dim3(128), 0, stream, xx, ldx, ww, yy, ldy, rstd, D, eps, add_one);
    else e = launch_pdl(rmsnorm_fwd_row_kernel<8>, dim3(rows), dim3(128), 0, stream, xx, ldx, ww, yy, ldy, rstd, D, eps, add_one);
    return e == cudaSuccess ? 0 : -5;
  }
  const int block = 256;
  if (D <= 128 && rows >= 8192) {
    const int t = D <= 64 ? 8 : 16;
    const int grid = grid_for((long long)rows * t, 256 * 2, 148 * 16);
    auto run = [&](auto kernel) {
      kernel<<<grid, 256, 0, stream>>>((const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)w, (__nv_bfloat16*)y, ldy, rstd, rows, D, eps,
                                       add_one);
    };
    if (t == 8) run(rmsnorm_fwd_narrow_kernel<8>);
    else run(rmsnorm_fwd_narrow_kernel<16>);
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
  }
  rmsnorm_fwd_kernel<<<grid_for((long long)rows * 32, block), block, 0, stream>>>(
      (const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)w, (__nv_bfloat16*)y, ldy, rstd, rows, D,
      eps, add_one);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// add: null, or [rows, D] bf16 (row stride ldadd, 16-byte pieces) that dx takes on top, dx itself among them
TB_API int tb_rmsnorm_bwd_add(const void* dy, long long lddy, const void* x, long long ldx,
                          const void* w, const float* rstd, void* dx, long long lddx, float* dw,
                          int rows, int D, float add_one, const void* add, long long ldadd, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D % 8) return -2;
  if (!dx && !dw) return 0;
  // dx and dw: up to 256 columns by lanes of a warp, up to 16384 by threads of a block; the SMs are filled once, so that the sums over
  // columns meet in few atomics (a second block an SM pays from 16384 rows on: 4096 x 512 11.6 us with two, 8.8 with one, 16384 x 512
  // 17.6 and 18.2).
  // dx alone gains nothing from sums that stay in registers; a warp a row / here, us: 16384 x 1536 34 / 38, 4096 x 2304 12.2 / 16.6,
  // 524288 x 256 151 / 226, 4096 x 16384 123 / 156. It comes here where a warp a row is too few warps or too wide a
  // row for their registers (128 x 4096 8.1 / 4.1, 4096 x 8192 64 / 39, 16384 x 4096 109 / 97), or leaves half of it idle (524288 x 128 142 / 116).
  // dw alone needs no weight and no rows of 16-byte pieces: that call keeps the kernel for wide rows.
#define RMS_BWD_ARGS                                                                                                          \
  (const __nv_bfloat16*)dy, lddy, (const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)w, rstd, (__nv_bfloat16*)dx, lddx, dw, rows, D, \
      add_one, (const __nv_bfloat16*)add, ldadd
  const bool narrow = dx && (dw ? D <= 256 : D <= 128 && rows >= 4096);
  const bool fits = dx && D > 256 && D <= 16384;
  const bool by_row = dw ? fits && !(reinterpret_cast<uintptr_t>(dw) & 15)
                         : fits && D > 2048 && (rows <= 512 || (D > 4096 ? D <= 8192 || rows <= 2048 : D > 3072 && rows >= 8192));
  if (!narrow && !by_row) {
    const int block = 256;
    if (dx)
      rmsnorm_bwd_dx_kernel<<<grid_for((long long)rows * 32, block), block, 0, stream>>>(
          (const __nv_bfloat16*)dy, lddy, (const __nv_bfloat16*)x, ldx, (const __nv_bfloat16*)w, rstd,
          (__nv_bfloat16*)dx, lddx, rows, D, add_one, (const __nv_bfloat16*)add, ldadd);
    if (dw) {
      dim3 grid((D + 127) / 128, (unsigned)min(128, (rows + 3) / 4));
      rmsnorm_bwd_dw_kernel<<<grid, 256, 0, stream>>>((const __nv_bfloat16*)dy, lddy,
                                                      (const __nv_bfloat16*)x, ldx, rstd, dw, rows, D);
    }
  } else if (narrow) {
    const int t = D <= 64 ? 8 : D <= 128 ? 16 : 32;
    // four rows a lane once that fills the SMs
    const int grid = max(grid_for((long long)rows * t, 256 * 4, 148 * 6), grid_for((long long)rows * t, 256, 148));
    if (t == 8) rmsnorm_bwd_narrow_kernel<8><<<grid, 256, 0, stream>>>(RMS_BWD_ARGS);
    else if (t == 16) rmsnorm_bwd_narrow_kernel<16><<<grid, 256, 0, stream>>>(RMS_BWD_ARGS);
    else rmsnorm_bwd_narrow_kernel<32><<<grid, 256, 0, stream>>>(RMS_BWD_ARGS);
  } else {
    const int vecs = D / 8, vpt = vecs <= 512 ? 1 : vecs <= 1024 ? 2 : 4;
    const int threads = ((vecs + vpt - 1) / vpt + 31) / 32 * 32, most = vpt == 1 ? 1024 : 512;
    const int groups = min(RMS_GROUPS, most / threads);
    const int grid = min((rows + groups - 1) / groups, 148 * (rows >= 16384 ? most / (threads * groups) : 1));
    const dim3 block(threads, groups);
    const size_t smem = groups > 1 ? (size_t)D * 4 : 0;      // at most 16 KB: more than one group has at most 4096 columns
    if (vpt == 1) rmsnorm_bwd_row_kernel<1><<<grid, block, smem, stream>>>(RMS_BWD_ARGS);
    else if (vpt == 2) rmsnorm_bwd_row_kernel<2><<<grid, block, smem, stream>>>(RMS_BWD_ARGS);
    else rmsnorm_bwd_row_kernel<4><<<grid, block, smem, stream>>>(RMS_BWD_ARGS);
  }
#undef RMS_BWD_ARGS
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

TB_API int tb_rmsnorm_bwd(const void* dy, long long lddy, const void* x, long long ldx, const void* w, const float* rstd, void* dx,
                          long long lddx, float* dw, int rows, int D, float add_one, int accumulate_dx, cudaStream_t stream) {
  return tb_rmsnorm_bwd_add(dy, lddy, x, ldx, w, rstd, dx, lddx, dw, rows, D, add_one, accumulate_dx ? dx : nullptr, lddx, stream);
}

TB_API int tb_rope(void* x, long long ld, const int* pos, const float* cos_t, const float* sin_t,
                   long long tokens, int heads, int H, int backward, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (H % 4) return -2;
  const long long units = rope_units(tokens, heads, H);
  // whole 16-byte pieces of both halves; a unit's number, and a turn's step beyond the last, fit 32 bits. Fewer units than these are
  // one short round of either kernel, of which the one by pairs has more threads (64 x 32 heads of 128, 4096 units: 2.2 us, 2.5 by
  // vectors; 256 x 32, 16384 units: 3.4, 2.7).
  if (rope_by_vectors(units) && H % 16 == 0 && ld % 8 == 0 &&
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(cos_t) | reinterpret_cast<uintptr_t>(sin_t)) & 15) == 0) {
    rope_vec_kernel<<<grid_for(units, 256), 256, 0, stream>>>((__nv_bfloat16*)x, ld, pos, cos_t, sin_t, (unsigned)units, heads, H,
                                                              backward ? -1.f : 1.f);
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
  }
  const long long total = tokens * heads * (H / 4);
  rope_kernel<<<grid_for(total, 256), 256, 0, stream>>>((__nv_bfloat16*)x, ld, pos, cos_t, sin_t,
                                                       tokens, heads, H, backward ? -1.f : 1.f);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

TB_API int tb_glu_fwd(const void* g, long long ldg, const void* u, long long ldu, void* h,
                      long long ldh, long long rows, int F, int kind, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (F % 8) return -2;
  return launch_pdl(glu_fwd_kernel, dim3(grid_for(rows * (F / 8), 256)), dim3(256), 0, stream, (const __nv_bfloat16*)g, ldg,
                    (const __nv_bfloat16*)u, ldu, (__nv_bfloat16*)h, ldh, rows, F, kind) == cudaSuccess ? 0 : -5;
}

TB_API int tb_glu_bwd(const void* dh, long long lddh, const void* g, long long ldg, const void* u,
                      long long ldu, void* dg, long long lddg, void* du, long long lddu,
                      long long rows, int F, int kind, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (F % 8) return -2;
  glu_bwd_kernel<<<grid_for(rows * (F / 8), 256), 256, 0, stream>>>(
      (const __nv_bfloat16*)dh, lddh, (const __nv_bfloat16*)g, ldg, (const __nv_bfloat16*)u, ldu,
      (__nv_bfloat16*)dg, lddg, (__nv_bfloat16*)du, lddu, rows, F, kind);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

TB_API int tb_embedding_fwd(const int* ids, const void* table, long long ldt, void* out,
                            long long ldo, long long tokens, int D, int vocab, float scale,
                            cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (D % 8) return -2;
  return launch_pdl(embedding_fwd_kernel, dim3(grid_for(tokens * (D / 8), 256)), dim3(256), 0, stream, ids,
                    (const __nv_bfloat16*)table, ldt, (__nv_bfloat16*)out, ldo, tokens, D, vocab, scale) == cudaSuccess ? 0 : -5;
}

namespace {
template <typename T>
int launch_embedding_bwd(const int* ids, const void* dout, long long ldo, void* dtable, long long ldt, long long tokens, int D,
                         int vocab, float scale, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (D % 2) return -2;
  const bool vec = D % 8 == 0 && ldo % 8 == 0 && ldt % 8 == 0 &&
                   ((reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dtable)) & 15) == 0;
  auto run = [&](auto kernel, int per) {
    kernel<<<grid_for(tokens * (D / per), 256), 256, 0, stream>>>(ids, (const __nv_bfloat16*)dout, ldo, (T*)dtable, ldt, tokens, D,
                                                                  vocab, scale);
  };
  if (vec) run(embedding_bwd_kernel<T>, 8);
  else run(embedding_bwd_pairs_kernel<T>, 2);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
}  // namespace

TB_API int tb_embedding_bwd(const int* ids, const void* dout, long long ldo, void* dtable,
                            long long ldt, long long tokens, int D, int vocab, float scale,
                            cudaStream_t stream) {
  return launch_embedding_bwd<__nv_bfloat16>(ids, dout, ldo, dtable, ldt, tokens, D, vocab, scale, stream);
}
// into a 32-bit table
TB_API int tb_embedding_bwd_f32(const int* ids, const void* dout, long long ldo, void* dtable, long long ldt, long long tokens, int D,
                                int vocab, float scale, cudaStream_t stream) {
  return launch_embedding_bwd<float>(ids, dout, ldo, dtable, ldt, tokens, D, vocab, scale, stream);
}

TB_API int tb_add_bf16(const void* a, const void* b, void* y, long long n, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (n % 8) return -2;
  add_kernel<<<grid_for(n / 8, 256), 256, 0, stream>>>((const __nv_bfloat16*)a,
                                                       (const __nv_bfloat16*)b, (__nv_bfloat16*)y, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
