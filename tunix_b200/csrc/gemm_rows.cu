// bf16 GEMM of a few rows (decode of one to four sequences).
//
//   C[M,N] = epilogue( A[M,K] * B[N,K]^T ),  A and B K-major, M <= 4
//
// At this height the product is a stream of the weight: a tile of the tensor cores is 128 rows high, and a tile's K loop is a
// chain of dependent stages in the few CTAs that N / 32 columns make. Here a warp owns R weight rows over a share of K, reads them
// 16 bytes a lane with every load of several steps in flight, and multiplies in fp32 on the CUDA cores (16 multiply-adds a
// 16-byte load at M = 2: an eighth of their rate at HBM speed). The KW warps that share a group of rows are summed through
// shared memory.
//
// Bound by latency (one wave: launch, one round of loads, one reduction) up to about 10 MB of weights and by HBM above. B200, one
// row, in a graph with cold weights, tensor cores -> here: 256 x 1536 8.7 -> 2.4 us, 1536 x 1536 9.7 -> 3.7, 1536 x 8960 13.4 -> 7.6,
// 4096 x 4096 12.2 -> 7.5, 4096 x 12288 24.2 -> 17.7; four rows 8.9 -> 3.4, 9.6 -> 4.7, 13.5 -> 9.2.
#include "common.cuh"

using namespace tb;

namespace {

enum { GF_OUT_F32 = 4, GF_ACCUM = 8, GF_BIAS = 16, GF_RESIDUAL = 32 };

struct RowsArgs {
  const __nv_bfloat16 *A, *B;
  long long lda, ldb, ldc, ldr;
  int N, K, flags, kw;              // kw: warps that share a group of rows (1, 2, 4 or 8)
  void* C;
  const __nv_bfloat16 *bias, *resid;
  float alpha;
};

constexpr int WARPS = 8, STEP = 256;       // elements of K that a warp reads of a row at a time

__device__ __forceinline__ uint4 ld_stream(const __nv_bfloat16* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <int M, int R, int U>
__global__ void __launch_bounds__(WARPS * 32)
gemm_rows_kernel(const RowsArgs a) {
  __shared__ float part[WARPS][R * M];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = WARPS / a.kw;                                      // groups of rows in this block
  const int n0 = (blockIdx.x * per + warp / a.kw) * R;
  const int k0 = (warp % a.kw) * STEP + lane * 8, stride = a.kw * STEP;
  pdl_trigger();
  pdl_wait();
  float acc[R][M];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) acc[r][m] = 0.f;
  if (n0 < a.N) {
    const __nv_bfloat16* b[R];
#pragma unroll
    for (int r = 0; r < R; ++r) b[r] = a.B + (long long)min(n0 + r, a.N - 1) * a.ldb;
    for (int k = k0; k < a.K; k += U * stride) {
      uint4 w[U][R], x[U][M];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int at = k + u * stride;
#pragma unroll
        for (int r = 0; r < R; ++r) w[u][r] = at < a.K ? ld_stream(b[r] + at) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int at = k + u * stride;
#pragma unroll
        for (int m = 0; m < M; ++m)
          x[u][m] = at < a.K ? *reinterpret_cast<const uint4*>(a.A + m * a.lda + at) : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int m = 0; m < M; ++m) {
          const uint32_t xs[4] = {x[u][m].x, x[u][m].y, x[u][m].z, x[u][m].w};
#pragma unroll
          for (int r = 0; r < R; ++r) {
            const uint32_t ws[4] = {w[u][r].x, w[u][r].y, w[u][r].z, w[u][r].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              acc[r][m] = fmaf(bf16_lo(ws[i]), bf16_lo(xs[i]), acc[r][m]);
              acc[r][m] = fmaf(bf16_hi(ws[i]), bf16_hi(xs[i]), acc[r][m]);
            }
          }
        }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) {
      acc[r][m] = warp_sum(acc[r][m]);
      if (lane == 0) part[warp][r * M + m] = acc[r][m];
    }
  __syncthreads();
  // one output a thread: group g of the block, row r of the group, row m of A
  if (threadIdx.x >= per * R * M) return;
  const int g = threadIdx.x / (R * M), rm = threadIdx.x % (R * M);
  const int n = (blockIdx.x * per + g) * R + rm / M, m = rm % M;
  if (n >= a.N) return;
  float o = 0.f;
  for (int w = 0; w < a.kw; ++w) o += part[g * a.kw + w][rm];
  o *= a.alpha;
  if (a.flags & GF_BIAS) o += __bfloat162float(a.bias[n]);
  if (a.flags & GF_RESIDUAL) o += __bfloat162float(a.resid[m * a.ldr + n]);
  if (a.flags & GF_OUT_F32) {
    float* c = reinterpret_cast<float*>(a.C) + m * a.ldc + n;
    *c = (a.flags & GF_ACCUM) ? o + *c : o;
  } else {
    __nv_bfloat16* c = reinterpret_cast<__nv_bfloat16*>(a.C) + m * a.ldc + n;
    *c = __float2bfloat16((a.flags & GF_ACCUM) ? o + __bfloat162float(*c) : o);
  }
}

}  // namespace

// Returns 1 when the problem was launched here, 0 when it is not one of this kernel's (the caller goes on), a negative code on
// error. Same conventions as tb_gemm_bf16.
int tb_gemm_rows_try(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                     int flags, const void* bias, const void* resid, long long ldr, float alpha, cudaStream_t stream) {
  // Rows of 16-byte pieces; no other flag than the epilogue's. Above these numbers of weights the stream of the weight bounds both
  // kernels and the multiply-adds of further rows only add to it. us, here / on the tensor cores: one row, 32768 x 4096 43.5 / 48.0,
  // 49152 x 4096 69.6 / 66.3, 151936 x 896 47.6 / 46.0; two, 16384 x 4096 24.8 / 27.1, 24576 x 4096 37.5 / 37.8; three, 4096 x 4096
  // 9.9 / 12.3, 6144 x 4096 14.7 / 14.8; four, 12.6 / 12.3 and 14.7 / 14.7. Three and four rows of many short columns already meet
  // there below: four, 9728 x 896 8.4 / 8.8, 16384 x 1024 14.4 / 10.9, 65536 x 256 14.1 / 11.7 (1024 x 16384 12.3 / 18.6).
  if (M > 4 || K % 8 || (flags & ~(GF_OUT_F32 | GF_ACCUM | GF_BIAS | GF_RESIDUAL))) return 0;
  const long long most = (M == 1 ? 128LL : M == 2 ? 64LL : N <= 4096 ? 16LL : 12LL) << 20;
  if ((long long)N * K > most) return 0;
  RowsArgs a;
  a.A = reinterpret_cast<const __nv_bfloat16*>(A); a.B = reinterpret_cast<const __nv_bfloat16*>(B);
  a.lda = lda; a.ldb = ldb; a.ldc = ldc; a.ldr = ldr; a.N = N; a.K = K; a.flags = flags; a.C = C;
  a.bias = reinterpret_cast<const __nv_bfloat16*>(bias); a.resid = reinterpret_cast<const __nv_bfloat16*>(resid); a.alpha = alpha;
  constexpr int R = 4;
  // K is shared by as many warps as it takes to give every SM eight blocks, as long as each warp has a step of its own
  const int groups = (N + R - 1) / R;
  a.kw = 1;
  while (a.kw < WARPS && (long long)groups * a.kw / WARPS < 8 * 148 && a.kw * 2 * STEP <= K) a.kw *= 2;
  const int per = WARPS / a.kw;
  const dim3 grid((groups + per - 1) / per), block(WARPS * 32);
  cudaError_t e;
  // one step in flight and many blocks, but for one row of few columns, which does not fill the SMs (1536 x 8960: 8.8 -> 7.6 us)
  switch (M) {
    case 1:
      e = N <= 2048 ? launch_pdl(gemm_rows_kernel<1, R, 2>, grid, block, 0, stream, a)
                    : launch_pdl(gemm_rows_kernel<1, R, 1>, grid, block, 0, stream, a);
      break;
    case 2: e = launch_pdl(gemm_rows_kernel<2, R, 1>, grid, block, 0, stream, a); break;
    case 3: e = launch_pdl(gemm_rows_kernel<3, R, 1>, grid, block, 0, stream, a); break;
    default: e = launch_pdl(gemm_rows_kernel<4, R, 1>, grid, block, 0, stream, a); break;
  }
  return e == cudaSuccess ? 1 : -5;
}
