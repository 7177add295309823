// Rows of a language-model head that count: the rows whose target is not negative, moved together, so that the head's products
// run over them alone. Their number stays on the device.
//
//   plan     pos[r] = place of row r among the rows that count, or -1; count = how many there are
//   gather   dst[pos[r]] = src[r], and the targets; 63 rows of zeros behind them (the weight gradient contracts over
//            whole blocks of 64, from the first row of any chunk)
//   scatter  dst[r] = src[pos[r]], 0 for rows that do not count
//
// Bound by HBM (4096 rows of 4096: 34 MB read and written); the head's four products of the rows left out cost 1.1 ms a 1000 rows by
// 32768 x 4096.
#include "common.cuh"

using namespace tb;

namespace {

__global__ void __launch_bounds__(1024)
plan_kernel(const int* __restrict__ targets, int rows, int* __restrict__ pos, int* __restrict__ count) {
  __shared__ int s_warp[32], s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_base = 0;
  __syncthreads();
  for (int r0 = 0; r0 < rows; r0 += 4096) {
    // four rows a thread, in order
    const int r = r0 + threadIdx.x * 4;
    int n = 0, on[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      on[i] = r + i < rows && targets[r + i] >= 0;
      n += on[i];
    }
    int sum = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    if (lane == 31) s_warp[warp] = sum;
    __syncthreads();
    if (warp == 0) {
      int v = s_warp[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int w = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += w;
      }
      s_warp[lane] = v;
    }
    __syncthreads();
    int at = s_base + (warp ? s_warp[warp - 1] : 0) + sum - n;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (r + i < rows) {
        pos[r + i] = on[i] ? at : -1;
        at += on[i];
      }
    __syncthreads();
    if (threadIdx.x == 0) s_base += s_warp[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) *count = s_base;
}

// a warp a row; warps past the rows write the zeros behind the last
__global__ void gather_rows_kernel(const __nv_bfloat16* __restrict__ src, long long lds, const int* __restrict__ targets, const int* __restrict__ pos,
                                   const int* __restrict__ count, int rows, int D, __nv_bfloat16* __restrict__ dst, int* __restrict__ out_targets) {
  const int lane = threadIdx.x & 31;
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  int to;
  if (r < rows) {
    to = pos[r];
    if (to < 0) return;
  } else {
    to = *count + (r - rows);
    if (to >= rows) return;
  }
  for (int c = lane * 8; c < D; c += 256)
    *reinterpret_cast<uint4*>(dst + (long long)to * D + c) =
        r < rows ? *reinterpret_cast<const uint4*>(src + (long long)r * lds + c) : make_uint4(0u, 0u, 0u, 0u);
  if (lane == 0) out_targets[to] = r < rows ? targets[r] : -1;
}

__global__ void scatter_rows_kernel(const __nv_bfloat16* __restrict__ src, const int* __restrict__ pos, int rows, int D,
                                    __nv_bfloat16* __restrict__ dst) {
  const int lane = threadIdx.x & 31;
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= rows) return;
  const int from = pos[r];
  for (int c = lane * 8; c < D; c += 256)
    *reinterpret_cast<uint4*>(dst + (long long)r * D + c) =
        from >= 0 ? *reinterpret_cast<const uint4*>(src + (long long)from * D + c) : make_uint4(0u, 0u, 0u, 0u);
}

// the same for one number a row, up to two of them: gather dst[pos[r]] = src[r], or scatter dst[r] = src[pos[r]] or 0
__global__ void move_numbers_kernel(const float* __restrict__ a, float* __restrict__ to_a, const float* __restrict__ b, float* __restrict__ to_b,
                                    const int* __restrict__ pos, int rows, int gather) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  const int p = pos[r];
  if (gather) {
    if (p < 0) return;
    if (a) to_a[p] = a[r];
    if (b) to_b[p] = b[r];
  } else {
    if (a) to_a[r] = p >= 0 ? a[p] : 0.f;
    if (b) to_b[r] = p >= 0 ? b[p] : 0.f;
  }
}

}  // namespace

// h_out [rows, D] contiguous, targets_out [rows]: *count rows are filled, and 63 more with zeros. D % 8 == 0, 16-byte aligned rows.
TB_API int tb_scored_gather(const void* h, long long ldh, const int* targets, int rows, int D, int* pos, int* count, void* h_out,
                            int* targets_out, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D % 8 || ldh % 8 || ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(h_out)) & 15)) return -2;
  plan_kernel<<<1, 1024, 0, stream>>>(targets, rows, pos, count);
  gather_rows_kernel<<<(rows + 63 + 7) / 8, 256, 0, stream>>>((const __nv_bfloat16*)h, ldh, targets, pos, count, rows, D, (__nv_bfloat16*)h_out,
                                                              targets_out);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
TB_API int tb_scored_scatter(const void* src, const int* pos, int rows, int D, void* dst, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (D % 8 || ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15)) return -2;
  scatter_rows_kernel<<<(rows + 7) / 8, 256, 0, stream>>>((const __nv_bfloat16*)src, pos, rows, D, (__nv_bfloat16*)dst);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
TB_API int tb_scored_numbers(const float* a, float* to_a, const float* b, float* to_b, const int* pos, int rows, int gather,
                             cudaStream_t stream) {
  if (rows <= 0) return 0;
  move_numbers_kernel<<<(rows + 255) / 256, 256, 0, stream>>>(a, to_a, b, to_b, pos, rows, gather);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
