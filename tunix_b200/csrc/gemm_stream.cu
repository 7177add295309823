// bf16 GEMM with one side of at most 64 (decode steps, the low-rank factors of adapters): a stream of the long operand.
//
//   C[M,N] = epilogue( A[M,K] * B[N,K]^T ),  min(M, N) <= 64, each operand K-major or MN-major
//
// The long operand is the left one of the product: 128 of its rows are a tile's lanes in TMEM and the short side is its columns, so a tile
// costs what the short side costs and the accumulator is as small as the result. The K range of a tile is V partial products (partial p
// sums k blocks [p KB / V, (p + 1) KB / V), and the partials are added in their order), spread over the S CTAs of a cluster:
//
//   * grid (S, tiles), cluster (S, 1, 1); CTA z owns partials [z V / S, (z + 1) V / S), each with an accumulator in TMEM
//   * warp 0: TMA into a ring of 6 to 10 stages of 16 KB of the long operand and the k block of the short one; warp 1: one-thread tcgen05.mma
//   * warps 2..5: the partial tiles from TMEM straight into the shared memory of the CTAs that sum their columns (CTA o has the o-th
//     share of the padded columns): stores cross the cluster once and nobody waits for a remote load
//   * one cluster barrier; each CTA sums its columns of all partial tiles and writes them
//
// V. Few rows by a K-major weight, the products of decode steps, have the partial products of gemm_splitk.cu, which took them before and takes
// what is left out here: both give the same bits, whoever runs a step. For the others V is S; they were one sum over all of K, which the
// tensor cores cut off at every step, so that V of them are nearer to 64 bits (64 x 4096 x 12288, fp32 out: 1.4e-5 -> below 1e-5).
//
// Bound by fixed costs (launch, first loads, the exchange) up to some 20 MB of the long operand and by HBM above.
// Every wait is bounded; a timeout sets *status and falls through to the cluster barriers, which every thread reaches on every path.
#include "common.cuh"

using namespace tb;

namespace {

constexpr int TILE = 128, BK = 64, UMMA_K = 16, MAX_STAGES = 10;
constexpr int W_BYTES = TILE * BK * 2;
constexpr int COLS = 16;                 // columns that a CTA sums at most
constexpr int MAX_PARTS = 8, TMEM_COLS = 128;                          // accumulators of a CTA: V / S (rounded up) of P columns, see the choice of S
constexpr int DATA_BYTES = 224 * 1024;   // ring (6 to 10 stages of 18 to 24 KB) and partial sums (up to 64 KB)
constexpr int SMEM_BYTES = DATA_BYTES + 256 + 1024;

enum { GF_A_MN = 1, GF_B_MN = 2, GF_OUT_F32 = 4, GF_ACCUM = 8, GF_BIAS = 16, GF_RESIDUAL = 32 };

struct StreamArgs {
  int rows, cols, K, flags, S, V, P, log_share, stages;    // rows: of the long operand; P: cols padded to 16, 32 or 64; log_share: of P / S / 4
  int w_mn, x_mn;          // the long and the short operand are MN-major
  int tall;                // C is [rows, cols], else [cols, rows]
  int x_bytes;             // of a k block of the short operand
  void* C;
  long long ldc;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* resid;
  long long ldr;
  float alpha;
  int* status;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Place (in 16-byte pieces) of four columns in a partial tile of 128 rows of `pieces` (1, 2, 4, ...): the pieces of a row are turned so that
// eight rows in a column meet eight banks.
__device__ __forceinline__ int piece_at(int row, int piece, int pieces) {
  return row * pieces + ((piece + (pieces < 8 ? row * pieces / 8 : row)) & (pieces - 1));
}

__global__ void __launch_bounds__(192, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const StreamArgs args) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  const int stages = args.stages, stage_bytes = W_BYTES + args.x_bytes;
  const uint32_t part_base = smem_base + stages * stage_bytes, bar_base = smem_base + DATA_BYTES;
  const float4* const part = reinterpret_cast<const float4*>(smem_al + stages * stage_bytes);   // [V][128 rows][columns of a CTA]
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (MAX_STAGES + s); };
  const uint32_t tfull_bar = bar_base + 8u * (2 * MAX_STAGES);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_al + DATA_BYTES + 8 * (2 * MAX_STAGES + 1));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = args.rows, cols = args.cols, S = args.S, V = args.V, P = args.P;
  const int z = blockIdx.x, n0 = blockIdx.y * TILE;                              // z: rank in the cluster
  const int num_kb = (args.K + BK - 1) / BK;
  const int p_begin = z * V / S, here = (z + 1) * V / S - p_begin;                // this CTA's partial products: from k block kb_of(p) on
  auto kb_of = [&](int p) { return (int)((long long)p * num_kb / V); };
  const int kb_begin = kb_of(p_begin), kb_end = kb_of(p_begin + here);
  const int pieces = P / S / 4;                        // of four columns that a CTA sums (powers of two)

  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(tfull_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
    prefetch_tensormap(&tmX);
    prefetch_tensormap(&tmW);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32((const void*)tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cluster_arrive();                                    // this CTA runs: its shared memory may be written from now on
  const uint32_t tmem = *tmem_slot;
  pdl_wait();

  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb_begin; kb < kb_end; ++kb) {
        if (!mbar_wait_bounded(empty_bar(stage), phase ^ 1, abort_flag, args.status, ST_TIMEOUT_PRODUCER)) break;
        const uint32_t sw = smem_base + stage * stage_bytes;
        mbar_expect_tx(full_bar(stage), stage_bytes);
        if (args.w_mn) {
          tma_load_2d(sw, &tmW, full_bar(stage), n0, kb * BK);
          tma_load_2d(sw + W_BYTES / 2, &tmW, full_bar(stage), n0 + 64, kb * BK);
        } else {
          tma_load_2d(sw, &tmW, full_bar(stage), kb * BK, n0);
        }
        tma_load_2d(sw + W_BYTES, &tmX, full_bar(stage), args.x_mn ? 0 : kb * BK, args.x_mn ? kb * BK : 0);
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
    cluster_wait();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(TILE, args.x_mn ? 64 : P, args.w_mn, args.x_mn);   // an MN-major run is 64 wide
      const uint32_t w_lbo = args.w_mn ? 8192u : 16u, x_lbo = args.x_mn ? 8192u : 16u;
      const uint32_t w_step = args.w_mn ? 2048u : 32u, x_step = args.x_mn ? 2048u : 32u;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      int p = p_begin, kb_next = kb_of(p + 1);
      uint32_t d = tmem, more = 0;                     // accumulator of partial p, and whether it holds something
      for (int kb = kb_begin; kb < kb_end; ++kb) {
        if (kb == kb_next) {                           // (no partial product is empty)
          kb_next = kb_of(++p + 1);
          d += P;
          more = 0;
        }
        if (!mbar_wait_bounded(full_bar(stage), phase, abort_flag, args.status, ST_TIMEOUT_MMA)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sw = smem_base + stage * stage_bytes, sx = sw + W_BYTES;
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_f16_ss(d, make_smem_desc(sw + k * w_step, w_lbo, 1024), make_smem_desc(sx + k * x_step, x_lbo, 1024), idesc, more | (k > 0));
        more = 1;
        umma_commit(empty_bar(stage));
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(tfull_bar);
    }
    __syncwarp();
    cluster_wait();
  } else {
    const int q = warp & 3, r = q * 32 + lane;
    // this thread's row of the sum, and what its results take from memory: asked for before the products are there
    const int n = n0 + r, col0 = z * pieces * 4;
    const bool out_f32 = args.flags & GF_OUT_F32, accum = args.flags & GF_ACCUM;
    const bool has_bias = args.flags & GF_BIAS, has_res = args.flags & GF_RESIDUAL;
    const long long step = args.tall ? 1 : args.ldc, at0 = args.tall ? (long long)n * args.ldc + col0 : (long long)col0 * args.ldc + n;
    const long long rstep = args.tall ? 1 : args.ldr, rat0 = args.tall ? (long long)n * args.ldr + col0 : (long long)col0 * args.ldr + n;
    float row_bias = 0.f, early[COLS];
    if (has_bias && !args.tall && n < rows) row_bias = __bfloat162float(args.bias[n]);
#pragma unroll
    for (int i = 0; i < COLS; ++i)
      early[i] = has_res && n < rows && i < pieces * 4 && col0 + i < cols ? __bfloat162float(args.resid[rat0 + i * rstep]) : 0.f;
    const bool ok = mbar_wait_warp(tfull_bar, 0, abort_flag, args.status, ST_TIMEOUT_EPILOGUE);
    tc_fence_after();
    cluster_wait();                                    // the peers run
#pragma unroll 1
    for (int p = 0; p < here; ++p) {
#pragma unroll 1
      for (int c = 0; c < cols; c += 16) {
        uint32_t v[16];
        if (ok) {
          tmem_ld_32x16(tmem + ((uint32_t)(q * 32) << 16) + p * P + c, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = 0u;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int piece = c / 4 + i, o = piece >> args.log_share;                 // the CTA that sums these columns
          const uint32_t to = part_base + (uint32_t)(((p_begin + p) * TILE * pieces + piece_at(r, piece & (pieces - 1), pieces)) << 4);
          if (piece * 4 < cols) st_cluster(map_to_cta(to, (uint32_t)o), v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
      }
    }
    tc_fence_before();
    cluster_arrive();
    cluster_wait();                                    // every partial sum of this CTA's columns is in its shared memory
    auto sum = [&](int piece) {
      float o[4] = {0.f, 0.f, 0.f, 0.f};
      const float4* p = part + piece_at(r, piece, pieces);
      for (int s = 0; s < V; ++s) {
        const float4 v = p[s * TILE * pieces];
        o[0] += v.x;
        o[1] += v.y;
        o[2] += v.z;
        o[3] += v.w;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int local = piece * 4 + i, col = col0 + local;
        if (col >= cols) break;
        o[i] *= args.alpha;
        if (has_bias) o[i] += args.tall ? __bfloat162float(args.bias[col]) : row_bias;
        o[i] += early[local];
        if (out_f32) {
          float* c = reinterpret_cast<float*>(args.C) + at0 + local * step;
          *c = accum ? *c + o[i] : o[i];
        } else {
          __nv_bfloat16* c = reinterpret_cast<__nv_bfloat16*>(args.C) + at0 + local * step;
          *c = __float2bfloat16(accum ? o[i] + __bfloat162float(*c) : o[i]);
        }
      }
    };
    if (n < rows) {
#pragma unroll
      for (int piece = 0; piece < COLS / 4; ++piece)
        if (piece < pieces && col0 + piece * 4 < cols) sum(piece);
    }
  }
  if (warp < 2) {
    cluster_arrive();
    cluster_wait();
  }

  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);   // let TMA copies that may still be in flight land
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

cudaLaunchConfig_t stream_config(int S, int tiles, cudaStream_t stream, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S, tiles, 1);
  cfg.blockDim = dim3(192, 1, 1);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = tb_pdl_enabled() ? 1 : 0;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cfg;
}

}  // namespace

int tb_gemm_splitk_split(int M, int N, int K, int flags);

// Returns 1 when the problem was launched here, 0 when it is not one of this kernel's (the caller goes on), a negative code on error.
// Same conventions as tb_gemm_bf16, whose caller has checked alignment and strides.
int tb_gemm_stream_try(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int flags,
                       const void* bias, const void* resid, long long ldr, float alpha, int* status, cudaStream_t stream) {
  if (flags & ~(GF_A_MN | GF_B_MN | GF_OUT_F32 | GF_ACCUM | GF_BIAS | GF_RESIDUAL)) return 0;
  const bool tall = M > N;
  const int rows = tall ? M : N, cols = tall ? N : M, num_kb = (K + BK - 1) / BK;
  if (cols > 64 || rows < TILE || K < 512) return 0;
  int parts = 0;                                       // 0: as many as CTAs
  if (!tall && !(flags & (GF_A_MN | GF_B_MN))) {
    parts = tb_gemm_splitk_split(M, N, K, flags);
    if (parts < 0) return parts;
    if (parts < 2 || parts > MAX_PARTS || alpha != 1.f) return 0;      // (a product by alpha may join the sum behind it in one rounding, or not)
  }
  const int tiles = (rows + TILE - 1) / TILE;
  static DeviceOnce once;
  static int clusters[9] = {0};                        // co-resident clusters per size, asked of the runtime once
  if (once.first()) {
    if (cudaFuncSetAttribute(gemm_stream_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) return -5;
    for (int s = 1; s <= 8; s *= 2) {
      cudaLaunchAttribute attr[2];
      cudaLaunchConfig_t q = stream_config(s, 1, nullptr, attr);
      q.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, gemm_stream_kernel, &q) != cudaSuccess || n <= 0) {
        cudaGetLastError();
        n = -1;
      }
      clusters[s] = n;
    }
  }
  // One wave of clusters; of few rows each CTA with whole partial products, of the others with four k blocks or more; and at most 16
  // columns to sum (a thread's results leave one by one; beyond that, and at short contractions, narrow tiles are faster). Of those sizes the
  // one with the shortest stream: a CTA draws up to about 60 bytes a nanosecond, all together what HBM gives; every further CTA of a cluster
  // adds to the exchange. us in a graph with cold weights, other kernels -> here: 64 rows by 4096 x 4096 16.1 -> 14.5, 4096 x 12288 30.1 -> 27.0,
  // 1536 x 8960 16.5 -> 12.1, 3072 x 8192 18.5 -> 18.3; 16 rows 13.0 -> 11.2, 25.6 -> 22.4, 14.3 -> 9.4, 16.3 -> 13.3 (with V = S, and so other bits, 10.4,
  // 21.1, 9.1, 12.9); factors of rank 16 of 4004 tokens, [4004, 3584] by [16, 3584] 17.3 -> 7.3, [4004, 14336]^T by [4004, 16] 29.6 -> 26.0, by [14336, 16]
  // 54.4 -> 23.5. Left out: 64 rows by 6144 x 4096 and 8192 x 4096 (32 columns a CTA; 18.4 and 22.5 in the other kernels).
  int best = 0, pad = 0;
  double cost = 0.0;
  for (int s = 1; s <= 8; s *= 2) {
    const int p = cols <= 16 && s <= 4 ? 16 : cols <= 32 ? 32 : 64;       // four columns a CTA or more
    if (clusters[s] < tiles || num_kb / s < 4 || p / s > COLS || (K < 768 && p > 16)) continue;
    if (parts && (parts < s || (parts + s - 1) / s * p > TMEM_COLS)) continue;
    const int most = parts ? (parts + s - 1) / s * ((num_kb + parts - 1) / parts) : (num_kb + s - 1) / s;       // k blocks of a CTA
    const double rate = 6400.0 / (tiles * s), t = most * (W_BYTES * 1e-3) / (rate < 60.0 ? rate : 60.0) + 0.25 * s;
    if (best == 0 || t < cost) {
      best = s;
      pad = p;
      cost = t;
    }
  }
  if (best == 0) return 0;
  StreamArgs a;
  a.rows = rows; a.cols = cols; a.K = K; a.flags = flags; a.S = best; a.V = parts ? parts : best; a.C = C; a.ldc = ldc; a.tall = tall;
  a.w_mn = (flags & (tall ? GF_A_MN : GF_B_MN)) != 0;
  a.x_mn = (flags & (tall ? GF_B_MN : GF_A_MN)) != 0;
  a.P = pad;
  a.x_bytes = (a.x_mn ? 64 : a.P) * BK * 2;             // an MN-major block is 64 wide, zeros past its columns
  a.log_share = 0;
  while ((a.P / best / 4) >> (a.log_share + 1)) ++a.log_share;
  a.stages = (DATA_BYTES - a.V * TILE * (pad / best) * 4) / (W_BYTES + a.x_bytes);
  if (a.stages > MAX_STAGES) a.stages = MAX_STAGES;
  a.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  a.resid = reinterpret_cast<const __nv_bfloat16*>(resid);
  a.ldr = ldr; a.alpha = alpha; a.status = status;
  const void *W = tall ? A : B, *X = tall ? B : A;
  const long long ldw = tall ? lda : ldb, ldx = tall ? ldb : lda;
  CUtensorMap tmX, tmW;
  if (a.x_mn ? tb_make_tmap_2d_bf16(&tmX, X, K, cols, ldx, BK, 64, 1) : tb_make_tmap_2d_bf16(&tmX, X, cols, K, ldx, a.P, BK, 1)) return -3;
  if (a.w_mn ? tb_make_tmap_2d_bf16(&tmW, W, K, rows, ldw, BK, 64, 1) : tb_make_tmap_2d_bf16(&tmW, W, rows, K, ldw, TILE, BK, 1)) return -4;
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = stream_config(best, tiles, stream, attr);
  return cudaLaunchKernelEx(&cfg, gemm_stream_kernel, tmX, tmW, a) == cudaSuccess ? 1 : -5;
}
