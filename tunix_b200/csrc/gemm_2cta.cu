// Two-SM bf16 GEMM for sm_100a: a pair of CTAs (a 2-CTA cluster) computes one 256 x 256 output tile with
// `tcgen05.mma.cta_group::2`.
//
//   C[M,N] = epilogue( A[M,K] * B[N,K]^T )            fp32 accumulation in TMEM
//
// Why: with one CTA per tile a 128 x 256 tile has to pull 48 KiB of operands through the SM's L2 port for every
// 512 tensor-core cycles, more than the port delivers, and the tensor pipe idles a quarter of the time (ncu:
// 74 % active on the single-CTA kernel). In a CTA pair each CTA stages its own 128 rows of A and only HALF of
// the B tile (128 of its 256 rows); the pair's MMA reads both halves, so every CTA moves 32 KiB per 512 cycles
// for the same math. No TMA multicast is involved: each CTA loads its own halves.
//
//   * cluster (2,1,1); CTA rank 0 is the leader and issues every MMA, rank 1 contributes shared memory and TMEM
//   * warp 0 (both CTAs): TMA producer for the CTA's own A / B halves; the loads carry `.cta_group::2` so that
//     their transaction bytes complete on the LEADER's full barrier, which the leader's producer arms with the
//     bytes of both CTAs
//   * warp 1 (leader): one thread issues 4 MMAs (M 256, N 256, K 16) per stage, then commits the stage's empty
//     barrier in both CTAs (two plain commits, own and peer address) and, per tile, the accumulator-full barrier
//     in both CTAs
//   * warps 2..5 (both CTAs): epilogue for the CTA's 128 rows, TMEM double-buffered; "accumulator free" arrives
//     on the leader's barrier from all eight epilogue warps (remote mbarrier arrive for the peer)
//   * 6 stages x 32 KiB, TMEM 2 x 256 columns per CTA, every wait bounded, cluster barrier before teardown
//
// Operand layouts (K-major / MN-major) and epilogue flags are those of gemm.cu.
#include "activation.cuh"
#include "common.cuh"
#include <cstdlib>

using namespace tb;

namespace {

constexpr int BM = 256, BN = 256, BK = 64, UMMA_K = 16;
constexpr int HM = 128, HN = 128;                  // rows of A and of B staged by one CTA
constexpr int STAGES = 6;
constexpr int A_BYTES = HM * BK * 2, B_BYTES = HN * BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int BLOCK_BYTES = 32 * 128;              // 32 rows of 64 bf16 or 32 fp32 results
constexpr int STAGING_BYTES = 4 * 2 * BLOCK_BYTES; // two blocks per epilogue warp
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + STAGING_BYTES + 256 + 1024;

enum { GF_A_MN = 1, GF_B_MN = 2, GF_OUT_F32 = 4, GF_ACCUM = 8, GF_BIAS = 16, GF_RESIDUAL = 32 };

// Grouped products (mixtures of experts): the tiles come from a list in device memory, as in gemm.cu, planned for 256 rows a tile.
struct TileDesc {          // must match gemm.cu
  int m0, n0, m_end, kb0, kb1, b_row0;
  long long c_off;
};

struct Args2 {
  const TileDesc* tiles;   // null: a dense problem
  const int* num_tiles_dev;
  int M, N, K, flags;
  // Rows that exist, known on the device: *limit - limit_off (null: all). Tiles of A rows past it are passed over, or with limit_k the
  // contraction ends there (its last block is whole: zeros in one operand).
  const int* limit;
  int limit_off, limit_k;
  int adds;              // C takes the result, and nothing else, on top: every warp passes over tiles with nothing to contract
  int group;             // tiles are walked in groups of this many rows of tiles (negative: columns), see tile_group
  // further products accumulated into the same TMEM tile, C += A_i[M, K_i] * B_i[N, K_i]^T with the layouts of A and B (a low-rank adapter
  // update carried by the base projection's GEMM, the input gradients of projections that share their input); 0 when absent
  int K2, K3;
  void* C;
  long long ldc;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* resid;
  long long ldr;
  float alpha;
  int* status;
  int tma_c;               // the result leaves in blocks through maps.c
  // Gated feed-forward layers: B is the gate projection in maps.b[0] and the up projection in maps.b[1], a tile's columns 128 of
  // each (N = their rows), and act(gate) * up leaves through maps.c[0], with gate and up through maps.c[1] and [2] if glu_keep.
  int glu, glu_kind, glu_keep;
  // log-softmax epilogue (lm_head): instead of writing C, every tile leaves per row the online-softmax state of its
  // 256 columns and the target column's value, so logits never reach memory. partial: fp32 [M, num_n, 4] =
  // (max, sum exp(z - max), sum exp(z - max) z, z[target] or -inf when the target is in another tile).
  const int* targets;
  float* partial;
  float inv_temp, softcap;
  // logit-gradient epilogue (lm_head backward): the accumulator z is turned in registers into
  //   dz = dlogp (1[j == target] - p_j) - dent p_j (z_j - lse + entropy),  p_j = exp(z_j - lse),
  // chained through temperature and soft-cap, and written as bf16; the fp32 logits never reach memory.
  // dz_lse != nullptr selects it; dz_dlogp / dz_dent / dz_ent may be null.
  const float* dz_lse;
  const float* dz_dlogp;
  const float* dz_dent;
  const float* dz_ent;
};

constexpr int SEGS = 3;
struct Maps2 {
  CUtensorMap a[SEGS], b[SEGS];
  CUtensorMap c[3];        // of the results, in blocks of 32 rows and 128 bytes
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_result), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma2_f16_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on a barrier (own or peer, cluster address) when the MMAs issued so far by this thread have retired
__device__ __forceinline__ void umma2_commit(uint32_t bar_cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr) : "memory");
}
// TMA tile load into this CTA's shared memory whose bytes complete on a barrier given by cluster address
__device__ __forceinline__ void tma2_load_2d(uint32_t smem_dst, const CUtensorMap* tm, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(tm)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

__global__ void __launch_bounds__(192, 1)
gemm2_kernel(const __grid_constant__ Maps2 maps, const Args2 args) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_al = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + STAGES * STAGE_BYTES + STAGING_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };                       // used in the leader only
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };           // one per CTA
  auto tfull_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + s); };       // one per CTA
  auto tempty_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + 2 + s); };  // used in the leader only
  volatile uint32_t* tmem_ptr_smem =
      reinterpret_cast<volatile uint32_t*>(smem_al + STAGES * STAGE_BYTES + STAGING_BYTES + 8 * (2 * STAGES + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int M = args.M, N = args.N, K = args.K;
  const bool glu = args.glu;
  const int tile_n = glu ? BN / 2 : BN;
  const int num_m = (M + BM - 1) / BM, num_n = (N + tile_n - 1) / tile_n;
  const int num_kb1 = (K + BK - 1) / BK;                         // k-blocks of the main operands ...
  const int num_kb2 = num_kb1 + (args.K2 + BK - 1) / BK;         // ... followed by those of the second ...
  const int num_kb = num_kb2 + (args.K3 + BK - 1) / BK;          // ... and the third product
  const bool grouped = args.tiles != nullptr;
  const int num_tiles = grouped ? *args.num_tiles_dev : num_m * num_n;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const bool a_mn = args.flags & GF_A_MN, b_mn = args.flags & GF_B_MN;
  const int lim = args.limit ? *args.limit - args.limit_off : 0x7fffffff;
  const int row_lim = args.limit_k ? 0x7fffffff : lim, kb_lim = args.limit_k ? max(0, min(num_kb, (lim + BK - 1) / BK)) : num_kb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(tfull_bar(s), 1);
      mbar_init(tempty_bar(s), 8);       // four epilogue warps in each CTA of the pair
    }
    *abort_flag = 0;
    mbar_fence_init();
    for (int i = 0; i < SEGS; ++i)
      if (i == 0 || (i == 1 ? args.K2 : args.K3) > 0) {
        prefetch_tensormap(&maps.a[i]);
        prefetch_tensormap(&maps.b[i]);
      }
  }
  if (warp == 1) {
    tmem_alloc2(smem_u32((const void*)tmem_ptr_smem), 2 * BN);
    tmem_relinquish2();
  }
  tc_fence_before();
  cluster_sync_all();                    // barriers of both CTAs exist before anyone signals across
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;

  // first row and column, end of the rows, k-blocks, what is added to B's row, and the row of C that row 0 of the output is
  struct Tile {
    int m0, n0, m_end, kb0, kb1, b_row0, c_row0;
  };
  auto tile_at = [&](int t) -> Tile {
    if (grouped) {
      const TileDesc d = args.tiles[t];
      return {d.m0, d.n0, d.m_end, d.kb0, d.kb1, d.b_row0, d.c_off ? (int)(d.c_off / args.ldc) : 0};
    }
    const bool by_n = args.group < 0;
    const int size = by_n ? -args.group : args.group, along = by_n ? num_n : num_m, across = by_n ? num_m : num_n;
    const int g = t / (size * across), first = g * size, r = t - first * across, here = min(size, along - first);
    const int a = first + r % here, b = r / here;
    return {(by_n ? b : a) * BM, (by_n ? a : b) * tile_n, M, 0, kb_lim, 0, 0};
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (own halves of A and B)
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        const Tile tile = tile_at(t);
        if (tile.m0 >= row_lim) continue;
        const int m0 = tile.m0 + (int)rank * HM, n0 = tile.n0 + (glu ? 0 : (int)rank * HN);
        for (int kb = tile.kb0; kb < tile.kb1; ++kb) {
          if (!mbar_wait_bounded(empty_bar(stage), phase ^ 1, abort_flag, args.status, ST_TIMEOUT_PRODUCER)) {
            ok = false;
            break;
          }
          const uint32_t sa = smem_base + stage * STAGE_BYTES;
          const uint32_t sb = sa + A_BYTES;
          const uint32_t fb = mapa_u32(full_bar(stage), 0);           // the leader's barrier for this stage
          if (leader) mbar_expect_tx(full_bar(stage), 2 * STAGE_BYTES);
          // the maps zero-fill past the end of their contraction, so a rank below 64 costs one padded k-block
          const int seg = kb < num_kb1 || grouped && args.K2 == 0 ? 0 : kb < num_kb2 ? 1 : 2;
          const CUtensorMap *ta = &maps.a[seg], *tb_ = &maps.b[glu ? (int)rank : seg];
          const int k0 = (kb - (seg == 0 ? 0 : seg == 1 ? num_kb1 : num_kb2)) * BK;
          if (!a_mn) {
            tma2_load_2d(sa, ta, fb, k0, m0);
          } else {
#pragma unroll
            for (int j = 0; j < HM / 64; ++j) tma2_load_2d(sa + j * 8192, ta, fb, m0 + 64 * j, k0);
          }
          if (!b_mn) {
            tma2_load_2d(sb, tb_, fb, k0, n0 + tile.b_row0);
          } else {
#pragma unroll
            for (int j = 0; j < HN / 64; ++j) tma2_load_2d(sb + j * 8192, tb_, fb, n0 + 64 * j, k0 + tile.b_row0);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer (leader CTA only)
    if (leader && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(BM, BN, a_mn ? 1 : 0, b_mn ? 1 : 0);
      const uint32_t a_lbo = a_mn ? 8192u : 16u, b_lbo = b_mn ? 8192u : 16u;
      const uint32_t a_kstep = a_mn ? 2048u : 32u, b_kstep = b_mn ? 2048u : 32u;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int t = pair; t < num_tiles && ok; t += num_pairs) {
        int kb0 = 0, kb1 = kb_lim;
        if (args.limit && tile_at(t).m0 >= row_lim) continue;
        if (grouped) {
          kb0 = args.tiles[t].kb0;
          kb1 = args.tiles[t].kb1;
        }
        if (args.adds && kb1 <= kb0) continue;
        if (!mbar_wait_bounded(tempty_bar(acc), acc_phase ^ 1, abort_flag, args.status, ST_TIMEOUT_MMA)) break;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_bounded(full_bar(stage), phase, abort_flag, args.status, ST_TIMEOUT_MMA)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_base + stage * STAGE_BYTES;
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            const uint64_t ad = make_smem_desc(sa + k * a_kstep, a_lbo, 1024);
            const uint64_t bd = make_smem_desc(sb + k * b_kstep, b_lbo, 1024);
            umma2_f16_ss(tmem_d, ad, bd, idesc, kb > kb0 || k > 0 ? 1u : 0u);
          }
          umma2_commit(empty_bar(stage));                              // frees the stage here ...
          umma2_commit(mapa_u32(empty_bar(stage), 1));                 // ... and in the peer
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma2_commit(tfull_bar(acc));
        umma2_commit(mapa_u32(tfull_bar(acc), 1));
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue (own 128 rows)
    const int q = warp & 3;
    int acc = 0;
    uint32_t acc_phase = 0;
    const bool out_f32 = args.flags & GF_OUT_F32, accum = args.flags & GF_ACCUM;
    const bool has_bias = args.flags & GF_BIAS, has_res = args.flags & GF_RESIDUAL;
    const float alpha = args.alpha;
    const bool c_al16 = (reinterpret_cast<uintptr_t>(args.C) & 15) == 0;
    const bool r_al16 = (reinterpret_cast<uintptr_t>(args.resid) & 15) == 0;
    const uint32_t tempty_leader0 = mapa_u32(tempty_bar(0), 0), tempty_leader1 = mapa_u32(tempty_bar(1), 0);
    const bool b_al16 = (reinterpret_cast<uintptr_t>(args.bias) & 15) == 0;
    uint8_t* const staging = smem_al + STAGES * STAGE_BYTES + q * 2 * BLOCK_BYTES;
    int block = 0;                         // the staging block that is written next
    const bool lse_mode = args.partial != nullptr;
    const bool dz_mode = args.dz_lse != nullptr;
    for (int t = pair; t < num_tiles; t += num_pairs) {
      const Tile tile = tile_at(t);
      if (tile.m0 >= row_lim) continue;
      const int row = tile.m0 + (int)rank * HM + q * 32 + lane, row_end = tile.m_end, c_row = tile.c_row0 + row;
      const int n0 = tile.n0;
      const bool none = tile.kb1 <= tile.kb0;              // an expert without rows: its part of a sum over rows is zero
      if (none && args.adds) continue;                     // [32768, 4096] in fp32, zeros added 246 us, left alone 18
      float dz_l = 0.f, dz_gl = 0.f, dz_ge = 0.f, dz_en = 0.f;
      int dz_t = -1;
      if (dz_mode && row < row_end) {
        dz_l = args.dz_lse[row];
        dz_ge = args.dz_dent ? args.dz_dent[row] : 0.f;
        dz_en = (args.dz_dent && args.dz_ent) ? args.dz_ent[row] : 0.f;
        dz_t = args.targets ? args.targets[row] : -1;
        if (dz_t < 0 || dz_t >= N) dz_t = -1;
        dz_gl = (dz_t >= 0 && args.dz_dlogp) ? args.dz_dlogp[row] : 0.f;
      }
      if (!mbar_wait_warp(tfull_bar(acc), acc_phase, abort_flag, args.status, ST_TIMEOUT_EPILOGUE)) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * BN + ((uint32_t)(q * 32) << 16);
      if (lse_mode) {
        // one thread owns one row of the tile: the softmax statistics of its 256 columns need no communication
        float mx = -INFINITY, sm = 0.f, sz = 0.f, zt = -INFINITY;
        const int tgt = row < row_end ? args.targets[row] : -1;
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          const int col0 = n0 + c * 32;
          if (col0 >= N) break;
          uint32_t r[32];
          tmem_ld_32x32(taddr + c * 32, r);
          tmem_ld_wait();
          float cm = -INFINITY;
          float z[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            float v = __uint_as_float(r[i]) * alpha;
            if (args.softcap > 0.f) v = args.softcap * tanhf(v / args.softcap);
            v *= args.inv_temp;
            z[i] = (col0 + i < N) ? v : -INFINITY;
            cm = fmaxf(cm, z[i]);
          }
          if (tgt >= col0 && tgt < col0 + 32) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (col0 + i == tgt) zt = z[i];
          }
          const float nm = fmaxf(mx, cm);
          const float corr = (mx == -INFINITY) ? 0.f : __expf(mx - nm);
          float s2 = 0.f, z2 = 0.f;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const float e = (z[i] == -INFINITY) ? 0.f : __expf(z[i] - nm);
            s2 += e;
            z2 += e * (z[i] == -INFINITY ? 0.f : z[i]);
          }
          sm = sm * corr + s2;
          sz = sz * corr + z2;
          mx = nm;
        }
        if (row < row_end)
          *reinterpret_cast<float4*>(args.partial + ((long long)row * num_n + n0 / BN) * 4) = make_float4(mx, sm, sz, zt);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc == 0 ? tempty_leader0 : tempty_leader1);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        continue;
      }
      const int row0 = row - lane;
      // a block of the staging memory, once its last store has read it; and its store (what lies past M or N is left out by TMA)
      auto acquire = [&] {
        if (lane == 0) tma_store_wait_read<1>();
        __syncwarp();
        return staging + block * BLOCK_BYTES + lane * 128;
      };
      auto release = [&](const CUtensorMap* to, int col0, bool sum) {
        fence_proxy_async_smem();
        __syncwarp();
        if (row0 >= row_end) return;
        if (lane == 0) {
          const uint32_t from = smem_u32(staging + block * BLOCK_BYTES);
          if (sum) tma_reduce_add_2d(to, from, col0, tile.c_row0 + row0);
          else tma_store_2d(to, from, col0, tile.c_row0 + row0);
          tma_store_commit();
        }
        block ^= 1;
      };
      auto put = [&](uint8_t* to, int half, const float (&v)[32]) {       // 32 bf16 results of the lane's row
#pragma unroll
        for (int g = 0; g < 4; ++g)
          *reinterpret_cast<uint4*>(to + (((half * 4 + g) ^ (lane & 7)) << 4)) =
              make_uint4(pack_bf16(v[8 * g], v[8 * g + 1]), pack_bf16(v[8 * g + 2], v[8 * g + 3]),
                         pack_bf16(v[8 * g + 4], v[8 * g + 5]), pack_bf16(v[8 * g + 6], v[8 * g + 7]));
      };
      auto get = [&](int col, float (&v)[32]) {                           // 32 columns of the accumulator
        uint32_t r[32];
        __syncwarp();
        tmem_ld_32x32(taddr + col, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = none ? 0.f : __uint_as_float(r[i]) * alpha;
      };
      if (glu) {
#pragma unroll 1
        for (int c = 0; c < BN / 2; c += 64) {
          if (n0 + c >= N) break;
          // gate and up as they are kept, rounded in pairs: the activation is that of the rows that a backward reads, and of the separate kernels
          uint32_t g[32], u[32];
          auto columns = [&](int col, uint32_t (&to)[32]) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              float v[32];
              get(col + half * 32, v);
#pragma unroll
              for (int i = 0; i < 16; ++i) to[half * 16 + i] = pack_bf16(v[2 * i], v[2 * i + 1]);
            }
          };
          auto leave = [&](int o, const uint32_t (&v)[32]) {
            uint8_t* const to = acquire();
#pragma unroll
            for (int i = 0; i < 8; ++i)
              *reinterpret_cast<uint4*>(to + ((i ^ (lane & 7)) << 4)) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            release(&maps.c[o], n0 + c, false);
          };
          columns(BN / 2 + c, u);
          if (args.glu_keep) leave(2, u);
          columns(c, g);
          if (args.glu_keep) leave(1, g);
#pragma unroll
          for (int i = 0; i < 32; ++i)
            g[i] = pack_bf16(act_fwd(bf16_lo(g[i]), args.glu_kind) * bf16_lo(u[i]), act_fwd(bf16_hi(g[i]), args.glu_kind) * bf16_hi(u[i]));
          leave(0, g);
        }
      } else {
        // 32 columns of the row, up to what is stored
        auto finish = [&](float (&v)[32], int col0) {
          const bool full = (col0 + 32 <= N);
          if (dz_mode) {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              float capped = v[i], chain = args.inv_temp;
              if (args.softcap > 0.f) {
                const float th = tanhf(v[i] / args.softcap);
                capped = args.softcap * th;
                chain *= (1.f - th * th);
              }
              const float z = capped * args.inv_temp;
              const float p = __expf(z - dz_l);
              float d = dz_gl * ((col0 + i == dz_t ? 1.f : 0.f) - p);
              if (dz_ge != 0.f) d -= dz_ge * p * (z - dz_l + dz_en);
              v[i] = row < row_lim ? d * chain : 0.f;
            }
          }
          if (has_bias) {
            if (full && b_al16) {
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                const uint4 u = reinterpret_cast<const uint4*>(args.bias + col0)[g];
                const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  v[g * 8 + 2 * j] += bf16_lo(w[j]);
                  v[g * 8 + 2 * j + 1] += bf16_hi(w[j]);
                }
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (col0 + i < N) v[i] += __bfloat162float(args.bias[col0 + i]);
            }
          }
          if (has_res) {
            const __nv_bfloat16* rp = args.resid + (long long)c_row * args.ldr + col0;
            if (full && (args.ldr % 8 == 0) && r_al16) {
#pragma unroll
              for (int g = 0; g < 4; ++g) {
                const uint4 u = reinterpret_cast<const uint4*>(rp)[g];
                const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  v[g * 8 + 2 * j] += bf16_lo(w[j]);
                  v[g * 8 + 2 * j + 1] += bf16_hi(w[j]);
                }
              }
            } else {
              for (int i = 0; i < 32; ++i)
                if (col0 + i < N) v[i] += __bfloat162float(rp[i]);
            }
          }
        };
        if (args.tma_c) {
          // Blocks of 32 rows and 128 bytes leave through shared memory and TMA, two in flight a warp: whole lines, and no thread waits for C
          // or its address. us in a loop, bf16 results by a lane a row -> here: 4096^3 110 -> 107, 8192 x 1024 x 4096 with B MN-major 65 -> 58, added to
          // bf16 4096^3 118 -> 113, 4096 x 14336 x 4096 385 -> 364; added to fp32, by rows of lanes before, 404 -> 389.
#pragma unroll 1
          for (int c = 0; c < BN; c += out_f32 ? 32 : 64) {
            const int col0 = n0 + c;
            if (col0 >= N) break;
            uint8_t* const to = acquire();
            float v[32];
            if (out_f32) {
              get(c, v);
              if (row < row_end) finish(v, col0);
#pragma unroll
              for (int g = 0; g < 8; ++g)
                *reinterpret_cast<float4*>(to + ((g ^ (lane & 7)) << 4)) = make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
            } else {
#pragma unroll
              for (int half = 0; half < 2; ++half) {
                get(c + half * 32, v);
                if (row < row_end) finish(v, col0 + half * 32);
                put(to, half, v);
              }
            }
            release(&maps.c[0], col0, out_f32 && accum);
          }
        } else {
#pragma unroll 1
          for (int c = 0; c < BN / 32; ++c) {
            const int col0 = n0 + c * 32;
            if (col0 >= N) break;
            float v[32];
            get(c * 32, v);
            if (row < row_end) {
              finish(v, col0);
              const bool full = (col0 + 32 <= N);
              if (out_f32) {
                float* cp = reinterpret_cast<float*>(args.C) + (long long)c_row * args.ldc + col0;
                if (full && (args.ldc % 4 == 0) && c_al16) {
#pragma unroll
                  for (int g = 0; g < 8; ++g) {
                    float4 o = make_float4(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3]);
                    if (accum) {
                      const float4 p = reinterpret_cast<float4*>(cp)[g];
                      o.x += p.x; o.y += p.y; o.z += p.z; o.w += p.w;
                    }
                    reinterpret_cast<float4*>(cp)[g] = o;
                  }
                } else {
                  for (int i = 0; i < 32; ++i)
                    if (col0 + i < N) cp[i] = accum ? cp[i] + v[i] : v[i];
                }
              } else {
                __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(args.C) + (long long)c_row * args.ldc + col0;
                if (full && (args.ldc % 8 == 0) && c_al16) {
#pragma unroll
                  for (int g = 0; g < 4; ++g) {
                    if (accum) {
                      const uint4 u = reinterpret_cast<uint4*>(cp)[g];
                      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                      for (int j = 0; j < 4; ++j) {
                        v[g * 8 + 2 * j] += bf16_lo(w[j]);
                        v[g * 8 + 2 * j + 1] += bf16_hi(w[j]);
                      }
                    }
                    uint4 o;
                    o.x = pack_bf16(v[g * 8 + 0], v[g * 8 + 1]);
                    o.y = pack_bf16(v[g * 8 + 2], v[g * 8 + 3]);
                    o.z = pack_bf16(v[g * 8 + 4], v[g * 8 + 5]);
                    o.w = pack_bf16(v[g * 8 + 6], v[g * 8 + 7]);
                    reinterpret_cast<uint4*>(cp)[g] = o;
                  }
                } else {
                  for (int i = 0; i < 32; ++i)
                    if (col0 + i < N) cp[i] = __float2bfloat16(v[i] + (accum ? __bfloat162float(cp[i]) : 0.f));
                }
              }
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc == 0 ? tempty_leader0 : tempty_leader1);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if (lane == 0) tma_store_wait_read<0>();
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);   // let TMA copies that may still be in flight land
  }
  cluster_sync_all();                    // the peer may still read this CTA's shared memory / write its TMEM
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc2(tmem_base, 2 * BN);
  }
}

int g_sms2 = 0;
// The order of the tiles: groups of at most 16 rows (or columns) of tiles, a group's tiles column by column, in the direction that
// reads the fewest 256-wide panels of A and B: a group's own once, all of the other operand once a group. 16 panels and the 4 or 5
// columns that 74 pairs work on at a time stay in L2; a side of up to 16 tiles is one group, and each panel of the other side is read in
// one go. Under the power cap a loop of products takes, against groups of 8 rows whatever the shape (us, bf16 out): 16384 x 4096 x 4096
// 432 -> 410, 8192 x 4096 x 4096 216 -> 210, 4096 x 14336 x 4096 388 -> 375, 4096 x 4096 x 14336 (dgrad) 390 -> 375, 4096^3 115 -> 112.
// Groups of 32 lose again (8192 x 4096 x 4096 228, 16384 x 12288 x 4096 1284 -> 1357).
int tile_group(int num_m, int num_n) {
  const int gm = (num_m + 15) / 16, gn = (num_n + 15) / 16;
  return num_m + (long long)gm * num_n <= num_n + (long long)gn * num_m ? (num_m + gm - 1) / gm : -((num_n + gn - 1) / gn);
}
struct LseArgs {           // log-softmax epilogue request; partial == nullptr for a plain GEMM
  const int* targets = nullptr;
  float* partial = nullptr;
  float inv_temp = 1.f, softcap = 0.f;
  const float* dz_lse = nullptr;       // logit-gradient epilogue when set
  const float* dz_dlogp = nullptr;
  const float* dz_dent = nullptr;
  const float* dz_ent = nullptr;
};
struct GluArgs {           // gated form where `up` is given: B is the gate projection, up the other; g and u take the two unless null
  int kind = 0;
  const void* up = nullptr;
  long long ldup = 0;
  void *g = nullptr, *u = nullptr;
  long long ldg = 0, ldu = 0;
};
struct Limit {             // see Args2::limit
  const int* at = nullptr;
  int off = 0, k = 0;
};
struct Product {           // a further product of the sum; K == 0 when absent
  const void *A = nullptr, *B = nullptr;
  int K = 0;
  long long lda = 0, ldb = 0;
};

// partial [M, num_n, 4] -> logp[row] = z[target] - lse (0 for targets outside [0, V)), lse, entropy = lse - E[z]
__global__ void lse_combine_kernel(const float* __restrict__ partial, const int* __restrict__ targets, int M, int num_n,
                                   int V, float* __restrict__ logp, float* __restrict__ lse_out, float* __restrict__ ent_out,
                                   const int* __restrict__ limit) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= M || (limit && row >= *limit)) return;
  const int lane = threadIdx.x & 31;
  float mx = -INFINITY, sm = 0.f, sz = 0.f, zt = -INFINITY;
  for (int j = lane; j < num_n; j += 32) {
    const float4 p = *reinterpret_cast<const float4*>(partial + ((long long)row * num_n + j) * 4);
    const float nm = fmaxf(mx, p.x);
    const float a = (mx == -INFINITY) ? 0.f : __expf(mx - nm), b = (p.x == -INFINITY) ? 0.f : __expf(p.x - nm);
    sm = sm * a + p.y * b;
    sz = sz * a + p.z * b;
    mx = nm;
    zt = fmaxf(zt, p.w);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, mx, o), os = __shfl_xor_sync(0xffffffffu, sm, o);
    const float oz = __shfl_xor_sync(0xffffffffu, sz, o), ot = __shfl_xor_sync(0xffffffffu, zt, o);
    const float nm = fmaxf(mx, om);
    const float a = (mx == -INFINITY) ? 0.f : __expf(mx - nm), b = (om == -INFINITY) ? 0.f : __expf(om - nm);
    sm = sm * a + os * b;
    sz = sz * a + oz * b;
    mx = nm;
    zt = fmaxf(zt, ot);
  }
  if (lane == 0) {
    const float lse = mx + logf(sm);
    const int t = targets[row];
    if (logp) logp[row] = (t >= 0 && t < V) ? zt - lse : 0.f;
    if (lse_out) lse_out[row] = lse;
    if (ent_out) ent_out[row] = lse - sz / sm;
  }
}

}  // namespace

namespace {
bool setup_2cta() {
  static DeviceOnce once;
  if (once.first()) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms2, cudaDevAttrMultiProcessorCount, dev);
    if (cudaFuncSetAttribute(gemm2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) return false;
  }
  return true;
}

int start_2cta(const Maps2& maps, const Args2& a, int tiles, cudaStream_t stream) {
  const int pairs = g_sms2 / 2, use_pairs = tiles < pairs ? tiles : pairs;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * use_pairs, 1, 1);
  cfg.blockDim = dim3(192, 1, 1);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, gemm2_kernel, maps, a) == cudaSuccess ? 1 : -5;
}

// Worth it when the pairs have most of a wave of 256 x 256 tiles (tile_n columns) and the K loop amortises the prologue.
bool takes_2cta(int M, int N, int K, int tile_n) {
  static const bool off = getenv("TUNIX_B200_NO_2CTA") != nullptr;
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + tile_n - 1) / tile_n);
  return !off && N >= tile_n && M >= 256 && K >= 256 && tiles >= (g_sms2 / 2 * 3) / 5;
}

int launch_2cta(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                int flags, const void* bias, const void* resid, long long ldr, float alpha, int* status,
                cudaStream_t stream, const LseArgs& lse, const Product& p2 = Product{}, const Product& p3 = Product{},
                const GluArgs& glu = GluArgs{}, const Limit& limit = Limit{}) {
  if (!setup_2cta()) return -5;
  const int tile_n = glu.up ? BN / 2 : BN;
  const int num_m = (M + BM - 1) / BM, num_n = (N + tile_n - 1) / tile_n;
  if (!takes_2cta(M, N, K, tile_n)) return 0;
  const bool a_mn = flags & GF_A_MN, b_mn = flags & GF_B_MN;
  // (the up projection takes the place of a second product: both read all of A)
  const Product sum[SEGS] = {{A, B, K, lda, ldb}, glu.up ? Product{A, glu.up, K, lda, glu.ldup} : p2, p3};
  Maps2 maps;
  for (int i = 0; i < SEGS; ++i) {
    const Product& q = sum[i];
    if (q.K <= 0) {                                       // never loaded from
      maps.a[i] = maps.a[0];
      maps.b[i] = maps.b[0];
      continue;
    }
    if ((q.lda % 8) || (q.ldb % 8) || ((reinterpret_cast<uintptr_t>(q.A) | reinterpret_cast<uintptr_t>(q.B)) & 15)) return -2;
    int r;
    if (!a_mn) r = tb_make_tmap_2d_bf16(&maps.a[i], q.A, M, q.K, q.lda, HM, BK, 1);
    else       r = tb_make_tmap_2d_bf16(&maps.a[i], q.A, q.K, M, q.lda, BK, 64, 1);
    if (r) return -3;
    if (!b_mn) r = tb_make_tmap_2d_bf16(&maps.b[i], q.B, N, q.K, q.ldb, HN, BK, 1);
    else       r = tb_make_tmap_2d_bf16(&maps.b[i], q.B, q.K, N, q.ldb, BK, 64, 1);
    if (r) return -4;
  }
  Args2 a = {};
  const bool adds = (flags & (GF_ACCUM | GF_BIAS | GF_RESIDUAL)) == GF_ACCUM;
  // Results in whole 16-byte pieces leave through TMA, columns included: what TMA leaves out past N it leaves out by such pieces. A sum into bf16 takes what is there as its residual, once and before the rounding
  const bool f32 = flags & GF_OUT_F32;
  a.tma_c = C != nullptr && (reinterpret_cast<uintptr_t>(C) & 15) == 0 && ldc % (f32 ? 4 : 8) == 0 && N % (f32 ? 4 : 8) == 0 &&
            (f32 || (flags & (GF_ACCUM | GF_RESIDUAL)) != (GF_ACCUM | GF_RESIDUAL));
  for (CUtensorMap& c : maps.c) c = maps.a[0];
  if (a.tma_c) {
    if (f32 ? tb_make_tmap_2d_f32(&maps.c[0], C, M, N, ldc, 32, 32) : tb_make_tmap_2d_bf16(&maps.c[0], C, M, N, ldc, 32, 64, 1)) return -4;
    if (!f32 && (flags & GF_ACCUM)) {
      flags = (flags & ~GF_ACCUM) | GF_RESIDUAL;
      resid = C;
      ldr = ldc;
    }
  }
  a.glu = glu.up != nullptr;
  a.glu_kind = glu.kind;
  a.glu_keep = glu.g != nullptr;
  if (glu.up) {
    if (!a.tma_c) return 0;
    auto rows_of_16 = [](const void* p, long long ld) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 8 == 0; };
    if (glu.g) {
      if (!rows_of_16(glu.g, glu.ldg) || !rows_of_16(glu.u, glu.ldu)) return 0;
      if (tb_make_tmap_2d_bf16(&maps.c[1], glu.g, M, N, glu.ldg, 32, 64, 1) || tb_make_tmap_2d_bf16(&maps.c[2], glu.u, M, N, glu.ldu, 32, 64, 1))
        return -4;
    }
  }
  a.K2 = p2.K;
  a.K3 = p3.K;
  a.group = tile_group(num_m, num_n);
  a.limit = limit.at; a.limit_off = limit.off; a.limit_k = limit.k; a.adds = adds;
  a.M = M; a.N = N; a.K = K; a.flags = flags; a.C = C; a.ldc = ldc;
  a.bias = reinterpret_cast<const __nv_bfloat16*>(bias);
  a.resid = reinterpret_cast<const __nv_bfloat16*>(resid);
  a.ldr = ldr; a.alpha = alpha; a.status = status;
  a.targets = lse.targets; a.partial = lse.partial; a.inv_temp = lse.inv_temp; a.softcap = lse.softcap;
  a.dz_lse = lse.dz_lse; a.dz_dlogp = lse.dz_dlogp; a.dz_dent = lse.dz_dent; a.dz_ent = lse.dz_ent;
  return start_2cta(maps, a, num_m * num_n, stream);
}
}  // namespace

// Returns 1 when the problem was launched here, 0 when it is left to the single-CTA kernel, negative on error.
int tb_gemm_2cta_try(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                     long long ldc, int flags, const void* bias, const void* resid, long long ldr, float alpha,
                     int* status, cudaStream_t stream) {
  return launch_2cta(A, B, C, M, N, K, lda, ldb, ldc, flags, bias, resid, ldr, alpha, status, stream, LseArgs{});
}

// C = epilogue(A * B^T + A2 * B2^T (+ A3 * B3^T)): products accumulated into the same TMEM tile (a base projection with a low-rank update, the
// input gradient of projections that share their input). A2 [M, K2] or [K2, M], B2 [N, K2] or [K2, N] and so on, laid out like A and B; K3 may
// be 0. The output's rounding and its passes over memory happen once.
// Returns 1 when launched, 0 when the problem is too small for the two-SM kernel (the caller then runs the products one by one), negative on
// error.
TB_API int tb_gemm_bf16_ext(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                            long long ldc, int flags, const void* bias, const void* resid, long long ldr, float alpha,
                            const void* A2, const void* B2, int K2, long long lda2, long long ldb2, const void* A3, const void* B3, int K3,
                            long long lda3, long long ldb3, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K2 <= 0 || (K2 % 8) || K3 < 0 || (K3 % 8) || (lda % 8) || (ldb % 8) || (reinterpret_cast<uintptr_t>(A) & 15) ||
      (reinterpret_cast<uintptr_t>(B) & 15))
    return -2;
  return launch_2cta(A, B, C, M, N, K, lda, ldb, ldc, flags, bias, resid, ldr, alpha, status, stream, LseArgs{}, {A2, B2, K2, lda2, ldb2},
                     {A3, B3, K3, lda3, ldb3});
}

// Grouped products on SM pairs over a tile list planned for 256 rows a tile (see tb_gemm_grouped_bf16, whose arguments these are). C is
// [c_rows, ldc]-strided with whole 16-byte pieces, all experts' outputs one below the other. A2 / B2 (K2 > 0): a second product of the same
// layouts and tiles, contracted over K2 behind the K of the first; the list's k-blocks count both.
// up (not null): B and up are the stacked gate and up projections, tiles 128 columns wide, C takes act(gate) * up, g and u (null: not kept)
// the two. All [c_rows, N] with stride ldc.
// The weights of 512 rows an expert are read once a tile of 256 rows instead of 128, and the pair's halves of B fit the L2 -> SM port.
TB_API int tb_gemm_grouped_pair(const void* A, long long a_rows, long long a_cols, long long lda, const void* B, long long b_rows,
                                long long b_cols, long long ldb, void* C, long long c_rows, long long ldc, int N, int flags, const void* tiles,
                                const int* num_tiles_dev, int max_tiles, int K, const void* A2, const void* B2, int K2, int glu_kind,
                                const void* up, void* g, void* u, int* status, cudaStream_t stream) {
  if (max_tiles <= 0) return 0;
  const bool f32 = flags & GF_OUT_F32, a_mn = flags & GF_A_MN, b_mn = flags & GF_B_MN;
  uintptr_t ptrs = 0;
  for (const void* p : {A, B, (const void*)C, A2, B2, up, (const void*)g, (const void*)u}) ptrs |= reinterpret_cast<uintptr_t>(p);
  if (lda % 8 || ldb % 8 || ldc % (f32 ? 4 : 8) || N % (f32 ? 4 : 8) || (ptrs & 15) || (K2 > 0 && K % BK) || (up && f32)) return -2;
  if (!setup_2cta()) return -5;
  Maps2 maps;
  const void *as[SEGS] = {A, K2 > 0 ? A2 : A, A}, *bs[SEGS] = {B, up ? up : K2 > 0 ? B2 : B, B};
  for (int i = 0; i < SEGS; ++i) {
    if (a_mn ? tb_make_tmap_2d_bf16(&maps.a[i], as[i], a_rows, a_cols, lda, BK, 64, 1)
             : tb_make_tmap_2d_bf16(&maps.a[i], as[i], a_rows, a_cols, lda, HM, BK, 1)) return -3;
    if (b_mn ? tb_make_tmap_2d_bf16(&maps.b[i], bs[i], b_rows, b_cols, ldb, BK, 64, 1)
             : tb_make_tmap_2d_bf16(&maps.b[i], bs[i], b_rows, b_cols, ldb, HN, BK, 1)) return -4;
  }
  const void* outs[3] = {C, up && g ? g : C, up && g ? u : C};
  for (int i = 0; i < 3; ++i)
    if (f32 ? tb_make_tmap_2d_f32(&maps.c[i], outs[i], c_rows, N, ldc, 32, 32) : tb_make_tmap_2d_bf16(&maps.c[i], outs[i], c_rows, N, ldc, 32, 64, 1))
      return -4;
  Args2 a = {};
  a.tiles = reinterpret_cast<const TileDesc*>(tiles);
  a.num_tiles_dev = num_tiles_dev;
  a.N = N; a.K = K; a.K2 = K2; a.flags = flags; a.C = C; a.ldc = ldc; a.alpha = 1.f; a.status = status; a.tma_c = 1; a.group = 1;
  a.inv_temp = 1.f; a.adds = (flags & GF_ACCUM) != 0;
  if (!f32 && (flags & GF_ACCUM)) {
    a.flags = (flags & ~GF_ACCUM) | GF_RESIDUAL;
    a.resid = reinterpret_cast<const __nv_bfloat16*>(C);
    a.ldr = ldc;
  }
  a.glu = up != nullptr; a.glu_kind = glu_kind; a.glu_keep = g != nullptr;
  const int rc = start_2cta(maps, a, max_tiles, stream);
  return rc == 1 ? 0 : rc;
}

int tb_gemm_splitk_split(int M, int N, int K, int flags);   // gemm_splitk.cu

// h [M, F] = act(x Wg^T) * (x Wu^T), both products and the activation in one launch; gate and up projections [M, F] are written too where
// g and u are given. x [M, K], Wg and Wu [F, K], bf16; F % 8 == 0. Returns 1 when launched, 0 when the call is left to separate kernels
// (too small, or rows that are not whole 16-byte pieces), negative on error.
// us, two products and the activation by itself -> here, gate and up kept / not kept: 4096 x 14336 x 4096 677 -> 635 / 608, 16384 x 12288 x 4096 2260 ->
// 2180 / 2050, 2048 x 8960 x 1536 103 -> 93 / 88, 512 x 8192 x 3072 60 -> 48 / 47. Gate and up are read from the accumulator once, as pairs of bf16
// (a rounding at a time, each read twice: 2048 x 8960 x 1536 in a loop 156, against 138 by themselves). Below K = 1536 three results of a tile took
// longer than its products: 2331 x 4864 x 896 59 -> 63 / 53. The activation's gradient in the epilogue of dy Wd was slower
// everywhere (4096 x 14336 x 4096 442 -> 519): its rows of gate and up arrive by a lane a row.
TB_API int tb_gemm_glu(const void* x, const void* wg, const void* wu, void* h, int M, int F, int K, long long ldx, long long ldwg,
                       long long ldwu, long long ldh, void* g, void* u, long long ldg, long long ldu, int kind, int* status,
                       cudaStream_t stream) {
  if (M <= 0 || F <= 0 || K < 1536 || F % 8) return 0;
  const int split = tb_gemm_splitk_split(M, F, K, 0);   // a few hundred rows by narrow layers of 8192 and more: sums in parts, which are nearer to
  if (split != 0) return split < 0 ? split : 0;         // 64 bits than one, stay with the kernel that makes them
  GluArgs a;
  a.kind = kind; a.up = wu; a.ldup = ldwu; a.g = g; a.u = u; a.ldg = ldg; a.ldu = ldu;
  return launch_2cta(x, wg, h, M, F, K, ldx, ldwg, ldh, 0, nullptr, nullptr, 0, 1.f, status, stream, LseArgs{}, Product{}, Product{}, a);
}

// log p(target) (and optionally lse / entropy) of z = softcap(h W^T) / temperature without materialising z:
// the two-SM GEMM's epilogue leaves per-tile softmax statistics, a small kernel merges them.
// h [M, K] bf16 (row stride ldh), w [V, K] bf16 (row stride ldw), targets int32 [M] (negative = ignored),
// partial: fp32 scratch of M * ceil(V / 256) * 4 elements. Returns 1 when run here, 0 when the problem does not
// qualify for the two-SM kernel (the caller uses its chunked path), negative on error. limit (device, null: M): rows from *limit on are left out.
TB_API int tb_lm_head_lse(const void* h, long long ldh, const void* w, long long ldw, int M, int V, int K,
                          const int* targets, float inv_temp, float softcap, float* partial, float* logp, float* lse,
                          float* entropy, int* status, const int* limit, cudaStream_t stream) {
  LseArgs lse_args;
  lse_args.targets = targets; lse_args.partial = partial; lse_args.inv_temp = inv_temp; lse_args.softcap = softcap;
  const int rc = launch_2cta(h, w, nullptr, M, V, K, ldh, ldw, 0, 0, nullptr, nullptr, 0, 1.0f, status, stream, lse_args, Product{},
                             Product{}, GluArgs{}, Limit{limit, 0, 0});
  if (rc != 1) return rc;
  const int num_n = (V + BN - 1) / BN;
  lse_combine_kernel<<<(M + 7) / 8, 256, 0, stream>>>(partial, targets, M, num_n, V, logp, lse, entropy, limit);
  return cudaGetLastError() == cudaSuccess ? 1 : -5;
}

// dz [M, V] (bf16, row stride ldo) = gradient of sum_rows(dlogp * logp + dent * entropy) (rows from *limit - limit_off on, if given, are left
// out, or zero in a tile with others) with respect to the raw
// logits h W^T, computed in the epilogue of the two-SM GEMM that recomputes those logits: lse (and entropy, when dent
// is given) are the row statistics saved by the forward pass. dlogp / dent / entropy may be null. Returns 1 when run
// here, 0 when the problem does not qualify for the two-SM kernel, negative on error.
TB_API int tb_lm_head_dlogits(const void* h, long long ldh, const void* w, long long ldw, int M, int V, int K,
                              const int* targets, const float* lse, const float* entropy, const float* dlogp,
                              const float* dent, float inv_temp, float softcap, void* out, long long ldo, int* status,
                              const int* limit, int limit_off, cudaStream_t stream) {
  if (!lse || !out) return -2;
  LseArgs e;
  e.targets = targets; e.inv_temp = inv_temp; e.softcap = softcap;
  e.dz_lse = lse; e.dz_dlogp = dlogp; e.dz_dent = dent; e.dz_ent = entropy;
  return launch_2cta(h, w, out, M, V, K, ldh, ldw, ldo, 0, nullptr, nullptr, 0, 1.0f, status, stream, e, Product{}, Product{}, GluArgs{},
                     Limit{limit, limit_off, 0});
}

// Whether the kernel takes a product of these sizes in rows of whole 16-byte pieces: 1 or 0, or a negative code.
TB_API int tb_two_sm_takes(int M, int N, int K) { return setup_2cta() ? takes_2cta(M, N, K, BN) : -5; }

// tb_gemm_bf16 for the first *limit - limit_off rows of A alone (the other rows of C are left as they are), or with limit_k for that much of the
// contraction (zeros up to the next multiple of 64 in one operand). Returns 1 when launched, 0 when the two-SM kernel does not take the
// sizes (nothing is launched), negative on error.
TB_API int tb_gemm_limited(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int flags,
                           const int* limit, int limit_off, int limit_k, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  return launch_2cta(A, B, C, M, N, K, lda, ldb, ldc, flags, nullptr, nullptr, 0, 1.f, status, stream, LseArgs{}, Product{}, Product{}, GluArgs{},
                     Limit{limit, limit_off, limit_k});
}
