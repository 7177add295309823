// Flash-attention backward for sm_100a on tcgen05 tensor cores.
//
// One CTA owns 128 keys of one kv head and walks over every (query head of the group,
// 64-row query tile) that can see them. All five GEMMs of the backward run on tcgen05 with
// the accumulators in TMEM; the transposed orientation (keys on TMEM lanes) makes every
// element-wise step thread-local (one thread per key row):
//
//   St  = K  Q^T          [128 keys x 64 queries]     P  = exp(z - lse)
//   dPt = V  dO^T         [128 x 64]                  dS = P * (dP - delta) * scale
//   dV += Pt  dO          [128 x HO]   (accumulates in TMEM over all query tiles / heads)
//   dK += dSt Q           [128 x HO]
//   dQt = K^T dS^T        [HO  x 64]   -> fp32 atomics into dQ (coalesced along the head dim)
//
// HO = min(H, 128): for head_dim 256 two CTAs share the keys, each producing one 128-column
// half of dK / dV / dQ (S and dP need the full contraction and are computed by both).
// Masks and soft-cap as in the forward kernel. Waits are bounded (common.cuh).
//
// Counterpart in the reference: autodiff of the attention in tunix/models/*/model.py
// (e.g. tunix/models/llama3/model.py:379-396); no hand-written backward exists there.
#include "segments.cuh"

using namespace tb;

namespace {

constexpr int BK_ = 128;  // keys per CTA
constexpr int BQ_ = 64;   // queries per iteration
constexpr int RG_ = 2;    // row-thread groups
constexpr float LOG2E = 1.4426950408889634f;

struct BwdArgs {
  int B, Tq, Tk, N, KH;
  float scale, softcap;
  int causal, window, q_off;
  const int* seg_q;
  const int* seg_k;
  const float* lse;     // [B, N, Tq]
  const float* delta;   // [B, N, Tq]
  float* dQ;            // fp32 [B*Tq, N*H], zero-initialised by the caller
  __nv_bfloat16* dK;    // [B*Tk, KH*H]
  __nv_bfloat16* dV;
  long long lddk, lddv;
  int* status;
};

template <int H>
struct BwdCfg {
  static constexpr bool PIPE = (H <= 128);          // software-pipelined schedule (needs room for more than one query tile)
  static constexpr int HS = H / 64;
  static constexpr int HO = H < 128 ? H : 128;
  static constexpr int NHALF = H / HO;
  static constexpr int NST = PIPE ? 3 : 1;          // Q / dO tile stages
  static constexpr int NDS = PIPE ? 2 : 1;          // dSt staging buffers
  static constexpr int SEG_BLOCKS = PIPE ? 2048 : 64;       // query tiles that the list can hold (what shared memory leaves)
  static constexpr int KV_BYTES = HS * BK_ * 128;
  static constexpr int Q_BYTES = HS * BQ_ * 128;
  static constexpr int P_BYTES = BK_ * 128;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = OFF_K + KV_BYTES;
  static constexpr int OFF_Q = OFF_V + KV_BYTES;
  static constexpr int OFF_DO = OFF_Q + NST * Q_BYTES;
  static constexpr int OFF_PT = OFF_DO + NST * Q_BYTES;
  static constexpr int OFF_DST = OFF_PT + P_BYTES;
  static constexpr int OFF_STAT = OFF_DST + NDS * P_BYTES;   // [3][2][64] lse and delta of three query tiles
  static constexpr int OFF_BAR = OFF_STAT + 3 * 2 * 64 * 4;
  static constexpr int SMEM_BYTES = OFF_BAR + 192 + 1024;
  // TMEM columns: St (two buffers if PIPE), dPt, dQt, dV, dK
  static constexpr int TM_DPT = PIPE ? 128 : 64;
  static constexpr int TM_DQT = TM_DPT + 64;
  static constexpr int TM_DV = TM_DQT + 64;
  static constexpr int TM_DK = TM_DV + HO;
  static constexpr int TMEM_COLS = 512;
  __host__ __device__ static constexpr int tm_st(int it) { return PIPE ? (it & 1) * 64 : 0; }
};

// Bound by the chain S -> P -> dS -> dK / dQ of one CTA an SM (512 TMEM columns, 208 KB), of which the products are 1280 cycles
// a tile at the tensor cores' rate. B200, 32 / 8 heads of 128, causal, the whole backward (with delta and the fp32 dQ passes),
// before -> after these roles, this schedule and the order of the grid: 2 x 2048 546 -> 279 us, 8 x 2048 1546 -> 1147,
// 1 x 16384 8569 -> 6620 (runs differ by 4 %); rollouts padded at both ends 8 x 1024 864 -> 375; packed rows 3 x 777 with 14 / 2 heads
// of 64 375 -> 110; 4 x 1001, 16 / 8 heads of 256, soft-cap 610 -> 376. Pt and dSt as operands in TMEM were tried: 3 to 5 % less at
// 1 x 16384 and 2 x 2048, nothing beyond what runs differ by at 8 x 2048 and in packed rows, and with heads of 64 between nothing and a
// loss of 14 %, once a vote before each store to TMEM and a barrier of the issuer's were added (the row warps' wait for dV of the tile
// before is also what keeps one that is ahead from arriving twice for a tile).
//
// Roles: row threads (P and dS), four warps that add dQt to dQ and fetch lse / delta of later tiles, one issuer.
// Schedule (PIPE): St runs two query tiles ahead and dPt of the next tile is the first product behind dSt, so the row threads go
// from dS of one tile to P of the next without a wait; dK, dQt and the next St follow while they work. dQt leaves through its own
// warps, off the row threads' path.
// The BQ_ query columns of a key row are split over RG_ threads (one per warpgroup), so the element-wise work between the MMAs
// runs on 128 * RG_ threads.
template <int H>
__global__ void __launch_bounds__(128 * RG_ + 160, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                const BwdArgs a) {
  using C_ = BwdCfg<H>;
  constexpr int CW_ = BQ_ / RG_;           // query columns per row thread
  constexpr int NROW_ = 128 * RG_;         // row threads per CTA (plus the issuer warp)
  constexpr int HO = C_::HO;
  constexpr int NST = C_::NST;
  constexpr bool PIPE = C_::PIPE;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t sbase = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* sptr = smem_raw + (sbase - smem_u32(smem_raw));
  const uint32_t sK = sbase + C_::OFF_K, sV = sbase + C_::OFF_V, sQ = sbase + C_::OFF_Q,
                 sdO = sbase + C_::OFF_DO, sPt = sbase + C_::OFF_PT, sdSt = sbase + C_::OFF_DST,
                 bars = sbase + C_::OFF_BAR;
  // barriers (8 bytes each): 0 KV | 1-3 Q[3] | 4-6 Qfree[3] | 7-8 St[2] | 9 dPt | 10 Pt | 11 dSt | 12 dQ | 13 dQ drained |
  //                          14 dV | 15-17 stats[3] ; tmem slot + abort flag ; 20 everything retired
  const uint32_t barKV = bars, barQ0 = bars + 8, barQF0 = bars + 32, barSt0 = bars + 56, bardPt = bars + 72,
                 barPt = bars + 80, bardSt = bars + 88, bardQ = bars + 96, barDQfree = bars + 104, bardV = bars + 112,
                 barStat0 = bars + 120, barDone = bars + 160;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sptr + C_::OFF_BAR + 144);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sptr + C_::OFF_BAR + 148);
  float* s_stat = reinterpret_cast<float*>(sptr + C_::OFF_STAT);

  const int warp = threadIdx.x >> 5;
  // heavy (early) causal tiles of all heads and rows first: a last wave of light ones
  const unsigned heads = (unsigned)a.KH * C_::NHALF, head = blockIdx.x % heads;
  const int kt = blockIdx.x / (heads * a.B);
  const int half = (C_::NHALF > 1) ? (head % C_::NHALF) : 0;
  const int kvh = head / C_::NHALF;
  const int b = blockIdx.x / heads % a.B;
  const int G = a.N / a.KH;
  const int k0 = kt * BK_;

  // query tiles that can see keys [k0, k0+128)
  int q_lo = 0, q_hi = a.Tq;
  if (a.causal) q_lo = max(0, k0 - a.q_off);
  if (a.window > 0) q_hi = min(a.Tq, k0 + BK_ + a.window - 1 - a.q_off);
  const int qt0 = q_lo / BQ_;
  int nq = q_hi > qt0 * BQ_ ? (q_hi - qt0 * BQ_ + BQ_ - 1) / BQ_ : 0;
  __shared__ SegList<C_::SEG_BLOCKS> s_list;
  const bool listed = a.seg_k && a.seg_q && nq <= C_::SEG_BLOCKS;
  if (listed)
    nq = build_seg_list(s_list, a.seg_k + (long long)b * a.Tk + k0, min(BK_, a.Tk - k0), a.seg_q + (long long)b * a.Tq, a.Tq, qt0, nq);
  const int nit = nq * G;
  // walks the query tiles of a head, head after head
  struct Walk {
    int n, i, base;
    bool same;                             // the ids of keys and queries are all one
  };
  auto tile_at = [&](Walk& w) {
    const int e = listed ? s_list.id[w.i] : 0;             // without a list a tile's number has no mark, and may take more than 15 bits
    w.base = (qt0 + (listed ? e & SEG_ID : w.i)) * BQ_;
    w.same = listed && (e & SEG_SAME);
  };
  auto first_tile = [&] {
    Walk w{kvh * G, 0, 0, false};
    if (nit > 0) tile_at(w);
    return w;
  };
  auto next_tile = [&](Walk& w) {
    if (++w.i == nq) {
      w.i = 0;
      ++w.n;
    }
    tile_at(w);
  };

  if (threadIdx.x == 0) {
    mbar_init(barKV, 1);
    for (int s = 0; s < 3; ++s) {
      mbar_init(barQ0 + 8 * s, 1);
      mbar_init(barQF0 + 8 * s, 1);
      mbar_init(barStat0 + 8 * s, 64);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(barSt0 + 8 * s, 1);
    }
    mbar_init(bardPt, 1);
    mbar_init(bardV, 1);
    mbar_init(barDone, 1);
    mbar_init(barPt, NROW_);
    mbar_init(bardSt, NROW_);
    mbar_init(bardQ, 1);
    mbar_init(barDQfree, 128);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == 4 * RG_ + 4) {
    tmem_alloc(smem_u32((const void*)tmem_slot), C_::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (warp == 4 * RG_ + 4) {
    // ------------------------------------------------------------ issuer warp
    if (nit > 0 && elect_one()) {
      const uint32_t idesc_s = make_idesc_bf16(128, BQ_, 0, 0);     // K-major x K-major, N = 64
      const uint32_t idesc_dv = make_idesc_bf16(128, HO, 0, 1);     // A K-major, B MN-major, N = HO
      const uint32_t idesc_dq = make_idesc_bf16(128, BQ_, 1, 1);    // both MN-major, N = 64
      const uint32_t col_off = half * (HO / 64) * (BQ_ * 128);      // slab offset of this half in Q/dO tiles
      const uint32_t k_half = sK + half * (HO / 64) * (BK_ * 128);
      Walk wl = first_tile();              // of the next load
      auto load_q = [&](int it) {
        const int st = it % NST;
        const uint32_t bar = barQ0 + 8 * st;
        mbar_expect_tx(bar, 2 * C_::Q_BYTES);
#pragma unroll
        for (int c = 0; c < C_::HS; ++c) {
          tma_load_2d(sQ + st * C_::Q_BYTES + c * (BQ_ * 128), &tmQ, bar, wl.n * H + 64 * c, b * a.Tq + wl.base);
          tma_load_2d(sdO + st * C_::Q_BYTES + c * (BQ_ * 128), &tmdO, bar, wl.n * H + 64 * c, b * a.Tq + wl.base);
        }
        if (it + 1 < nit) next_tile(wl);
      };
      // St = K Q^T ; dPt = V dO^T  (contraction over the full head dim)
      auto issue_s = [&](int it) {
        const uint32_t q_s = sQ + (it % NST) * C_::Q_BYTES;
#pragma unroll
        for (int kk = 0; kk < H / 16; ++kk) {
          const uint64_t ad = make_smem_desc(sK + (kk >> 2) * (BK_ * 128) + (kk & 3) * 32, 16, 1024);
          const uint64_t bd = make_smem_desc(q_s + (kk >> 2) * (BQ_ * 128) + (kk & 3) * 32, 16, 1024);
          umma_f16_ss(tmem + C_::tm_st(it), ad, bd, idesc_s, kk != 0);
        }
        umma_commit(barSt0 + (PIPE ? 8 * (it & 1) : 0));
      };
      auto issue_dp = [&](int it) {
        const uint32_t do_s = sdO + (it % NST) * C_::Q_BYTES;
#pragma unroll
        for (int kk = 0; kk < H / 16; ++kk) {
          const uint64_t ad = make_smem_desc(sV + (kk >> 2) * (BK_ * 128) + (kk & 3) * 32, 16, 1024);
          const uint64_t bd = make_smem_desc(do_s + (kk >> 2) * (BQ_ * 128) + (kk & 3) * 32, 16, 1024);
          umma_f16_ss(tmem + C_::TM_DPT, ad, bd, idesc_s, kk != 0);
        }
        umma_commit(bardPt);
      };
      // dV += Pt dO   (A = Pt K-major over 64 queries, B = dO MN-major, this CTA's column half)
      auto issue_dv = [&](int it) {
        const uint32_t do_s = sdO + (it % NST) * C_::Q_BYTES;
#pragma unroll
        for (int kk = 0; kk < BQ_ / 16; ++kk) {
          const uint64_t ad = make_smem_desc(sPt + kk * 32, 16, 1024);
          const uint64_t bd = make_smem_desc(do_s + col_off + kk * 2048, BQ_ * 128, 1024);
          umma_f16_ss(tmem + C_::TM_DV, ad, bd, idesc_dv, (it | kk) != 0);
        }
        umma_commit(bardV);
      };
      // dK += dSt Q
      auto issue_dk = [&](int it) {
        const uint32_t q_s = sQ + (it % NST) * C_::Q_BYTES;
        const uint32_t ds = sdSt + (PIPE ? (it & 1) : 0) * C_::P_BYTES;
#pragma unroll
        for (int kk = 0; kk < BQ_ / 16; ++kk) {
          const uint64_t ad = make_smem_desc(ds + kk * 32, 16, 1024);
          const uint64_t bd = make_smem_desc(q_s + col_off + kk * 2048, BQ_ * 128, 1024);
          umma_f16_ss(tmem + C_::TM_DK, ad, bd, idesc_dv, (it | kk) != 0);
        }
      };
      // dQt = K^T dS^T
      auto issue_dq = [&](int it) {
        const uint32_t ds = sdSt + (PIPE ? (it & 1) : 0) * C_::P_BYTES;
#pragma unroll
        for (int kk = 0; kk < BK_ / 16; ++kk) {
          // A = K^T: M (head dim) contiguous, 64-wide M chunks BK_*128 bytes apart; 16 keys per step
          const uint64_t ad = make_smem_desc(k_half + kk * 2048, BK_ * 128, 1024);
          const uint64_t bd = make_smem_desc(ds + kk * 2048, BK_ * 128, 1024);
          umma_f16_ss(tmem + C_::TM_DQT, ad, bd, idesc_dq, kk != 0);
        }
        umma_commit(barQF0 + 8 * (it % NST));
        umma_commit(bardQ);
      };
#define BWD_WAIT(bar, par, code) \
  if (!mbar_wait_bounded((bar), (par), abort_flag, a.status, (code))) { ok = false; break; }
      bool ok = true;
      mbar_expect_tx(barKV, 2 * C_::KV_BYTES);
#pragma unroll
      for (int c = 0; c < C_::HS; ++c) {
        tma_load_2d(sK + c * (BK_ * 128), &tmK, barKV, kvh * H + 64 * c, b * a.Tk + k0);
        tma_load_2d(sV + c * (BK_ * 128), &tmV, barKV, kvh * H + 64 * c, b * a.Tk + k0);
      }
      for (int i = 0; i < NST && i < nit; ++i) load_q(i);
      ok = mbar_wait_bounded(barKV, 0, abort_flag, a.status, ST_TIMEOUT_PRODUCER);
      if (PIPE) {
        ok = ok && mbar_wait_bounded(barQ0, 0, abort_flag, a.status, ST_TIMEOUT_PRODUCER);
        if (ok) {
          tc_fence_after();
          issue_s(0);
          issue_dp(0);
        }
        if (nit > 1 && ok) {
          ok = mbar_wait_bounded(barQ0 + 8, 0, abort_flag, a.status, ST_TIMEOUT_PRODUCER);
          if (ok) {
            tc_fence_after();
            issue_s(1);
          }
        }
        for (int it = 0; it < nit && ok; ++it) {
          BWD_WAIT(barPt, it & 1, ST_TIMEOUT_MMA);
          tc_fence_after();
          issue_dv(it);
          if (it >= 1 && it + 2 < nit) {
            // the stage of tile it-1 is free once its dK / dQt retired
            BWD_WAIT(barQF0 + 8 * ((it - 1) % NST), ((it - 1) / NST) & 1, ST_TIMEOUT_MMA);
            load_q(it + 2);
          }
          // dS of this tile is stored: its dPt has been read
          BWD_WAIT(bardSt, it & 1, ST_TIMEOUT_MMA);
          tc_fence_after();
          if (it + 1 < nit) issue_dp(it + 1);
          issue_dk(it);
          if (it >= 1) BWD_WAIT(barDQfree, (it - 1) & 1, ST_TIMEOUT_MMA);
          tc_fence_after();
          issue_dq(it);
          if (it + 2 < nit) {
            BWD_WAIT(barQ0 + 8 * ((it + 2) % NST), ((it + 2) / NST) & 1, ST_TIMEOUT_PRODUCER);
            tc_fence_after();
            issue_s(it + 2);
          }
        }
      } else {
        for (int it = 0; it < nit && ok; ++it) {
          if (it >= 1) {
            BWD_WAIT(barQF0, (it - 1) & 1, ST_TIMEOUT_MMA);
            load_q(it);
          }
          BWD_WAIT(barQ0, it & 1, ST_TIMEOUT_PRODUCER);
          tc_fence_after();
          issue_s(it);
          issue_dp(it);
          BWD_WAIT(barPt, it & 1, ST_TIMEOUT_MMA);
          tc_fence_after();
          issue_dv(it);
          BWD_WAIT(bardSt, it & 1, ST_TIMEOUT_MMA);
          tc_fence_after();
          issue_dk(it);
          if (it >= 1) BWD_WAIT(barDQfree, (it - 1) & 1, ST_TIMEOUT_MMA);
          tc_fence_after();
          issue_dq(it);
        }
      }
      if (ok) umma_commit(barDone);
#undef BWD_WAIT
    }
  } else if (warp >= 4 * RG_) {
    // ------------------------------------------- dQ and the row statistics
    const int r = threadIdx.x - NROW_;     // lane = head-dim index (within this CTA's half); column = query
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const long long ld = (long long)a.N * H;
    Walk w = first_tile(), ws = w;         // of the tile that is drained, and of the next statistics
    auto fetch = [&](float& v_lse, float& v_delta) {
      const int qi = ws.base + r;
      const bool in = r < 64 && qi < a.Tq;
      const long long o = ((long long)b * a.N + ws.n) * a.Tq + qi;
      v_lse = in ? a.lse[o] * LOG2E : INFINITY;
      v_delta = in ? a.delta[o] : 0.f;
    };
    auto put = [&](int it, float v_lse, float v_delta) {
      if (r < 64) {
        float* d = s_stat + (it % 3) * 128;
        d[r] = v_lse;
        d[64 + r] = v_delta;
        mbar_arrive(barStat0 + 8 * (it % 3));
      }
    };
    float v_lse, v_delta;
    for (int it = 0; it < 3 && it < nit; ++it) {
      fetch(v_lse, v_delta);
      put(it, v_lse, v_delta);
      if (it + 1 < nit) next_tile(ws);
    }
    bool ok = true;
    for (int it = 0; it < nit && ok; ++it) {
      if (it + 3 < nit) fetch(v_lse, v_delta);
      if (!mbar_wait_warp(bardQ, it & 1, abort_flag, a.status, ST_TIMEOUT_EPILOGUE)) { ok = false; break; }
      tc_fence_after();
      if (it + 3 < nit) {                  // dQt of this tile is there: its dS is, and nobody reads its statistics any more
        put(it + 3, v_lse, v_delta);
        if (it + 4 < nit) next_tile(ws);
      }
      uint32_t t[2][32];
#pragma unroll
      for (int j = 0; j < 2; ++j) tmem_ld_32x32(tmem + lane_addr + C_::TM_DQT + 32 * j, t[j]);
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(barDQfree);
      if (r < HO) {
        float* dq = a.dQ + ((long long)b * a.Tq + w.base) * ld + (long long)w.n * H + half * HO + r;
        if (w.base + BQ_ <= a.Tq) {
#pragma unroll
          for (int i = 0; i < BQ_; ++i) atomicAdd(dq + i * ld, __uint_as_float(t[i >> 5][i & 31]));
        } else {
#pragma unroll
          for (int i = 0; i < BQ_; ++i)
            if (w.base + i < a.Tq) atomicAdd(dq + i * ld, __uint_as_float(t[i >> 5][i & 31]));
        }
      }
      if (it + 1 < nit) next_tile(w);
    }
  } else {
    // ------------------------------------------------------- per-key-row math
    const int r = threadIdx.x & 127;     // key row in tile == TMEM lane
    const int hq = threadIdx.x >> 7;     // which CW_ query columns of the row this thread works on
    const int c0 = hq * CW_;
    const int kp = k0 + r;
    const bool key_valid = kp < a.Tk;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const int my_seg = (a.seg_k && key_valid) ? a.seg_k[(long long)b * a.Tk + kp] : 0;
    bool ok = true;
    const float sc2 = a.scale * LOG2E, inv_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;
    Walk w = first_tile();
    for (int it = 0; it < nit && ok; ++it) {
      const float* st_lse = s_stat + (it % 3) * 128 + c0;      // this thread's columns
      const float* st_delta = st_lse + 64;
      const int q0 = w.base + c0;
      // does any (key, query) pair of this tile need masking?
      const int qpos_lo = w.base + a.q_off, qpos_hi = w.base + BQ_ - 1 + a.q_off;
      const bool by_seg = a.seg_k != nullptr && !w.same;
      const bool need_mask = (k0 + BK_ > a.Tk) || (w.base + BQ_ > a.Tq) || by_seg || (a.causal && (k0 + BK_ - 1 > qpos_lo)) ||
                             (a.window > 0 && (k0 <= qpos_hi - a.window));
      uint32_t keep[CW_ / 32];             // the queries that see this key, one bit each
      if (need_mask) {
        int lo = 0, hi = key_valid ? a.Tq - q0 : 0;
        if (a.causal) lo = kp - a.q_off - q0;
        if (a.window > 0) hi = min(hi, kp + a.window - a.q_off - q0);
#pragma unroll
        for (int j = 0; j < CW_ / 32; ++j) {
          keep[j] = bits_below(hi - 32 * j) & ~bits_below(lo - 32 * j);
          if (by_seg && a.seg_q) seg_bits(a.seg_q + (long long)b * a.Tq, q0 + 32 * j, a.Tq, my_seg, keep[j]);
          else if (by_seg && my_seg != 0) keep[j] = 0;
        }
      }

      // One answer for a warp ahead of the aligned loads from TMEM, and before anybody leaves the loop: the votes over segment ids
      // above need every lane.
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(barStat0 + 8 * (it % 3), (it / 3) & 1, abort_flag, a.status, ST_TIMEOUT_EPILOGUE) &&
                                       mbar_wait_bounded(barSt0 + (PIPE ? 8 * (it & 1) : 0), (PIPE ? it >> 1 : it) & 1, abort_flag,
                                                         a.status, ST_TIMEOUT_EPILOGUE));
      if (!ok) break;
      tc_fence_after();
      float p[CW_];
      uint32_t pk[CW_ / 2];
      {
        uint32_t t[CW_ / 32][32];
#pragma unroll
        for (int j = 0; j < CW_ / 32; ++j) tmem_ld_32x32(tmem + lane_addr + C_::tm_st(it) + c0 + 32 * j, t[j]);
        tmem_ld_wait();
        if (a.softcap > 0.f) {
#pragma unroll
          for (int i = 0; i < CW_; ++i) {
            // as in the forward, whose row sums it then matches. Also the closer form in this file's fast-math build: against 64 bits,
            // cap 50, scores up to 150, the capped score is off by 3.2e-6 rms (1.4e-5 at most), with tanhf by 1.3e-4 (3.9e-4); the
            // cap's derivative by 1.1e-7 and 4.2e-6.
            const float z = cap_score(__uint_as_float(t[i >> 5][i & 31]) * a.scale, a.softcap, inv_cap);
            t[i >> 5][i & 31] = __float_as_uint(z * inv_cap);
            p[i] = exp2f(fmaf(z, LOG2E, -st_lse[i]));
          }
        } else {
#pragma unroll
          for (int i = 0; i < CW_; ++i) p[i] = exp2f(fmaf(__uint_as_float(t[i >> 5][i & 31]), sc2, -st_lse[i]));
        }
        if (need_mask) {
#pragma unroll
          for (int i = 0; i < CW_; ++i)
            if (!(keep[i >> 5] >> (i & 31) & 1)) p[i] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < CW_ / 2; ++i) pk[i] = pack_bf16(p[2 * i], p[2 * i + 1]);
        if (a.softcap > 0.f) {             // dS passes through the cap's derivative
#pragma unroll
          for (int i = 0; i < CW_; ++i) {
            const float th = __uint_as_float(t[i >> 5][i & 31]);
            p[i] *= 1.f - th * th;
          }
        }
      }
      // dV of the tile before has read the buffer of Pt (without PIPE it retired before this tile's St)
      bool free = true;                    // a failed wait is acted upon at the next vote
      if (PIPE && it >= 1) free = mbar_wait_bounded(bardV, (it - 1) & 1, abort_flag, a.status, ST_TIMEOUT_EPILOGUE);
      {
        uint8_t* prow = sptr + C_::OFF_PT + r * 128;
#pragma unroll
        for (int c = 0; c < CW_ / 8; ++c)
          *reinterpret_cast<uint4*>(prow + (((c + c0 / 8) ^ (r & 7)) << 4)) =
              make_uint4(pk[4 * c], pk[4 * c + 1], pk[4 * c + 2], pk[4 * c + 3]);
        fence_proxy_async_smem();
        tc_fence_before();
        mbar_arrive(barPt);
      }
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(bardPt, it & 1, abort_flag, a.status, ST_TIMEOUT_EPILOGUE) && free);
      if (!ok) break;
      tc_fence_after();
      {
        uint32_t t[CW_ / 32][32];
#pragma unroll
        for (int j = 0; j < CW_ / 32; ++j) tmem_ld_32x32(tmem + lane_addr + C_::TM_DPT + c0 + 32 * j, t[j]);
        tmem_ld_wait();
        // (dSt of the tile before last was read by products that retired before this dPt)
        uint8_t* drow = sptr + C_::OFF_DST + (PIPE ? (it & 1) : 0) * C_::P_BYTES + r * 128;
#pragma unroll
        for (int c = 0; c < CW_ / 8; ++c) {
          float d[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int i = 8 * c + e;
            const float dp = __uint_as_float(t[i >> 5][i & 31]);
            d[e] = p[i] * (dp - st_delta[i]) * a.scale;
          }
          uint4 v;
          v.x = pack_bf16(d[0], d[1]);
          v.y = pack_bf16(d[2], d[3]);
          v.z = pack_bf16(d[4], d[5]);
          v.w = pack_bf16(d[6], d[7]);
          *reinterpret_cast<uint4*>(drow + (((c + c0 / 8) ^ (r & 7)) << 4)) = v;
        }
        fence_proxy_async_smem();
        tc_fence_before();
        mbar_arrive(bardSt);
      }
      if (it + 1 < nit) next_tile(w);
    }
    if (nit > 0 && ok) ok = mbar_wait_warp(barDone, 0, abort_flag, a.status, ST_TIMEOUT_EPILOGUE);
    // ------------------------------------------------------------- dK / dV
    tc_fence_after();
    __nv_bfloat16* dkrow = a.dK + ((long long)b * a.Tk + kp) * a.lddk + (long long)kvh * H + half * HO;
    __nv_bfloat16* dvrow = a.dV + ((long long)b * a.Tk + kp) * a.lddv + (long long)kvh * H + half * HO;
#pragma unroll 1
    for (int c = hq; c < HO / 32; c += RG_) {      // the row's output columns are shared out between its threads
      uint32_t o[32];
#pragma unroll 1
      for (int which = 0; which < 2; ++which) {
        if (nit > 0 && ok) {
          tmem_ld_32x32(tmem + lane_addr + (which ? C_::TM_DK : C_::TM_DV) + c * 32, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = 0;
        }
        if (key_valid) {
          __nv_bfloat16* dst = (which ? dkrow : dvrow) + c * 32;
#pragma unroll
          for (int g4 = 0; g4 < 4; ++g4) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(o[8 * g4 + 0]), __uint_as_float(o[8 * g4 + 1]));
            v.y = pack_bf16(__uint_as_float(o[8 * g4 + 2]), __uint_as_float(o[8 * g4 + 3]));
            v.z = pack_bf16(__uint_as_float(o[8 * g4 + 4]), __uint_as_float(o[8 * g4 + 5]));
            v.w = pack_bf16(__uint_as_float(o[8 * g4 + 6]), __uint_as_float(o[8 * g4 + 7]));
            *reinterpret_cast<uint4*>(dst + g4 * 8) = v;
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  if (warp == 4 * RG_ + 4) {
    tc_fence_after();
    tmem_dealloc(tmem, C_::TMEM_COLS);
  }
}

// delta[b, n, t] = sum_h dO * O: H / 8 lanes a row, 8 columns a lane, two rows of a lane in flight. Bound by HBM: O and dO once.
// B200, a warp a row and 4-byte loads before: 1 x 16384 x 32 heads of 128 117 -> 53 us, 8 x 1024 62 -> 29, 4 x 1001 x 16 of 256 17.5 -> 15.9.
template <int H, typename I>          // I: of a row number
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ o, long long ldo, const __nv_bfloat16* __restrict__ dout, long long lddo,
                  float* __restrict__ delta, int B, int T, int N) {
  constexpr int L = H / 8, PER = 256 / L, U = 2;
  const int sub = threadIdx.x % L;
  const I total = (I)B * T * N, step = (I)gridDim.x * PER;
  // every lane of a warp makes the same number of turns: the shuffles below need all of them
  for (I w0 = (I)blockIdx.x * PER; w0 < total; w0 += U * step) {
    uint4 x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const I w = w0 + threadIdx.x / L + u * step;
      x[u] = y[u] = make_uint4(0u, 0u, 0u, 0u);
      if (w < total) {
        const I bt = w / N;
        const int c = (int)(w - bt * N) * H + sub * 8;
        x[u] = __ldg(reinterpret_cast<const uint4*>(o + (long long)bt * ldo + c));
        y[u] = __ldg(reinterpret_cast<const uint4*>(dout + (long long)bt * lddo + c));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const I w = w0 + threadIdx.x / L + u * step;
      const uint32_t xs[4] = {x[u].x, x[u].y, x[u].z, x[u].w}, ys[4] = {y[u].x, y[u].y, y[u].z, y[u].w};
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) acc += bf16_lo(xs[k]) * bf16_lo(ys[k]) + bf16_hi(xs[k]) * bf16_hi(ys[k]);
#pragma unroll
      for (int s = L / 2; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
      if (sub == 0 && w < total) {
        const I bt = w / N, b = bt / T;
        delta[((long long)b * N + (w - bt * N)) * T + (bt - b * T)] = acc;
      }
    }
  }
}

// The same by pairs, a warp a row, for rows that are not whole 16-byte pieces and other head sizes.
__global__ void attn_delta_pairs_kernel(const __nv_bfloat16* __restrict__ o, long long ldo, const __nv_bfloat16* __restrict__ dout,
                                        long long lddo, float* __restrict__ delta, int B, int T, int N, int H) {
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const long long total = (long long)B * T * N;
  for (long long w = (long long)blockIdx.x * warps + (threadIdx.x >> 5); w < total; w += (long long)gridDim.x * warps) {
    const long long bt = w / N, n = w - bt * N, b = bt / T;
    const __nv_bfloat16 *po = o + bt * ldo + n * H, *pd = dout + bt * lddo + n * H;
    float acc = 0.f;
    for (int c = lane * 2; c < H; c += 64) {
      const uint32_t x = *reinterpret_cast<const uint32_t*>(po + c), y = *reinterpret_cast<const uint32_t*>(pd + c);
      acc += bf16_lo(x) * bf16_lo(y) + bf16_hi(x) * bf16_hi(y);
    }
    acc = warp_sum(acc);
    if (lane == 0) delta[(b * N + n) * T + (bt - b * T)] = acc;
  }
}

int launch_delta(const void* o, long long ldo, const void* dout, long long lddo, float* delta, int B, int T, int N, int H,
                 cudaStream_t stream) {
  const long long total = (long long)B * T * N;
  if (total <= 0) return 0;
  const bool vec = ldo % 8 == 0 && lddo % 8 == 0 && ((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(dout)) & 15) == 0;
  if (!vec || (H != 64 && H != 128 && H != 256)) {
    const long long blocks = (total + 7) / 8;
    attn_delta_pairs_kernel<<<(int)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, stream>>>(
        (const __nv_bfloat16*)o, ldo, (const __nv_bfloat16*)dout, lddo, delta, B, T, N, H);
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
  }
  auto run = [&](auto kernel, int per) {
    const long long blocks = (total + 2 * per - 1) / (2 * per);
    kernel<<<(int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, stream>>>((const __nv_bfloat16*)o, ldo, (const __nv_bfloat16*)dout, lddo,
                                                                           delta, B, T, N);
  };
  const bool small = total < (1LL << 30);             // row numbers, and what a turn adds to them, in 32 bits
  if (H == 64) small ? run(attn_delta_kernel<64, uint32_t>, 32) : run(attn_delta_kernel<64, long long>, 32);
  else if (H == 128) small ? run(attn_delta_kernel<128, uint32_t>, 16) : run(attn_delta_kernel<128, long long>, 16);
  else small ? run(attn_delta_kernel<256, uint32_t>, 8) : run(attn_delta_kernel<256, long long>, 8);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

template <int H>
int launch_bwd(const void* q, const void* k, const void* v, const void* dout, const BwdArgs& a,
               long long ldq, long long ldk, long long ldv, long long lddo, cudaStream_t stream) {
  using C_ = BwdCfg<H>;
  CUtensorMap tq, tk, tv, tdo;
  if (tb_make_tmap_2d_bf16(&tq, q, (uint64_t)a.B * a.Tq, (uint64_t)a.N * H, ldq, BQ_, 64, 1)) return -3;
  if (tb_make_tmap_2d_bf16(&tdo, dout, (uint64_t)a.B * a.Tq, (uint64_t)a.N * H, lddo, BQ_, 64, 1)) return -3;
  if (tb_make_tmap_2d_bf16(&tk, k, (uint64_t)a.B * a.Tk, (uint64_t)a.KH * H, ldk, BK_, 64, 1)) return -3;
  if (tb_make_tmap_2d_bf16(&tv, v, (uint64_t)a.B * a.Tk, (uint64_t)a.KH * H, ldv, BK_, 64, 1)) return -3;
  static DeviceOnce once;
  if (once.first() &&
      cudaFuncSetAttribute(attn_bwd_kernel<H>, cudaFuncAttributeMaxDynamicSharedMemorySize, C_::SMEM_BYTES) != cudaSuccess)
    return -5;
  const long long ctas = (long long)a.KH * C_::NHALF * a.B * ((a.Tk + BK_ - 1) / BK_);
  if (ctas > 0x7fffffffLL) return -2;
  const dim3 grid((unsigned)ctas);
  attn_bwd_kernel<H><<<grid, 128 * RG_ + 160, C_::SMEM_BYTES, stream>>>(tq, tk, tv, tdo, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

}  // namespace

TB_API int tb_attn_delta(const void* o, long long ldo, const void* dout, long long lddo, float* delta,
                         int B, int T, int N, int H, cudaStream_t stream) {
  return launch_delta(o, ldo, dout, lddo, delta, B, T, N, H, stream);
}

// dq_accum: fp32 [B*Tq, N*H] zero-initialised; dk, dv: bf16 [B*Tk, KH*H] (fully written).
TB_API int tb_attn_bwd(const void* q, const void* k, const void* v, const void* dout, const float* lse,
                       const float* delta, float* dq_accum, void* dk, void* dv, int B, int Tq, int Tk,
                       int N, int KH, int H, long long ldq, long long ldk, long long ldv, long long lddo,
                       long long lddk, long long lddv, float scale, float softcap, int causal, int window,
                       int q_off, const int* seg_q, const int* seg_k, int* status, cudaStream_t stream) {
  if (B <= 0 || Tk <= 0 || KH <= 0) return 0;
  if (N % KH || (ldq % 8) || (ldk % 8) || (ldv % 8) || (lddo % 8) || (lddk % 8) || (lddv % 8)) return -2;
  BwdArgs a;
  a.B = B; a.Tq = Tq; a.Tk = Tk; a.N = N; a.KH = KH;
  a.scale = scale; a.softcap = softcap; a.causal = causal; a.window = window; a.q_off = q_off;
  a.seg_q = seg_q; a.seg_k = seg_k; a.lse = lse; a.delta = delta; a.dQ = dq_accum;
  a.dK = reinterpret_cast<__nv_bfloat16*>(dk); a.dV = reinterpret_cast<__nv_bfloat16*>(dv);
  a.lddk = lddk; a.lddv = lddv; a.status = status;
  switch (H) {
    case 64: return launch_bwd<64>(q, k, v, dout, a, ldq, ldk, ldv, lddo, stream);
    case 128: return launch_bwd<128>(q, k, v, dout, a, ldq, ldk, ldv, lddo, stream);
    case 256: return launch_bwd<256>(q, k, v, dout, a, ldq, ldk, ldv, lddo, stream);
    default: return -2;
  }
}

// ---------------------------------------------------------------------------------------------
// Allocation-free entry point (declared in noalloc.h; it has no counterpart in the reference).
//
// tb_attn_bwd above expects its caller to hand it two scratch buffers (delta and the fp32 dQ
// accumulator), which in this package come from torch's caching allocator. Some callers cannot
// allocate device memory at all: code running inside a CUDA-graph capture or a stream-ordered
// region where cudaMalloc is illegal, a serving process whose memory pool is owned and fully
// reserved by another component, or a plain C/C++ host that links this library without torch.
// For them the scratch lives in the library image itself.
// ---------------------------------------------------------------------------------------------
#include "noalloc.h"
#include <cstdio>
#include <mutex>

namespace {

// Fixed scratch, resident on every GPU that loads this library until the process exits.
static __device__ __align__(256) float g_noalloc_dq_scratch[TB_NOALLOC_MAX_DQ_ELEMS];
static __device__ __align__(256) float g_noalloc_delta_scratch[TB_NOALLOC_MAX_ROWS];

constexpr int kMaxDevices = 64;
float* g_noalloc_dq_ptr[kMaxDevices] = {nullptr};
float* g_noalloc_delta_ptr[kMaxDevices] = {nullptr};
std::mutex g_noalloc_setup_mutex;          // two host threads may make the first call on a device at once
thread_local char g_noalloc_error[256] = "";   // each host thread reads the message of its own last call

__global__ void noalloc_zero_kernel(float* p, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    p[i] = 0.f;
}
__global__ void noalloc_cast_kernel(const float* __restrict__ in, __nv_bfloat16* __restrict__ out, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16(in[i]);
}

int noalloc_fail(int code, const char* msg) {
  snprintf(g_noalloc_error, sizeof(g_noalloc_error), "%s", msg);
  return code;
}

// In host code the array names above are host-side stand-ins, not device addresses; the real
// addresses are looked up once per device, with that device current.
int noalloc_setup(int dev) {
  std::lock_guard<std::mutex> lock(g_noalloc_setup_mutex);
  if (g_noalloc_dq_ptr[dev] && g_noalloc_delta_ptr[dev]) return 0;
  float* p = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&p, g_noalloc_dq_scratch);
  if (e != cudaSuccess || !p) return noalloc_fail(-10, "cudaGetSymbolAddress(dq scratch) failed");
  g_noalloc_dq_ptr[dev] = p;
  p = nullptr;
  e = cudaGetSymbolAddress((void**)&p, g_noalloc_delta_scratch);
  if (e != cudaSuccess || !p) return noalloc_fail(-10, "cudaGetSymbolAddress(delta scratch) failed");
  g_noalloc_delta_ptr[dev] = p;
  return 0;
}

}  // namespace

TB_API const char* tb_noalloc_last_error() { return g_noalloc_error; }

TB_API int tb_attn_bwd_noalloc(const void* q, const void* k, const void* v, const void* o, const void* dout,
                               const float* lse, void* dq, void* dk, void* dv, int B, int Tq, int Tk, int N,
                               int KH, int H, float scale, float softcap, int causal, int window,
                               int* status, cudaStream_t stream) {
  g_noalloc_error[0] = 0;
  if (B <= 0 || Tq <= 0 || Tk <= 0 || N <= 0 || KH <= 0 || N % KH) return noalloc_fail(-2, "bad shape");
  if (H != 64 && H != 128 && H != 256) return noalloc_fail(-2, "head dim must be 64, 128 or 256");
  const long long dq_elems = (long long)B * Tq * N * H;
  const long long rows = (long long)B * N * Tq;
  if (dq_elems > TB_NOALLOC_MAX_DQ_ELEMS || rows > TB_NOALLOC_MAX_ROWS) {
    snprintf(g_noalloc_error, sizeof(g_noalloc_error),
             "problem too large for the built-in scratch: B*Tq*N*H = %lld (max %lld), B*N*Tq = %lld (max %lld)",
             dq_elems, (long long)TB_NOALLOC_MAX_DQ_ELEMS, rows, (long long)TB_NOALLOC_MAX_ROWS);
    return -11;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return noalloc_fail(-10, "no current device");
  if (int rc = noalloc_setup(dev)) return rc;
  float* dq32 = g_noalloc_dq_ptr[dev];
  float* delta = g_noalloc_delta_ptr[dev];
  const long long ldq = (long long)N * H, ldkv = (long long)KH * H;
  // The scratch keeps the previous call's contents: the dQ accumulator must start at zero.
  noalloc_zero_kernel<<<592, 256, 0, stream>>>(dq32, dq_elems);
  if (int rc = launch_delta(o, ldq, dout, ldq, delta, B, Tq, N, H, stream)) return noalloc_fail(rc, "row sums: launch failed");
  BwdArgs a;
  a.B = B; a.Tq = Tq; a.Tk = Tk; a.N = N; a.KH = KH;
  a.scale = scale; a.softcap = softcap; a.causal = causal; a.window = window; a.q_off = Tk - Tq;
  a.seg_q = nullptr; a.seg_k = nullptr; a.lse = lse; a.delta = delta; a.dQ = dq32;
  a.dK = reinterpret_cast<__nv_bfloat16*>(dk); a.dV = reinterpret_cast<__nv_bfloat16*>(dv);
  a.lddk = ldkv; a.lddv = ldkv; a.status = status;
  int rc;
  switch (H) {
    case 64: rc = launch_bwd<64>(q, k, v, dout, a, ldq, ldkv, ldkv, ldq, stream); break;
    case 128: rc = launch_bwd<128>(q, k, v, dout, a, ldq, ldkv, ldkv, ldq, stream); break;
    default: rc = launch_bwd<256>(q, k, v, dout, a, ldq, ldkv, ldkv, ldq, stream); break;
  }
  if (rc) return noalloc_fail(rc, "backward launch failed");
  noalloc_cast_kernel<<<592, 256, 0, stream>>>(dq32, (__nv_bfloat16*)dq, dq_elems);
  return cudaGetLastError() == cudaSuccess ? 0 : noalloc_fail(-5, "kernel launch failed");
}
