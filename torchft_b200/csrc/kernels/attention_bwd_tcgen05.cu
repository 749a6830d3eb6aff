// Causal grouped-query attention, backward pass, on the 5th-generation tensor cores.
//
// One CTA owns one (batch, kv head, 128-key block) and walks over every query head of the
// group and every 64-query tile that can see the block.  Scores are formed transposed, keys on
// the TMEM lanes and queries on the columns, so every MMA has M = 128:
//
//   S^T  = K  Q^T            [keys x q]      A = K   (K-major)      B = Q   (K-major)
//   dP^T = V  dO^T           [keys x q]      A = V   (K-major)      B = dO  (K-major)
//   P^T  = exp2(c S^T - lse),  dS^T = scale * P^T (dP^T - delta)     (softmax warps)
//   dV  += P^T  dO           [keys x d]      A = P^T (K-major)      B = dO  (MN-major)
//   dK  += dS^T Q            [keys x d]      A = dS^T (K-major)     B = Q   (MN-major)
//   dQ^T = K^T  dS^T         [d x q]         A = K   (MN-major)     B = dS^T (MN-major)
//
// P^T and dS^T go back, as packed bf16, into the TMEM columns their scores came from and are the
// A operands of the dV and dK MMAs straight from tensor memory; dS^T is also written to shared
// memory (128-byte swizzle) as the MN-major B operand of the dQ^T MMA.  dK and dV stay in TMEM for the
// whole CTA; dQ^T is drained every tile and added to an fp32 accumulator in global memory (four
// queries of a head-dim element per reduction, 512 consecutive bytes per warp instruction).
//
// Warps: 0 = TMA (K, V once; Q, dO, lse, delta per tile, 3 stages), 1 = MMA issue, 2..9 and 10..17 =
// two softmax groups that take the tiles in turn (and together store dK, dV at the end), 18..21 = dQ
// drain.  S^T and dP^T have two buffers each, and dQ^T of a tile takes the place of its dP^T, which fills
// the 512 TMEM columns:
//   issue order   dQ(t-1) dV(t-1) dK(t-1) | S(t+1) dP(t+1) | dQ(t) ...
// so that the softmax of one tile runs beside that of the other, and dQ(t-1) is drained under dV(t-1),
// dK(t-1) and S(t+1), before dP(t+1) needs its columns.  All waits are bounded.
//
// What bounds it: a tile's MMAs take 1650 cycles by themselves, a tile 3300.  The exponentials, the stores
// of dS^T and the reductions can each be taken out for 0 to 3 %, so the difference is taken to be the
// instruction stream of the MMA warp and its waits next to 21 other warps.  704 threads leave 80 registers a
// thread, and the softmax spills: 40 bytes of stores and 72 of loads at head dim 128, 48 and 156 at 64
// (ptxas); what that costs is not measured.
// 8 x 2048, 32/8 heads of 64: 930 us with one softmax group of 16 warps and scalar reductions, 777 us with
// two (442 TFLOP/s); 1 x 8192, heads of 128: 1706 us either way.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <math.h>

#include "ftb200_common.cuh"
#include "tcgen05_helpers.cuh"

namespace {

using namespace ftb200::tc;

constexpr int BKV = 128;
constexpr int BQ = 64;
constexpr int NUM_THREADS = 704;
constexpr int SOFTMAX_WARPS = 16;
constexpr int DRAIN_WARPS = 4;
constexpr int GROUP_WARPS = SOFTMAX_WARPS / 2;  // softmax warps per tile
constexpr int CPT = BQ / 2;        // query columns per thread: two threads per key row and tile
constexpr int CHUNK = 16;          // of them at a time
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t COL_S = 0, COL_DP = 128, COL_DV = 256, COL_DK = 384;  // dQ^T where dP^T was
constexpr uint32_t KV_SLAB = BKV * 128;        // 16 KB: [128 rows x 128 B], 64 head-dim elements per row
constexpr uint32_t Q_SLAB = BQ * 128;          // 8 KB: [64 rows x 128 B]
constexpr uint32_t PT_TILE = BKV * BQ * 2;     // 16 KB, one slab of [128 key rows x 64 q]
constexpr int QDO_STAGES = 3;  // a stage is held until the tile's dV/dK MMAs are done, two tiles after its load began
constexpr uint32_t PDS_BYTES = PT_TILE;        // dS^T only: P^T never leaves tensor memory
constexpr uint32_t STATS_BYTES = 2 * BQ * 4;   // per stage: lse[64], delta[64]

// Shared-memory layout for head dim D (64 or 128): K and V tiles of D/64 slabs each, then the Q/dO stages, the
// dS^T buffers, the statistics and the barriers.
template <int D>
struct Lay {
  static constexpr int SLABS = D / 64;
  static constexpr uint32_t KV_TILE = SLABS * KV_SLAB;
  static constexpr uint32_t Q_TILE = SLABS * Q_SLAB;
  static constexpr uint32_t OFF_K = 0, OFF_V = KV_TILE;
  static constexpr uint32_t OFF_STAGE = 2 * KV_TILE;    // per stage: Q, dO
  static constexpr uint32_t STAGE_BYTES = 2 * Q_TILE;
  static constexpr uint32_t OFF_PDS = OFF_STAGE + QDO_STAGES * STAGE_BYTES;  // per buffer: dS^T
  static constexpr uint32_t OFF_STATS = OFF_PDS + 2 * PDS_BYTES;
  static constexpr uint32_t OFF_MISC = OFF_STATS + QDO_STAGES * STATS_BYTES;
  static constexpr uint32_t SMEM_BYTES = OFF_MISC + 256 + 1024;
  static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB of shared memory a CTA can have");
};

enum : int {
  BAR_KV = 0,
  BAR_QDO_FULL = 1,   // +stage (3)
  BAR_QDO_EMPTY = 4,  // +stage (3)
  BAR_S_FULL = 7,     // +buf
  BAR_DP_FULL = 9,    // +buf
  BAR_PDS_FULL = 11,  // +buf
  BAR_DQ_FULL = 13,   // +buf
  BAR_DQ_EMPTY = 15,  // +buf
  BAR_DKV_DONE = 17,
  NUM_BARS = 18,
};

struct BwdParams {
  int batch, seq, n_heads, n_kv_heads;
  int causal;
  float scale, scale_log2;
  const float* neg_lse2;   // [batch, n_heads, seq], -log2(e) times the forward's log-sum-exp
  const float* neg_delta;  // [batch, n_heads, seq], -scale times delta
  float* dq_acc;           // fp32, zeroed; per 64-query tile and head: [16][D][4 queries]
  __nv_bfloat16* dK;   // rows batch*seq, row stride ld_dk
  __nv_bfloat16* dV;
  long long ld_dk, ld_dv;
  int* status;
};

__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void red_add_v4(float* dst, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

template <int D>
__global__ void __launch_bounds__(NUM_THREADS, 1)
attention_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                     const BwdParams p) {
  using Ly = Lay<D>;
  constexpr int SLABS = Ly::SLABS;
  constexpr uint32_t KV_TILE = Ly::KV_TILE, Q_TILE = Ly::Q_TILE, OFF_K = Ly::OFF_K, OFF_V = Ly::OFF_V;
  constexpr uint32_t OFF_STAGE = Ly::OFF_STAGE, STAGE_BYTES = Ly::STAGE_BYTES, OFF_PDS = Ly::OFF_PDS;
  constexpr uint32_t OFF_STATS = Ly::OFF_STATS, OFF_MISC = Ly::OFF_MISC;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_MISC);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_MISC + 192);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + OFF_MISC + 196);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar_base = smem_u32(bars);
  auto bar = [&](int i) { return bar_base + 8u * i; };

  // early key blocks see the most queries under a causal mask: schedule them first
  const int per_block = p.batch * p.n_kv_heads;
  const int jb = static_cast<int>(blockIdx.x) / per_block;
  const int bh = static_cast<int>(blockIdx.x) % per_block;
  const int b = bh / p.n_kv_heads, hk = bh % p.n_kv_heads;
  const int rep = p.n_heads / p.n_kv_heads;
  const int n_qtiles = p.seq / BQ;
  const int first_q = p.causal ? (jb * BKV) / BQ : 0;
  const int T = rep * (n_qtiles - first_q);
  const int kv_row0 = b * p.seq + jb * BKV;
  // tiles in order: the queries of a head that see the block, then the next head of the group
  struct TileWalk {
    int h, qt;
  };
  auto next_tile = [&](TileWalk& w) {
    if (++w.qt == n_qtiles) {
      w.qt = first_q;
      ++w.h;
    }
  };

  if (threadIdx.x == 0) {
    mbar_init(bar(BAR_KV), 1);
    for (int s = 0; s < QDO_STAGES; ++s) {
      mbar_init(bar(BAR_QDO_FULL + s), 1);
      mbar_init(bar(BAR_QDO_EMPTY + s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar(BAR_S_FULL + s), 1);
      mbar_init(bar(BAR_DP_FULL + s), 1);
      mbar_init(bar(BAR_PDS_FULL + s), GROUP_WARPS);
      mbar_init(bar(BAR_DQ_FULL + s), 1);
      mbar_init(bar(BAR_DQ_EMPTY + s), DRAIN_WARPS);
    }
    mbar_init(bar(BAR_DKV_DONE), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (elect_one()) {
      mbar_expect_tx(bar(BAR_KV), 2 * KV_TILE);
#pragma unroll
      for (int sl = 0; sl < SLABS; ++sl) {
        tma_load_2d(smem_base + OFF_K + sl * KV_SLAB, &tmK, bar(BAR_KV), hk * D + 64 * sl, kv_row0);
        tma_load_2d(smem_base + OFF_V + sl * KV_SLAB, &tmV, bar(BAR_KV), hk * D + 64 * sl, kv_row0);
      }
    }
    __syncwarp();
    bool ok = true;
    TileWalk w{hk * rep, first_q};
    for (int t = 0; t < T && ok; ++t, next_tile(w)) {
      const int st = t % QDO_STAGES;
      const uint32_t use = static_cast<uint32_t>(t / QDO_STAGES);
      if (!mbar_wait_warp(bar(BAR_QDO_EMPTY + st), (use & 1u) ^ 1u, abort_flag)) {
        ok = false;
        break;
      }
      const int h = w.h, qt = w.qt;
      const int q_row0 = b * p.seq + qt * BQ;
      const uint32_t sq = smem_base + OFF_STAGE + st * STAGE_BYTES;
      const uint32_t sdo = sq + Q_TILE;
      const uint32_t sst = smem_base + OFF_STATS + st * STATS_BYTES;
      const long long stat_off = (static_cast<long long>(b) * p.n_heads + h) * p.seq + qt * BQ;
      if (elect_one()) {
        mbar_expect_tx(bar(BAR_QDO_FULL + st), 2 * Q_TILE + STATS_BYTES);
#pragma unroll
        for (int sl = 0; sl < SLABS; ++sl) {
          tma_load_2d(sq + sl * Q_SLAB, &tmQ, bar(BAR_QDO_FULL + st), h * D + 64 * sl, q_row0);
          tma_load_2d(sdo + sl * Q_SLAB, &tmDO, bar(BAR_QDO_FULL + st), h * D + 64 * sl, q_row0);
        }
        bulk_load_1d(sst, p.neg_lse2 + stat_off, BQ * 4, bar(BAR_QDO_FULL + st));
        bulk_load_1d(sst + BQ * 4, p.neg_delta + stat_off, BQ * 4, bar(BAR_QDO_FULL + st));
      }
      __syncwarp();
    }
    if (!ok) {
      const uint64_t t0 = ftb200::globaltimer_ns();
      while (ftb200::globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    const uint32_t F = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(128 >> 4) << 24);
    const uint32_t idesc_st = F | (static_cast<uint32_t>(BQ >> 3) << 17);                             // N = 64, K-major both
    const uint32_t idesc_kv = F | (1u << 16) | (static_cast<uint32_t>(D >> 3) << 17);                 // N = D, B MN-major
    const uint32_t idesc_dq = F | (1u << 15) | (1u << 16) | (static_cast<uint32_t>(BQ >> 3) << 17);   // N = 64, both MN-major
    // descriptor bases: one per buffer and operand role, constants per K step (the issue loop
    // must stay short: these MMAs are too small to hide descriptor arithmetic)
    constexpr uint32_t HI = smem_desc_hi(1024);
    const uint32_t k_km = smem_desc_lo(smem_base + OFF_K, 16);        // K as K-major A (S^T)
    const uint32_t v_km = smem_desc_lo(smem_base + OFF_V, 16);        // V as K-major A (dP^T)
    // K as MN-major A (dQ^T): M = 128 runs over the head dim.  With head dim 64 the second 64 rows of that MMA
    // read the slab behind K's only one, which is V's: lanes 64..127 of dQ^T then hold a product nobody reads.
    const uint32_t k_mn = smem_desc_lo(smem_base + OFF_K, KV_SLAB);
    const uint32_t q_km0 = smem_desc_lo(smem_base + OFF_STAGE, 16);             // Q, stage 0, K-major B
    const uint32_t q_mn0 = smem_desc_lo(smem_base + OFF_STAGE, Q_SLAB);         // Q, stage 0, MN-major B
    const uint32_t ds_mn0 = smem_desc_lo(smem_base + OFF_PDS, PT_TILE);  // dS^T, buffer 0, MN-major B
    constexpr uint32_t STAGE16 = STAGE_BYTES >> 4, QT16 = Q_TILE >> 4, PDS16 = PDS_BYTES >> 4;
    bool ok = mbar_wait_warp(bar(BAR_KV), 0, abort_flag);
    for (int t = 0; t <= T && ok; ++t) {
      if (t < T) {
        // S and dP of tile t; the MMAs that read P and dS of tile t - 2 from the same S buffer were issued before
        const int st = t & 1, qs = t % QDO_STAGES;
        const uint32_t use = static_cast<uint32_t>(t >> 1);
        if (!mbar_wait_warp(bar(BAR_QDO_FULL + qs), static_cast<uint32_t>(t / QDO_STAGES) & 1u, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t qb_km = q_km0 + qs * STAGE16;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t a_off = ((kk >> 2) * KV_SLAB + (kk & 3) * 32) >> 4, b_off = ((kk >> 2) * Q_SLAB + (kk & 3) * 32) >> 4;
            umma_bf16_lh(tmem_base + COL_S + st * BQ, k_km + a_off, HI, qb_km + b_off, HI, idesc_st, kk != 0);
          }
          umma_commit(bar(BAR_S_FULL + st));
        }
        __syncwarp();
        if (!mbar_wait_warp(bar(BAR_DQ_EMPTY + st), (use & 1u) ^ 1u, abort_flag)) {  // dQ of tile t - 2 drained
          ok = false;
          break;
        }
        tc_fence_after();
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t a_off = ((kk >> 2) * KV_SLAB + (kk & 3) * 32) >> 4, b_off = ((kk >> 2) * Q_SLAB + (kk & 3) * 32) >> 4;
            umma_bf16_lh(tmem_base + COL_DP + st * BQ, v_km + a_off, HI, qb_km + QT16 + b_off, HI, idesc_st, kk != 0);
          }
          umma_commit(bar(BAR_DP_FULL + st));
        }
        __syncwarp();
      }
      if (t >= 1) {
        const int u = t - 1, pb = u & 1, qs = u % QDO_STAGES;
        const uint32_t use = static_cast<uint32_t>(u >> 1);
        if (!mbar_wait_warp(bar(BAR_PDS_FULL + pb), use & 1u, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t qb_mn = q_mn0 + qs * STAGE16;
        const uint32_t dsb_mn = ds_mn0 + pb * PDS16;
        // queries 16k..16k+15 of tile u: P^T in columns 16k..16k+7 of its score buffer, dS^T in 16k+8..16k+15
        const uint32_t pt_tmem = tmem_base + COL_S + pb * BQ;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < BKV / 16; ++kk) {  // dQ^T = K^T dS^T, over dP^T of the tile (read by the softmax)
            umma_bf16_lh(tmem_base + COL_DP + pb * BQ, k_mn + ((kk * 2048) >> 4), HI, dsb_mn + ((kk * 2048) >> 4), HI, idesc_dq, kk != 0);
          }
          umma_commit(bar(BAR_DQ_FULL + pb));
#pragma unroll
          for (int kk = 0; kk < BQ / 16; ++kk) {  // dV += P^T dO
            umma_bf16_tmem_a(tmem_base + COL_DV, pt_tmem + kk * 16, qb_mn + QT16 + ((kk * 2048) >> 4), HI, idesc_kv, (u | kk) != 0);
          }
#pragma unroll
          for (int kk = 0; kk < BQ / 16; ++kk) {  // dK += dS^T Q
            umma_bf16_tmem_a(tmem_base + COL_DK, pt_tmem + kk * 16 + 8, qb_mn + ((kk * 2048) >> 4), HI, idesc_kv, (u | kk) != 0);
          }
          umma_commit(bar(BAR_QDO_EMPTY + qs));
        }
        __syncwarp();
      }
    }
    if (ok && elect_one()) umma_commit(bar(BAR_DKV_DONE));
    __syncwarp();
  } else if (warp >= 18) {
    // ---------------- dQ drain (warps 18..21): TMEM lane = head-dim index ----------------
    const int quarter = warp & 3;
    const int dcol = quarter * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    TileWalk w{hk * rep, first_q};
    for (int u = 0; u < T; ++u, next_tile(w)) {
      const int buf = u & 1;
      if (!mbar_wait_warp(bar(BAR_DQ_FULL + buf), static_cast<uint32_t>(u >> 1) & 1u, abort_flag)) break;
      tc_fence_after();
      uint32_t v[BQ];
      const bool mine = quarter * 32 < D;  // head dim 64: only lanes 0..63 of dQ^T are real
      if (mine) {
        tmem_ld32(tmem_base + COL_DP + buf * BQ + lane_addr, v);
        tmem_ld32(tmem_base + COL_DP + buf * BQ + 32 + lane_addr, v + 32);
        tmem_wait_ld();
      }
      tc_fence_before();
      mbar_arrive_warp(bar(BAR_DQ_EMPTY + buf));
      if (mine) {
        // four queries of one head-dim element lie together: a warp adds 512 consecutive bytes per instruction
        const long long tile = (static_cast<long long>(b) * n_qtiles + w.qt) * p.n_heads + w.h;
        float* dst = p.dq_acc + tile * (BQ * D) + dcol * 4;
#pragma unroll
        for (int c = 0; c < BQ / 4; ++c)
          red_add_v4(dst + c * (D * 4), __uint_as_float(v[4 * c]), __uint_as_float(v[4 * c + 1]), __uint_as_float(v[4 * c + 2]),
                     __uint_as_float(v[4 * c + 3]));
      }
    }
  } else {
    // ---------------- softmax, dK/dV store (warps 2..17) ----------------
    const int quarter = warp & 3;
    const int sw = (warp - 2) >> 2;       // four warps with the same columns
    const int grp = sw >> 1, g = sw & 1;  // which tiles (even or odd), which 32 of the tile's 64 queries
    const int row = quarter * 32 + lane;  // key within the block
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    bool ok = true;
    const unsigned long long scale2 = f2_pack(p.scale_log2, p.scale_log2), dscale2 = f2_pack(p.scale, p.scale);
    const int key = jb * BKV + row;
    TileWalk w{hk * rep, first_q};
    if (grp == 1) next_tile(w);
    const uint32_t s_addr = tmem_base + COL_S + grp * BQ + g * CPT + lane_addr;
    const uint32_t dp_addr = tmem_base + COL_DP + grp * BQ + g * CPT + lane_addr;
    uint8_t* drow = smem + OFF_PDS + grp * PDS_BYTES + row * 128;
    for (int t = grp; t < T; t += 2, next_tile(w), next_tile(w)) {
      const uint32_t use = static_cast<uint32_t>(t >> 1);
      const int qs = t % QDO_STAGES;
      // the tile's statistics arrived with Q and dO
      if (!mbar_wait_warp(bar(BAR_S_FULL + grp), use & 1u, abort_flag) ||
          !mbar_wait_warp(bar(BAR_QDO_FULL + qs), static_cast<uint32_t>(t / QDO_STAGES) & 1u, abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after();
      // pairs of -log2(e) lse and -scale delta, as the packed arithmetic takes them
      const ulonglong2* stats2 = reinterpret_cast<const ulonglong2*>(smem + OFF_STATS + qs * STATS_BYTES) + g * (CPT / 4);
      const int q0 = w.qt * BQ + g * CPT;
      const bool diag = (p.causal != 0) && (q0 < jb * BKV + BKV);
#pragma unroll
      for (int cc = 0; cc < CPT / CHUNK; ++cc) {
        uint32_t sv[CHUNK], dp[CHUNK];
        tmem_ld16(s_addr + cc * CHUNK, sv);
        if (cc > 0) tmem_ld16(dp_addr + cc * CHUNK, dp);
        tmem_wait_ld();
        float pe[CHUNK];
#pragma unroll
        for (int c = 0; c < CHUNK / 4; ++c) {
          const ulonglong2 l4 = stats2[cc * (CHUNK / 4) + c];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int qi = 4 * c + 2 * e;
            const unsigned long long x2 =
                f2_fma(f2_pack(__uint_as_float(sv[qi]), __uint_as_float(sv[qi + 1])), scale2, e == 0 ? l4.x : l4.y);
            f2_unpack(x2, pe[qi], pe[qi + 1]);
            pe[qi] = exp2f(pe[qi]);
            pe[qi + 1] = exp2f(pe[qi + 1]);
          }
        }
        if (diag) {
#pragma unroll
          for (int c = 0; c < CHUNK; ++c)
            if (key > q0 + cc * CHUNK + c) pe[c] = 0.f;
        }
        if (cc == 0) {
          if (!mbar_wait_warp(bar(BAR_DP_FULL + grp), use & 1u, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          tmem_ld16(dp_addr, dp);
          tmem_wait_ld();
        }
        uint32_t pds[CHUNK];  // P^T, dS^T
#pragma unroll
        for (int c = 0; c < CHUNK / 4; ++c) {
          const ulonglong2 d4 = stats2[BQ / 4 + cc * (CHUNK / 4) + c];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int qi = 4 * c + 2 * e;
            // dS = P (scale dP - scale delta)
            const unsigned long long ds2 =
                f2_mul(f2_pack(pe[qi], pe[qi + 1]),
                       f2_fma(f2_pack(__uint_as_float(dp[qi]), __uint_as_float(dp[qi + 1])), dscale2, e == 0 ? d4.x : d4.y));
            float s0, s1;
            f2_unpack(ds2, s0, s1);
            __nv_bfloat162 a = __floats2bfloat162_rn(pe[qi], pe[qi + 1]);
            __nv_bfloat162 d2 = __floats2bfloat162_rn(s0, s1);
            pds[qi / 2] = *reinterpret_cast<uint32_t*>(&a);
            pds[CHUNK / 2 + qi / 2] = *reinterpret_cast<uint32_t*>(&d2);
          }
        }
        // the dS^T buffer is free once dQ^T of the group's tile before is complete
        if (cc == 0 && !mbar_wait_warp(bar(BAR_DQ_FULL + grp), (use & 1u) ^ 1u, abort_flag)) {
          ok = false;
          break;
        }
        // P^T and dS^T replace the scores this thread has just read (its own 16 columns)
        tmem_st16(s_addr + cc * CHUNK, pds);
#pragma unroll
        for (int c = 0; c < CHUNK / 8; ++c) {
          const int chunk = ((g * (CPT / 8) + cc * (CHUNK / 8) + c) ^ (row & 7)) << 4;
          *reinterpret_cast<uint4*>(drow + chunk) = make_uint4(pds[CHUNK / 2 + 4 * c], pds[CHUNK / 2 + 4 * c + 1],
                                                               pds[CHUNK / 2 + 4 * c + 2], pds[CHUNK / 2 + 4 * c + 3]);
        }
      }
      if (!ok) break;
      fence_async_smem();
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(bar(BAR_PDS_FULL + grp));
    }
    if (ok && mbar_wait_warp(bar(BAR_DKV_DONE), 0, abort_flag)) {
      tc_fence_after();
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        constexpr int CW = D / 4;  // head-dim columns per thread
        const uint32_t col = (which == 0 ? COL_DV : COL_DK) + sw * CW;
        __nv_bfloat16* base = which == 0 ? p.dV : p.dK;
        const long long ld = which == 0 ? p.ld_dv : p.ld_dk;
        __nv_bfloat16* dst = base + static_cast<long long>(kv_row0 + row) * ld + hk * D + sw * CW;
        uint32_t v[CW];
        if constexpr (CW == 32)
          tmem_ld32(tmem_base + col + lane_addr, v);
        else
          tmem_ld16(tmem_base + col + lane_addr, v);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < CW / 8; ++c) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[8 * c + e]);
          reinterpret_cast<ftb200::bf16x8*>(dst)[c] = ftb200::pack8(f);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag && p.status != nullptr) atomicExch(p.status, FTB200_ST_TIMEOUT);
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// Before the main kernel, one pass over O and dO: neg_delta[b, h, s] = -scale sum_d dO O, neg_lse2 = -log2(e) lse, and the dQ
// accumulator zeroed.  A thread takes 8 elements (16 bytes of each), D / 8 neighbouring lanes a (row, head).
template <int D>
__global__ void __launch_bounds__(256) attention_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o,
                                                                 const __nv_bfloat16* __restrict__ d_o,
                                                                 const float* __restrict__ lse, float* __restrict__ neg_lse2,
                                                                 float* __restrict__ neg_delta, float4* __restrict__ dq_acc,
                                                                 int seq, int n_heads, long long pieces, long long ld_o,
                                                                 long long ld_do, float scale) {
  constexpr int LANES = D / 8;
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool live = i < pieces;
  const int per_row = n_heads * LANES;
  const int r = static_cast<int>((live ? i : 0) / per_row);  // batch * seq rows fit an int (the host checks)
  const int c = static_cast<int>((live ? i : 0) - static_cast<long long>(r) * per_row);
  float s = 0.f;
  if (live) {
    float x[8], y[8];
    ftb200::unpack8(*reinterpret_cast<const ftb200::bf16x8*>(o + r * ld_o + c * 8), x);
    ftb200::unpack8(*reinterpret_cast<const ftb200::bf16x8*>(d_o + r * ld_do + c * 8), y);
    dq_acc[2 * i] = make_float4(0.f, 0.f, 0.f, 0.f);
    dq_acc[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int e = 0; e < 8; ++e) s = fmaf(x[e], y[e], s);
  }
#pragma unroll
  for (int k = LANES / 2; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
  if (live && c % LANES == 0) {
    const long long at = (static_cast<long long>(r / seq) * n_heads + c / LANES) * seq + r % seq;
    neg_delta[at] = -s * scale;
    neg_lse2[at] = lse[at] * -1.4426950408889634f;
  }
}

// dq (bf16, row stride ld) = accumulator (fp32, per 64-query tile and head [16][D][4 queries]); a thread takes 8
// head-dim elements of 4 queries.
template <int D>
__global__ void __launch_bounds__(256) attention_dq_cast_kernel(const float4* __restrict__ acc, __nv_bfloat16* __restrict__ dq,
                                                                long long pieces, int n_heads, long long ld) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= pieces) return;
  const int d8 = static_cast<int>(i % (D / 8));
  const long long g = i / (D / 8);  // (tile, head, group of 4 queries)
  const int q4 = static_cast<int>(g & 15);
  const long long th = g >> 4;
  const int h = static_cast<int>(th % n_heads);
  const long long row0 = th / n_heads * 64 + q4 * 4;
  float4 v[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) v[e] = acc[g * D + d8 * 8 + e];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float f[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = k == 0 ? v[e].x : k == 1 ? v[e].y : k == 2 ? v[e].z : v[e].w;
    *reinterpret_cast<ftb200::bf16x8*>(dq + (row0 + k) * ld + h * D + d8 * 8) = ftb200::pack8(f);
  }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(sym);
    }
  }
  return fn;
}

int encode_rows(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows) {
  auto fn = encode_fn();
  if (fn == nullptr) return FTB200_E_DRIVER;
  cuuint64_t gdim[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t gstride[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2] = {64u, static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), gdim, gstride, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : FTB200_E_DRIVER;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

// Scratch the backward pass needs, in bytes: fp32 dQ accumulator, -scale delta, -log2(e) lse.
// (sized for head dim 128; enough for 64 as well)
FTB200_API long long ftb200_attention_bwd_scratch_bytes(int batch, int seq, int n_heads) {
  const long long rows = static_cast<long long>(batch) * seq;
  return rows * n_heads * 128 * 4 + 2 * rows * n_heads * 4;
}

namespace {

template <int D>
int attention_bwd_impl(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                       void* dq, void* dk, void* dv, void* scratch, int batch, int seq, int n_heads, int n_kv_heads,
                       long long ld_q, long long ld_k, long long ld_v, long long ld_o, long long ld_do, long long ld_dq,
                       long long ld_dk, long long ld_dv, float scale, int causal, int* status, cudaStream_t stream) {
  constexpr uint32_t SMEM_BYTES = Lay<D>::SMEM_BYTES;
  const long long rows = static_cast<long long>(batch) * seq;
  float* dq_acc = reinterpret_cast<float*>(scratch);
  float* neg_delta = dq_acc + rows * n_heads * D;
  float* neg_lse2 = neg_delta + rows * n_heads;
  if (rows > 0x7fffffffLL) return FTB200_E_TOOBIG;
  CUtensorMap tq, tk, tv, tdo;
  int rc = encode_rows(&tq, q, rows, static_cast<long long>(n_heads) * D, ld_q, BQ);
  if (rc == 0) rc = encode_rows(&tdo, d_o, rows, static_cast<long long>(n_heads) * D, ld_do, BQ);
  if (rc == 0) rc = encode_rows(&tk, k, rows, static_cast<long long>(n_kv_heads) * D, ld_k, BKV);
  if (rc == 0) rc = encode_rows(&tv, v, rows, static_cast<long long>(n_kv_heads) * D, ld_v, BKV);
  if (rc != 0) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(attention_bwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) !=
        cudaSuccess)
      return FTB200_E_CUDA;
    attr_set = true;
  }
  const long long pieces = rows * n_heads * (D / 8);
  if ((pieces + 255) / 256 > 0x7fffffffLL) return FTB200_E_TOOBIG;
  attention_bwd_prep_kernel<D><<<static_cast<unsigned>((pieces + 255) / 256), 256, 0, stream>>>(
      reinterpret_cast<const __nv_bfloat16*>(o), reinterpret_cast<const __nv_bfloat16*>(d_o), lse, neg_lse2, neg_delta,
      reinterpret_cast<float4*>(dq_acc), seq, n_heads, pieces, ld_o, ld_do, scale);
  BwdParams p;
  p.batch = batch; p.seq = seq; p.n_heads = n_heads; p.n_kv_heads = n_kv_heads; p.causal = causal;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.neg_lse2 = neg_lse2; p.neg_delta = neg_delta; p.dq_acc = dq_acc;
  p.dK = reinterpret_cast<__nv_bfloat16*>(dk); p.dV = reinterpret_cast<__nv_bfloat16*>(dv);
  p.ld_dk = ld_dk; p.ld_dv = ld_dv; p.status = status;
  const long long grid = static_cast<long long>(batch) * n_kv_heads * (seq / BKV);
  if (grid > 0x7fffffffLL) return FTB200_E_TOOBIG;
  attention_bwd_kernel<D><<<static_cast<unsigned>(grid), NUM_THREADS, SMEM_BYTES, stream>>>(tq, tk, tv, tdo, p);
  attention_dq_cast_kernel<D><<<static_cast<unsigned>((pieces / 4 + 255) / 256), 256, 0, stream>>>(
      reinterpret_cast<const float4*>(dq_acc), reinterpret_cast<__nv_bfloat16*>(dq), pieces / 4, n_heads, ld_dq);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

}  // namespace

// q, k, v, o, d_o as in the forward pass (2-D views, row strides in elements); dq, dk, dv are
// written (not accumulated).  lse is the forward's [batch, n_heads, seq].  scratch: at least
// ftb200_attention_bwd_scratch_bytes, 16-byte aligned.  Head dim 64 or 128.
FTB200_API int ftb200_attention_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                                    const float* lse, void* dq, void* dk, void* dv, void* scratch, int batch, int seq,
                                    int n_heads, int n_kv_heads, int head_dim, long long ld_q, long long ld_k,
                                    long long ld_v, long long ld_o, long long ld_do, long long ld_dq, long long ld_dk,
                                    long long ld_dv, float scale, int causal, int* status, cudaStream_t stream) {
  if ((head_dim != 64 && head_dim != 128) || batch <= 0 || seq <= 0 || seq % BKV != 0 || n_heads <= 0 ||
      n_kv_heads <= 0 || n_heads % n_kv_heads != 0)
    return FTB200_E_BADARG;
  const void* ptrs[] = {q, k, v, o, d_o, dq, dk, dv, scratch};
  for (const void* x : ptrs)
    if (!aligned16(x)) return FTB200_E_ALIGN;
  const long long lds[] = {ld_q, ld_k, ld_v, ld_o, ld_do, ld_dq, ld_dk, ld_dv};
  for (long long x : lds)
    if (x & 7) return FTB200_E_ALIGN;
  if (head_dim == 64)
    return attention_bwd_impl<64>(q, k, v, o, d_o, lse, dq, dk, dv, scratch, batch, seq, n_heads, n_kv_heads, ld_q, ld_k,
                                  ld_v, ld_o, ld_do, ld_dq, ld_dk, ld_dv, scale, causal, status, stream);
  return attention_bwd_impl<128>(q, k, v, o, d_o, lse, dq, dk, dv, scratch, batch, seq, n_heads, n_kv_heads, ld_q, ld_k,
                                 ld_v, ld_o, ld_do, ld_dq, ld_dk, ld_dv, scale, causal, status, stream);
}
