// Causal grouped-query attention, backward pass, on the 5th-generation tensor cores.
//
// One CTA owns one (batch, kv head, 128-key block) and walks over every query head of the
// group (where that would leave SMs idle, over a share of them: head_split) and every 128-query tile that can
// see the block.  Scores are formed transposed, keys on the TMEM lanes and queries on the columns, so every MMA has M = 128:
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
// whole CTA; dQ^T is drained every tile: a drain warp puts its 32 head-dim elements into shared memory, a quarter of the queries
// at a time, and each quarter is added to an fp32 accumulator in global memory by one bulk reduction of 4 KB.
//
// Warps: 0 = TMA (K, V once; Q with lse and delta, dO per tile), 1 = MMA issue, 4..7 = dQ drain, 8..15 = softmax (two
// threads per key, 64 queries each; together they store dK, dV at the end).  Issue order of a tile t:
//   dV(t) S(t+1) dK(t) dQ(t) dP(t+1)
// so that the exponentials of t + 1 run under dK(t), dQ(t) and dP(t+1), and dS(t) is formed under dV(t) and S(t+1).  At head
// dim 128 the 512 TMEM columns are full and dQ^T takes the place of its dP^T, so dP(t+1) waits until it is drained; at
// head dim 64 it has columns of its own.
//
// What bounds it: at head dim 128 the sum of dQ^T.  A tile's 64 KB leave an SM at about 21 bytes a cycle as bulk reductions
// (whatever their size, 4 or 16 KB) and at 25 as red.v4; the latter go through the load/store pipe that the softmax needs
// for dS^T and the statistics, whose second half then takes 2570 cycles instead of 1020 (800 with no reductions at all).  A
// tile takes 3750 cycles: 4890 with red.v4, 3250 with no reductions, 2600 for its 40 MMAs, 2048 + 1000 for what they, the
// TMA and the softmax move through shared memory at 128 bytes a cycle.  dO has one stage there, as the staging of dQ^T takes
// the second one's place.  At head dim 64 it is the chain of the softmax, 2830 cycles a tile
// (the slope over one CTA's chain of 32, 64 and 128 tiles).  Starts, ends and the last wave included a tile costs an SM 4210
// cycles at 1 x 8192 and 3650 at 8 x 2048, heads of 64.
// The warp's index and the TMEM base are read from lane 0 (shfl): then the branch and the addresses are known to be the
// same in all lanes and the MMAs' descriptors stay in uniform registers (1494 -> 1437 us, 650 -> 605 us).
// 1 x 8192, 32/8 heads of 128: 1705 us with 64-query tiles, 1290 us (1065 TFLOP/s) with these; 8 x 2048, heads of 64: 785 -> 592 us.
//
// Sequences of any length: the tensor maps have the sequence as a dimension of its own, so a tile's rows beyond its end are
// zeros.  The statistics and the dQ accumulator are laid out for whole tiles; a query beyond the end has the log-sum-exp
// +infinity there, so its probabilities are zero, and dQ, dK and dV beyond the end are not stored.
//
// Every mbarrier wait is bounded; on expiry the CTA records FTB200_ST_TIMEOUT in the caller's
// status word, frees its TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <math.h>

#include "ftb200_common.cuh"
#include "tcgen05_helpers.cuh"

namespace {

using namespace ftb200::tc;

constexpr int BKV = 128;
constexpr int BQ = 128;
constexpr int NUM_THREADS = 512;
constexpr int SOFTMAX_WARPS = 8;
constexpr int DRAIN_WARPS = 4;
// Registers: a CTA is launched with 128 a thread (65536 / 512, checked on the host) and shares them out by warpgroup:
// TMA and MMA issue, drain (128 elements of dQ^T in flight), two of softmax (a thread keeps 64 probabilities).
constexpr int LAUNCH_REGS = 128, ISSUE_REGS = 48, DRAIN_REGS = 144, SOFTMAX_REGS = 160;
static_assert(ISSUE_REGS + DRAIN_REGS + 2 * SOFTMAX_REGS <= 4 * LAUNCH_REGS, "more registers than the CTA is launched with");
constexpr int CPT = BQ / 2;        // query columns per softmax thread: two threads per key row
constexpr int CHUNK = 16;          // of them at a time where dP^T is read
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t SLAB = 128 * 128;           // 16 KB: [128 rows x 128 B], 64 elements per row
constexpr int STAGES = 2;                      // of Q; of dO as well at head dim 64
constexpr uint32_t DS_BYTES = BKV * BQ * 2;    // dS^T, two slabs of 64 queries
constexpr uint32_t STATS_BYTES = 2 * BQ * 4;   // per stage of Q: lse[128], delta[128]
constexpr int DQ_PARTS = 4;                    // a drain warp's 32 x 128 elements of dQ^T leave in so many bulk reductions,
constexpr uint32_t DQ_PART_BYTES = 32 * BQ * 4 / DQ_PARTS;  // from two buffers of its own

// Shared-memory layout and TMEM columns for head dim D (64 or 128): K and V tiles of D/64 slabs each, then the Q and
// dO stages, dS^T, the statistics and the barriers.
template <int D>
struct Lay {
  static constexpr int SLABS = D / 64;
  static constexpr uint32_t TILE = SLABS * SLAB;  // 128 rows of K, V, Q or dO
  static constexpr uint32_t OFF_K = 0, OFF_V = TILE;
  static constexpr uint32_t OFF_Q = 2 * TILE;               // per stage: Q
  static constexpr int DO_STAGES = D == 128 ? 1 : 2;         // one: it is free from dV on and needed again three products later
  static constexpr uint32_t OFF_DO = OFF_Q + STAGES * TILE;  // per stage: dO
  static constexpr uint32_t OFF_DS = OFF_DO + DO_STAGES * TILE;
  static constexpr uint32_t OFF_DQ = OFF_DS + DS_BYTES;      // per drain warp: two parts of dQ^T
  static constexpr uint32_t OFF_STATS = OFF_DQ + DRAIN_WARPS * 2 * DQ_PART_BYTES;
  static constexpr uint32_t OFF_MISC = OFF_STATS + STAGES * STATS_BYTES;
  static constexpr uint32_t SMEM_BYTES = OFF_MISC + 256;
  static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB of shared memory a CTA can have");
  static constexpr uint32_t COL_S = 0, COL_DP = 128, COL_DV = 256, COL_DK = 256 + D;
  // head dim 128 fills the 512 columns: dQ^T takes the place of its dP^T (and of dS^T, once dK has read it)
  static constexpr bool DQ_OVER_DP = D == 128;
  static constexpr uint32_t COL_DQ = DQ_OVER_DP ? COL_DP : 256 + 2 * D;
};

enum : int {
  BAR_KV = 0,
  BAR_Q_FULL = 1,    // +stage
  BAR_Q_EMPTY = 3,   // +stage
  BAR_DO_FULL = 5,   // +stage
  BAR_DO_EMPTY = 7,  // +stage
  BAR_S_FULL = 9,
  BAR_P_READY = 10,
  BAR_DP_FULL = 11,
  BAR_DS_READY = 12,
  BAR_DQ_FULL = 13,
  BAR_DQ_EMPTY = 14,
  BAR_DKV_DONE = 15,
  NUM_BARS = 16,
};

struct BwdParams {
  int batch, seq, n_heads, n_kv_heads;
  int causal;
  float scale, scale_log2;
  const float* neg_lse2;   // [batch, n_heads, whole tiles of seq], -log2(e) times the forward's log-sum-exp
  const float* neg_delta;  // the same, -scale times delta
  float* dq_acc;           // fp32, zeroed; per 128 queries and head: [D / 32][32 groups of 4 queries][32][4 queries]
  __nv_bfloat16* dK;   // rows batch*seq, row stride ld_dk
  __nv_bfloat16* dV;
  long long ld_dk, ld_dv;
  int split;           // CTAs that share the query heads of a kv head
  float4* dkv_part;    // split > 1: their dV and dK, fp32, per (batch, kv head, key block, share) [2][D / 4][128 keys][4]
  const float4* rope;  // null, or (cos, sin) pairs [seq][D / 2]: dQ and dK are rotated back
  int* status;
};

// Eight elements (four pairs) rotated back by their angles (cos, sin, cos, sin).
__device__ __forceinline__ void rotate_back(float* f, const float4& c0, const float4& c1) {
  const float cosv[4] = {c0.x, c0.z, c1.x, c1.z}, sinv[4] = {c0.y, c0.w, c1.y, c1.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float a = f[2 * e], b = f[2 * e + 1];
    f[2 * e] = a * cosv[e] + b * sinv[e];
    f[2 * e + 1] = b * cosv[e] - a * sinv[e];
  }
}

__device__ __forceinline__ void bulk_load_1d(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// Adds `bytes` of shared memory to global memory as fp32.  The calling thread's bulk group has to be committed.
__device__ __forceinline__ void bulk_add_f32(float* dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes)
               : "memory");
}

template <int D>
__global__ void __launch_bounds__(NUM_THREADS, 1)
attention_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                     const BwdParams p) {
  using Ly = Lay<D>;
  constexpr int SLABS = Ly::SLABS;
  constexpr uint32_t TILE = Ly::TILE;
  extern __shared__ __align__(1024) uint8_t smem[];  // swizzled tiles start at multiples of 1024 (checked)
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Ly::OFF_MISC);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Ly::OFF_MISC + 192);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + Ly::OFF_MISC + 196);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar_base = smem_u32(bars);
  auto bar = [&](int i) { return bar_base + 8u * i; };

  // tiles have to start at their swizzle atom; there is no room to move them up to it
  if ((smem_base & 1023u) != 0) {
    ftb200::wait_for_previous();
    if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, FTB200_ST_BOUNDS);
    return;
  }

  // early key blocks see the most queries under a causal mask: schedule them first
  const int per_block = p.batch * p.n_kv_heads * p.split;
  const int jb = static_cast<int>(blockIdx.x) / per_block;
  const int share = static_cast<int>(blockIdx.x) % p.split;
  const int bh = static_cast<int>(blockIdx.x) % per_block / p.split;
  const int b = bh / p.n_kv_heads, hk = bh % p.n_kv_heads;
  const int rep = p.n_heads / p.n_kv_heads / p.split;  // of this CTA
  const int h0 = (hk * p.split + share) * rep;
  const int n_qtiles = (p.seq + BQ - 1) / BQ;
  const int first_q = p.causal ? jb : 0;
  const int T = rep * (n_qtiles - first_q);
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
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar(BAR_Q_FULL + s), 1);
      mbar_init(bar(BAR_Q_EMPTY + s), 1);
      mbar_init(bar(BAR_DO_FULL + s), 1);
      mbar_init(bar(BAR_DO_EMPTY + s), 1);
    }
    mbar_init(bar(BAR_S_FULL), 1);
    mbar_init(bar(BAR_P_READY), SOFTMAX_WARPS);
    mbar_init(bar(BAR_DP_FULL), 1);
    mbar_init(bar(BAR_DS_READY), SOFTMAX_WARPS);
    mbar_init(bar(BAR_DQ_FULL), 1);
    mbar_init(bar(BAR_DQ_EMPTY), DRAIN_WARPS);
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
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  ftb200::wait_for_previous();

  if (warp < 4) {
    regs_dec<ISSUE_REGS>();
    if (warp == 0) {
      // ---------------- TMA producer ----------------
      if (elect_one()) {
        mbar_expect_tx(bar(BAR_KV), 2 * TILE);
#pragma unroll
        for (int sl = 0; sl < SLABS; ++sl) {
          tma_load_3d(smem_base + Ly::OFF_K + sl * SLAB, &tmK, bar(BAR_KV), hk * D + 64 * sl, jb * BKV, b);
          tma_load_3d(smem_base + Ly::OFF_V + sl * SLAB, &tmV, bar(BAR_KV), hk * D + 64 * sl, jb * BKV, b);
        }
      }
      __syncwarp();
      bool ok = true;
      TileWalk w{h0, first_q};
      for (int t = 0; t < T && ok; ++t, next_tile(w)) {
        const int st = t % STAGES;
        const uint32_t was = static_cast<uint32_t>(t / STAGES) & 1u ^ 1u;
        const int dst = t % Ly::DO_STAGES;
        const int q0 = w.qt * BQ;
        const long long stat_off = ((static_cast<long long>(b) * p.n_heads + w.h) * n_qtiles + w.qt) * BQ;
        const uint32_t sq = smem_base + Ly::OFF_Q + st * TILE, sdo = smem_base + Ly::OFF_DO + dst * TILE;
        const uint32_t sst = smem_base + Ly::OFF_STATS + st * STATS_BYTES;
        if (!mbar_wait_warp(bar(BAR_Q_EMPTY + st), was, abort_flag)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          mbar_expect_tx(bar(BAR_Q_FULL + st), TILE + STATS_BYTES);
#pragma unroll
          for (int sl = 0; sl < SLABS; ++sl)
            tma_load_3d(sq + sl * SLAB, &tmQ, bar(BAR_Q_FULL + st), w.h * D + 64 * sl, q0, b);
          bulk_load_1d(sst, p.neg_lse2 + stat_off, BQ * 4, bar(BAR_Q_FULL + st));
          bulk_load_1d(sst + BQ * 4, p.neg_delta + stat_off, BQ * 4, bar(BAR_Q_FULL + st));
        }
        __syncwarp();
        if (!mbar_wait_warp(bar(BAR_DO_EMPTY + dst), static_cast<uint32_t>(t / Ly::DO_STAGES) & 1u ^ 1u, abort_flag)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          mbar_expect_tx(bar(BAR_DO_FULL + dst), TILE);
#pragma unroll
          for (int sl = 0; sl < SLABS; ++sl)
            tma_load_3d(sdo + sl * SLAB, &tmDO, bar(BAR_DO_FULL + dst), w.h * D + 64 * sl, q0, b);
        }
        __syncwarp();
      }
      ftb200::start_next();
      if (!ok) {
        const uint64_t t0 = ftb200::globaltimer_ns();
        while (ftb200::globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
      }
      __syncwarp();
    } else if (warp == 1) {
      // ---------------- MMA issuer ----------------
      const uint32_t F = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(128 >> 4) << 24);
      const uint32_t idesc_st = F | (static_cast<uint32_t>(BQ >> 3) << 17);                            // N = 128, K-major both
      const uint32_t idesc_kv = F | (1u << 16) | (static_cast<uint32_t>(D >> 3) << 17);                // N = D, B MN-major
      const uint32_t idesc_dq = F | (1u << 15) | (1u << 16) | (static_cast<uint32_t>(BQ >> 3) << 17);  // N = 128, both MN-major
      constexpr uint32_t HI = smem_desc_hi(1024);
      const uint32_t k_km = smem_desc_lo(smem_base + Ly::OFF_K, 16);  // K as K-major A (S^T)
      const uint32_t v_km = smem_desc_lo(smem_base + Ly::OFF_V, 16);  // V as K-major A (dP^T)
      // K as MN-major A (dQ^T): M = 128 runs over the head dim.  With head dim 64 the second 64 rows of that MMA
      // read the slab behind K's only one, which is V's: lanes 64..127 of dQ^T then hold a product nobody reads.
      const uint32_t k_mn = smem_desc_lo(smem_base + Ly::OFF_K, SLAB);
      const uint32_t q_km0 = smem_desc_lo(smem_base + Ly::OFF_Q, 16), q_mn0 = smem_desc_lo(smem_base + Ly::OFF_Q, SLAB);
      const uint32_t do_km0 = smem_desc_lo(smem_base + Ly::OFF_DO, 16), do_mn0 = smem_desc_lo(smem_base + Ly::OFF_DO, SLAB);
      const uint32_t ds_mn = smem_desc_lo(smem_base + Ly::OFF_DS, SLAB);
      constexpr uint32_t TILE16 = TILE >> 4;
      // queries 16k..16k+15 of P^T (of dS^T): 8 columns at the start of the half of S^T (dP^T) that the writing thread read
      auto pt_col = [](int kk) { return (kk >> 2) * 64 + (kk & 3) * 8; };

      auto score = [&](uint32_t d_col, uint32_t a_km, uint32_t b_km, int full) {  // S^T or dP^T
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = ((kk >> 2) * SLAB + (kk & 3) * 32) >> 4;
            umma_bf16_lh(tmem_base + d_col, a_km + off, HI, b_km + off, HI, idesc_st, kk != 0);
          }
          umma_commit(bar(full));
        }
        __syncwarp();
      };
      auto from_tmem = [&](uint32_t d_col, uint32_t a_col, uint32_t b_mn, bool first, int freed) {  // dV or dK
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < BQ / 16; ++kk)
            umma_bf16_tmem_a(tmem_base + d_col, tmem_base + a_col + pt_col(kk), b_mn + ((kk * 2048) >> 4), HI, idesc_kv,
                             !first || kk != 0);
          umma_commit(bar(freed));
        }
        __syncwarp();
      };
      auto wait = [&](int which, uint32_t parity) {
        const bool w = mbar_wait_warp(bar(which), parity, abort_flag);
        tc_fence_after();
        return w;
      };
      // S^T of the next tile is issued ahead of the products that wait for this tile's dS^T, so that its softmax runs
      // under them; the columns of S^T are free for it as P^T's reader, dV, was issued before.
      bool ok = wait(BAR_KV, 0) && wait(BAR_Q_FULL, 0);
      if (ok) score(Ly::COL_S, k_km, q_km0, BAR_S_FULL);
      ok = ok && wait(BAR_DO_FULL, 0);
      if (ok) score(Ly::COL_DP, v_km, do_km0, BAR_DP_FULL);
      for (int t = 0; t < T && ok; ++t) {
        const int st = t % STAGES, nst = (t + 1) % STAGES;
        const uint32_t odd = static_cast<uint32_t>(t) & 1u, nph = static_cast<uint32_t>((t + 1) / STAGES) & 1u;
        const int dst = t % Ly::DO_STAGES, ndst = (t + 1) % Ly::DO_STAGES;
        if (!(ok = wait(BAR_P_READY, odd))) break;
        from_tmem(Ly::COL_DV, Ly::COL_S, do_mn0 + dst * TILE16, t == 0, BAR_DO_EMPTY + dst);
        if (t + 1 < T) {
          if (!(ok = wait(BAR_Q_FULL + nst, nph))) break;
          score(Ly::COL_S, k_km, q_km0 + nst * TILE16, BAR_S_FULL);
        }
        if (!(ok = wait(BAR_DS_READY, odd))) break;
        from_tmem(Ly::COL_DK, Ly::COL_DP, q_mn0 + st * TILE16, t == 0, BAR_Q_EMPTY + st);
        if (!Ly::DQ_OVER_DP && !(ok = wait(BAR_DQ_EMPTY, odd ^ 1u))) break;  // dQ^T of tile t - 1 drained
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < BKV / 16; ++kk)  // dQ^T = K^T dS^T
            umma_bf16_lh(tmem_base + Ly::COL_DQ, k_mn + ((kk * 2048) >> 4), HI, ds_mn + ((kk * 2048) >> 4), HI, idesc_dq, kk != 0);
          umma_commit(bar(BAR_DQ_FULL));
        }
        __syncwarp();
        if (t + 1 < T) {
          if (!(ok = wait(BAR_DO_FULL + ndst, static_cast<uint32_t>((t + 1) / Ly::DO_STAGES) & 1u))) break;
          if (Ly::DQ_OVER_DP && !(ok = wait(BAR_DQ_EMPTY, odd))) break;  // dQ^T of tile t drained
          score(Ly::COL_DP, v_km, do_km0 + ndst * TILE16, BAR_DP_FULL);
        }
      }
      if (ok && elect_one()) umma_commit(bar(BAR_DKV_DONE));
      __syncwarp();
    }
  } else if (warp < 8) {
    // ---------------- dQ drain: TMEM lane = head-dim index ----------------
    regs_inc<DRAIN_REGS>();
    const int quarter = warp & 3;
    const uint32_t dq_addr = tmem_base + Ly::COL_DQ + (static_cast<uint32_t>(quarter * 32) << 16);
    const bool mine = quarter * 32 < D;  // head dim 64: only lanes 0..63 of dQ^T are real
    const uint32_t off = Ly::OFF_DQ + quarter * 2 * DQ_PART_BYTES;
    constexpr int PER = BQ / 4 / DQ_PARTS;  // groups of four queries in a part
    TileWalk w{h0, first_q};
    for (int u = 0; u < T; ++u, next_tile(w)) {
      if (!mbar_wait_warp(bar(BAR_DQ_FULL), static_cast<uint32_t>(u) & 1u, abort_flag)) break;
      tc_fence_after();
      uint32_t v[BQ];
      if (mine) {
#pragma unroll
        for (int c = 0; c < BQ / 32; ++c) tmem_ld32(dq_addr + c * 32, v + c * 32);
        tmem_wait_ld();
      }
      tc_fence_before();
      mbar_arrive_warp(bar(BAR_DQ_EMPTY));
      if (mine) {
        const long long tile = (static_cast<long long>(b) * n_qtiles + w.qt) * p.n_heads + w.h;
        float* dst = p.dq_acc + tile * (BQ * D) + quarter * (32 * BQ);
#pragma unroll
        for (int part = 0; part < DQ_PARTS; ++part) {
          const uint32_t buf = off + (part & 1) * DQ_PART_BYTES;
          // the reduction that read this buffer last, two before this one, has read it
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          __syncwarp();
#pragma unroll
          for (int c = 0; c < PER; ++c) {
            const uint32_t* x = v + (part * PER + c) * 4;
            *reinterpret_cast<uint4*>(smem + buf + (c * 32 + lane) * 16) = make_uint4(x[0], x[1], x[2], x[3]);
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            bulk_add_f32(dst + part * (DQ_PART_BYTES / 4), smem_base + buf, DQ_PART_BYTES);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
  } else {
    // ---------------- softmax, dK/dV store ----------------
    regs_inc<SOFTMAX_REGS>();
    const int quarter = warp & 3;
    const int g = (warp - 8) >> 2;        // which 64 of the tile's queries
    const int row = quarter * 32 + lane;  // key within the block
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    bool ok = true;
    const unsigned long long scale2 = f2_pack(p.scale_log2, p.scale_log2), dscale2 = f2_pack(p.scale, p.scale);
    TileWalk w{h0, first_q};
    const uint32_t s_addr = tmem_base + Ly::COL_S + g * CPT + lane_addr;
    const uint32_t dp_addr = tmem_base + Ly::COL_DP + g * CPT + lane_addr;
    const bool beyond = jb * BKV + row >= p.seq;  // this key
    uint8_t* drow = smem + Ly::OFF_DS + g * SLAB + row * 128;
    for (int t = 0; t < T && ok; ++t, next_tile(w)) {
      const uint32_t odd = static_cast<uint32_t>(t) & 1u;
      const int st = t % STAGES;
      // the tile's statistics arrived with Q
      if (!mbar_wait_warp(bar(BAR_Q_FULL + st), static_cast<uint32_t>(t / STAGES) & 1u, abort_flag) ||
          !mbar_wait_warp(bar(BAR_S_FULL), odd, abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after();
      // pairs of -log2(e) lse and -scale delta, as the packed arithmetic takes them
      const ulonglong2* lse2 = reinterpret_cast<const ulonglong2*>(smem + Ly::OFF_STATS + st * STATS_BYTES) + g * (CPT / 4);
      const ulonglong2* delta2 = lse2 + BQ / 4;
      float pe[CPT];
      {
        uint32_t sv[CPT];
        tmem_ld32(s_addr, sv);
        tmem_ld32(s_addr + 32, sv + 32);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < CPT / 4; ++c) {
          const ulonglong2 l4 = lse2[c];
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
      }
      if (p.causal != 0 && w.qt == jb) {  // the diagonal tile: queries before the key
#pragma unroll
        for (int c = 0; c < CPT; ++c)
          if (row > g * CPT + c) pe[c] = 0.f;
      } else if (beyond) {  // no causal mask leaves it out
#pragma unroll
        for (int c = 0; c < CPT; ++c) pe[c] = 0.f;
      }
      {
        uint32_t pt[CPT / 2];
#pragma unroll
        for (int c = 0; c < CPT / 2; ++c) {
          __nv_bfloat162 a = __floats2bfloat162_rn(pe[2 * c], pe[2 * c + 1]);
          pt[c] = *reinterpret_cast<uint32_t*>(&a);
        }
        tmem_st32(s_addr, pt);  // over scores that this thread has read
        tmem_wait_st();
      }
      tc_fence_before();
      mbar_arrive_warp(bar(BAR_P_READY));

      if (!mbar_wait_warp(bar(BAR_DP_FULL), odd, abort_flag)) {  // dK and dQ^T of tile t - 1 are complete too: dS^T is free
        ok = false;
        break;
      }
      tc_fence_after();
      uint32_t dp[2][CHUNK];
      tmem_ld16(dp_addr, dp[0]);
      tmem_wait_ld();
#pragma unroll
      for (int cc = 0; cc < CPT / CHUNK; ++cc) {
        if (cc + 1 < CPT / CHUNK) tmem_ld16(dp_addr + (cc + 1) * CHUNK, dp[(cc + 1) & 1]);
        const uint32_t* d = dp[cc & 1];
        uint32_t ds[CHUNK / 2];
#pragma unroll
        for (int c = 0; c < CHUNK / 4; ++c) {
          const ulonglong2 d4 = delta2[cc * (CHUNK / 4) + c];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int qi = 4 * c + 2 * e;
            // dS = P (scale dP - scale delta)
            const unsigned long long ds2 =
                f2_mul(f2_pack(pe[cc * CHUNK + qi], pe[cc * CHUNK + qi + 1]),
                       f2_fma(f2_pack(__uint_as_float(d[qi]), __uint_as_float(d[qi + 1])), dscale2, e == 0 ? d4.x : d4.y));
            float s0, s1;
            f2_unpack(ds2, s0, s1);
            __nv_bfloat162 x = __floats2bfloat162_rn(s0, s1);
            ds[qi / 2] = *reinterpret_cast<uint32_t*>(&x);
          }
        }
        if (cc + 1 < CPT / CHUNK) tmem_wait_ld();
        tmem_st8(dp_addr + cc * (CHUNK / 2), ds);  // over columns that this thread has read
#pragma unroll
        for (int c = 0; c < CHUNK / 8; ++c) {
          const int at = ((cc * (CHUNK / 8) + c) ^ (row & 7)) << 4;
          *reinterpret_cast<uint4*>(drow + at) = make_uint4(ds[4 * c], ds[4 * c + 1], ds[4 * c + 2], ds[4 * c + 3]);
        }
      }
      fence_async_smem();
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive_warp(bar(BAR_DS_READY));
    }
    if (ok && mbar_wait_warp(bar(BAR_DKV_DONE), 0, abort_flag)) {
      tc_fence_after();
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        constexpr int CW = D / 2;  // head-dim columns per thread
        const uint32_t col = (which == 0 ? Ly::COL_DV : Ly::COL_DK) + g * CW;
        __nv_bfloat16* base = which == 0 ? p.dV : p.dK;
        const long long ld = which == 0 ? p.ld_dv : p.ld_dk;
        __nv_bfloat16* dst = base + (static_cast<long long>(b) * p.seq + jb * BKV + row) * ld + hk * D + g * CW;
        uint32_t v[CW];
#pragma unroll
        for (int c = 0; c < CW / 32; ++c) tmem_ld32(tmem_base + col + c * 32 + lane_addr, v + c * 32);
        tmem_wait_ld();
        if (p.split > 1) {
          float4* part = p.dkv_part + ((static_cast<long long>(bh) * n_qtiles + jb) * p.split + share) * (2 * D / 4 * BKV) +
                         (which * D / 4 + g * CW / 4) * BKV + row;
#pragma unroll
          for (int c = 0; c < CW / 4; ++c)
            part[c * BKV] = make_float4(__uint_as_float(v[4 * c]), __uint_as_float(v[4 * c + 1]), __uint_as_float(v[4 * c + 2]),
                                        __uint_as_float(v[4 * c + 3]));
          continue;
        }
#pragma unroll
        for (int c = 0; c < CW / 8; ++c) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[8 * c + e]);
          if (beyond) continue;
          if (which == 1 && p.rope != nullptr) {
            const float4* cs = p.rope + static_cast<long long>(jb * BKV + row) * (D / 4) + g * (CW / 4) + 2 * c;
            rotate_back(f, cs[0], cs[1]);
          }
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
// accumulator zeroed.  A thread takes 8 elements (16 bytes of each), D / 8 neighbouring lanes a (row, head); `pieces` counts the
// rows of whole tiles.
template <int D>
__global__ void __launch_bounds__(256) attention_bwd_prep_kernel(const __nv_bfloat16* o,
                                                                 const __nv_bfloat16* d_o,
                                                                 const float* lse, float* neg_lse2,
                                                                 float* neg_delta, float4* dq_acc,
                                                                 int seq, int n_heads, long long pieces, long long ld_o,
                                                                 long long ld_do, float scale) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  constexpr int LANES = D / 8;
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool live = i < pieces;
  const int per_row = n_heads * LANES;
  const int rt = static_cast<int>((live ? i : 0) / per_row);  // rows of whole tiles fit an int (the host checks)
  const int c = static_cast<int>((live ? i : 0) - static_cast<long long>(rt) * per_row);
  const int seq_t = (seq + BQ - 1) / BQ * BQ;
  const int b = rt / seq_t, pos = rt - b * seq_t;
  const bool inside = pos < seq;
  const long long r = static_cast<long long>(b) * seq + pos;
  float s = 0.f;
  if (live) {
    dq_acc[2 * i] = make_float4(0.f, 0.f, 0.f, 0.f);
    dq_acc[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (live && inside) {
    float x[8], y[8];
    ftb200::unpack8(*reinterpret_cast<const ftb200::bf16x8*>(o + r * ld_o + c * 8), x);
    ftb200::unpack8(*reinterpret_cast<const ftb200::bf16x8*>(d_o + r * ld_do + c * 8), y);
#pragma unroll
    for (int e = 0; e < 8; ++e) s = fmaf(x[e], y[e], s);
  }
#pragma unroll
  for (int k = LANES / 2; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
  if (live && c % LANES == 0) {
    const long long bh = static_cast<long long>(b) * n_heads + c / LANES;
    neg_delta[bh * seq_t + pos] = inside ? -s * scale : 0.f;
    neg_lse2[bh * seq_t + pos] = inside ? lse[bh * seq + pos] * -1.4426950408889634f : -INFINITY;
  }
}

// dq (bf16, row stride ld) = accumulator (fp32, per 128 queries and head [D / 32][32 groups of 4 queries][32][4 queries]),
// rotated back with `rope`.  A warp takes 64 head-dim elements, two a lane, of CAST_GROUPS groups of four queries: 512
// consecutive bytes a half warp and load, 128 a warp and store.  (Eight elements of a group a lane: 44 us for 8 x 2048, 32 heads
// of 64, against 27.)
constexpr int CAST_GROUPS = 4;

template <int D>
__device__ __forceinline__ void cast_dq(long long wi, const float4* acc, __nv_bfloat16* dq, long long warps, int n_heads, long long ld,
                                        int seq, const float2* rope) {
  constexpr int PER_HEAD = (D / 64) * (32 / CAST_GROUPS);  // warps per tile and head
  if (wi >= warps) return;
  const int lane = threadIdx.x & 31;
  const long long th = wi / PER_HEAD;
  const int part = static_cast<int>(wi - th * PER_HEAD);
  const int slab = part / (32 / CAST_GROUPS) * 2 + (lane >> 4), q4 = part % (32 / CAST_GROUPS) * CAST_GROUPS;
  const int d = slab * 32 + 2 * (lane & 15);
  const int n_qtiles = (seq + BQ - 1) / BQ;
  const int tile = static_cast<int>(th / n_heads);
  const int h = static_cast<int>(th - static_cast<long long>(tile) * n_heads);
  const int pos0 = tile % n_qtiles * BQ + q4 * 4;  // in its sequence
  const float4* src = acc + th * (32 * D) + slab * 1024 + q4 * 32 + 2 * (lane & 15);
  float4 v[CAST_GROUPS][2];
#pragma unroll
  for (int u = 0; u < CAST_GROUPS; ++u) {
    v[u][0] = __ldcs(src + u * 32);
    v[u][1] = __ldcs(src + u * 32 + 1);
  }
  __nv_bfloat16* dst = dq + (static_cast<long long>(tile / n_qtiles) * seq + pos0) * ld + h * D + d;
#pragma unroll
  for (int u = 0; u < CAST_GROUPS; ++u) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int q = u * 4 + k;
      if (pos0 + q >= seq) return;
      float a = k == 0 ? v[u][0].x : k == 1 ? v[u][0].y : k == 2 ? v[u][0].z : v[u][0].w;
      float b = k == 0 ? v[u][1].x : k == 1 ? v[u][1].y : k == 2 ? v[u][1].z : v[u][1].w;
      if (rope != nullptr) {
        const float2 cs = rope[static_cast<long long>(pos0 + q) * (D / 2) + d / 2];
        const float x = a;
        a = x * cs.x + b * cs.y;
        b = b * cs.x - x * cs.y;
      }
      *reinterpret_cast<__nv_bfloat162*>(dst + q * ld) = __floats2bfloat162_rn(a, b);
    }
  }
}

// dK and dV of a key block (bf16) from the shares' sums, added in their order; dK is rotated back with `rope`.  A block takes 32
// head-dim elements of dV (piece < D / 32) or dK, a thread 16 of them of one key.
template <int D>
__device__ __forceinline__ void cast_dkv(int block, int piece, const BwdParams& p) {
  const int tiles = (p.seq + BKV - 1) / BKV;
  const int bh = block / tiles, jb = block % tiles;
  const int which = piece / (D / 32);
  const int key = threadIdx.x >> 1, d0 = piece % (D / 32) * 32 + (threadIdx.x & 1) * 16;
  const int pos = jb * BKV + key;
  if (pos >= p.seq) return;
  const float4* src = p.dkv_part + static_cast<long long>(block) * p.split * (2 * D / 4 * BKV) + (which * D / 4 + d0 / 4) * BKV + key;
  float f[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) f[e] = 0.f;
  for (int s = 0; s < p.split; ++s, src += 2 * D / 4 * BKV) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float4 x = src[c * BKV];
      f[4 * c] += x.x;
      f[4 * c + 1] += x.y;
      f[4 * c + 2] += x.z;
      f[4 * c + 3] += x.w;
    }
  }
  if (which == 1 && p.rope != nullptr) {
    const float4* cs = p.rope + static_cast<long long>(pos) * (D / 4) + d0 / 4;
    rotate_back(f, cs[0], cs[1]);
    rotate_back(f + 8, cs[2], cs[3]);
  }
  const int b = bh / p.n_kv_heads, hk = bh % p.n_kv_heads;
  __nv_bfloat16* dst = (which == 0 ? p.dV : p.dK) + (static_cast<long long>(b) * p.seq + pos) * (which == 0 ? p.ld_dv : p.ld_dk) + hk * D + d0;
  reinterpret_cast<ftb200::bf16x8*>(dst)[0] = ftb200::pack8(f);
  reinterpret_cast<ftb200::bf16x8*>(dst)[1] = ftb200::pack8(f + 8);
}

// What follows the main kernel, in one launch: blocks below dkv_blocks add up and cast dK and dV (where heads are shared), the others
// cast dQ.  In two launches a step of two layers on 256 tokens took 297 us instead of 292, one of four layers of width 1024 on
// 3 x 1000 tokens 1982 instead of 1962.
template <int D>
__global__ void __launch_bounds__(256) attention_bwd_cast_kernel(const float4* acc, __nv_bfloat16* dq, long long warps, long long ld_dq,
                                                                 int dkv_blocks, const BwdParams p) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  const int block = static_cast<int>(blockIdx.x);
  if (block < dkv_blocks)
    cast_dkv<D>(block / (2 * D / 32), block % (2 * D / 32), p);
  else
    cast_dq<D>(static_cast<long long>(block - dkv_blocks) * 8 + (threadIdx.x >> 5), acc, dq, warps, p.n_heads, ld_dq, p.seq,
               reinterpret_cast<const float2*>(p.rope));
}

// How many CTAs share the query heads of a kv head: one where every SM has a CTA anyway, else as many as divide the heads and stay
// at four CTAs a SM.  The CTA of the first key block walks over all of a head's tiles, so its heads are the longest chain; what
// sharing costs is dK and dV in fp32, written and read once more.  Whole pass, us: 3 x 1000, 8/2 heads of 128 (48 CTAs) 102 -> 48;
// 1 x 1024, 8/2 of 128 (16) 92 -> 37; 1 x 1536, 32/8 of 128 (96) 146 -> 99; 2 x 2048, 16/4 of 128 (128) 188 -> 144; 1 x 2048,
// 32/8 of 64 (128) 133 -> 98.  Beyond one CTA a SM it loses: 2 x 2048, 32/8 of 128 (256) 222 -> 238.
int head_split(long long ctas, int rep) {
  const int sms = ftb200::sm_count();
  int split = 1;
  if (ctas <= sms)
    for (int s = 2; s <= rep; ++s)
      if (rep % s == 0 && ctas * s <= 4LL * sms) split = s;
  return split;
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

// [batch, seq, cols] bf16 view with row stride ld (elements); box = 64 columns x 128 rows, 128-byte swizzle
int encode_rows(CUtensorMap* map, const void* base, long long batch, long long seq, long long cols, long long ld) {
  auto fn = encode_fn();
  if (fn == nullptr) return FTB200_E_DRIVER;
  cuuint64_t gdim[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(seq), static_cast<cuuint64_t>(batch)};
  cuuint64_t gstride[2] = {static_cast<cuuint64_t>(ld) * 2, static_cast<cuuint64_t>(seq) * ld * 2};
  cuuint32_t box[3] = {64u, 128u, 1u};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), gdim, gstride, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : FTB200_E_DRIVER;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

// Scratch the backward pass needs, in bytes: fp32 dQ accumulator, -scale delta, -log2(e) lse, and the shares' dV and dK where the
// query heads are shared out.  (sized for head dim 128; enough for 64 as well)
FTB200_API long long ftb200_attention_bwd_scratch_bytes(int batch, int seq, int n_heads, int n_kv_heads) {
  if (batch <= 0 || seq <= 0 || n_heads <= 0 || n_kv_heads <= 0 || n_heads % n_kv_heads != 0) return 0;
  const long long tiles = (static_cast<long long>(seq) + BQ - 1) / BQ, rows = batch * tiles * BQ;
  const long long ctas = batch * tiles * n_kv_heads;
  const int split = head_split(ctas, n_heads / n_kv_heads);
  return rows * n_heads * 128 * 4 + 2 * rows * n_heads * 4 + (split > 1 ? ctas * split * (2 * 128 * BKV * 4) : 0);
}

namespace {

template <int D>
int attention_bwd_impl(const void* q, const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                       void* dq, void* dk, void* dv, void* scratch, int batch, int seq, int n_heads, int n_kv_heads,
                       long long ld_q, long long ld_k, long long ld_v, long long ld_o, long long ld_do, long long ld_dq,
                       long long ld_dk, long long ld_dv, float scale, int causal, const float* cos_sin, int* status,
                       cudaStream_t stream) {
  constexpr uint32_t SMEM_BYTES = Lay<D>::SMEM_BYTES;
  const long long tiles = (static_cast<long long>(seq) + BQ - 1) / BQ;
  const long long rows = batch * tiles * BQ;
  float* dq_acc = reinterpret_cast<float*>(scratch);
  float* neg_delta = dq_acc + rows * n_heads * D;
  float* neg_lse2 = neg_delta + rows * n_heads;
  const int split = head_split(batch * tiles * n_kv_heads, n_heads / n_kv_heads);
  if (rows > 0x7fffffffLL) return FTB200_E_TOOBIG;
  CUtensorMap tq, tk, tv, tdo;
  int rc = encode_rows(&tq, q, batch, seq, static_cast<long long>(n_heads) * D, ld_q);
  if (rc == 0) rc = encode_rows(&tdo, d_o, batch, seq, static_cast<long long>(n_heads) * D, ld_do);
  if (rc == 0) rc = encode_rows(&tk, k, batch, seq, static_cast<long long>(n_kv_heads) * D, ld_k);
  if (rc == 0) rc = encode_rows(&tv, v, batch, seq, static_cast<long long>(n_kv_heads) * D, ld_v);
  if (rc != 0) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(attention_bwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) !=
        cudaSuccess)
      return FTB200_E_CUDA;
    // the warpgroups share out what a CTA is launched with: with fewer registers a thread the increase would wait for good
    cudaFuncAttributes attr;
    if (cudaFuncGetAttributes(&attr, attention_bwd_kernel<D>) != cudaSuccess) return FTB200_E_CUDA;
    if (attr.numRegs < LAUNCH_REGS) return FTB200_E_REGS;
    attr_set = true;
  }
  const long long pieces = rows * n_heads * (D / 8);
  if ((pieces + 255) / 256 > 0x7fffffffLL) return FTB200_E_TOOBIG;
  ftb200::launch_after(attention_bwd_prep_kernel<D>, static_cast<unsigned>((pieces + 255) / 256), 256, 0, stream,
      reinterpret_cast<const __nv_bfloat16*>(o), reinterpret_cast<const __nv_bfloat16*>(d_o), lse, neg_lse2, neg_delta,
      reinterpret_cast<float4*>(dq_acc), seq, n_heads, pieces, ld_o, ld_do, scale);
  BwdParams p;
  p.batch = batch; p.seq = seq; p.n_heads = n_heads; p.n_kv_heads = n_kv_heads; p.causal = causal;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.neg_lse2 = neg_lse2; p.neg_delta = neg_delta; p.dq_acc = dq_acc;
  p.dK = reinterpret_cast<__nv_bfloat16*>(dk); p.dV = reinterpret_cast<__nv_bfloat16*>(dv);
  p.ld_dk = ld_dk; p.ld_dv = ld_dv; p.status = status;
  p.rope = reinterpret_cast<const float4*>(cos_sin);
  p.split = split;
  p.dkv_part = reinterpret_cast<float4*>(neg_lse2 + rows * n_heads);
  const long long grid = static_cast<long long>(batch) * n_kv_heads * tiles * split;
  if (grid > 0x7fffffffLL) return FTB200_E_TOOBIG;
  ftb200::launch_after(attention_bwd_kernel<D>, static_cast<unsigned>(grid), NUM_THREADS, SMEM_BYTES, stream, tq, tk, tv, tdo,
      p);
  const long long cast_warps = batch * tiles * n_heads * (D / 64) * (32 / CAST_GROUPS);
  const long long dkv_blocks = split > 1 ? static_cast<long long>(batch) * n_kv_heads * tiles * (2 * D / 32) : 0;
  const long long cast_blocks = dkv_blocks + (cast_warps + 7) / 8;  // fewer than the first kernel's
  ftb200::launch_after(attention_bwd_cast_kernel<D>, static_cast<unsigned>(cast_blocks), 256, 0, stream,
      reinterpret_cast<const float4*>(dq_acc), reinterpret_cast<__nv_bfloat16*>(dq), cast_warps, ld_dq,
      static_cast<int>(dkv_blocks), p);
  return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
}

}  // namespace

// q, k, v, o, d_o as in the forward pass (2-D views, row strides in elements); dq, dk, dv are
// written (not accumulated).  lse is the forward's [batch, n_heads, seq].  scratch: at least
// ftb200_attention_bwd_scratch_bytes, 16-byte aligned.  Head dim 64 or 128.  cos_sin: null, or fp32 [seq][head_dim / 2]
// pairs of the angles that q and k were rotated by (pair (2i, 2i + 1) of a head by the i-th angle of its row's position):
// dq and dk are then the gradients of the values before the rotation, rotated back in fp32 ahead of the rounding to bf16.
FTB200_API int ftb200_attention_bwd(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                                    const float* lse, void* dq, void* dk, void* dv, void* scratch, int batch, int seq,
                                    int n_heads, int n_kv_heads, int head_dim, long long ld_q, long long ld_k,
                                    long long ld_v, long long ld_o, long long ld_do, long long ld_dq, long long ld_dk,
                                    long long ld_dv, float scale, int causal, const float* cos_sin, int* status,
                                    cudaStream_t stream) {
  if ((head_dim != 64 && head_dim != 128) || batch <= 0 || seq <= 0 || n_heads <= 0 ||
      n_kv_heads <= 0 || n_heads % n_kv_heads != 0)
    return FTB200_E_BADARG;
  const void* ptrs[] = {q, k, v, o, d_o, dq, dk, dv, scratch, cos_sin};
  for (const void* x : ptrs)
    if (!aligned16(x)) return FTB200_E_ALIGN;
  const long long lds[] = {ld_q, ld_k, ld_v, ld_o, ld_do, ld_dq, ld_dk, ld_dv};
  for (long long x : lds)
    if (x & 7) return FTB200_E_ALIGN;
  if (head_dim == 64)
    return attention_bwd_impl<64>(q, k, v, o, d_o, lse, dq, dk, dv, scratch, batch, seq, n_heads, n_kv_heads, ld_q, ld_k,
                                  ld_v, ld_o, ld_do, ld_dq, ld_dk, ld_dv, scale, causal, cos_sin, status, stream);
  return attention_bwd_impl<128>(q, k, v, o, d_o, lse, dq, dk, dv, scratch, batch, seq, n_heads, n_kv_heads, ld_q, ld_k,
                                 ld_v, ld_o, ld_do, ld_dq, ld_dk, ld_dv, scale, causal, cos_sin, status, stream);
}
