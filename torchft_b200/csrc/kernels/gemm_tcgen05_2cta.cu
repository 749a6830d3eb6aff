// bf16 GEMM with 2-SM tensor-core instructions (tcgen05.mma.cta_group::2).
//
// Same contract as the 1-CTA kernel in gemm_tcgen05.cu.  Two CTAs of a cluster share
// one 256x256 output tile (256x128 where the output is small, see plan_tiles): each stages its own 128 rows of A and its own 128 of the 256
// B columns (32 KiB per 64-deep K slab instead of 48 KiB), the pair's leader issues one
// M=256 MMA that reads both halves of B, and each CTA's TMEM receives the accumulator of
// its own 128 rows.  Per SM that is a third less shared-memory fill traffic per FLOP and
// room for a 6-stage ring, which is what the 1-CTA kernel lacks: its tensor pipe idles
// ~40% of the time waiting for operand tiles in flight.
//
// Synchronisation inside the pair:
//   full[s]   (leader)  both CTAs' TMA loads complete_tx on the leader's barrier
//   empty[s]  (each)    the leader's tcgen05.commit arrives on both CTAs' barriers
//   tfull[a]  (each)    likewise, after the last MMA of a tile
//   tempty[a] (leader)  the 2 x 4 epilogue warps of the pair arrive (remote arrive
//                       from the peer)
// All waits are bounded as in the 1-CTA kernel.
//
// A last wave that leaves most pairs idle is split over K (SPLIT, see plan_tiles): a cluster of S pairs takes one of its
// tiles, each pair a share of the K slabs, and after them the S accumulators meet through distributed shared memory:
// every CTA owns the 32-column chunks c of its 128 rows with c * S / chunks == its pair and gets the other pairs' values
// of them copied into its operand ring, which is free by then:
//   ready     (each)    the S - 1 CTAs with the same rows in the other pairs have finished their products (remote arrive)
//   got       (each)    their values have arrived (complete_tx of the copies)
// The values are added in the order of the pairs, so the result does not depend on which one was first.
//
// All-gather fused into the GEMM (ftb200_gemm_bf16_gather): B is a weight whose rows lie
// spread over the ranks of a shard group, as one contiguous piece of a flat parameter unit
// that the ranks shard evenly.  Four extra warps per CTA pull the weight out of the owners'
// shard buffers over NVLink (plain 16-byte peer loads) into the local gathered unit, 16 KiB
// at a time in row order, and count the finished pieces per block of 128 B rows; the TMA
// producer of a tile waits (bounded) for the count of its 128 rows and then loads them from
// local memory, so the tensor cores work on the first tiles while the rest of the weight
// is still crossing the links, and every remote byte crosses them once.  The pieces are
// handed out through a counter, so the CTAs that are running pull everything whether or
// not the whole grid is resident.
#include <algorithm>
#include <atomic>
#include <cuda.h>
#include <cudaTypedefs.h>

#include "ftb200_common.cuh"
#include "tcgen05_helpers.cuh"

namespace {

constexpr int BM = 128;  // rows per CTA (256 per pair)
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr uint32_t A_BYTES = BM * BK * 2;

// What becomes of a tile.
enum Epilogue : int {
  EPI_STORE = 0,    // it is stored (added to fp32 or rows that TMA does not take, with the activation of its columns' pairs, scattered: GemmParams)
  EPI_DSWIGLU = 1,  // it is the gradient of silu(gate) * up: the gate/up pairs it belongs to are replaced by their gradients
  EPI_LOSS = 2,     // its rows' maximum, sum of exponentials and target value are noted; it is not stored
  EPI_ADD = 3,      // it is added to what bf16 C holds
};

// A pair's tile has 256 or 128 columns; the K ring fills 192 KB with 6 or 8 stages.  The gradient of the activation needs
// twice the staging area (two 64-column pieces of gate/up pairs) and leaves it 5 or 6.
template <int BN_, int EPI>
struct Tile {
  static constexpr int BN = BN_;        // columns per pair
  static constexpr int BNH = BN / 2;    // of B's rows, per CTA
  static constexpr bool DS = EPI == EPI_DSWIGLU;
  static constexpr int STAGES = BN == 256 ? (DS ? 5 : 6) : (DS ? 6 : 8);
  static constexpr uint32_t B_BYTES = BNH * BK * 2;
  static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr uint32_t STAGE_WARP_BYTES = 32 * (DS ? 512 : 256);  // epilogue: 32 rows x 128 bf16 per warp (256)
  static constexpr uint32_t OFF_STAGING = STAGES * STAGE_BYTES, OFF_MISC = OFF_STAGING + 4 * STAGE_WARP_BYTES;
  static constexpr uint32_t SMEM_BYTES = OFF_MISC + 256 + 1024;
  static_assert(SMEM_BYTES <= 232448, "exceeds the 227 KB of shared memory a CTA can have");
  static_assert(DS || OFF_STAGING == 196608, "a shared tile's exchange fills the ring");
};
constexpr uint32_t RING_BYTES = 196608;
constexpr int GATHER_BLOCK = 128;  // B rows whose pieces the all-gather counts together: a CTA's half of a 256-column tile
constexpr int NUM_THREADS = 192;
constexpr int GATHER_WARPS = 4;  // only launched by the all-gather variant
constexpr int NUM_THREADS_GATHER = NUM_THREADS + 32 * GATHER_WARPS;
constexpr int GATHER_PIECE_V = 1024;  // 16-byte vectors per piece (16 KiB)
constexpr uint32_t TMEM_COLS = 512;
constexpr int GROUP_M = 8;  // in 256-row pair tiles (the all-gather variant uses twice that)

using namespace ftb200::tc;

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ uint32_t cluster_nctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}

// Orders nothing: with release semantics it would first wait for the kernel's stores to arrive, 1200 cycles at its end.
__device__ __forceinline__ void cluster_sync_relaxed() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

// TMA tile load issued by one CTA of a pair; the completion bytes are signalled on a
// barrier that may live in the partner CTA (address in the cluster window).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                 int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
      "[%2];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
      : "memory");
}

__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// Stores a tile of shared memory; what lies beyond the tensor is left out.  The calling thread's bulk group has to be
// committed.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(src), "r"(c0), "r"(c1)
               : "memory");
}

__device__ __forceinline__ void umma_bf16_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrive (once all MMAs issued so far have completed) on the barrier at the same
// shared-memory offset in both CTAs of the pair.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar, uint32_t lead_cta) {
  const uint16_t mask = static_cast<uint16_t>(3u << lead_cta);
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(mask)
               : "memory");
}

struct GemmParams {
  int M, N, K;
  int a_mn, b_mn;
  int out_fp32;
  int accumulate;
  int tma_out;                 // bf16 output through tmC (rows and columns beyond M and N are clipped)
  long long ldc;
  void* C;
  int* status;
  // fused SwiGLU: output columns are (gate, up) pairs; aux[row, j] = silu(C[row,2j]) * C[row,2j+1]
  void* aux;
  long long ld_aux;
  // EPI_LOSS, per row: [tiles of a row] (maximum, sum of exponentials over it), the target's value, the target
  float2* row_stats;
  float* target_value;
  const long long* target;
  // fused reduce-scatter epilogue: C is not written locally; every 16-byte piece of the
  // (contiguous, row-major) result goes to the rank that owns that slice of the flat
  // gradient unit, into that rank's staging area for source rank `sc_src`.
  int sc_world;                // 0 = off
  int sc_src;
  long long sc_shard;          // elements per shard (multiple of 8)
  long long sc_off;            // element offset of C inside the flat unit (multiple of 8)
  void* sc_peers[8];           // base of every rank's staging area (peer-mapped), [world][shard] elements
  int group_m;                 // tile order: this many 256-row tiles share a B tile before the next B tile
  // fused all-gather of B (see the head of the file); B points into the local gathered unit
  int ga_world;                // 0 = off
  long long ga_shard;          // elements per shard
  long long ga_off;            // element offset of B inside the flat unit (multiple of 8)
  const void* ga_peers[8];     // every rank's shard buffer (peer-mapped; [rank] is local)
  void* ga_dst;                // == B
  unsigned int* ga_sync;       // [0] next piece to hand out, [1 + c] pieces done of 128-row block c (zeroed per launch)
  int whole;                   // SPLIT: this many tiles are worked on by one pair each, the rest by a cluster each
};

// Bounded mbarrier wait that also acquires what other CTAs of the cluster wrote before they arrived.
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  const uint64_t t0 = ftb200::globaltimer_ns();
  for (uint32_t polls = 1;; ++polls) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (__all_sync(0xffffffffu, ok != 0)) return true;
    if ((polls & 255u) == 0) {
      const bool give_up = *abort_flag != 0 || ftb200::globaltimer_ns() - t0 > WAIT_LIMIT_NS;
      if (__any_sync(0xffffffffu, give_up)) {
        *abort_flag = 1;
        return false;
      }
    }
  }
}

// After a wait that ran out: copies in flight land in shared memory, so the CTA stays until they have.
__device__ __forceinline__ void sleep_200us() {
  const uint64_t t0 = ftb200::globaltimer_ns();
  while (ftb200::globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
}

// Bounded wait until *p >= want (device-scope acquire).
__device__ __forceinline__ bool count_wait(const unsigned int* p, unsigned int want, volatile int* abort_flag) {
  const uint64_t t0 = ftb200::globaltimer_ns();
  uint32_t spins = 0;
  for (;;) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    if (v >= want) return true;
    if ((++spins & 15u) == 0) {
      if (*abort_flag) return false;
      if (ftb200::globaltimer_ns() - t0 > WAIT_LIMIT_NS) {
        *abort_flag = 1;
        return false;
      }
      __nanosleep(64);
    }
  }
}

// The same for a whole warp whose loop has to stay converged.  One lane polls: 32 of them would load the word that the
// gather warps add to 32 times as often.  What it acquired is ordered before what the other lanes do next.
__device__ __forceinline__ bool count_wait_warp(const unsigned int* p, unsigned int want, volatile int* abort_flag) {
  const bool ok = (threadIdx.x & 31) != 0 || count_wait(p, want, abort_flag);
  __syncwarp();
  return __all_sync(0xffffffffu, ok);
}

// silu(gate) * up of four (gate, up) pairs: the activation of the rounded values, so that a later recompute from C agrees.
__device__ __forceinline__ uint2 silu_mul(const ftb200::bf16x8& packed) {
  float g[8], sv[4];
  ftb200::unpack8(packed, g);
#pragma unroll
  for (int e = 0; e < 4; ++e) sv[e] = g[2 * e] / (1.f + __expf(-g[2 * e])) * g[2 * e + 1];
  __nv_bfloat162 lo = __floats2bfloat162_rn(sv[0], sv[1]), hi = __floats2bfloat162_rn(sv[2], sv[3]);
  uint2 o;
  o.x = *reinterpret_cast<uint32_t*>(&lo);
  o.y = *reinterpret_cast<uint32_t*>(&hi);
  return o;
}

// Asynchronous copy from this CTA's shared memory to another's, counted by a barrier there.
__device__ __forceinline__ void copy_to_cta(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}

// Split last wave: a chunk is 32 columns of a CTA's 128 rows, a warp's share of it 32 rows.  With S pairs a CTA gets at
// most MAX_IN of them (S = 3: two pairs' values of three chunks) and sends at most as many, in a ring of twice that.
constexpr uint32_t CHUNK_BYTES = 128 * 32 * 4, SHARE_BYTES = CHUNK_BYTES / 4;
constexpr int MAX_IN = 6;
constexpr int MAX_SPLIT = 4;  // 8 CTAs: the largest cluster that every part takes
static_assert(2 * MAX_IN * CHUNK_BYTES <= RING_BYTES, "the ring holds what comes and what goes");

// Clusters of two CTAs (SPLIT: of 2 S), set at the launch.
template <int BN_, bool SPLIT, int EPI>
__global__ void __launch_bounds__(SPLIT ? NUM_THREADS : NUM_THREADS_GATHER, 1)
gemm_bf16_tcgen05_2cta_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                              const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmAux,
                              const GemmParams p) {
  using TL = Tile<BN_, EPI>;
  constexpr uint32_t OFF_STAGING = TL::OFF_STAGING, OFF_MISC = TL::OFF_MISC, STAGE_WARP_BYTES = TL::STAGE_WARP_BYTES;
  constexpr int BN = TL::BN, BNH = TL::BNH, STAGES = TL::STAGES;
  constexpr uint32_t STAGE_BYTES = TL::STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_MISC);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 6);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t cluster_rank = cluster_ctarank();
  const uint32_t rank = cluster_rank & 1u;  // in the pair
  const uint32_t lead_cta = cluster_rank - rank;
  const bool leader = rank == 0;
  const int S = SPLIT ? static_cast<int>(cluster_nctarank() >> 1) : 1;  // pairs that share a tile of the last wave
  const int pair = SPLIT ? static_cast<int>(cluster_rank >> 1) : 0;

  const uint32_t smem_base = smem_u32(smem);
  const uint32_t bar_base = smem_u32(bars);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + s); };
  auto tempty_bar = [&](int s) { return bar_base + 8u * (2 * STAGES + 2 + s); };
  const uint32_t ready_bar = bar_base + 8u * (2 * STAGES + 4), got_bar = bar_base + 8u * (2 * STAGES + 5);
  auto pairs_bar = [&](int q, int half) { return bar_base + 8u * (2 * STAGES + 7 + 2 * q + half); };  // EPI_DSWIGLU, EPI_ADD

  if (warp == 0) {
    if (lane < 2 * STAGES) mbar_init(bar_base + 8u * lane, 1);                             // full, empty
    if (lane >= 16 && lane < 20) mbar_init(tfull_bar(lane - 16), lane < 18 ? 1 : 2 * 4);  // tfull, tempty (one arrival a warp)
    if (lane == 20) *abort_flag = 0;
    if ((EPI == EPI_DSWIGLU || EPI == EPI_ADD) && lane >= 24) mbar_init(pairs_bar(0, lane - 24), 1);
    if (SPLIT && lane == 21) mbar_init(ready_bar, S - 1);
    if (SPLIT && lane == 22) mbar_init(got_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (lane == 0) {
      prefetch_map(&tmA);
      prefetch_map(&tmB);
      if (p.tma_out && EPI != EPI_DSWIGLU) prefetch_map(&tmC);
      if (p.tma_out && p.aux != nullptr) prefetch_map(&tmAux);
    }
    __syncwarp();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }

  const int num_m = (p.M + 2 * BM - 1) / (2 * BM);
  const int num_n = (p.N + BN - 1) / BN;
  const int num_tiles = num_m * num_n;
  const int num_k = (p.K + BK - 1) / BK;
  const int group_m = p.group_m;
  const int tiles_per_group = group_m * num_n;
  const int pair_id = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  const int whole = SPLIT ? p.whole : num_tiles;
  // The tiles of this pair in turn: t, and the K slabs of it that are this pair's.
  struct Work {
    int t, k0, k1;
    bool shared;
  };
  auto have_work = [&](Work& w) {
    if (!SPLIT || w.t < whole) return w.t < whole;
    if (w.shared) return false;  // one shared tile a cluster at most, after its whole ones
    w.t = whole + pair_id / S;
    w.k0 = num_k * pair / S;
    w.k1 = num_k * (pair + 1) / S;
    w.shared = true;
    return w.t < num_tiles;
  };
  auto next_work = [&](Work& w) {
    if (!w.shared) w.t += num_pairs;
  };
  const Work first{pair_id, 0, num_k, false};

  auto tile_coords = [&](int t, int& m0, int& n0) {
    const int g = t / tiles_per_group;
    const int first_m = g * group_m;
    const int gsz = min(num_m - first_m, group_m);
    const int r = t - g * tiles_per_group;
    m0 = (first_m + r % gsz) * (2 * BM) + static_cast<int>(rank) * BM;  // this CTA's rows
    n0 = (r / gsz) * BN;
  };
  int m0, n0;
  tile_coords(pair_id, m0, n0);  // of the first tile, while the barriers and the TMEM are on their way

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_relaxed();  // the partner's barriers exist (they were fenced) before anything signals them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  ftb200::wait_for_previous();

  if (warp == 0) {
    // ---------------- TMA producer (both CTAs) ----------------
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (Work w = first; have_work(w) && ok; next_work(w)) {
      if (w.t != pair_id) tile_coords(w.t, m0, n0);
      const int nb = n0 + static_cast<int>(rank) * BNH;  // this CTA's half of the B tile
      if (BNH == GATHER_BLOCK && p.ga_world > 0 && nb < p.N) {
        // these 128 rows of B are local once all their pieces are counted; the loads below go through the
        // async proxy, the pieces were written through the generic one
        if (!count_wait_warp(p.ga_sync + 1 + nb / GATHER_BLOCK, static_cast<unsigned int>(p.K / 64), abort_flag)) {
          ok = false;
          break;
        }
        asm volatile("fence.proxy.async.global;" ::: "memory");
      }
      for (int kb = w.k0; kb < w.k1; ++kb) {
        if (!mbar_wait_warp(empty_bar(stage), phase ^ 1u, abort_flag)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          const uint32_t sa = smem_base + stage * STAGE_BYTES;
          const uint32_t sb = sa + A_BYTES;
          const int k0 = kb * BK;
          if (leader) mbar_expect_tx(full_bar(stage), 2 * STAGE_BYTES);
          const uint32_t fb = map_to_cta(full_bar(stage), lead_cta);
          if (p.a_mn == 0) {
            tma_load_2d_pair(sa, &tmA, fb, k0, m0);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d_pair(sa + j * (BK * 128), &tmA, fb, m0 + 64 * j, k0);
          }
          if (p.b_mn == 0) {
            tma_load_2d_pair(sb, &tmB, fb, k0, nb);
          } else {
#pragma unroll
            for (int j = 0; j < BNH / 64; ++j) tma_load_2d_pair(sb + j * (BK * 128), &tmB, fb, nb + 64 * j, k0);
          }
        }
        __syncwarp();
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (p.ga_world == 0 && p.sc_world == 0) ftb200::start_next();
    if (!ok) sleep_200us();
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (leader) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(p.a_mn) << 15) |
                             (static_cast<uint32_t>(p.b_mn) << 16) | (static_cast<uint32_t>(BN >> 3) << 17) |
                             (static_cast<uint32_t>((2 * BM) >> 4) << 24);
      const uint32_t a_lbo = p.a_mn ? BK * 128 : 16, a_step = p.a_mn ? 2048 : 32;
      const uint32_t b_lbo = p.b_mn ? BK * 128 : 16, b_step = p.b_mn ? 2048 : 32;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (Work w = first; have_work(w) && ok; next_work(w)) {
        if (!mbar_wait_warp(tempty_bar(acc), acc_phase ^ 1u, abort_flag)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = w.k0; kb < w.k1; ++kb) {
          if (!mbar_wait_warp(full_bar(stage), phase, abort_flag)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (elect_one()) {
            const uint32_t sa = smem_base + stage * STAGE_BYTES;
            const uint32_t sb = sa + A_BYTES;
#pragma unroll
            for (int kk = 0; kk < BK / UMMA_K; ++kk) {
              const uint64_t adesc = make_smem_desc(sa + kk * a_step, a_lbo, 1024);
              const uint64_t bdesc = make_smem_desc(sb + kk * b_step, b_lbo, 1024);
              umma_bf16_pair(d_tmem, adesc, bdesc, idesc, ((kb - w.k0) | kk) != 0 ? 1u : 0u);
            }
            umma_commit_pair(empty_bar(stage), lead_cta);
            if (kb == w.k1 - 1) umma_commit_pair(tfull_bar(acc), lead_cta);
          }
          __syncwarp();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp >= 6) {
    // ---------------- all-gather of B (warps 6..9 of both CTAs, all-gather variant only) ----------------
    if (p.ga_world > 0) {
      const long long total_v = static_cast<long long>(p.N) * p.K / 8;
      const long long pieces = (total_v + GATHER_PIECE_V - 1) / GATHER_PIECE_V;
      const unsigned int pieces_per_block = static_cast<unsigned int>(p.K / 64);  // 128 rows x K x 2 B / 16 KiB
      uint4* dstv = reinterpret_cast<uint4*>(p.ga_dst);
      for (;;) {
        unsigned int piece = 0;
        if (lane == 0) piece = atomicAdd(p.ga_sync, 1u);
        piece = __shfl_sync(0xffffffffu, piece, 0);
        if (piece >= pieces) break;
        const long long v0 = static_cast<long long>(piece) * GATHER_PIECE_V;
        const long long flat0 = p.ga_off + v0 * 8;
        const long long owner0 = flat0 / p.ga_shard;
        const long long rem0 = flat0 - owner0 * p.ga_shard;
#pragma unroll 1
        for (int b = 0; b < GATHER_PIECE_V / 256; ++b) {
          uint4 v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int i = b * 256 + u * 32 + lane;
            v[u] = make_uint4(0u, 0u, 0u, 0u);
            if (v0 + i < total_v) {
              long long rem = rem0 + static_cast<long long>(i) * 8;
              long long owner = owner0;
              if (rem >= p.ga_shard) {  // a piece is shorter than a shard: at most one boundary inside it
                rem -= p.ga_shard;
                ++owner;
              }
              if (FTB_IN_RANGE(owner, p.ga_world))
                v[u] = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p.ga_peers[owner]) + rem);
            }
          }
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int i = b * 256 + u * 32 + lane;
            if (v0 + i < total_v) dstv[v0 + i] = v[u];
          }
        }
        asm volatile("fence.proxy.async.global;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          __threadfence();
          atomicAdd(p.ga_sync + 1 + piece / pieces_per_block, 1u);
        }
      }
    }
  } else {
    // ---------------- epilogue (warps 2..5 of both CTAs) ----------------
    const int q = warp & 3;
    int acc = 0;
    uint32_t acc_phase = 0;
    const bool vec_ok = p.out_fp32 ? ((p.ldc & 3) == 0) : ((p.ldc & 7) == 0);
    uint32_t pairs_phase = 0;  // EPI_DSWIGLU, EPI_ADD: bit h, of half h
    for (Work w = first; have_work(w); next_work(w)) {
      if (w.t != pair_id) tile_coords(w.t, m0, n0);
      if (EPI == EPI_DSWIGLU || (EPI == EPI_ADD && !(SPLIT && w.shared))) {
        // 64 columns at a time: the 128 gate/up columns they belong to (EPI_ADD: what C holds there) come by TMA, two pieces ahead
        // (the first two under the tile's products), are replaced in place by their gradients (the sums), and leave by TMA.
        // A thread that reads its row of C piece by piece where it writes it waits for memory 32 times in a row: 8192 x 1024 x
        // 750 added to C 63.5 -> 24.6 us (stored: 20.5), 1024 x 256 x 64 20.5 -> 10.2, 128256 x 2048 x 2048 1546 -> 695.
        constexpr int BOXES = EPI == EPI_DSWIGLU ? 2 : 1;  // 64 columns each, of a piece
        const CUtensorMap* map = EPI == EPI_DSWIGLU ? &tmAux : &tmC;
        const int row0 = m0 + q * 32;
        const uint32_t stg = OFF_STAGING + q * STAGE_WARP_BYTES;
        auto inside = [&](int c) { return n0 + c * 64 < p.N && row0 < p.M; };
        auto fetch = [&](int c) {
          mbar_expect_tx(pairs_bar(q, c & 1), STAGE_WARP_BYTES / 2);
#pragma unroll
          for (int h = 0; h < BOXES; ++h)
            tma_load_2d(smem_base + stg + (c & 1) * (STAGE_WARP_BYTES / 2) + h * 4096, map, pairs_bar(q, c & 1),
                        BOXES * (n0 + c * 64) + 64 * h, row0);
        };
        if (lane == 0) {
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the tile before has left the staging area
          if (inside(0)) fetch(0);
          if (inside(1)) fetch(1);
        }
        __syncwarp();
        if (!mbar_wait_warp(tfull_bar(acc), acc_phase, abort_flag)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr0 = tmem_base + acc * BN + (static_cast<uint32_t>(q * 32) << 16);
        bool ok = true;
#pragma unroll 1
        for (int c = 0; c < BN / 64; ++c) {
          uint32_t v[64];
          tmem_ld32(taddr0 + c * 64, v);
          tmem_ld32(taddr0 + c * 64 + 32, v + 32);
          if (c > 0 && c + 1 < BN / 64 && lane == 0 && inside(c + 1)) {
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // piece c - 1 has left
            fetch(c + 1);
          }
          __syncwarp();
          tmem_wait_ld();
          if (c + 1 == BN / 64) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(map_to_cta(tempty_bar(acc), lead_cta));
          }
          if (!inside(c)) continue;
          if (!mbar_wait_warp(pairs_bar(q, c & 1), (pairs_phase >> (c & 1)) & 1u, abort_flag)) {
            ok = false;
            break;
          }
          pairs_phase ^= 1u << (c & 1);
          uint8_t* prow = smem + stg + (c & 1) * (STAGE_WARP_BYTES / 2) + lane * 128;
#pragma unroll
          for (int j = 0; j < 8 * BOXES; ++j) {
            ftb200::bf16x8* at = reinterpret_cast<ftb200::bf16x8*>(prow + (j >> 3) * 4096 + (((j & 7) ^ (lane & 7)) << 4));
            float f[8], o[8];
            ftb200::unpack8(*at, f);
            if (EPI == EPI_ADD) {
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = __uint_as_float(v[(8 * j + e) & 63]) + f[e];
              *at = ftb200::pack8(o);
              continue;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float d = __uint_as_float(v[4 * j + e]), g = f[2 * e], u = f[2 * e + 1];
              const float sg = 1.f / (1.f + __expf(-g));
              const float silu = g * sg;
              o[2 * e] = d * u * (sg + silu * (1.f - sg));
              o[2 * e + 1] = d * silu;
            }
            *at = ftb200::pack8(o);
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
#pragma unroll
            for (int h = 0; h < BOXES; ++h)
              if (n0 + c * 64 + 32 * h < p.N)
                tma_store_2d(map, smem_base + stg + (c & 1) * (STAGE_WARP_BYTES / 2) + h * 4096, BOXES * (n0 + c * 64) + 64 * h,
                             row0);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
        if (!ok) break;
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1u;
        }
        continue;
      }
      if (!mbar_wait_warp(tfull_bar(acc), acc_phase, abort_flag)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int row = m0 + q * 32 + lane;
      const uint32_t taddr0 = tmem_base + acc * BN + (static_cast<uint32_t>(q * 32) << 16);
      const uint32_t stg = OFF_STAGING + q * STAGE_WARP_BYTES;
      if (EPI == EPI_LOSS || (EPI == EPI_STORE && p.tma_out && !(SPLIT && w.shared))) {
        // bf16 output: 64 columns at a time go, one row a thread, into a 128-byte-swizzled piece of the warp's staging area
        // and leave by TMA (which clips what lies beyond M and N), while the next 64 come out of tensor memory.  Nothing hides
        // the last tile's epilogue: 5800 cycles for 256 columns that leave a row-major staging area as row segments, 4100
        // this way, all in all 14.2 -> 12.6 us for 3000 x 1536 x 1024, 17.3 -> 14.5 us for 1024 x 1024 x 3000.
        constexpr int PIECES = BN / 64;
        float row_max = -INFINITY, row_sum = 0.f;  // EPI_LOSS: over the tile's columns
        long long target = -1;
        if (EPI == EPI_LOSS && row < p.M) target = p.target[row];
        uint32_t r[2][64];
        tmem_ld32(taddr0, r[0]);
        tmem_ld32(taddr0 + 32, r[0] + 32);
#pragma unroll
        for (int c = 0; c < PIECES; ++c) {
          tmem_wait_ld();
          if (c + 1 < PIECES) {
            tmem_ld32(taddr0 + (c + 1) * 64, r[(c + 1) & 1]);
            tmem_ld32(taddr0 + (c + 1) * 64 + 32, r[(c + 1) & 1] + 32);
          } else {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(map_to_cta(tempty_bar(acc), lead_cta));
          }
          const uint32_t* v = r[c & 1];
          const bool inside = n0 + c * 64 < p.N && m0 + q * 32 < p.M;
          // With an activation the two halves of the area are one for C and one for 64 columns of aux, which two pieces fill.
          const bool with_aux = EPI == EPI_STORE && p.aux != nullptr;
          const uint32_t piece = with_aux ? stg : stg + (c & 1) * (STAGE_WARP_BYTES / 2);
          if (lane == 0) {  // what was stored from this half last has been read
            if (with_aux)
              asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            else
              asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          }
          __syncwarp();
          uint8_t* prow = smem + piece + lane * 128;
          uint8_t* arow = smem + stg + STAGE_WARP_BYTES / 2 + lane * 128;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[8 * j + e]);
            const ftb200::bf16x8 packed = ftb200::pack8(f);
            *reinterpret_cast<ftb200::bf16x8*>(prow + ((j ^ (lane & 7)) << 4)) = packed;
            if (with_aux) *reinterpret_cast<uint2*>(arow + ((((c & 1) * 4 + (j >> 1)) ^ (lane & 7)) << 4) + (j & 1) * 8) = silu_mul(packed);
          }
          if (EPI == EPI_LOSS && inside) {
            // of the rounded values, as they are stored; columns beyond N are left out
            const int left = p.N - (n0 + c * 64);
            float f[8], top = row_max;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (8 * j < left) {  // N is a multiple of 8
                ftb200::unpack8(*reinterpret_cast<const ftb200::bf16x8*>(prow + ((j ^ (lane & 7)) << 4)), f);
#pragma unroll
                for (int e = 0; e < 8; ++e) top = fmaxf(top, f[e]);
              }
            }
            const float base = top == -INFINITY ? 0.f : top;
            row_sum *= __expf(row_max - base);
            row_max = top;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (8 * j < left) {
                ftb200::unpack8(*reinterpret_cast<const ftb200::bf16x8*>(prow + ((j ^ (lane & 7)) << 4)), f);
#pragma unroll
                for (int e = 0; e < 8; ++e) row_sum += __expf(f[e] - base);
              }
            }
            const long long at = target - (n0 + c * 64);
            if (at >= 0 && at < 64 && at < left)
              p.target_value[row] = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(
                  prow + (((static_cast<int>(at) >> 3) ^ (lane & 7)) << 4) + (at & 7) * 2));
          }
          fence_async_smem();
          __syncwarp();
          if (EPI != EPI_LOSS && lane == 0 && inside) {
            tma_store_2d(&tmC, smem_base + piece, n0 + c * 64, m0 + q * 32);
            if (with_aux && ((c & 1) || n0 + (c + 1) * 64 >= p.N))
              tma_store_2d(&tmAux, smem_base + stg + STAGE_WARP_BYTES / 2, (n0 + (c & ~1) * 64) >> 1, m0 + q * 32);
          }
          if (lane == 0) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        if (EPI == EPI_LOSS && row < p.M)
          p.row_stats[static_cast<long long>(row) * num_n + n0 / BN] = make_float2(row_max, row_sum);
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1u;
        }
        continue;
      }
      if constexpr (EPI != EPI_STORE && !(EPI == EPI_ADD && SPLIT)) continue;
      auto store_chunk = [&](int c, const uint32_t* r) {  // 32 columns of the thread's row
        const int col0 = n0 + c * 32;
        if (row < p.M && col0 < p.N) {
          const bool full = vec_ok && (col0 + 32 <= p.N);
          if (p.out_fp32) {
            float* dst = reinterpret_cast<float*>(p.C) + static_cast<long long>(row) * p.ldc + col0;
            if (full) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float4 v = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                       __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
                if (p.accumulate) {
                  const float4 o = reinterpret_cast<const float4*>(dst)[j];
                  v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
                }
                reinterpret_cast<float4*>(dst)[j] = v;
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                if (col0 + j < p.N) {
                  const float v = __uint_as_float(r[j]);
                  dst[j] = p.accumulate ? dst[j] + v : v;
                }
              }
            }
          } else {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.C) + static_cast<long long>(row) * p.ldc + col0;
            if (full) {
              ftb200::bf16x8 old[4];
              if (EPI == EPI_ADD) {  // all on their way before the first store
#pragma unroll
                for (int j = 0; j < 4; ++j) old[j] = reinterpret_cast<const ftb200::bf16x8*>(dst)[j];
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                float f[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[8 * j + e]);
                if (p.accumulate) {
                  float o[8];
                  ftb200::unpack8(EPI == EPI_ADD ? old[j] : reinterpret_cast<const ftb200::bf16x8*>(dst)[j], o);
#pragma unroll
                  for (int e = 0; e < 8; ++e) f[e] += o[e];
                }
                const ftb200::bf16x8 packed = ftb200::pack8(f);
                reinterpret_cast<ftb200::bf16x8*>(dst)[j] = packed;
                if (p.aux != nullptr)
                  *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.aux) + static_cast<long long>(row) * p.ld_aux +
                                            (col0 >> 1) + 4 * j) = silu_mul(packed);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                if (col0 + j < p.N) {
                  float v = __uint_as_float(r[j]);
                  if (p.accumulate) v += __bfloat162float(dst[j]);
                  dst[j] = __float2bfloat16(v);
                }
              }
            }
          }
        }
      };
      if (SPLIT && w.shared) {
        // A chunk is kept as a share of each warp, four columns of its 32 rows after another.  It is written to this CTA's own
        // ring and copied from there; remote stores of 16 bytes a thread are no faster and no simpler to count.
        constexpr int CHUNKS = BN / 32;
        auto owner = [&](int c) { return c * S / CHUNKS; };
        auto first_of = [&](int j) { return (j * CHUNKS + S - 1) / S; };
        const int mine0 = first_of(pair), mine = first_of(pair + 1) - mine0;  // this CTA's chunks
        const uint32_t in = smem_base + q * SHARE_BYTES + static_cast<uint32_t>(lane) * 16;
        if (q == 2) {
          if (lane == 0) mbar_expect_tx(got_bar, (S - 1) * mine * CHUNK_BYTES);
          __syncwarp();
          // this CTA's products are done: its ring may be written
          if (lane < S && lane != pair) mbar_arrive_cluster(map_to_cta(ready_bar, 2 * lane + rank));
          __syncwarp();
        }
        bool told = false;  // the others' rings are free
        int out = 0;
        for (int c = 0; c < CHUNKS; ++c) {
          const int j = owner(c);
          if (j == pair) continue;
          uint32_t r[32];
          tmem_ld32(taddr0 + c * 32, r);
          const uint32_t from = smem_base + (MAX_IN + out++) * CHUNK_BYTES + q * SHARE_BYTES;
          tmem_wait_ld();
#pragma unroll
          for (int v = 0; v < 8; ++v)
            *reinterpret_cast<uint4*>(smem + (from - smem_base) + v * 512 + lane * 16) = make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
          fence_async_smem();
          if (!told && !mbar_wait_cluster(ready_bar, 0, abort_flag)) break;
          told = true;
          __syncwarp();
          if (lane == 0) {  // the owner keeps the chunks of the other pairs in their order
            const int slot = (pair - (pair > j)) * (first_of(j + 1) - first_of(j)) + c - first_of(j);
            copy_to_cta(map_to_cta(smem_base + slot * CHUNK_BYTES + q * SHARE_BYTES, 2 * j + rank), from, SHARE_BYTES,
                        map_to_cta(got_bar, 2 * j + rank));
          }
        }
        if (!mbar_wait_warp(got_bar, 0, abort_flag)) break;
#pragma unroll 1
        for (int c = mine0; c < mine0 + mine; ++c) {
          uint32_t own[32], r[32];
          tmem_ld32(taddr0 + c * 32, own);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < MAX_SPLIT; ++j) {
            if (j >= S) break;
            const uint8_t* slot = smem + (in - smem_base) + ((j - (j > pair)) * mine + c - mine0) * CHUNK_BYTES;
#pragma unroll
            for (int v = 0; v < 8; ++v) {
              float4 x = make_float4(__uint_as_float(own[4 * v]), __uint_as_float(own[4 * v + 1]), __uint_as_float(own[4 * v + 2]),
                                     __uint_as_float(own[4 * v + 3]));
              if (j != pair) x = *reinterpret_cast<const float4*>(slot + v * 512);
              r[4 * v] = __float_as_uint(j == 0 ? x.x : __uint_as_float(r[4 * v]) + x.x);
              r[4 * v + 1] = __float_as_uint(j == 0 ? x.y : __uint_as_float(r[4 * v + 1]) + x.y);
              r[4 * v + 2] = __float_as_uint(j == 0 ? x.z : __uint_as_float(r[4 * v + 2]) + x.z);
              r[4 * v + 3] = __float_as_uint(j == 0 ? x.w : __uint_as_float(r[4 * v + 3]) + x.w);
            }
          }
          store_chunk(c, r);
        }
      } else if (p.sc_world > 0) {
        // Scattered to the owners' memory: the tile goes through a per-warp staging area so that every store instruction
        // covers two 256-byte row segments.  One 16-byte piece per thread and row would touch 32 rows per instruction: an
        // NVLink packet each, which throttles the kernel.
        const int half = lane >> 4, ch = lane & 15;
#pragma unroll 1
        for (int cg = 0; cg < BN / 128; ++cg) {
#pragma unroll 1
          for (int cc = 0; cc < 4; ++cc) {
            uint32_t r[32];
            tmem_ld32(taddr0 + (cg * 4 + cc) * 32, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float f[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[8 * j + e]);
              *reinterpret_cast<ftb200::bf16x8*>(smem + stg + lane * 256 + (((cc * 4 + j) ^ (lane & 15)) << 4)) = ftb200::pack8(f);
            }
          }
          __syncwarp();
          const int gcol = n0 + cg * 128 + ch * 8;
#pragma unroll 4
          for (int it = 0; it < 16; ++it) {
            const int rr = it * 2 + half;
            const int grow = m0 + q * 32 + rr;
            const ftb200::bf16x8 v = *reinterpret_cast<const ftb200::bf16x8*>(smem + stg + rr * 256 + ((ch ^ (rr & 15)) << 4));
            if (grow < p.M && gcol + 8 <= p.N) {
              const long long flat = p.sc_off + static_cast<long long>(grow) * p.ldc + gcol;
              const long long owner = flat / p.sc_shard;
              const long long rem = flat - owner * p.sc_shard;
              if (!FTB_IN_RANGE(owner, p.sc_world)) continue;
              __nv_bfloat16* base = reinterpret_cast<__nv_bfloat16*>(p.sc_peers[owner]);
              *reinterpret_cast<ftb200::bf16x8*>(base + static_cast<long long>(p.sc_src) * p.sc_shard + rem) = v;
            }
          }
          __syncwarp();
        }
      } else {
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(taddr0 + c * 32, r);
          tmem_wait_ld();
          store_chunk(c, r);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(map_to_cta(tempty_bar(acc), lead_cta));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // no store reads the staging area any more
    if (*abort_flag) sleep_200us();  // this warp's loads and copies that nobody waited for have ended then
    __syncwarp();
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag && p.status != nullptr) atomicExch(p.status, FTB200_ST_TIMEOUT);
  cluster_sync_relaxed();  // no CTA retires while another may still touch its barriers, operands or ring
  // what another pair copied into this CTA's ring may still be on its way if this one has given up waiting for it
  if (SPLIT) {
    if (*abort_flag) sleep_200us();
    __syncwarp();
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// One row: C[n] = sum_k a[k] B[n, k] of a K-major B.  Bound by reading B once; a warp takes ROWS rows of it, GEMV_LOADS loads of
// 16 bytes of each in flight a lane, and `a` comes from L1.  The tile kernel reads B at 4.3 TB/s for a row, 255 rows of every
// tile being padding: 128256 x 4096 246 -> 163 us (6.5 TB/s),
// 8192 x 1024 12.1 -> 6.2, 1024 x 256 6.0 -> 2.5.
constexpr int GEMV_ROWS = 2, GEMV_LOADS = 4, GEMV_THREADS = 256;

__global__ void __launch_bounds__(GEMV_THREADS)
gemv_bf16_kernel(const ftb200::bf16x8* a, const ftb200::bf16x8* B, __nv_bfloat16* C, int N,
                 int K8, long long ldb8) {
  ftb200::wait_for_previous();
  ftb200::start_next();
  const int lane = threadIdx.x & 31;
  const int n0 = (static_cast<int>(blockIdx.x) * (GEMV_THREADS / 32) + (threadIdx.x >> 5)) * GEMV_ROWS;
  if (n0 >= N) return;
  const ftb200::bf16x8* row[GEMV_ROWS];
#pragma unroll
  for (int r = 0; r < GEMV_ROWS; ++r) row[r] = B + min(n0 + r, N - 1) * ldb8;
  float sum[GEMV_ROWS][2] = {};
  for (int k0 = lane; k0 < K8; k0 += 32 * GEMV_LOADS) {
    uint4 b[GEMV_ROWS][GEMV_LOADS];
    ftb200::bf16x8 x[GEMV_LOADS];
#pragma unroll
    for (int u = 0; u < GEMV_LOADS; ++u) {
      const bool in = k0 + 32 * u < K8;
#pragma unroll
      for (int r = 0; r < GEMV_ROWS; ++r)
        b[r][u] = in ? __ldcs(reinterpret_cast<const uint4*>(row[r] + k0 + 32 * u)) : make_uint4(0u, 0u, 0u, 0u);
      if (in) x[u] = a[k0 + 32 * u];
    }
#pragma unroll
    for (int u = 0; u < GEMV_LOADS; ++u) {
      if (k0 + 32 * u >= K8) break;
      float f[8];
      ftb200::unpack8(x[u], f);
#pragma unroll
      for (int r = 0; r < GEMV_ROWS; ++r) {
        float g[8];
        ftb200::unpack8(*reinterpret_cast<const ftb200::bf16x8*>(&b[r][u]), g);
#pragma unroll
        for (int e = 0; e < 8; ++e) sum[r][e & 1] = fmaf(f[e], g[e], sum[r][e & 1]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < GEMV_ROWS; ++r) {
    const float s = ftb200::warp_sum(sum[r][0] + sum[r][1]);
    if (lane == 0 && n0 + r < N) C[n0 + r] = __float2bfloat16(s);
  }
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
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

int encode_2d(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_cols,
              int box_rows) {
  auto fn = get_encode_fn();
  if (fn == nullptr) return FTB200_E_DRIVER;
  cuuint64_t gdim[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t gstride[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(box_cols), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), gdim, gstride, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : FTB200_E_DRIVER;
}

}  // namespace

// Same arguments as ftb200_gemm_bf16; pairs of CTAs cooperate on 256x256 tiles.
struct ScatterSpec {
  int world = 0;
  int src = 0;
  long long shard = 0;
  long long off = 0;
  void* const* peers = nullptr;
};

struct EpilogueSpec {
  int kind = EPI_STORE;
  float2* row_stats = nullptr;
  float* target_value = nullptr;
  const long long* target = nullptr;
};

struct GatherSpec {
  int world = 0;
  long long shard = 0;
  long long off = 0;
  const void* const* peers = nullptr;
  unsigned int* sync = nullptr;
};

template <int BN, bool SPLIT, int EPI>
static cudaError_t prepare_2cta() {
  static std::atomic<bool> done{false};
  if (done.load(std::memory_order_acquire)) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(gemm_bf16_tcgen05_2cta_kernel<BN, SPLIT, EPI>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<BN, EPI>::SMEM_BYTES);
  if (e == cudaSuccess) done.store(true, std::memory_order_release);
  return e;
}

// attrs: room for two.
static void cluster_launch(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attrs, int ctas, int pairs_per_cluster, int threads,
                           uint32_t smem, cudaStream_t stream) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = 2 * pairs_per_cluster;
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = 1;
}

// How many clusters of `split` pairs fit the chip at once (clusters do not span its processing clusters, whose number of
// SMs is no multiple of every size).
template <int BN>
static int resident_clusters(int split) {
  static std::atomic<int> known[MAX_SPLIT + 1];
  int n = known[split].load(std::memory_order_relaxed);
  if (n == 0) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attrs[2];
    cluster_launch(cfg, attrs, 2 * split, split, NUM_THREADS, Tile<BN, EPI_STORE>::SMEM_BYTES, nullptr);
    if (prepare_2cta<BN, true, EPI_STORE>() != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, gemm_bf16_tcgen05_2cta_kernel<BN, true, EPI_STORE>, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = -1;
    }
    known[split].store(n, std::memory_order_relaxed);
  }
  return n;
}

struct TilePlan {
  int columns;  // of a pair's tile
  int split;    // pairs that share a tile of the last wave (1: none do)
  int whole;    // tiles before them
  int ctas;
};

// Columns of a pair's tile: 128 where the narrow tiles of the whole output fit the pairs at once, 256 elsewhere.  A narrow
// tile takes about 0.7 of a wide one's time (it asks the L2 for 96 bytes a cycle and SM instead of 64), so it pays where
// it only puts idle pairs to work: 1024 x 1024 x 3000 26.0 -> 17.3 us, 256 x 1024 x 256 9.8 -> 6.3 us; but 3000 x 5632 x
// 1024 36.0 -> 40.6 us, 1536 x 4096 x 14336 146 -> 169 us.
// And whether the last wave (the whole output, where it is less than one) is split over K, by an estimate of the time in
// units of one 64-deep slab of a 256-column tile (0.3 us): the waves' slabs and, for a shared tile, SPLIT_COST: about
// 9 us go into the meeting of its accumulators, whatever K is.  1536 x 4096 x 14336 (96 tiles on 74 pairs) 144 -> 123 us,
// 1536 x 4096 x 28672 290 -> 240, 3072 x 2048 x 8192 84 -> 77, 750 x 1024 x 8192 30 -> 25, 77 x 4096 x 14336 52 -> 44; where the
// estimate says no: 500 x 4096 x 4096 20 -> 27, 1536 x 1024 x 3000 15 -> 22, 1000 x 2048 x 2048 13 -> 20.
static TilePlan plan_tiles(int M, int N, int K, int pairs, bool may_split) {
  constexpr float NARROW = 0.7f, SPLIT_COST = 32.f;
  const int rows = (M + 2 * BM - 1) / (2 * BM), slabs = (K + BK - 1) / BK;
  const int wide = rows * ((N + 255) / 256), narrow = rows * ((N + 127) / 128);
  TilePlan best{narrow <= pairs ? 128 : 256, 1, 0, 2 * pairs};
  float least = best.columns == 128 ? slabs * NARROW : static_cast<float>((wide + pairs - 1) / pairs) * slabs;
  if (!may_split || slabs < 16) return best;
  for (int columns = 128; columns <= 256; columns += 128) {
    const int tiles = columns == 128 ? narrow : wide;
    const float slab = columns == 128 ? NARROW : 1.f;
    for (int split = 2; split <= MAX_SPLIT && 4 * split <= slabs; ++split) {
      const int clusters = columns == 128 ? resident_clusters<128>(split) : resident_clusters<256>(split);
      if (clusters <= 0) continue;
      const int waves = tiles / (clusters * split), rest = tiles - waves * clusters * split;
      if (rest == 0 || rest > clusters) continue;
      const float cost = (waves * slabs + (slabs + split - 1) / split) * slab + SPLIT_COST;
      if (cost < least) {
        least = cost;
        best = TilePlan{columns, split, waves * clusters * split, 2 * split * (waves > 0 ? clusters : rest)};
      }
    }
  }
  return best;
}

template <int BN, bool SPLIT, int EPI>
static int launch_2cta(const void* A, const void* B, long long lda, long long ldb, int ctas, int split, int threads,
                       const GemmParams& p, cudaStream_t stream) {
  CUtensorMap tmA, tmB, tmC, tmAux;
  int rc;
  if (!p.a_mn)
    rc = encode_2d(&tmA, A, p.M, p.K, lda, BK, BM);
  else
    rc = encode_2d(&tmA, A, p.K, p.M, lda, 64, BK);
  if (rc) return rc;
  if (!p.b_mn)
    rc = encode_2d(&tmB, B, p.N, p.K, ldb, BK, BN / 2);
  else
    rc = encode_2d(&tmB, B, p.K, p.N, ldb, 64, BK);
  if (rc) return rc;
  tmC = tmAux = tmA;  // not used without tma_out
  if (p.tma_out) {
    if (p.C != nullptr) rc = encode_2d(&tmC, p.C, p.M, p.N, p.ldc, 64, 32);
    if (rc == 0 && p.aux != nullptr)
      rc = encode_2d(&tmAux, p.aux, p.M, EPI == EPI_DSWIGLU ? 2 * p.N : p.N / 2, p.ld_aux, 64, 32);
    if (rc) return rc;
  }
  if (prepare_2cta<BN, SPLIT, EPI>() != cudaSuccess) return FTB200_E_CUDA;
  const int tiles = ((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + BN - 1) / BN);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attrs[2];
  cluster_launch(cfg, attrs, SPLIT ? ctas : std::min(2 * tiles, ctas), split, threads, Tile<BN, EPI>::SMEM_BYTES, stream);
  if (p.ga_world == 0 && p.sc_world == 0) {  // as ftb200::launch_after does
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
  }
  return cudaLaunchKernelEx(&cfg, gemm_bf16_tcgen05_2cta_kernel<BN, SPLIT, EPI>, tmA, tmB, tmC, tmAux, p) == cudaSuccess
             ? 0
             : FTB200_E_CUDA;
}

static int gemm_2cta_impl(const void* A, const void* B, void* C, int M, int N, int K, int a_mn_major, int b_mn_major,
                          long long lda, long long ldb, long long ldc, int flags, int* status, int max_ctas, void* aux,
                          long long ld_aux, cudaStream_t stream, const ScatterSpec* sc = nullptr,
                          const GatherSpec* ga = nullptr, const EpilogueSpec* ep = nullptr) {
  if (M <= 0 || N <= 0 || K <= 0 || A == nullptr || B == nullptr || (C == nullptr && sc == nullptr && ep == nullptr)) return FTB200_E_BADARG;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda & 7) || (ldb & 7))
    return FTB200_E_ALIGN;
  if ((reinterpret_cast<uintptr_t>(C) & 15)) return FTB200_E_ALIGN;
  if (M == 1 && !a_mn_major && !b_mn_major && flags == 0 && (K & 7) == 0 && aux == nullptr && sc == nullptr && ga == nullptr &&
      ep == nullptr && max_ctas <= 0) {
    constexpr int PER_BLOCK = GEMV_ROWS * GEMV_THREADS / 32;
    ftb200::launch_after(gemv_bf16_kernel, (N + PER_BLOCK - 1) / PER_BLOCK, GEMV_THREADS, 0, stream,
        reinterpret_cast<const ftb200::bf16x8*>(A), reinterpret_cast<const ftb200::bf16x8*>(B),
        reinterpret_cast<__nv_bfloat16*>(C), N, K / 8, ldb / 8);
    return cudaGetLastError() == cudaSuccess ? 0 : FTB200_E_CUDA;
  }
  GemmParams p;
  p.M = M; p.N = N; p.K = K;
  p.a_mn = a_mn_major ? 1 : 0;
  p.b_mn = b_mn_major ? 1 : 0;
  p.out_fp32 = flags & 1;
  p.accumulate = (flags >> 1) & 1;
  p.ldc = ldc;
  p.C = C;
  p.status = status;
  p.aux = aux;
  p.ld_aux = ld_aux;
  p.row_stats = ep != nullptr ? ep->row_stats : nullptr;
  p.target_value = ep != nullptr ? ep->target_value : nullptr;
  p.target = ep != nullptr ? ep->target : nullptr;
  p.sc_world = 0;
  p.sc_src = 0;
  p.sc_shard = 0;
  p.sc_off = 0;
  for (int i = 0; i < 8; ++i) p.sc_peers[i] = nullptr;
  if (sc != nullptr) {
    p.sc_world = sc->world;
    p.sc_src = sc->src;
    p.sc_shard = sc->shard;
    p.sc_off = sc->off;
    for (int i = 0; i < sc->world && i < 8; ++i) p.sc_peers[i] = sc->peers[i];
  }
  // TMA wants 16-byte rows; what else comes (fp32, other strides) takes the general path of the epilogue
  p.tma_out = sc == nullptr && !p.out_fp32 && (ldc & 7) == 0 && ldc >= N && (N & 7) == 0 &&
              (aux == nullptr || ((ld_aux & 7) == 0 && ld_aux >= N / 2 && (reinterpret_cast<uintptr_t>(aux) & 15) == 0));
  const bool add = p.tma_out && p.accumulate && ga == nullptr && aux == nullptr;
  if (p.accumulate && !add) p.tma_out = 0;
  p.group_m = GROUP_M;
  p.whole = 0;
  p.ga_world = 0;
  p.ga_shard = 0;
  p.ga_off = 0;
  p.ga_dst = nullptr;
  p.ga_sync = nullptr;
  for (int i = 0; i < 8; ++i) p.ga_peers[i] = nullptr;
  if (ga != nullptr) {
    p.ga_world = ga->world;
    p.ga_shard = ga->shard;
    p.ga_off = ga->off;
    p.ga_dst = const_cast<void*>(B);
    p.ga_sync = ga->sync;
    for (int i = 0; i < ga->world && i < 8; ++i) p.ga_peers[i] = ga->peers[i];
    // Sixteen row tiles share a B tile before the next B tile (eight without the gather).  The whole weight is
    // needed by the end of the first group of row tiles; with M = 8192 that group is half of the GEMM instead of
    // a quarter, which halves the link bandwidth the gather needs to stay ahead, and costs ~2.5 % of the GEMM's
    // speed in L2 locality (measured; all of M per B tile costs ~9 %).
    p.group_m = 2 * GROUP_M;
    if (cudaMemsetAsync(ga->sync, 0, sizeof(unsigned int) * (1 + static_cast<size_t>(N) / GATHER_BLOCK), stream) != cudaSuccess)
      return FTB200_E_CUDA;
  }
  int ctas = ftb200::sm_count() & ~1;
  if (max_ctas > 0 && max_ctas < ctas) ctas = std::max(2, max_ctas & ~1);
  if (ga != nullptr) return launch_2cta<256, false, EPI_STORE>(A, B, lda, ldb, ctas, 1, NUM_THREADS_GATHER, p, stream);
  if (ep != nullptr) {
    p.tma_out = 1;  // the entry has looked at what TMA wants
    const bool narrow = plan_tiles(M, N, K, ctas / 2, false).columns == 128;
    if (ep->kind == EPI_DSWIGLU)
      return narrow ? launch_2cta<128, false, EPI_DSWIGLU>(A, B, lda, ldb, ctas, 1, NUM_THREADS, p, stream)
                    : launch_2cta<256, false, EPI_DSWIGLU>(A, B, lda, ldb, ctas, 1, NUM_THREADS, p, stream);
    return narrow ? launch_2cta<128, false, EPI_LOSS>(A, B, lda, ldb, ctas, 1, NUM_THREADS, p, stream)
                  : launch_2cta<256, false, EPI_LOSS>(A, B, lda, ldb, ctas, 1, NUM_THREADS, p, stream);
  }
  // scattered and activated outputs leave through the staging area, which a shared tile does not
  const TilePlan plan = plan_tiles(M, N, K, ctas / 2, sc == nullptr && aux == nullptr && max_ctas <= 0);
  p.whole = plan.whole;
  if (add) {
    if (plan.split > 1)
      return plan.columns == 128 ? launch_2cta<128, true, EPI_ADD>(A, B, lda, ldb, plan.ctas, plan.split, NUM_THREADS, p, stream)
                                 : launch_2cta<256, true, EPI_ADD>(A, B, lda, ldb, plan.ctas, plan.split, NUM_THREADS, p, stream);
    return plan.columns == 128 ? launch_2cta<128, false, EPI_ADD>(A, B, lda, ldb, ctas, 1, NUM_THREADS, p, stream)
                               : launch_2cta<256, false, EPI_ADD>(A, B, lda, ldb, ctas, 1, NUM_THREADS, p, stream);
  }
  if (plan.split > 1) {
    if (plan.columns == 128) return launch_2cta<128, true, EPI_STORE>(A, B, lda, ldb, plan.ctas, plan.split, NUM_THREADS, p, stream);
    return launch_2cta<256, true, EPI_STORE>(A, B, lda, ldb, plan.ctas, plan.split, NUM_THREADS, p, stream);
  }
  if (plan.columns == 128) return launch_2cta<128, false, EPI_STORE>(A, B, lda, ldb, ctas, 1, NUM_THREADS, p, stream);
  return launch_2cta<256, false, EPI_STORE>(A, B, lda, ldb, ctas, 1, NUM_THREADS, p, stream);
}

FTB200_API int ftb200_gemm_bf16_2cta(const void* A, const void* B, void* C, int M, int N, int K, int a_mn_major,
                                     int b_mn_major, long long lda, long long ldb, long long ldc, int flags, int* status,
                                     int max_ctas, cudaStream_t stream) {
  return gemm_2cta_impl(A, B, C, M, N, K, a_mn_major, b_mn_major, lda, ldb, ldc, flags, status, max_ctas, nullptr, 0, stream);
}

// Forward GEMM of a gated MLP with the activation fused into the epilogue: B's rows are
// interleaved (gate_0, up_0, gate_1, up_1, ...), C [M,N] receives the pre-activations and
// aux [M,N/2] receives silu(gate) * up.  bf16 output, N a multiple of 32, no accumulate.
FTB200_API int ftb200_gemm_bf16_swiglu(const void* A, const void* B, void* C, void* aux, int M, int N, int K, long long lda,
                                       long long ldb, long long ldc, long long ld_aux, int* status, int max_ctas,
                                       cudaStream_t stream) {
  if (aux == nullptr || (N % 32) || (ldc & 7) || (ld_aux & 3) || (reinterpret_cast<uintptr_t>(aux) & 7)) return FTB200_E_ALIGN;
  return gemm_2cta_impl(A, B, C, M, N, K, 0, 0, lda, ldb, ldc, 0, status, max_ctas, aux, ld_aux, stream);
}

static bool aligned16(const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15) == 0; }

// Backward of a gated MLP's down projection and activation: D[M,N] = dY[M,K] . W[K,N] (W row-major, as it is stored for the
// forward product) is the gradient of silu(gate) * up and is not stored; gu [M, 2 N], the interleaved (gate, up) pairs of
// the forward pass, is overwritten by their gradients.  N and ld_gu multiples of 8.
FTB200_API int ftb200_gemm_bf16_dswiglu(const void* dY, const void* W, void* gu, int M, int N, int K, long long ld_dy,
                                        long long ld_w, long long ld_gu, int* status, cudaStream_t stream) {
  if (gu == nullptr) return FTB200_E_BADARG;
  if ((N & 7) || (ld_gu & 7) || ld_gu < 2LL * N || !aligned16(gu)) return FTB200_E_ALIGN;
  if (N > 0x3fffffff) return FTB200_E_TOOBIG;
  EpilogueSpec ep;
  ep.kind = EPI_DSWIGLU;
  return gemm_2cta_impl(dY, W, nullptr, M, N, K, 0, 1, ld_dy, ld_w, N, 0, status, 0, gu, ld_gu, stream, nullptr, nullptr, &ep);
}

// Floats of scratch memory for ftb200_gemm_bf16_loss.
FTB200_API long long ftb200_gemm_bf16_loss_scratch_floats(int M, int N) {
  if (M <= 0 || N <= 0) return 0;
  const int columns = plan_tiles(M, N, 1, ftb200::sm_count() / 2, false).columns;
  return static_cast<long long>(M) * (2LL * ((N + columns - 1) / columns) + 1);
}

int ftb200_launch_cross_entropy_rows(const long long* target, const float2* row_stats, const float* target_value, float* loss,
                                     int tiles, int T, int V, cudaStream_t st);

// Cross-entropy of logits = A[M,K] . B[N,K]^T against target [M], which are not stored: loss[row] = logsumexp - logit of the
// target (0 for a negative target, a target beyond N counts as logit 0), of the logits rounded to bf16.  The product's epilogue
// notes every row's maximum, sum of exponentials and target value per tile in `scratch`
// (ftb200_gemm_bf16_loss_scratch_floats, 8-byte aligned); a second kernel finishes the rows.  1024 x 128256 x 2048: 474 us with
// the logits stored and read again, 346 without.  (With gradients the logits have to be stored, and reading them once instead
// of twice gains nothing at 8192 rows: 7335 us either way at K = 4096.)  N a multiple of 8.
FTB200_API int ftb200_gemm_bf16_loss(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb,
                                     const long long* target, float* loss, float* scratch, int* status, cudaStream_t stream) {
  if (target == nullptr || loss == nullptr || scratch == nullptr || M <= 0 || N <= 0) return FTB200_E_BADARG;
  if ((N & 7) || (reinterpret_cast<uintptr_t>(scratch) & 7)) return FTB200_E_ALIGN;
  const int columns = plan_tiles(M, N, K, ftb200::sm_count() / 2, false).columns;
  const int tiles = (N + columns - 1) / columns;
  EpilogueSpec ep;
  ep.kind = EPI_LOSS;
  ep.row_stats = reinterpret_cast<float2*>(scratch);
  ep.target_value = scratch + 2LL * M * tiles;
  ep.target = target;
  const int rc = gemm_2cta_impl(A, B, nullptr, M, N, K, 0, 0, lda, ldb, N, 0, status, 0, nullptr, 0, stream, nullptr, nullptr, &ep);
  if (rc != 0) return rc;
  return ftb200_launch_cross_entropy_rows(target, ep.row_stats, ep.target_value, loss, tiles, M, N, stream);
}

// GEMM whose epilogue is the reduce-scatter's transfer: the [M,N] result (row-major, row
// stride N) is one field of a flat gradient unit that `world` ranks shard evenly; each
// 16-byte piece is stored straight into the owner rank's staging area
// (peers[owner] + src_rank * shard_elems + offset-in-shard) over NVLink while the tensor
// cores work on the next tile.  A team round and a local sum over the `world` staging
// slices (ftb200_team_reduce_scatter on local pointers) finish the reduce-scatter.
// N must be a multiple of 32; shard_elems and unit_off multiples of 8.
FTB200_API int ftb200_gemm_bf16_scatter(const void* A, const void* B, int M, int N, int K, int a_mn_major, int b_mn_major,
                                        long long lda, long long ldb, void* const* peers, int world, int src_rank,
                                        long long shard_elems, long long unit_off, int* status, int max_ctas,
                                        cudaStream_t stream) {
  if (peers == nullptr || world < 1 || world > 8 || src_rank < 0 || src_rank >= world) return FTB200_E_BADARG;
  if ((N % 32) || (shard_elems % 8) || (unit_off % 8)) return FTB200_E_ALIGN;
  if (unit_off + static_cast<long long>(M) * N > shard_elems * world) return FTB200_E_TOOBIG;
  ScatterSpec sc;
  sc.world = world; sc.src = src_rank; sc.shard = shard_elems; sc.off = unit_off; sc.peers = peers;
  return gemm_2cta_impl(A, B, nullptr, M, N, K, a_mn_major, b_mn_major, lda, ldb, N, 0, status, max_ctas, nullptr, 0, stream, &sc);
}

// C[M,N] = A[M,K] . B[N,K]^T where B is still spread over the shard group: `B_local` points at the weight's place
// inside this rank's gathered copy of a flat parameter unit (`unit_off` elements from the unit's start, row stride
// K), `shard_peers[r]` at rank r's shard of that unit (`shard_elems` elements each; [rank] is local memory).  The
// kernel fills B_local from the shards while it multiplies (see the head of this file); after it, B_local is an
// ordinary gathered weight.  `sync_words`: 1 + N/128 32-bit words of scratch in local memory, zeroed here on
// `stream`; it may be shared by all calls on one stream.  aux / ld_aux: optional SwiGLU output as in
// ftb200_gemm_bf16_swiglu (then N must be a multiple of 32).  N a multiple of 128, K of 64, bf16 output.
// The caller orders the call after every rank's shard has been written (a team round) and keeps the shards
// unchanged until all ranks' calls have ended.
FTB200_API int ftb200_gemm_bf16_gather(const void* A, void* B_local, void* C, int M, int N, int K, long long lda,
                                       long long ldc, const void* const* shard_peers, int world, long long shard_elems,
                                       long long unit_off, unsigned int* sync_words, void* aux, long long ld_aux,
                                       int* status, int max_ctas, cudaStream_t stream) {
  if (shard_peers == nullptr || sync_words == nullptr || world < 1 || world > 8) return FTB200_E_BADARG;
  if ((N % GATHER_BLOCK) || (K % 64) || (shard_elems % 8) || (unit_off % 8) || (ldc & 7)) return FTB200_E_ALIGN;
  if (shard_elems < 8LL * GATHER_PIECE_V) return FTB200_E_BADARG;  // a piece may cross one shard boundary, not two
  if (unit_off + static_cast<long long>(N) * K > shard_elems * world) return FTB200_E_TOOBIG;
  for (int r = 0; r < world; ++r)
    if (shard_peers[r] == nullptr || (reinterpret_cast<uintptr_t>(shard_peers[r]) & 15)) return FTB200_E_ALIGN;
  if (aux != nullptr && ((N % 32) || (ld_aux & 3) || (reinterpret_cast<uintptr_t>(aux) & 7))) return FTB200_E_ALIGN;
  GatherSpec ga;
  ga.world = world; ga.shard = shard_elems; ga.off = unit_off; ga.peers = shard_peers; ga.sync = sync_words;
  return gemm_2cta_impl(A, B_local, C, M, N, K, 0, 0, lda, K, ldc, 0, status, max_ctas, aux, ld_aux, stream, nullptr, &ga);
}

FTB_DEFINE_BOUNDS_QUERY(gemm_2cta)
