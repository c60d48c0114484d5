// Block-scaled e4m3 GEMM for large problems and long contractions,
//     D[m,n] = sum_kb SA(m,kb) SB(n,kb) sum_{k in kb} A[m,k] B[n,k],
// with the scales brought into a ring in shared memory and eight wide promotion warps.  Two forms:
//   CG = 2  pairs of SMs (tcgen05 cta_group::2): a cluster of two CTAs computes a 256 x 256 tile.  CTA r of a pair owns rows 128 r.. of
//           the tile (its tensor memory holds their accumulators) and loads its 128 rows of A and half of the 256 rows of B; the
//           tensor cores read the other half of B from the partner's shared memory.
//   CG = 1  one SM, 128 x 192 or 128 x 128 tiles, with a scale per column.
// Promotion is as in gemm_fp8.cu: float32 scales, so every 128-deep contraction block is a chain of its own into a fresh accumulator
// buffer, which promotion warps read, scale and add in registers; the same operations in the same order, hence the same bits.
//
// Warp roles of a CTA (384 threads):
//   0-7   promotion + epilogue: warp w reads TMEM lanes 32 (w % 4).. (a hardware rule), columns BN / 2 (w / 4).. of the accumulator
//   8     TMA producer
//   9     MMA issuer (of a pair: in the first CTA only)
//   10    scales: the block's row and column scales go into the ring, as many blocks ahead as there are stages
//   11    the tile's bulk stores
//
// What bounds the pairs: for large problems the board's power cap (1000 W; 32768 x 2048 -> 6144 in a loop of half a second runs at
// 1.36-1.40 GHz), else the promotion warps, which never find an accumulator missing: on each scheduler 2 x 64 packed FMAs of two
// cycles (twice that with a scale per column) and the register writes of the TMEM loads, which hold the FMA pipe up: 375 cycles of a
// block's 512 on the tensor core alone (666 with column scales), measured without MMAs, TMA or barriers; about 700 (1000) with
// everything.  So the design keeps promotion short rather than wide:
//   - A pair moves 32 KB per SM and block from the L2 instead of 48, and one thread issues for two SMs.
//   - Eight warps of 128 columns instead of sixteen of 64 (registers handed over, 224 each): half the barrier operations, scale loads and
//     set-up per block.  1400 warp instructions per block of a tile instead of 1821.  (Sixteen: 434 us for the problem above, eight 415.)
//   - No scale is fetched by a promotion warp and none is waited for separately: the accumulator's barrier counts the MMAs' commit and
//     the scale warp's announcement.  (A barrier of its own for the scales: 630 instead of 560 us for the weight gradient.)
//   - A wait's outcome is looked at once a tile, not voted on in every block.
//   - The buffer goes back by an arrival with CTA scope on the first CTA's barrier.  With cluster scope the release is a fence that waits
//     for the SM's copies in flight: 700 us instead of 360.
//   - In the last block of a bf16 tile each piece is converted and staged as soon as it is complete (forward 421 -> 413 us).
// Forward 32768 x 2048 -> 6144 in a loop: 435 us with gemm_fp8.cu, 413 here (1.90 / 2.00 PFLOP/s); with a scale per column 555 / 512;
// its weight gradient 584 / 548 (six waves where 5.2 would do); in short bursts 383 / 346, 530 / 435, 530 / 480.
//
// One SM with column scales: gemm_fp8.cu's promotion warps fetch and stage the scales of every block themselves, here they find them.
// From twelve blocks on 1.05-1.4 times as fast in one wave (200 x 2048 -> 8192 9.6 / 8.8 us, 500 x 4096 -> 4096 19.4 / 14.7, weight gradient
// 768 x 3072 of 4096 tokens 15.6 / 14.6), below it loses 0.2 us: scales come later to the first block, and eight warps take longer
// over the last tile than sixteen.  The same with a scale per 128 columns (not built: 2 % slower below twelve blocks, +-2 % above).
//
// Tried and left out: the next block's barrier probed during a block (a try_wait that comes too early suspends the warp; with test_wait
// 2 % slower), a ready counter in shared memory polled instead of the barrier (5 % slower), 32-column pieces in two register buffers
// (spills), column-scale pieces in two register buffers (3 % slower: the FMA pipe, not the load's latency, is the limit).
//
// Every wait on an mbarrier is bounded, as in gemm_fp8.cu (codes of its roles; 9 = scales).
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "gemm_tiles.cuh"
#include "host_api.h"
#include "mbarrier.cuh"
#include "umma.cuh"

namespace tg {

// ---- cluster forms of the PTX wrappers ---------------------------------------------------

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// the same shared-memory offset in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster_if(uint32_t bar, uint32_t pred) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cluster.b64 _, [%0];\n\t}"
               ::"r"(bar), "r"(pred) : "memory");
}
// a load into this CTA's shared memory whose bytes are counted by a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_f8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives on the barrier at this offset in both CTAs once the MMAs issued before are done
__device__ __forceinline__ void umma_commit_both(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(uint16_t(3)) : "memory");
}
__device__ __forceinline__ void umma_commit_here(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
template <int CG>
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  if constexpr (CG == 2) tma_load_2d_pair(dst, map, bar, x, y);
  else tma_load_2d(dst, map, bar, x, y);
}
template <int CG>
__device__ __forceinline__ void umma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (CG == 2) umma_f8_pair(d_tmem, a_desc, b_desc, idesc, accumulate);
  else umma_f8(d_tmem, a_desc, b_desc, idesc, accumulate);
}
template <int CG>
__device__ __forceinline__ void commit(uint32_t bar) {
  if constexpr (CG == 2) umma_commit_both(bar);
  else umma_commit(bar);
}
// four bytes from memory to shared memory (any 4-byte alignment), through L1: a row scale's sector serves eight blocks
__device__ __forceinline__ void cp_async_4(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// ---- kernel --------------------------------------------------------------------------------

constexpr int kBandRows = 16;      // 128-row tiles per band of the numbering (see tile_coords)

// Compile-time plan of one variant: CG CTAs (a cluster of two, or one) on a tile of 128 CG rows x BN columns.
template <int CG, int BN_, int SB_GRAN, bool OUT_F32>
struct RingCfg {
  static constexpr int BN = BN_, sb_gran = SB_GRAN;
  static constexpr bool out_f32 = OUT_F32;
  static constexpr int promo_warps = 8;
  static constexpr int producer_warp = 8, issuer_warp = 9, scale_warp = 10, store_warp = 11;
  static constexpr int threads = 384;
  // 168 registers a thread at launch; the service warpgroup hands over what the two promotion warpgroups grow by
  static constexpr int launch_regs = 168, promo_regs = 224, service_regs = 56;
  static_assert(service_regs + 2 * promo_regs <= 3 * launch_regs, "register hand-over asks for more than is released");
  static constexpr int cols = BN / 2, pieces = cols / 16;      // accumulator columns of a warp, in pieces of 16
  // Column scales: the fragment layout of an MMA accumulator (a thread holds 4 rows x cols / 4 columns instead of one row), in which a
  // column scale is shared by 8 lanes instead of all 32.
  static constexpr bool frag = SB_GRAN == 1;
  static_assert(frag || pieces % 2 == 0, "two register buffers take turns");
  static constexpr int tmem_bufs = BN > 128 ? 2 : 4, tmem_stride = kTmemCols / tmem_bufs;
  static constexpr int b_boxes = CG == 2 ? 1 : (BN + 127) / 128;   // (a CTA of a pair loads half of B)
  static_assert(CG == 1 || BN == 256, "a pair's tile");
  static constexpr int stage_bytes = (1 + b_boxes) * kTileBytes;
  // output boxes: 32 rows of box_cols columns; warp_boxes of them are staged at a time
  static constexpr int esize = OUT_F32 ? 4 : 2;
  static constexpr int box_cols = cols % (128 / esize) == 0 ? 128 / esize : 32;
  static constexpr int box_row = box_cols * esize, box_bytes = 32 * box_row, box_pieces = box_cols / 16;
  static constexpr int warp_boxes = cols / box_cols * box_bytes <= 8192 ? cols / box_cols : BN == 256 ? 2 : 1;
  static constexpr int phases = cols / (warp_boxes * box_cols);
  static_assert(phases * warp_boxes * box_cols == cols && (box_row == 128 || (box_row == 64 && frag)), "output boxes");
  static constexpr int out_bytes = promo_warps * warp_boxes * box_bytes;
  // a ring slot: 128 row scales, then the column scales (BN, or one per 128 columns)
  static constexpr int slot_floats = 128 + (SB_GRAN == 1 ? BN : 4);
  static constexpr int static_reserve = 1024;
  static constexpr int stages_fit = (kSmemLimit - static_reserve - out_bytes - tmem_bufs * 4 * slot_floats) / (stage_bytes + 4 * slot_floats);
  static constexpr int stages = stages_fit > 6 ? 6 : stages_fit;
  // The scales of block i go into slot i % ring once the stage of block i is free, that is, once the MMAs of block i - stages are
  // done.  Those were issued after every promotion warp had given back the accumulator of block i - stages - tmem_bufs, which it does
  // after its last look at that block's scales.
  static constexpr int ring = stages + tmem_bufs;
  static constexpr int off_out = stages * stage_bytes;
  static constexpr int off_ring = off_out + out_bytes;
  static constexpr int smem_bytes = off_ring + ring * slot_floats * 4;
  static constexpr int n_bars = 2 * stages + 2 * tmem_bufs + 3;
  static_assert(n_bars <= 24, "control block too small");
  static_assert(stages >= 3 && stages >= tmem_bufs && smem_bytes + static_reserve <= kSmemLimit, "shared-memory plan");
};

struct RingProblem {
  CUtensorMap a, b, d;
  GemmParams p;
};

// The items of a problem that one unit (a CTA or a pair) works on: from `first` on in steps of `early_step` below early_end and of `step`
// from there on, while they are below n.
struct Walk {
  int first, early_step, early_end, step, n;
  __device__ __forceinline__ int next(int item) const { return item + (item < early_end ? early_step : step); }
};
__device__ __forceinline__ Walk walk_alone(int unit, int units, int n) { return Walk{unit, 0, 0, units, n}; }
// Two problems on the same units: the first one's items go round, and the units that its last round leaves idle take `rounds` rounds of the
// second one's meanwhile, before all take it up, the idle ones first.
__device__ __forceinline__ Walk walk_second(int unit, int units, int n1, int n2, int rounds) {
  const int busy = n1 % units, idle = units - busy, early_end = rounds * idle;
  if (busy == 0) return walk_alone(unit, units, n2);
  return Walk{unit >= busy ? unit - busy : early_end + idle + unit, idle, early_end, units, n2};
}

// C and D: the plans of the two problems (TWO) or C twice.
template <int CG, typename C, typename D, bool TWO, typename START>
__device__ __forceinline__ void ring_body(const RingProblem& one, const RingProblem& two, int rounds, START&& start) {
  constexpr int BN = C::BN, kStages = C::stages, kRing = C::ring, kBufs = C::tmem_bufs;
  static_assert(C::BN == D::BN && C::stages == D::stages && C::out_bytes == D::out_bytes && C::stage_bytes == D::stage_bytes, "one layout for both");
  constexpr int kSlot = C::slot_floats > D::slot_floats ? C::slot_floats : D::slot_floats;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(16) uint64_t ctl_bars[24];
  __shared__ uint32_t ctl_tmem_ptr;
  __shared__ int ctl_abort;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t full0 = smem_u32(ctl_bars), empty0 = full0 + 8u * kStages;
  const uint32_t tfull0 = empty0 + 8u * kStages, tempty0 = tfull0 + 8u * kBufs;
  const uint32_t drain_bar = tempty0 + 8u * kBufs, staged_bar = drain_bar + 8u, unstaged_bar = drain_bar + 16u;
  volatile uint32_t* tmem_ptr_smem = &ctl_tmem_ptr;
  volatile int* abort_flag = &ctl_abort;

  unsigned* const status = one.p.status;
  if ((sbase & 1023u) != 0) {   // the swizzled operand layout needs this alignment (both CTAs have the same layout)
    if (threadIdx.x == 0 && status != nullptr) atomicCAS(status, 0u, 6u);
    return;
  }

  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t rank = CG == 2 ? cluster_rank() : 0u;
  const int unit = int(blockIdx.x) / CG, units = int(gridDim.x) / CG;
  auto items_of = [](const GemmParams& p) { return p.tiles_m * p.tiles_n * p.ksplit; };
  const Walk walk1 = walk_alone(unit, units, items_of(one.p));
  const Walk walk2 = TWO ? walk_second(unit, units, items_of(one.p), items_of(two.p), rounds) : walk1;
  // is there an item after this one?
  auto followed = [&](const Walk& w, int item, bool first) { return w.next(item) < w.n || (TWO && first && walk2.first < walk2.n); };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full0 + 8u * s, 1);            // (the first CTA's counts the bytes of both)
      mbar_init(empty0 + 8u * s, 1);
    }
    for (int b = 0; b < kBufs; ++b) {
      mbar_init(tfull0 + 8u * b, 2);           // the block's MMAs and its scales
      mbar_init(tempty0 + 8u * b, CG * C::promo_warps);
    }
    mbar_init(drain_bar, 1);
    mbar_init(staged_bar, C::promo_warps);
    mbar_init(unstaged_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&one.a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&one.b)) : "memory");
  }
  if (warp == C::issuer_warp) {
    if constexpr (CG == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl_tmem_ptr)), "r"(uint32_t(kTmemCols)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      tmem_alloc(smem_u32(&ctl_tmem_ptr), kTmemCols);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  if constexpr (CG == 2) cluster_sync();              // both CTAs' barriers exist before either signals across
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  start();

  if (warp >= C::promo_warps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::service_regs));
    if (warp == C::producer_warp) {
      // ------------------------------ TMA producer -------------------------------------
      uint32_t s = 0, ph = 1;
      bool ok = true;
      const uint32_t full_leader = CG == 2 ? map_rank(full0, 0u) : full0;
      auto produce = [&](const RingProblem& q, const Walk& w) {
       const GemmParams& p = q.p;
       for (int item = w.first; ok && item < w.n; item = w.next(item)) {
        int ks, tile, tm, tn;
        item_split(p, item, p.tiles_m * p.tiles_n, ks, tile);
        tile_coords(p, tile, tm, tn);
        const int m0 = (tm * CG + int(rank)) * BM, n0 = tn * BN + int(rank) * 128;     // (past M or N: zeros)
        int k0 = range_first(p, ks) * BK;
        const int nkb = range_blocks(p, ks);
        for (int kb = 0; kb < nkb; ++kb, k0 += BK) {
          ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8u * s, ph, abort_flag, status, 1u));
          if (!ok) break;
          if (elect_one()) {
            const uint32_t dst = sbase + s * C::stage_bytes, fb = full_leader + 8u * s;
            // The first CTA announces the bytes of both.  The second's may land before that: its barrier phase is the same one,
            // since the stage was free in both CTAs only after the phase before had completed.
            if (rank == 0) mbar_expect_tx(full0 + 8u * s, CG * C::stage_bytes);
            tma_load<CG>(dst, &q.a, fb, p.a_mn ? m0 : k0, p.a_mn ? k0 : m0);
#pragma unroll
            for (int b = 0; b < C::b_boxes; ++b) {
              const int nb = n0 + b * 128;
              tma_load<CG>(dst + (1 + b) * kTileBytes, &q.b, fb, p.b_mn ? nb : k0, p.b_mn ? k0 : nb);
            }
          }
          __syncwarp();
          if (++s == kStages) { s = 0; ph ^= 1u; }
        }
       }
      };
      produce(one, walk1);
      if constexpr (TWO) produce(two, walk2);
    } else if (warp == C::issuer_warp) {
      // ------------------------------ MMA issuer (first CTA) ----------------------------
      if (rank == 0) {
        const uint64_t desc_a0 = make_smem_desc(sbase), desc_b0 = make_smem_desc(sbase + kTileBytes);
        const uint32_t desc_hi = uint32_t(desc_a0 >> 32);
        const uint32_t a_lo0 = uint32_t(desc_a0), b_lo0 = uint32_t(desc_b0);
        bool ok = true;
        const bool stage_lane = lane >= 16;      // one wait instruction per block: half the lanes poll either barrier
        uint32_t s = 0, sph = 0, buf = 0, bph = 1, soff = 0;
        auto issue = [&](const RingProblem& q, const Walk& w) {
          const GemmParams& p = q.p;
          // D f32 (bit 4), A/B e4m3 (0), major bits 15/16, N>>3 at 17, M>>4 at 24
          const uint32_t idesc = (1u << 4) | (uint32_t(p.a_mn) << 15) | (uint32_t(p.b_mn) << 16) | (uint32_t(BN >> 3) << 17) |
                                 (uint32_t(CG * BM >> 4) << 24);
          const uint32_t a_step = p.a_mn ? (UMMA_K * 128) >> 4 : UMMA_K >> 4;
          const uint32_t b_step = p.b_mn ? (UMMA_K * 128) >> 4 : UMMA_K >> 4;
          uint32_t total = 0;
          for (int item = w.first; item < w.n; item = w.next(item)) {
            int ks, tile;
            item_split(p, item, p.tiles_m * p.tiles_n, ks, tile);
            total += uint32_t(range_blocks(p, ks));
          }
          for (uint32_t it = 0; ok && it < total; ++it) {
            const uint32_t bar = stage_lane ? full0 + 8u * s : tempty0 + 8u * buf;
            const uint32_t par = stage_lane ? sph : bph;
            ok = __all_sync(0xffffffffu, mbar_wait(bar, par, abort_flag, status, stage_lane ? 3u : 2u));
            if (!ok) break;
            __syncwarp();                  // (the vote is no memory barrier, and the elected lane has seen one of the two only)
            tc_fence_after();
            if (elect_one()) {
              const uint32_t d_tmem = tmem_base + buf * uint32_t(C::tmem_stride);
#pragma unroll
              for (int k = 0; k < BK / UMMA_K; ++k)
                umma<CG>(d_tmem, (uint64_t(desc_hi) << 32) | (a_lo0 + soff + k * a_step),
                         (uint64_t(desc_hi) << 32) | (b_lo0 + soff + k * b_step), idesc, k > 0 ? 1u : 0u);
              if constexpr (CG == 1) commit<CG>(empty0 + 8u * s);
              commit<CG>(tfull0 + 8u * buf);
              if constexpr (CG == 2) commit<CG>(empty0 + 8u * s);
            }
            __syncwarp();
            soff += uint32_t(C::stage_bytes >> 4);
            if (++s == kStages) { s = 0; sph ^= 1u; soff = 0; }
            if (++buf == kBufs) { buf = 0; bph ^= 1u; }
          }
        };
        issue(one, walk1);
        if constexpr (TWO) issue(two, walk2);
        // nothing issued here may still be running when tensor memory is freed
        if (elect_one()) {
          if constexpr (CG == 2) umma_commit_here(drain_bar);
          else umma_commit(drain_bar);
          mbar_wait(drain_bar, 0u, abort_flag, status, 4u);
        }
        __syncwarp();
      }
    } else if (warp == C::scale_warp) {
      // ------------------------------ scales --------------------------------------------
      // Copies run as many blocks ahead of the announcement as there are accumulators: block j's scales are announced on its
      // accumulator's barrier, beside its MMAs, once that barrier is through with the block before.  The MMAs of block i wait for the
      // announcement of block i - tmem_bufs, which comes after the copy of block i: so while that copy waits for its stage, the stage's
      // barrier cannot go on to the phase after.  (The first blocks' MMAs wait for no announcement: their copies must not look at the
      // barrier, and need not.)
      uint32_t s = 0, ph = 1, slot = 0, buf = 0, bph = 1, copied = 0;
      bool ok = true;
      const uint32_t is_lane0 = lane == 0;
      auto announce = [&]() {
        ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8u * buf, bph, abort_flag, status, 9u));
        __syncwarp();                // every lane's copies, before lane 0 announces them (a vote is no memory barrier)
        mbar_arrive_if(tfull0 + 8u * buf, is_lane0);
        if (++buf == kBufs) { buf = 0; bph ^= 1u; }
      };
      auto copy = [&](const RingProblem& q, const Walk& w, auto cfg) {
       constexpr int SB_GRAN = decltype(cfg)::sb_gran;
       const GemmParams& p = q.p;
       for (int item = w.first; ok && item < w.n; item = w.next(item)) {
        int ks, tile, tm, tn;
        item_split(p, item, p.tiles_m * p.tiles_n, ks, tile);
        tile_coords(p, tile, tm, tn);
        const int m0 = (tm * CG + int(rank)) * BM, n0 = tn * BN;
        const uint32_t kb0 = uint32_t(range_first(p, ks));
        // element offsets (the host checks that they fit 32 bits); rows and columns past the end read a valid scale
        uint32_t sa_off[4], sb_off[SB_GRAN == 1 ? BN / 32 : 1];
#pragma unroll
        for (int i = 0; i < 4; ++i) sa_off[i] = uint32_t(min(m0 + lane + 32 * i, p.M - 1)) * uint32_t(p.sa_sm) + kb0 * uint32_t(p.sa_sk);
        if (SB_GRAN == 1) {
#pragma unroll
          for (int i = 0; i < BN / 32; ++i) sb_off[i] = uint32_t(min(n0 + lane + 32 * i, p.N - 1)) * uint32_t(p.sb_sn) + kb0 * uint32_t(p.sb_sk);
        } else {
          sb_off[0] = uint32_t(min(n0 / 128 + (lane & 1), (p.N - 1) / 128)) * uint32_t(p.sb_sn) + kb0 * uint32_t(p.sb_sk);
        }
        const int nkb = range_blocks(p, ks);
        for (int kb = 0; kb < nkb; ++kb) {
          if (copied >= uint32_t(kStages)) {
            ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8u * s, ph, abort_flag, status, 9u));
            if (!ok) break;
          }
          const uint32_t dst = sbase + C::off_ring + slot * uint32_t(kSlot * 4) + 4u * lane;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            cp_async_4(dst + 128u * i, p.sa + sa_off[i]);
            sa_off[i] += uint32_t(p.sa_sk);
          }
          if (SB_GRAN == 1) {
#pragma unroll
            for (int i = 0; i < BN / 32; ++i) {
              cp_async_4(dst + 512u + 128u * i, p.sb + sb_off[i]);
              sb_off[i] += uint32_t(p.sb_sk);
            }
          } else {
            if (lane < BN / 128) cp_async_4(dst + 512u, p.sb + sb_off[0]);
            sb_off[0] += uint32_t(p.sb_sk);
          }
          asm volatile("cp.async.commit_group;" ::: "memory");
          if (++s == kStages) { s = 0; ph ^= 1u; }
          if (++slot == kRing) slot = 0;
          if (++copied > kBufs) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kBufs) : "memory");
            announce();
            if (!ok) break;
          }
        }
      }
      };
      copy(one, walk1, C());
      if constexpr (TWO) copy(two, walk2, D());
      asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll 1
      for (uint32_t left = min(copied, uint32_t(kBufs)); ok && left > 0; --left) announce();
    } else {
      // ------------------------------ tile stores ----------------------------------------
      uint32_t sph = 0;
      bool ok = true;
      auto store = [&](const RingProblem& q, const Walk& w, bool first, auto cfg) {
        using Q = decltype(cfg);
        const GemmParams& p = q.p;
        for (int item = w.first; ok && item < w.n && followed(w, item, first); item = w.next(item)) {       // (all but the last)
          int ks, tile, tm, tn;
          item_split(p, item, p.tiles_m * p.tiles_n, ks, tile);
          tile_coords(p, tile, tm, tn);
#pragma unroll 1
          for (int phase = 0; phase < Q::phases; ++phase) {
            ok = __all_sync(0xffffffffu, mbar_wait(staged_bar, sph, abort_flag, status, 7u));
            if (!ok) break;
            sph ^= 1u;
            if (elect_one()) {
#pragma unroll 1
              for (int pw = 0; pw < Q::promo_warps; ++pw) {
#pragma unroll
                for (int h = 0; h < Q::warp_boxes; ++h)
                  tma_store_3d_nocommit(&q.d, sbase + C::off_out + uint32_t(pw * Q::warp_boxes + h) * Q::box_bytes,
                                        tn * BN + (pw >> 2) * Q::cols + (phase * Q::warp_boxes + h) * Q::box_cols,
                                        (tm * CG + int(rank)) * BM + (pw & 3) * 32, ks);
              }
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
              tma_store_wait_read();
              mbar_arrive(unstaged_bar);
            }
            __syncwarp();
          }
        }
      };
      store(one, walk1, true, C());
      if constexpr (TWO) store(two, walk2, false, D());
    }
  } else {
    // ------------------------------ promotion + epilogue --------------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::promo_regs));
    const int quarter = warp & 3, cg = warp >> 2;
    const int r = quarter * 32 + lane;
    const int fg = lane >> 2, fj = lane & 3;     // fragment coordinates: rows fg + 8 i, column pairs 8 k + 2 fj
    const float* ring = reinterpret_cast<const float*>(smem + C::off_ring);
    const uint32_t tcol0 = tmem_base + (uint32_t(quarter * 32) << 16) + uint32_t(cg * C::cols);
    const int sb_index = cg * C::cols / 128;
    static_assert(C::warp_boxes * C::box_bytes == D::warp_boxes * D::box_bytes, "one layout for both");
    const uint32_t wb = sbase + C::off_out + uint32_t(warp) * (C::warp_boxes * C::box_bytes);
    const uint32_t tempty_leader = CG == 2 ? map_rank(tempty0, 0u) : tempty0;
    const uint32_t is_lane0 = lane == 0;
    uint32_t buf = 0, bph = 0, uph = 1, slot = 0;
    // A wait that gives up has raised the abort flag, and every wait after it returns at once: the warps look at `ok` once a tile.
    bool ok = true;
    auto release = [&](uint32_t b) {
      tc_fence_before();
      __syncwarp();
      if constexpr (CG == 2) mbar_arrive_cluster_if(tempty_leader + 8u * b, is_lane0);
      else mbar_arrive_if(tempty_leader + 8u * b, is_lane0);
    };
    auto promote_items = [&](const RingProblem& prob, const Walk& w, bool first, auto cfg) {
     using Q = decltype(cfg);
     constexpr bool kFrag = Q::frag, OUT_F32 = Q::out_f32;
     const GemmParams& p = prob.p;
     const int n_tiles = p.tiles_m * p.tiles_n;
     for (int item = w.first; item < w.n; item = w.next(item)) {
      float2 acc[C::cols / 2];
#pragma unroll
      for (int j = 0; j < C::cols / 2; ++j) acc[j] = make_float2(0.f, 0.f);
      int nkb;
      {
        int ks, tile;
        item_split(p, item, n_tiles, ks, tile);
        nkb = range_blocks(p, ks);
      }
      // Rows in bf16: the last block stages each piece as soon as it is complete, beside the promotion of the next (forward and data
      // gradient 2 % faster at 8 and 16 blocks a tile; in fragments, whose stores are four bytes each, 0.5 % slower)
      constexpr bool kStageInBlock = Q::phases == 1 && !OUT_F32 && !kFrag;
      const int plain = kStageInBlock ? nkb - 1 : nkb;
      const bool last = !followed(w, item, first);
      auto rows_free = [&]() {      // the staging rows have been read (the first pass finds them free)
        ok &= mbar_wait(unstaged_bar, uph, abort_flag, status, 8u);
        __syncwarp();
        uph ^= 1u;
      };
      // Piece q (of the phase, which begins with piece q0 of the accumulator).  Fragments: rows fg + 8 i; bf16: 16-byte chunk 2 q + k of the
      // box's row, 4 fj bytes in; float32: chunk 4 q + 2 k + (fj >> 1), half fj & 1.  Rows: chunks 2 q, 2 q + 1 (float32: 4 q ...).
      // Swizzle: chunk xor the row's low three bits, with 64-byte rows xor the two above the lowest.
      const uint32_t st_base = wb + (kFrag ? uint32_t(fg) * Q::box_row + (OUT_F32 ? (uint32_t(fj >> 1) << 4) + 8u * uint32_t(fj & 1) : 4u * uint32_t(fj))
                                           : uint32_t(lane) * 128u);
      const uint32_t st_flip = (!kFrag ? uint32_t(lane & 7) : Q::box_row == 128 ? uint32_t(fg) : uint32_t(fg >> 1)) << 4;
      auto stage = [&](auto qc, auto q0c) {
        constexpr int qq = decltype(qc)::value, q0 = decltype(q0c)::value, q = qq % Q::box_pieces, box = (qq / Q::box_pieces) * Q::box_bytes;
        if constexpr (kFrag) {
          static_loop<4>([&](auto i) {
            static_loop<2>([&](auto k) {
              const float2 a = acc[(4 * (q0 + qq) + i.value) * 2 + k.value];
              if constexpr (OUT_F32) sts_swz_f32x2<box + i.value * 8 * Q::box_row + (4 * q + 2 * k.value) * 16>(st_base, st_flip, a);
              else sts_swz_b32<box + i.value * 8 * Q::box_row + (2 * q + k.value) * 16>(st_base, st_flip, pack_bf16x2(a.x, a.y));
            });
          });
        } else if constexpr (OUT_F32) {
          static_loop<4>([&](auto c) {
            const int j = 8 * (q0 + qq) + 2 * c.value;
            sts_swz_f32x4<box + (4 * q + c.value) * 16>(st_base, st_flip, acc[j], acc[j + 1]);
          });
        } else {
          static_loop<2>([&](auto c) {
            const int j = 8 * (q0 + qq) + 4 * c.value;
            sts_swz_v4<box + (2 * q + c.value) * 16>(st_base, st_flip, pack_bf16x2(acc[j].x, acc[j].y), pack_bf16x2(acc[j + 1].x, acc[j + 1].y),
                                                     pack_bf16x2(acc[j + 2].x, acc[j + 2].y), pack_bf16x2(acc[j + 3].x, acc[j + 3].y));
          });
        }
      };
      auto enter_block = [&]() {
        ok &= mbar_wait(tfull0 + 8u * buf, bph, abort_flag, status, 5u);
        __syncwarp();
        tc_fence_after();
        const float* sc = ring + slot * kSlot;
        if (++slot == kRing) slot = 0;
        return sc;
      };
      auto leave_block = [&]() {
        release(buf);
        if (++buf == kBufs) { buf = 0; bph ^= 1u; }
      };
      if constexpr (kFrag) {
        // acc[(4 q + i) * 2 + k] holds rows fg + 8 i, columns 16 q + 8 k + 2 fj (+1)
        auto block = [&](auto staging) {
          const float* sc = enter_block();
          const uint32_t taddr = tcol0 + buf * uint32_t(C::tmem_stride);
          float sa_r[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) sa_r[i] = sc[quarter * 32 + fg + 8 * i];
          const float* scol = sc + 128 + cg * C::cols + 2 * fj;
          static_loop<C::pieces>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            uint32_t v[16];
            float2 sb2[2];
            sb2[0] = *reinterpret_cast<const float2*>(scol + 16 * q);
            sb2[1] = *reinterpret_cast<const float2*>(scol + 16 * q + 8);
            tmem_ld_frag16(taddr + 16 * q, v);
            tmem_ld_frag16(taddr + (16u << 16) + 16 * q, v + 8);
            tmem_wait_ld16(v);
            if (q == C::pieces - 1) leave_block();         // (after the last look at the scales, see RingCfg::ring)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int o = 8 * (i >> 1) + 4 * k + 2 * (i & 1);
                const float2 pv = make_float2(__uint_as_float(v[o]), __uint_as_float(v[o + 1]));
                float2& a = acc[(4 * q + i) * 2 + k];
                a = __ffma2_rn(__fmul2_rn(pv, sb2[k]), make_float2(sa_r[i], sa_r[i]), a);
              }
            }
            if constexpr (decltype(staging)::value != 0) stage(qc, IntC<0>{});
          });
        };
#pragma unroll 1
        for (int kb = 0; kb < plain; ++kb) block(IntC<0>{});
        if constexpr (kStageInBlock) {
          rows_free();
          block(IntC<1>{});
        }
      } else {
        // two register buffers: the next piece is on its way while one is promoted, across blocks too
        uint32_t v[2][16];
        const float* sc = enter_block();
        float s = sc[r] * sc[128 + sb_index];
        uint32_t taddr = tcol0 + buf * uint32_t(C::tmem_stride);
        tmem_ld16(taddr, v[0]);
#pragma unroll 1
        for (int kb = 0; kb < plain; ++kb) {
          const bool more = kb + 1 < nkb;
#pragma unroll
          for (int q = 0; q < C::pieces - 1; ++q) {
            tmem_wait_ld16(v[q & 1]);
            tmem_ld16(taddr + 16 * (q + 1), v[(q + 1) & 1]);
            promote<128, 16>(acc + 8 * q, v[q & 1], nullptr, 0.f, s);
          }
          tmem_wait_ld16(v[1]);
          leave_block();
          float s_next = 0.f;
          if (more) {
            sc = enter_block();
            taddr = tcol0 + buf * uint32_t(C::tmem_stride);
            tmem_ld16(taddr, v[0]);
            s_next = sc[r] * sc[128 + sb_index];
          }
          promote<128, 16>(acc + 8 * (C::pieces - 1), v[1], nullptr, 0.f, s);
          s = s_next;
        }
        if constexpr (kStageInBlock) {
          rows_free();
          static_loop<C::pieces>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            tmem_wait_ld16(v[q & 1]);
            if constexpr (q + 1 < C::pieces) tmem_ld16(taddr + 16 * (q + 1), v[(q + 1) & 1]);
            else leave_block();
            promote<128, 16>(acc + 8 * q, v[q & 1], nullptr, 0.f, s);
            stage(qc, IntC<0>{});
          });
        }
      }
      if (!__all_sync(0xffffffffu, ok)) break;

      // ---- epilogue: registers -> this warp's swizzled staging rows -> bulk stores ----
      // The store warp hands a tile's boxes to the copy engine one after the other (40 cycles each), beside the next tile's first
      // blocks.  After the last tile nothing hides that: every warp issues its own.
      static_loop<Q::phases>([&](auto pc) {
        constexpr int phase = decltype(pc)::value;
        if constexpr (!kStageInBlock) {
          if (!last || phase == 0) {
            rows_free();
          } else {
            if (is_lane0) tma_store_wait_read();
            __syncwarp();
          }
          static_loop<Q::warp_boxes * Q::box_pieces>([&](auto qc) { stage(qc, IntC<phase * Q::warp_boxes * Q::box_pieces>{}); });
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> visible to the copy engine
        __syncwarp();
        if (!last) {
          mbar_arrive_if(staged_bar, is_lane0);
        } else if (is_lane0) {
          int ks, tile, tm, tn;
          item_split(p, item, n_tiles, ks, tile);
          tile_coords(p, tile, tm, tn);
#pragma unroll
          for (int h = 0; h < Q::warp_boxes; ++h)
            tma_store_3d_nocommit(&prob.d, wb + uint32_t(h) * Q::box_bytes, tn * BN + cg * C::cols + (phase * Q::warp_boxes + h) * Q::box_cols,
                                  (tm * CG + int(rank)) * BM + quarter * 32, ks);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        __syncwarp();
      });
      if (!__all_sync(0xffffffffu, ok)) break;
     }
    };
    promote_items(one, walk1, true, C());
    if constexpr (TWO) {
      if (__all_sync(0xffffffffu, ok)) promote_items(two, walk2, false, D());
    }
  }

  // ------------------------------ teardown ----------------------------------------------
  // the last bulk stores must have read their staging rows before the CTA's shared memory goes away
  if (warp < C::promo_warps && lane == 0) tma_store_wait_read();
  __syncwarp();
  tc_fence_before();
  if constexpr (CG == 2) cluster_sync();              // the partner no longer reads this CTA's shared memory or signals its barriers
  else __syncthreads();
  if (warp == C::issuer_warp) {
    __syncwarp();
    tc_fence_after();
    if constexpr (CG == 2)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(uint32_t(kTmemCols)) : "memory");
    else
      tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int CG, int BN, int SB_GRAN, bool OUT_F32>
__global__ void __launch_bounds__((RingCfg<CG, BN, SB_GRAN, OUT_F32>::threads), 1) gemm_ring_kernel(const __grid_constant__ RingProblem one) {
  using C = RingCfg<CG, BN, SB_GRAN, OUT_F32>;
  ring_body<CG, C, C, false>(one, one, 0, [] {
    grid_trigger();
    grid_wait();
  });
}

// A linear's weight gradient and then its data gradient on the same pairs, barriers and buffers running on from one to the other.  What
// bounds the two apart is their last rounds: 5000 x 1024 -> 4096 has 64 tiles of 40 blocks and 80 of 32 for 74 pairs.  The long items go
// first, and pairs that their last round leaves idle begin with the short ones.  With the quantisers, in a loop: 82 -> 67.5 us; 24576 x
// 1024 -> 1024 101 -> 85 us, -> 3072 226 -> 208, 8192 x 2048 -> 2048 101 -> 97.
template <bool OUT_F32>
__global__ void __launch_bounds__((RingCfg<2, 256, 1, OUT_F32>::threads), 1)
gemm_ring_two_kernel(const __grid_constant__ RingProblem one, const __grid_constant__ RingProblem two, int rounds) {
  ring_body<2, RingCfg<2, 256, 1, OUT_F32>, RingCfg<2, 256, 128, false>, true>(one, two, rounds, [] {
    grid_trigger();
    grid_wait();
  });
}

// ---- host ------------------------------------------------------------------------------

template <int CG, typename C>
static int prepare_ring(const tg_gemm_args* a, const GemmParams& p0, RingProblem& q) {
  GemmParams& p = q.p;
  p = p0;
  const int64_t a_inner = p.a_mn ? a->M : a->K, a_outer = p.a_mn ? a->K : a->M;
  const int64_t b_inner = p.b_mn ? a->N : a->K, b_outer = p.b_mn ? a->K : a->N;
  if (int rc = make_tmap(&q.a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->a, a_inner, a_outer, a->lda, 128, 128)) return rc;
  if (int rc = make_tmap(&q.b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->b, b_inner, b_outer, a->ldb, 128, 128)) return rc;
  if (int rc = make_output_map(&q.d, C::out_f32, a, p, C::box_cols, C::box_row)) return rc;
  p.tiles_m = int((a->M + CG * BM - 1) / (CG * BM));
  p.tiles_n = int((a->N + C::BN - 1) / C::BN);
  p.band = std::min(p.tiles_m, kBandRows / CG);
  return set_reciprocals(p);
}

// The launch of one of the kernels above; `units_of`, per device: how many units run at a time (a pair takes two SMs of one cluster group).
struct RingLaunch {
  cudaLaunchAttribute attrs[2];
  cudaLaunchConfig_t cfg = {};
  template <typename K>
  int prepare(K kern, int cg, int threads, int smem, std::atomic<int>* units_of, int& units, cudaStream_t st) {
    int dev = 0;
    TG_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return TG_ERR_SHAPE;
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = cg;
    attrs[0].val.clusterDim.y = attrs[0].val.clusterDim.z = 1;
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attrs;
    cfg.numAttrs = 1;
    cfg.stream = st;
    int fit = units_of[dev].load(std::memory_order_acquire);      // with the kernel's shared memory: set once per device
    if (fit == 0) {
      TG_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      fit = sm_count();
      if (cg == 2) {
        cfg.gridDim = dim3(unsigned(sm_count() & ~1));
        TG_CUDA_CHECK(cudaOccupancyMaxActiveClusters(&fit, kern, &cfg));
      }
      if (fit < 1) return record_cuda_error(cudaErrorLaunchOutOfResources, "no CTA pair fits on this device");
      units_of[dev].store(fit, std::memory_order_release);
    }
    units = std::max(1, std::min(fit, cg == 2 ? gemm_pairs() : gemm_sms()));
    return TG_OK;
  }
};

template <int CG, int BN, int SB_GRAN, bool OUT_F32>
static int launch_ring(const tg_gemm_args* a, const GemmParams& p, cudaStream_t st) {
  using C = RingCfg<CG, BN, SB_GRAN, OUT_F32>;
  static std::atomic<int> units_of[64];
  auto kern = gemm_ring_kernel<CG, BN, SB_GRAN, OUT_F32>;
  RingProblem q;
  RingLaunch l;
  int units = 0;
  if (int rc = prepare_ring<CG, C>(a, p, q)) return rc;
  if (int rc = l.prepare(kern, CG, C::threads, C::smem_bytes, units_of, units, st)) return rc;
  const int n_items = q.p.tiles_m * q.p.tiles_n * q.p.ksplit;
  l.cfg.gridDim = dim3(unsigned(CG * std::min(n_items, units)));
  if ((p.a_mn == 0 && a->M <= 256) || (n_items <= 4 * units && p.nkb <= 32)) l.cfg.numAttrs = 2;
  TG_CUDA_CHECK(cudaLaunchKernelEx(&l.cfg, kern, q));
  return TG_OK;
}

int ring_run(const tg_gemm_args* a, const GemmParams& p, bool pair, int bn, bool f32, cudaStream_t st) {
  if (pair && a->sb_gran_n == 1) return f32 ? launch_ring<2, 256, 1, true>(a, p, st) : launch_ring<2, 256, 1, false>(a, p, st);
  if (pair) return f32 ? launch_ring<2, 256, 128, true>(a, p, st) : launch_ring<2, 256, 128, false>(a, p, st);
  if (bn == 192) return launch_ring<1, 192, 1, false>(a, p, st);
  return f32 ? launch_ring<1, 128, 1, true>(a, p, st) : launch_ring<1, 128, 1, false>(a, p, st);
}

template <bool OUT_F32>
static int launch_ring_two(const tg_gemm_args* a, const GemmParams& pa, const tg_gemm_args* b, const GemmParams& pb, cudaStream_t st) {
  using C = RingCfg<2, 256, 1, OUT_F32>;
  using D = RingCfg<2, 256, 128, false>;
  static std::atomic<int> units_of[64];
  auto kern = gemm_ring_two_kernel<OUT_F32>;
  RingProblem one, two;
  RingLaunch l;
  int units = 0;
  if (int rc = prepare_ring<2, C>(a, pa, one)) return rc;
  if (int rc = prepare_ring<2, D>(b, pb, two)) return rc;
  if (int rc = l.prepare(kern, 2, C::threads, std::max(C::smem_bytes, D::smem_bytes), units_of, units, st)) return rc;
  const int n1 = one.p.tiles_m * one.p.tiles_n * one.p.ksplit, n2 = two.p.tiles_m * two.p.tiles_n;
  units = std::min(units, n1 + n2);
  l.cfg.gridDim = dim3(unsigned(2 * units));
  int rounds = 0;
  two_problems_us(n1, pair_item_us(true, pa.nkb + (pa.nkb_rem > 0)), n2, pair_item_us(false, pb.nkb), units, rounds);
  TG_CUDA_CHECK(cudaLaunchKernelEx(&l.cfg, kern, one, two, rounds));
  return TG_OK;
}

int ring_pair_two(const tg_gemm_args* a, const GemmParams& pa, bool f32, const tg_gemm_args* b, const GemmParams& pb, cudaStream_t st) {
  return f32 ? launch_ring_two<true>(a, pa, b, pb, st) : launch_ring_two<false>(a, pa, b, pb, st);
}

}  // namespace tg
