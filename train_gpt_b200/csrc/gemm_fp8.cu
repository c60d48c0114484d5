// Block-scaled e4m3 GEMM for sm_100a:  D[m,n] = sum_kb SA(m,kb) SB(n,kb) sum_{k in kb} A[m,k] B[n,k]
//
// Replaces jax.nn.scaled_matmul as train-gpt calls it (fp8.py:70-76) plus the bf16 cast of
// fp8.py:78, and -- with other operand orientations -- the backward GEMMs of fp8.py:96-97.
//
// The scales are float32 (amax/448), not powers of two, so the tensor core's own
// block-scale path (UE8M0 factors) cannot apply them bit-faithfully.  Instead every
// 128-deep contraction block is issued as its own tcgen05.mma chain into a fresh TMEM
// accumulator buffer, and sixteen "promotion" warps pull each finished buffer out of TMEM
// (tcgen05.ld), hand it back to the tensor core, multiply by SA*SB and add into float32
// register accumulators with packed f32x2 FMAs while the tensor core fills the next buffer.
//
// Tile: 128 rows x BN columns, BN = 256 (two 256-column TMEM buffers) or 128 (four).  The
// wide tile halves the shared-memory and L2 traffic per FLOP and doubles the tensor-core
// time per issued instruction, which is what keeps the single-thread issue loop and the
// barrier round trips off the critical path.
//
// Warp roles in the CTA (persistent, one CTA per SM; work items numbered in bands, see tile_coords):
//   warps 0..P-1 promotion + epilogue (P = 16, or 12 for 192-column tiles); warp w may touch TMEM
//                lanes 32*(w%4).. (a hardware rule) and owns accumulator columns (BN/4)*(w/4)..;
//                four warps per scheduler hide each other's TMEM-load latency.  Tiles leave through
//                bulk tensor stores (registers -> the warp's swizzled staging rows ->
//                cp.async.bulk.tensor, one box per 128 bytes of row), waited for only when the rows
//                are reused a tile later.
//   warp P       TMA producer: A (one 128 x 128-byte box) and B (BN/128 boxes), 128B swizzle
//   warp P+1     MMA issuer (owns the TMEM allocation): one lane-split barrier wait per block
//   warps P+2,3  (256-column tiles only) idle padding of the producer's warpgroup, so that it can
//                release registers to the promotion warpgroups with setmaxnreg: 96 -> 40 / 104.
//
// The loops of all three roles carry their state (stage, buffer, phase, scale offsets) instead of
// deriving it from a block counter, and the barriers live in static shared memory, so that a block
// costs the promotion warps little more than its 32 packed FMAs and 4 TMEM loads: the first builds
// spent four fifths of their instructions on address arithmetic and were bound by issue.
//
// Operand orientation is data, not code: the TMA box is 128 bytes x 128 rows for both
// K-major and MN-major storage (only the coordinates swap), and the shared-memory operand
// descriptors / instruction descriptor carry the major-ness, so dgrad and wgrad read the
// same buffers the forward wrote, untransposed.  Few output tiles with a long contraction are
// cut along the contraction (plan_gemm); few rows against a wide weight take the kernel of
// gemm_skinny.cu.
//
// Every wait on an mbarrier is bounded: when the limit runs out the waiting role raises a
// CTA-wide abort flag, stores a code in *status, and all roles fall through to the common
// teardown (TMEM is always freed).
#include <cuda.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "gemm_tiles.cuh"
#include "host_api.h"
#include "mbarrier.cuh"
#include "umma.cuh"

#ifndef TG_X_BAND
#define TG_X_BAND 16
#endif
#ifndef TG_X_PROMO_REGS
#define TG_X_PROMO_REGS 104
#endif
#ifndef TG_X_SERVICE_REGS
#define TG_X_SERVICE_REGS 40
#endif

namespace tg {

constexpr int kBandRows = TG_X_BAND;             // tile rows per band of the tile numbering (see tile_coords)

// Compile-time plan of one kernel variant.
template <int BN_, int SB_GRAN, bool OUT_F32>
struct Cfg {
  static constexpr int BN = BN_;
  // 192-column tiles run 12 promotion warps (14 warps in all: 128 registers per thread instead
  // of the 96 an 18-warp CTA gets), the others 16
  static constexpr int promo_warps = BN == 192 ? 12 : 16;
  // Warp layout: promotion warps 0..P-1 (whole warpgroups), then the TMA producer, then the MMA
  // issuer.  The 256-column tile pads that last warpgroup with two idle warps so that it can hand
  // registers over with setmaxnreg: 20 warps start at 96 registers per thread; the producer's
  // warpgroup drops to `service_regs` and each promotion warpgroup grows to `promo_regs`
  // (service_regs + 4 * promo_regs <= 5 * 96 per scheduler, so the growth never waits for
  // registers that nobody releases).
  static constexpr bool regsteal = BN == 256;
  static constexpr int producer_warp = promo_warps;
  static constexpr int issuer_warp = promo_warps + 1;
  static constexpr int warps = promo_warps + (regsteal ? 4 : 2);
  static constexpr int threads = 32 * warps;
  static constexpr int promo_regs = TG_X_PROMO_REGS, service_regs = TG_X_SERVICE_REGS;
  static_assert(service_regs + 4 * promo_regs <= 5 * 96, "register hand-over asks for more than is released");
  static constexpr int tmem_bufs = BN > 128 ? 2 : 4;
  static constexpr int tmem_stride = kTmemCols / tmem_bufs;   // columns between accumulator buffers
  static constexpr int cols_per_warp = BN / (promo_warps / 4);  // 64 or 32
  static constexpr int b_boxes = (BN + 127) / 128;
  static constexpr int stage_bytes = kTileBytes * (1 + b_boxes);
  static constexpr int esize = OUT_F32 ? 4 : 2;
  // epilogue: a warp stages its 32 rows x `phase_cols` columns at a time (rows of <= 128
  // bytes; a fourth pipeline stage bought with narrower staging rows measured no faster)
  static constexpr int row_bytes = cols_per_warp * esize;     // 64, 128 or 256
  static constexpr int phase_cap = 128;
  static constexpr int phase_row_bytes = row_bytes < phase_cap ? row_bytes : phase_cap;
  static constexpr int phases = row_bytes / phase_row_bytes;
  static constexpr int phase_cols = phase_row_bytes / esize;
  // tiles leave through bulk tensor stores: per promotion warp one 32-row box for bf16 (never waited
  // for inside the tile loop), two for float32 through the same staging rows
  static constexpr int warp_out_bytes = 32 * phase_row_bytes;
  static constexpr int out_bytes = promo_warps * warp_out_bytes;
  // per-column scales: float[warps][2][cols_per_warp column scales + 32 row scales], double-buffered
  static constexpr int sc_slot = cols_per_warp + 32;
  static constexpr int sb_bytes = SB_GRAN == 1 ? promo_warps * 2 * sc_slot * 4 : 0;
  // 64-column warps with per-column scales read TMEM in the MMA fragment layout (a thread holds 4 rows
  // x 16 columns instead of 1 x 64): a column scale is then shared by 8 lanes instead of all 32, and
  // the block's 64 of them cost 8 conflict-free 8-byte reads per thread instead of 16 broadcasts of 16
  // bytes, which a warp is served a quarter at a time (64 -> 16 shared-memory wavefronts per warp)
  static constexpr bool frag = SB_GRAN == 1 && cols_per_warp == 64;
  // the barriers, the TMEM pointer and the abort flag are static shared memory (fixed addresses: the
  // loops address them with immediates); the dynamic part starts at the next 1024-byte boundary
  static constexpr int static_reserve = 1024;
  static constexpr int stages_fit = (kSmemLimit - static_reserve - out_bytes - sb_bytes) / stage_bytes;
  static constexpr int stages = stages_fit > 6 ? 6 : stages_fit;
  // offsets from the 1024-aligned base of dynamic shared memory
  static constexpr int off_out = stages * stage_bytes;
  static constexpr int off_sb = off_out + out_bytes;
  // (handing the wide accumulator over in two 128-column halves, each with its own barriers
  // and N=128 MMAs, was tried: 7 % slower -- A is read twice and twice as many MMAs issue)
  // With one staging phase per tile and idle warps to spare, one of them issues the tile's bulk
  // stores: the copy engine accepts a promotion warp's 4 KB box only after the boxes before it (a
  // 64 KB tile takes it ~1000 cycles at the SM's write bandwidth), and the sixteen warps used to sit
  // in that queue instead of draining the next tile's accumulators.
  static constexpr bool store_warp_on = regsteal && phases == 1;
  static constexpr int store_warp = promo_warps + 2;
  static constexpr int n_bars = 2 * stages + 2 * tmem_bufs + 1 + 2;
  static constexpr int smem_bytes = off_sb + sb_bytes;       // dynamic shared memory
  static_assert(n_bars <= 24, "control block too small");
  static_assert(stages >= 3, "pipeline too shallow");
  static_assert(smem_bytes + static_reserve <= kSmemLimit, "shared-memory plan exceeds the 227 KB a CTA may use");
};

// ---- kernel ----------------------------------------------------------------------------

// Thread block `block` of `blocks` that share a problem.  `start` comes between what a kernel launched early may do and the rest.
template <int BN_, int SB_GRAN, bool OUT_F32, typename START>
__device__ __forceinline__ void gemm_body(const CUtensorMap& tmap_a, const CUtensorMap& tmap_b, const CUtensorMap& tmap_d, const GemmParams& p,
                                          int block, int blocks, START&& start) {
  using C = Cfg<BN_, SB_GRAN, OUT_F32>;
  constexpr int BN = C::BN, kStages = C::stages, kTmemBufs = C::tmem_bufs, kCols = C::cols_per_warp;
  constexpr int kPromoWarps = C::promo_warps;
  // operand stages (1024-byte aligned for the 128-byte swizzle), output staging, scale staging
  extern __shared__ __align__(1024) uint8_t smem[];
  // barriers, 8 bytes each: full[kStages], empty[kStages], tfull[kTmemBufs], tempty[kTmemBufs], drain, staged, unstaged
  __shared__ __align__(16) uint64_t ctl_bars[24];
  __shared__ uint32_t ctl_tmem_ptr;
  __shared__ int ctl_abort;
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = smem_u32(ctl_bars);
  const uint32_t full0 = bar0, empty0 = bar0 + 8u * kStages;
  const uint32_t tfull0 = bar0 + 16u * kStages, tempty0 = tfull0 + 8u * kTmemBufs;
  const uint32_t drain_bar = tempty0 + 8u * kTmemBufs;
  const uint32_t staged_bar = drain_bar + 8u, unstaged_bar = drain_bar + 16u;   // the store warp's pair (see Cfg::store_warp_on)
  volatile uint32_t* tmem_ptr_smem = &ctl_tmem_ptr;
  volatile int* abort_flag = &ctl_abort;
  if ((sbase & 1023u) != 0) {   // the swizzled operand layout needs this alignment; never seen, but not assumed
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0u, 6u);
    return;
  }

  // the warp index through a shuffle: the compiler then knows it is the same in every lane and keeps
  // what derives from it (role, TMEM address, barrier addresses) in uniform registers
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int n_tiles = p.tiles_m * p.tiles_n;
  const int n_items = n_tiles * p.ksplit;     // work item i = (tile i % n_tiles, contraction range i / n_tiles)
  const int first_item = block, item_step = blocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full0 + 8u * s, 1);
      mbar_init(empty0 + 8u * s, 1);
    }
    for (int b = 0; b < kTmemBufs; ++b) {
      mbar_init(tfull0 + 8u * b, 1);
      mbar_init(tempty0 + 8u * b, kPromoWarps);
    }
    mbar_init(drain_bar, 1);
    mbar_init(staged_bar, kPromoWarps);
    mbar_init(unstaged_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_a)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_b)) : "memory");
  }
  if (warp == C::issuer_warp) {
    tmem_alloc(smem_u32(&ctl_tmem_ptr), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  start();

  if (warp >= C::promo_warps) {
    if (C::regsteal) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::service_regs));
    if (warp == C::producer_warp) {
      // ------------------------------ TMA producer -------------------------------------
      // The whole warp walks the loop (uniform control flow); one elected lane issues.  Stage index
      // and phase are carried, not derived from a block counter (no modulo in the loop).
      uint32_t s = 0, ph = 1;                 // the first pass over the stages finds them all free
      bool ok = true;
      for (int item = first_item; ok && item < n_items; item += item_step) {
        int ks, tile, tm, tn;
        item_split(p, item, n_tiles, ks, tile);
        tile_coords(p, tile, tm, tn);
        const int m0 = tm * BM, n0 = tn * BN;
        int k0 = range_first(p, ks) * BK;
        const int nkb = range_blocks(p, ks);
        for (int kb = 0; kb < nkb; ++kb, k0 += BK) {
          ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8u * s, ph, abort_flag, p.status, 1u));
          if (!ok) break;
          if (elect_one()) {
            const uint32_t dst = sbase + s * C::stage_bytes, fb = full0 + 8u * s;
            mbar_expect_tx(fb, C::stage_bytes);
            tma_load_2d(dst, &tmap_a, fb, p.a_mn ? m0 : k0, p.a_mn ? k0 : m0);
#pragma unroll
            for (int b = 0; b < C::b_boxes; ++b) {
              const int nb = n0 + b * 128;  // a box wholly past N is still loaded: it arrives as zeros
              tma_load_2d(dst + (1 + b) * kTileBytes, &tmap_b, fb, p.b_mn ? nb : k0, p.b_mn ? k0 : nb);
            }
          }
          __syncwarp();
          if (++s == kStages) { s = 0; ph ^= 1u; }
        }
      }
    } else if (warp == C::issuer_warp) {
      // ------------------------------ MMA issuer ---------------------------------------
      // Blocks are independent: each has its own TMEM buffer and shared-memory stage.
      // instruction descriptor: D f32 (bit 4), A/B e4m3 (0), major bits 15/16, N>>3 at 17, M>>4 at 24
      const uint32_t idesc = (1u << 4) | (uint32_t(p.a_mn) << 15) | (uint32_t(p.b_mn) << 16) |
                             (uint32_t(BN >> 3) << 17) | (uint32_t(BM >> 4) << 24);
      // descriptor start-address step per UMMA_K: 32 bytes along a K-major row, 32 rows of 128 B otherwise
      const uint32_t a_step = p.a_mn ? (UMMA_K * 128) >> 4 : UMMA_K >> 4;
      const uint32_t b_step = p.b_mn ? (UMMA_K * 128) >> 4 : UMMA_K >> 4;
      // a descriptor's low word holds (address >> 4) in 14 bits: shared memory ends below 2^18, so
      // adding block offsets to the low word never carries out of the field
      const uint64_t desc_a0 = make_smem_desc(sbase), desc_b0 = make_smem_desc(sbase + kTileBytes);
      const uint32_t desc_hi = uint32_t(desc_a0 >> 32);
      const uint32_t a_lo0 = uint32_t(desc_a0), b_lo0 = uint32_t(desc_b0);
      uint32_t total = 0;                     // contraction blocks of all this block's work items
      for (int item = first_item; item < n_items; item += item_step) {
        int ks, tile;
        item_split(p, item, n_tiles, ks, tile);
        total += uint32_t(range_blocks(p, ks));
      }
      bool ok = true;
      // A barrier operation has tens of cycles of latency even when the barrier is already complete,
      // and this loop is a chain of them: it does ONE wait instruction per block, lanes 0-15 polling
      // the accumulator buffer's barrier and lanes 16-31 the stage's.
      const bool stage_lane = lane >= 16;
      uint32_t s = 0, sph = 0, buf = 0, bph = 1, soff = 0;
      for (uint32_t it = 0; ok && it < total; ++it) {
        const uint32_t bar = stage_lane ? full0 + 8u * s : tempty0 + 8u * buf;
        const uint32_t par = stage_lane ? sph : bph;
        ok = __all_sync(0xffffffffu, mbar_wait(bar, par, abort_flag, p.status, stage_lane ? 3u : 2u));
        if (!ok) break;
        __syncwarp();                  // (the vote is no memory barrier, and the elected lane has seen one of the two only)
        tc_fence_after();
        if (elect_one()) {
          const uint32_t d_tmem = tmem_base + buf * uint32_t(C::tmem_stride);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_f8(d_tmem, (uint64_t(desc_hi) << 32) | (a_lo0 + soff + k * a_step),
                    (uint64_t(desc_hi) << 32) | (b_lo0 + soff + k * b_step), idesc, k > 0 ? 1u : 0u);
          umma_commit(empty0 + 8u * s);      // shared-memory stage free once these MMAs retire
          umma_commit(tfull0 + 8u * buf);    // accumulator buffer ready for promotion
        }
        __syncwarp();
        soff += uint32_t(C::stage_bytes >> 4);
        if (++s == kStages) { s = 0; sph ^= 1u; soff = 0; }
        if (++buf == kTmemBufs) { buf = 0; bph ^= 1u; }
      }
      // make sure nothing issued here is still running when TMEM is freed
      if (elect_one()) {
        umma_commit(drain_bar);
        mbar_wait(drain_bar, 0u, abort_flag, p.status, 4u);
      }
      __syncwarp();
    } else if (C::store_warp_on && warp == C::store_warp) {
      // ------------------------------ tile store issuer -----------------------------------
      // Per tile: wait until all promotion warps have staged their rows, hand the sixteen boxes to the
      // copy engine, wait until it has read them, give the staging rows back.
      uint32_t sph = 0;
      for (int item = first_item; item < n_items; item += item_step) {
        int ks, tile, tm, tn;
        item_split(p, item, n_tiles, ks, tile);
        tile_coords(p, tile, tm, tn);
        if (!__all_sync(0xffffffffu, mbar_wait(staged_bar, sph, abort_flag, p.status, 7u))) break;
        sph ^= 1u;
        if (elect_one()) {
#pragma unroll 1
          for (int w = 0; w < kPromoWarps; ++w)
            tma_store_3d_nocommit(&tmap_d, sbase + C::off_out + uint32_t(w) * C::warp_out_bytes, tn * BN + (w >> 2) * kCols,
                                  tm * BM + (w & 3) * 32, ks);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          tma_store_wait_read();
          mbar_arrive(unstaged_bar);
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------ promotion + epilogue --------------------------------
    if (C::regsteal) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::promo_regs));
    const int pw = warp;                       // 0..kPromoWarps-1
    const int quarter = warp & 3;              // TMEM lanes this warp may touch
    const int cg = pw >> 2;                    // column group
    const int r = quarter * 32 + lane;         // row inside the tile
    const int c0 = cg * kCols;                 // first column inside the tile
    float* sb_stage = reinterpret_cast<float*>(smem + C::off_sb) + pw * (2 * C::sc_slot);  // warp-private, double-buffered
    constexpr bool kFrag = C::frag;
    const int fg = lane >> 2, fj = lane & 3;     // fragment coordinates: rows fg + 8 i, column pairs 8 k + 2 fj
    const uint32_t out_base = sbase + C::off_out + uint32_t(pw) * C::warp_out_bytes + uint32_t(lane) * C::phase_row_bytes;
    // TMA swizzle of this row: 16-byte chunk index XOR address bits 7.. (128B: 3 bits, 64B: 2, 32B: 1)
    const int swz = C::phase_row_bytes == 128 ? (lane & 7) : C::phase_row_bytes == 64 ? ((lane >> 1) & 3) : ((lane >> 2) & 1);
    bool ok = true;

    // The promotion loop is bound by instruction issue (four such warps share a scheduler, and per
    // block each has 32 packed FMAs and four TMEM loads of payload), so everything else in it is
    // carried incrementally: the accumulator buffer's barrier addresses, TMEM address and phase
    // are toggled, the scale pointers are bumped, and rows / columns outside the problem read a
    // clamped (valid) address instead of being predicated off.
    uint32_t buf = 0, bph = 0, uph = 0;
    const uint32_t tcol0 = tmem_base + (uint32_t(quarter * 32) << 16) + uint32_t(c0);

    // Per-tile state is ONE register pair of scale offsets, set one tile ahead so that the first scale
    // loads are in flight during the previous tile's epilogue; the epilogue derives the tile's
    // coordinates from the item number again rather than keeping them live through the loop.
    uint32_t sa_off = 0, sb_off = 0;           // element offsets into p.sa / p.sb (the host checks they fit 32 bits)
    // The scales of block k+1 are loaded at the top of block k's iteration, by volatile asm so
    // that the compiler cannot sink the loads to their use: with ordinary loads it did, and clock64
    // stamps showed ~450 cycles of exposed L2 latency per block in these warps.
    float sa_q0 = 0.f;
    float2 sb_q0 = make_float2(0.f, 0.f);
    // per-column scales: lane j stages column c0 + j (32-column warps) or the pair c0 + 2j, c0 + 2j + 1
    constexpr int kPerLane = kCols / 32;
    // One scale per 128 columns: its address changes line with every block, so a load per block
    // misses L1 every time and the loop would run at one L2 round trip per block.  Instead lane l
    // fetches the scale of block 32 g + l once per 32 blocks and a shuffle hands each block its value.
    float sb_grp = 0.f, sb_nxt = 0.f;
    int open_nkb = p.nkb;          // contraction blocks of the work item opened last (ranges of a split need not be equal)
    auto load_sb_lane = [&](int g) {
      float v = 0.f;
      const int kb = 32 * g + lane;
      if (kb < open_nkb) v = ld_f32(p.sb + sb_off + uint32_t(kb) * uint32_t(p.sb_sk));
      return v;
    };
    auto load_sb_cols = [&]() {     // per-column scales of the block sb_off points at
      float2 v;
      v.x = ld_f32(p.sb + sb_off);
      v.y = kPerLane == 2 ? ld_f32(p.sb + sb_off + uint32_t(p.sb_sn)) : 0.f;
      return v;
    };
    auto open_tile = [&](int item) {
      int ks, tile, tm, tn;
      item_split(p, item, n_tiles, ks, tile);
      const uint32_t kb_off = uint32_t(range_first(p, ks));
      open_nkb = range_blocks(p, ks);
      tile_coords(p, tile, tm, tn);
      const int n0 = tn * BN;
      const int m = min(tm * BM + r, p.M - 1);       // rows past M: a valid scale, results never stored
      sa_off = uint32_t(m) * uint32_t(p.sa_sm) + kb_off * uint32_t(p.sa_sk);
      if (SB_GRAN == 1) {
        const int col = min(n0 + c0 + kPerLane * lane, p.N - kPerLane);   // N % 8 == 0: a pair is in or out together
        sb_off = uint32_t(col) * uint32_t(p.sb_sn) + kb_off * uint32_t(p.sb_sk);
        sb_q0 = load_sb_cols();
        sb_off += uint32_t(p.sb_sk);
      } else {                                       // one scale per 128 columns
        const int nblk = min((n0 + c0) / 128, (p.N - 1) / 128);
        sb_off = uint32_t(nblk) * uint32_t(p.sb_sn) + kb_off * uint32_t(p.sb_sk);
        sb_grp = load_sb_lane(0);
      }
      sa_q0 = ld_f32(p.sa + sa_off);
      sa_off += uint32_t(p.sa_sk);
    };
    const uint32_t is_lane0 = lane == 0;
    auto release = [&](uint32_t b) {   // every partial sum of the buffer is in registers: hand it back to the tensor core
      tc_fence_before();
      __syncwarp();
      mbar_arrive_if(tempty0 + 8u * b, is_lane0);     // predicated, no branch
    };

    if (first_item < n_items) open_tile(first_item);
    for (int item = first_item; item < n_items; item += item_step) {
      float2 acc[kCols / 2];
#pragma unroll
      for (int j = 0; j < kCols / 2; ++j) acc[j] = make_float2(0.f, 0.f);

      const int nkb = open_nkb;    // set when this item was opened (before the previous tile's epilogue)
      // One contraction block.  `bsel` says which accumulator buffer it drains: a compile-time constant
      // in the two-buffer variants (the block loop below is unrolled by two, so barrier addresses, TMEM
      // address and staging slot are immediates), the carried counter otherwise.
      auto do_block = [&](auto bsel, int kb) -> bool {
        const uint32_t b = bsel.get(buf);
        const float sa_v = sa_q0;
        float2 sb_v = sb_q0;
        const bool more = kb + 1 < nkb;
        if (more) sa_q0 = ld_f32(p.sa + sa_off);
        sa_off += uint32_t(p.sa_sk);
        if (SB_GRAN == 1) {
          if (more) sb_q0 = load_sb_cols();
          sb_off += uint32_t(p.sb_sk);
        } else {
          const int kl = kb & 31;
          if (kl == 0) {
            if (kb != 0) sb_grp = sb_nxt;
            sb_nxt = load_sb_lane((kb >> 5) + 1);
          }
          sb_v.x = __shfl_sync(0xffffffffu, sb_grp, kl);
        }
        float* stage = sb_stage + (b & 1u) * C::sc_slot;      // two slots: consecutive blocks alternate
        if (SB_GRAN == 1) {
          if (kPerLane == 2) *reinterpret_cast<float2*>(stage + 2 * lane) = sb_v;
          else stage[lane] = sb_v.x;
          if (kFrag) stage[kCols + lane] = sa_v;   // row 32 * quarter + lane
          __syncwarp();
        }
        if (!__all_sync(0xffffffffu, mbar_wait(tfull0 + 8u * b, bph, abort_flag, p.status, 5u))) return false;
        tc_fence_after();
        const uint32_t taddr = tcol0 + b * uint32_t(C::tmem_stride);
        const float s_scalar = sa_v * sb_v.x;
        if (kFrag) {
          // acc[(4 q + i) * 2 + k] holds rows fg + 8 i, columns 16 q + 8 k + 2 fj (+1)
          float sa_r[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) sa_r[i] = stage[kCols + fg + 8 * i];
          auto promote_piece = [&](const uint32_t (&cur)[16], int q) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const float2 sb2 = *reinterpret_cast<const float2*>(stage + 16 * q + 8 * k + 2 * fj);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int o = 8 * (i >> 1) + 4 * k + 2 * (i & 1);
                const float2 pv = make_float2(__uint_as_float(cur[o]), __uint_as_float(cur[o + 1]));
                float2& a = acc[(4 * q + i) * 2 + k];
                a = __ffma2_rn(__fmul2_rn(pv, sb2), make_float2(sa_r[i], sa_r[i]), a);
              }
            }
          };
          {
            // two staging sets: the loads of piece q + 1 are in flight while piece q is promoted
            uint32_t va[16], vb[16];
            tmem_ld_frag16(taddr, va);
            tmem_ld_frag16(taddr + (16u << 16), va + 8);
            tmem_wait_ld16(va);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t (&cur)[16] = (q & 1) ? vb : va;
              uint32_t (&nxt)[16] = (q & 1) ? va : vb;
              if (q < 3) {
                tmem_ld_frag16(taddr + 16 * (q + 1), nxt);
                tmem_ld_frag16(taddr + (16u << 16) + 16 * (q + 1), nxt + 8);
              }
              promote_piece(cur, q);
              if (q < 3) tmem_wait_ld16(nxt);
              if (q == 2) release(b);        // every load of the buffer has landed
            }
          }
        } else if (kCols > 32) {
          // 64 columns in four 16-column pieces; the buffer goes back after the last load lands
          uint32_t v[16];
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            tmem_ld16(taddr + 16 * q, v);
            tmem_wait_ld16(v);
            promote<SB_GRAN, 16>(acc + 8 * q, v, stage + 16 * q, sa_v, s_scalar);
          }
          tmem_ld16(taddr + 48, v);
          tmem_wait_ld16(v);
          release(b);
          promote<SB_GRAN, 16>(acc + 24, v, stage + 48, sa_v, s_scalar);
        } else {
          uint32_t v[32];
          tmem_ld32(taddr, v);
          tmem_wait_ld(v);
          release(b);
          promote<SB_GRAN, 32>(acc, v, stage, sa_v, s_scalar);
        }
        // keep this block's FMAs above the next block's first instructions (no instruction is emitted)
        if constexpr (kTmemBufs == 2 && !kFrag) {
#pragma unroll
          for (int j = 0; j < kCols / 2; ++j) asm volatile("" : "+f"(acc[j].x), "+f"(acc[j].y));
        }
        return true;
      };
      // (unrolling the per-column-scale variant measured 7-10 % slower: its blocks overlap better as a rolled loop)
      if constexpr (kTmemBufs == 2 && !kFrag) {
        int kb = 0;
        if (buf != 0) {                      // a previous tile ended on an odd block: drain buffer 1 first
          ok = do_block(StaticBuf<1>{}, kb++);
          buf = 0;
          bph ^= 1u;
        }
        for (; ok && kb + 1 < nkb; kb += 2) {
          ok = do_block(StaticBuf<0>{}, kb) && do_block(StaticBuf<1>{}, kb + 1);
          bph ^= 1u;
        }
        if (ok && kb < nkb) {
          ok = do_block(StaticBuf<0>{}, kb);
          buf = 1;
        }
      } else {
        for (int kb = 0; ok && kb < nkb; ++kb) {
          ok = do_block(DynBuf{}, kb);
          if (++buf == kTmemBufs) { buf = 0; bph ^= 1u; }
        }
      }
      if (!ok) break;   // aborting: every other role sees the flag in its own wait

      // start the next tile's first scale loads before the stores of this one
      if (item + item_step < n_items) open_tile(item + item_step);
      int tile_m0 = 0, tile_n0 = 0, tile_ks = 0;
      if constexpr (!C::store_warp_on) {
        int tile, tm, tn;
        item_split(p, item, n_tiles, tile_ks, tile);
        tile_coords(p, tile, tm, tn);
        tile_m0 = tm * BM;
        tile_n0 = tn * BN;
      }

      // ---- epilogue: registers -> this warp's swizzled staging rows -> bulk tensor stores ----------
      // The warp's 32 rows x kCols columns leave as one box per 128 bytes of row (one box for bf16,
      // two for float32).  Lane 0 hands a box to the copy engine and the warp goes straight on; the
      // wait for the engine to have read the staging rows comes only before they are overwritten
      // (for the first box of a tile that is one whole tile later).  Rows past M and columns past N
      // are clipped by the tensor map, whose third coordinate is the contraction slice.
      constexpr int PRB = C::phase_row_bytes;
      const uint32_t wb = sbase + C::off_out + uint32_t(pw) * C::warp_out_bytes;
      if constexpr (C::store_warp_on) {
        // the staging rows are free once the store warp's boxes of the tile before have been read
        // (a whole tile ago: this does not wait in practice); first tile: nothing to wait for
        if (item != first_item) {
          ok = __all_sync(0xffffffffu, mbar_wait(unstaged_bar, uph, abort_flag, p.status, 8u));
          if (!ok) break;
          uph ^= 1u;
        }
      }
#pragma unroll
      for (int ph = 0; ph < C::phases; ++ph) {
        if constexpr (!C::store_warp_on) {
          if (lane == 0) tma_store_wait_read();
        }
        __syncwarp();
        if (kFrag && OUT_F32) {
          // thread (fg, fj) holds rows fg + 8 i, columns 16 qq + 8 k + 2 fj (+1) of the phase: 16-byte chunk
          // 4 qq + 2 k + (fj >> 1), 8-byte half fj & 1
          const uint32_t fbase = wb + uint32_t(fg) * PRB + (uint32_t(fj >> 1) << 4) + 8u * uint32_t(fj & 1);
          const uint32_t flip = uint32_t(fg & 7) << 4;
          static_loop<2>([&](auto qq) {
            static_loop<4>([&](auto i) {
              static_loop<2>([&](auto k) {
                const float2 a = acc[(4 * (2 * ph + qq.value) + i.value) * 2 + k.value];
                sts_swz_f32x2<i.value * 8 * PRB + (4 * qq.value + 2 * k.value) * 16>(fbase, flip, a);
              });
            });
          });
        } else if (kFrag) {
          // rows fg + 8 i, 16-byte chunk 2 q + k, 4 fj bytes in
          const uint32_t fbase = wb + uint32_t(fg) * PRB + 4u * uint32_t(fj);
          const uint32_t flip = uint32_t(fg & 7) << 4;
          static_loop<4>([&](auto q) {
            static_loop<4>([&](auto i) {
              static_loop<2>([&](auto k) {
                const float2 a = acc[(4 * q.value + i.value) * 2 + k.value];
                sts_swz_b32<i.value * 8 * PRB + (2 * q.value + k.value) * 16>(fbase, flip, pack_bf16x2(a.x, a.y));
              });
            });
          });
        } else if (OUT_F32) {
          static_loop<PRB / 16>([&](auto c) {     // 4 floats per 16-byte chunk
            const int j = ph * (C::phase_cols / 2) + 2 * c.value;
            sts_swz_f32x4<c.value * 16>(out_base, uint32_t(swz) << 4, acc[j], acc[j + 1]);
          });
        } else {
          static_loop<PRB / 16>([&](auto c) {     // 8 bf16 per 16-byte chunk
            const int j = ph * (C::phase_cols / 2) + 4 * c.value;
            sts_swz_v4<c.value * 16>(out_base, uint32_t(swz) << 4, pack_bf16x2(acc[j].x, acc[j].y),
                                     pack_bf16x2(acc[j + 1].x, acc[j + 1].y), pack_bf16x2(acc[j + 2].x, acc[j + 2].y),
                                     pack_bf16x2(acc[j + 3].x, acc[j + 3].y));
          });
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> visible to the copy engine
        __syncwarp();
        if constexpr (C::store_warp_on) {
          mbar_arrive_if(staged_bar, is_lane0);
        } else {
          if (lane == 0) tma_store_3d(&tmap_d, wb, tile_n0 + c0 + ph * C::phase_cols, tile_m0 + quarter * 32, tile_ks);
        }
      }
    }
  }

  // ------------------------------ teardown ----------------------------------------------
  // the last bulk stores must have read their staging rows before the CTA's shared memory goes away
  if (!C::store_warp_on && warp < C::promo_warps && lane == 0) tma_store_wait_read();
  tc_fence_before();
  __syncthreads();
  if (warp == C::issuer_warp) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

template <int BN, int SB_GRAN, bool OUT_F32>
__global__ void __launch_bounds__((Cfg<BN, SB_GRAN, OUT_F32>::threads), 1)
gemm_fp8_blockscaled_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                            const __grid_constant__ CUtensorMap tmap_d, const __grid_constant__ GemmParams p) {
  gemm_body<BN, SB_GRAN, OUT_F32>(tmap_a, tmap_b, tmap_d, p, int(blockIdx.x), int(gridDim.x), [] {
    grid_trigger();
    grid_wait();            // (both do nothing where the launch was an ordinary one)
  });
}

// Two problems of one wave together: the first n1 blocks work on the first, the others on the second.  A linear's data and weight
// gradient both start from the same quantised tensors, and where they are small each is a launch of 4 us that leaves most SMs idle.
struct GemmProblem {
  CUtensorMap a, b, d;
  GemmParams p;
};
template <int GRAN1, int GRAN2>
__global__ void __launch_bounds__((Cfg<128, GRAN1, false>::threads), 1)
gemm_two_kernel(const __grid_constant__ GemmProblem one, const __grid_constant__ GemmProblem two, int n1) {
  static_assert(Cfg<128, GRAN1, false>::threads == Cfg<128, GRAN2, false>::threads, "one thread block shape");
  auto start = [] {
    grid_trigger();
    grid_wait();
  };
  const int block = int(blockIdx.x);
  if (block < n1) gemm_body<128, GRAN1, false>(one.a, one.b, one.d, one.p, block, n1, start);
  else gemm_body<128, GRAN2, false>(two.a, two.b, two.d, two.p, block - n1, int(gridDim.x) - n1, start);
}

// ---- host ------------------------------------------------------------------------------

// The tensor maps of a problem, and what of its parameters follows from the tile.
template <int BN_, int SB_GRAN, bool OUT_F32>
static int prepare_gemm(const tg_gemm_args* a, GemmParams& p, CUtensorMap& ta, CUtensorMap& tb, CUtensorMap& td) {
  using C = Cfg<BN_, SB_GRAN, OUT_F32>;
  const int64_t a_inner = p.a_mn ? a->M : a->K, a_outer = p.a_mn ? a->K : a->M;
  const int64_t b_inner = p.b_mn ? a->N : a->K, b_outer = p.b_mn ? a->K : a->N;
  if (int rc = make_tmap(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->a, a_inner, a_outer, a->lda, 128, 128)) return rc;
  if (int rc = make_tmap(&tb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->b, b_inner, b_outer, a->ldb, 128, 128)) return rc;
  if (int rc = make_output_map(&td, OUT_F32, a, p, C::phase_cols, C::phase_row_bytes)) return rc;
  p.tiles_m = int((a->M + BM - 1) / BM);
  p.tiles_n = int((a->N + BN_ - 1) / BN_);
  p.band = p.tiles_m < kBandRows ? p.tiles_m : kBandRows;
  return set_reciprocals(p);
}

template <int BN_, int SB_GRAN, bool OUT_F32>
static int launch_gemm(const tg_gemm_args* a, GemmParams p, cudaStream_t st) {
  using C = Cfg<BN_, SB_GRAN, OUT_F32>;
  auto kern = gemm_fp8_blockscaled_kernel<BN_, SB_GRAN, OUT_F32>;
  CUtensorMap ta, tb, td;
  if (int rc = prepare_gemm<BN_, SB_GRAN, OUT_F32>(a, p, ta, tb, td)) return rc;
  const int n_items = p.tiles_m * p.tiles_n * p.ksplit;
  const int sms = gemm_sms();
  const int grid = n_items < sms ? n_items : sms;
  // the attribute is per device: set it once for each device this instantiation runs on
  static bool attr_set[64] = {};
  int dev = 0;
  TG_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return TG_ERR_SHAPE;
  if (!attr_set[dev]) {
    TG_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem_bytes));
    attr_set[dev] = true;
  }
  // Few tokens, or few short items per SM: kernels short enough for an early launch to show (4096 x 768 x 3072 with its backward
  // pass: 78.1 -> 74.9 us).  At every size a layer of 32768 x 2048 is 9 % slower.
  if ((p.a_mn == 0 && a->M <= 256) || (n_items <= 4 * sms && p.nkb <= 32)) {
    TG_CUDA_CHECK(launch_early(kern, grid, C::threads, C::smem_bytes, st, ta, tb, td, p));
    return TG_OK;
  }
  kern<<<grid, C::threads, C::smem_bytes, st>>>(ta, tb, td, p);
  TG_CUDA_CHECK(cudaGetLastError());
  return TG_OK;
}

// ---- split contraction -------------------------------------------------------------------
// A GEMM with few output tiles and a long contraction (the weight gradient: d_model x d_model
// outputs, tens of thousands of tokens contracted) leaves most SMs idle.  With caller-provided
// workspace the contraction is cut into S equal ranges, every (tile, range) pair becomes a work
// item writing float32 partial sums to its own slice of the workspace, and a second kernel adds
// the slices in range order (deterministic) and converts to the output type.

template <bool OUT_F32>
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* __restrict__ ws, void* __restrict__ d, int M, int N, long long ldd, int S,
                     long long slice_elems) {
  const long long quads = (long long)M * (N / 4);
  grid_trigger();
  grid_wait();
  ws = loads_below(ws);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < quads; i += (long long)gridDim.x * blockDim.x) {
    const long long m = i / (N / 4);
    const int n = int(i % (N / 4)) * 4;
    float4 acc = *reinterpret_cast<const float4*>(ws + m * N + n);
    for (int sl = 1; sl < S; ++sl) {
      const float4 v = *reinterpret_cast<const float4*>(ws + sl * slice_elems + m * N + n);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    if (OUT_F32) {
      *reinterpret_cast<float4*>(static_cast<float*>(d) + m * ldd + n) = acc;
    } else {
      *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(d) + m * ldd + n) =
          make_uint2(pack_bf16x2(acc.x, acc.y), pack_bf16x2(acc.z, acc.w));
    }
  }
}

// Tile width and number of contraction ranges of a problem, by modelled time.
//
// Wide tiles (256 columns with one scale per 128 columns, 192 with a scale per column) do a full GPU's work with a quarter less
// traffic and promotion overhead per output than 128; 128-column tiles cut a problem of one or two waves finer: 1024^3 is 32
// tiles of 256 on 148 SMs, or 64 of 128 (8.3 -> 6.5 us); 200 x 2048 x 8192 64 or 128 (12.7 -> 8.2).  A contraction cut into S
// ranges (the first nkb % S one block longer) fills the SMs of a problem with few tiles and pays for a second kernel that adds S
// float32 slices.
//
// The constants are microseconds measured on single GEMMs of 4 to 64 blocks: a launch with its ramps, a contraction block of a
// tile (wide tiles in fewer than three waves contend less; the forward with column scales waits longer for them than the weight
// gradient, whose scales were just written), a tile's set-up and stores, the reduction's launch and its bytes.
// The model is within 10-15 % of the measurements it was made from; a narrower tile or a cut has to win by 3 %.
//
// Contractions of fewer than eight blocks over five waves and more are bound by their stores: a tile then takes at least what its
// part of the result takes (`stores`, measured on 200 to 32768 rows, 512 to 8192 columns).  Wide against 128-column tiles,
// microseconds: weight gradient 8192 x 8192 of 64 tokens 29.0 / 31.9, of 256 37.4 / 42.1 and 8192 x 256 -> 8192 31.8 / 38.5 (both took the
// narrow ones without this term); 4096 x 128 -> 1024, two waves, 4.9 / 4.5.  Over 288 problems of fewer than eight blocks the width
// taken is 0.2 % slower than the better one on average (2.7 % without the term).
//
// A pair of SMs with a 256 x 256 tile (gemm_ring.cu) moves a third less from the L2 per block and promotes with fewer instructions, but it
// starts later and a wave of it is coarser.  Measured on 720 uncut problems of 130 to 32768 rows, in turn with the widths above: three
// waves of pairs and more 1.04-1.12 times as fast with a scale per 128 columns, 1.05-1.4 with a scale per column (8192 x 2048 -> 8192 147
// against 158 us and 176 against 230; weight gradient 2048 x 8192 of 8192 tokens 203 / 234), half a wave or less 0.66-0.76.  A
// contraction of one block is nothing to promote, and pairs lose there (20960 x 128 -> 896 11.6 / 14.1 us, with column scales 8192 x 128 -> 3072 13.6 / 16.5) but for
// a few waves of 256-column tiles with a scale per 128, where the two are within 2 % (17246 x 128 -> 896 10.8 / 10.9).  Two blocks: with a scale per
// 128 columns 8589 x 256 -> 4992 23.6 / 25.0; per column it depends on the last wave, as an item takes 2.1 us for its stores (8192 x 256 -> 3072 16.4 / 17.7, -> 4096
// 21.8 / 19.7).  Cut problems, 150 of them: weight gradient 23680 x 1920 x 2304 in four ranges 151 / 133 us, forward 303 x 6016 -> 1408 in five 12.6 / 15.3.
// Column scales that lie apart (apart_us), single SMs / pairs: 445 x 3456 -> 4736 13.0 / 21.0 us, 4992 x 3584 -> 1024 31.0 / 38.4, but cut in two
// 2176 x 7168 -> 3328 161 / 100 (its kernel fetches each scale when it needs it, one sector for one number) and 22016 x 1280 -> 1280 53.9 / 44.2.  Of 1100
// problems, 660 of them such, the rule takes pairs where single SMs are more than 2 % faster in five (at most 6 %).
//
// The tile width does not show in the result; the number of ranges does, in the last bit of float32 sums, and a training run
// amplifies that over its steps.  So where the tokens are whole blocks of 128, as a training step's are, the number of
// ranges is a rule of its own (training_ranges) that the tile width has no part in.
struct GemmPlan {
  int bn, S;
  int64_t bytes;     // workspace the cut needs
  bool pair;         // 256 x 256 tiles on pairs of SMs (gemm_ring.cu)
  bool ring;         // bn-wide tiles by gemm_ring.cu
  double us;         // modelled time
};
// S of 1 to 8 ranges of at least 8 blocks by waves of wide tiles x (blocks per item + 3 for an item's ramp and stores), plus for
// S > 1 the reduction over S float32 slices at 4 MB per block time.
static int training_ranges(const tg_gemm_args* a, int wide) {
  const int64_t nkb = a->K / BK, tiles = ((a->M + BM - 1) / BM) * ((a->N + wide - 1) / wide);
  const int sms = gemm_sms();
  int ranges = 1;
  double best = 0.0;
  for (int S = 1; S <= 8; ++S) {
    if (S > 1 && nkb / S < 8) break;
    double cost = double((tiles * S + sms - 1) / sms) * (double((nkb + S - 1) / S) + 3.0);
    if (S > 1) cost += double(4 * S + 2) * double(a->M) * double(a->N) / 4.0e6;
    if (S == 1 || cost < best * 0.98) { best = cost; ranges = S; }
  }
  return ranges;
}

// What a contraction block takes longer (or, in the ring, less long) than the figures of plan_gemm where the column scales of a block lie apart,
// each in a sector with those of the same column's next blocks (the data gradient of a weight that was quantised along its columns): by the
// number of blocks, that is, the distance between two columns' scales.
static double apart_us(bool pair, int bn, bool cut, bool ring, int64_t nkb) {
  const double far = double(std::max<int64_t>(nkb, 16) - 16);
  if (pair) return std::min(0.005 * far, 0.16);
  if (bn == 192 && cut) return std::min(std::max(0.04 * far - 0.32, 0.0), 0.6);
  if (!ring) return 0.0;
  return bn == 192 ? std::min(-0.04 + 0.004 * far, 0.11) : -0.04;
}

static GemmPlan plan_gemm(const tg_gemm_args* a) {
  const bool columns = a->sb_gran_n == 1;
  const int wide = a->N <= 128 ? 128 : columns ? 192 : 256;
  GemmPlan pl = {wide, 1, 0, false, false, 0.0};
  const int64_t nkb = (a->K + BK - 1) / BK;
  const int sms = gemm_sms();
  const bool whole = a->K % BK == 0 && (a->a_major == TG_MAJOR_MN || a->M % 128 == 0);      // (weight gradient: the tokens are K)
  const int fixed = whole ? training_ranges(a, wide) : 0;
  double best = 0.0;
  for (const int bn : {wide, 128}) {
    const int64_t tiles = ((a->M + BM - 1) / BM) * ((a->N + bn - 1) / bn);
    for (int S = 1; S <= 8; ++S) {
      if (S > 1 && nkb / S < 8) break;
      if (fixed != 0 && S != fixed) continue;
      const int64_t waves = (tiles * S + sms - 1) / sms;
      const double block = bn == 256 ? (waves < 3 ? 0.44 : 0.50) : bn == 192 ? 0.47 : !columns ? 0.355 : a->a_major == TG_MAJOR_K ? 0.42 : 0.38;
      const double tile = bn == 128 ? (columns ? 0.5 : 0.1) : 1.0;
      const double blocks = double((nkb + S - 1) / S);
      const double stores = nkb >= 8 || waves < 5 ? 0.0 : bn == 256 ? 2.0 : bn == 192 ? 1.4 : columns ? 0.65 + 0.38 * blocks : 0.75 + 0.29 * blocks;
      double us = 3.0 + double(waves) * std::max(block * blocks + tile, stores);
      if (S > 1) us += 3.5 + double(4 * S + 2) * double(a->M) * double(a->N) / 8.0e6;
      if (best == 0.0 || us < best * 0.97) {
        best = us;
        pl.bn = bn;
        pl.S = S;
      }
    }
    if (wide == 128) break;
  }
  if (pl.S > 1) pl.bytes = int64_t(pl.S) * a->M * a->N * int64_t(sizeof(float));
  const int64_t pairs = gemm_pairs();
  if (pairs > 0 && a->M > 128 && a->N > 128) {
    const int64_t items = ((a->M + 255) / 256) * ((a->N + 255) / 256) * pl.S, waves = (items + pairs - 1) / pairs;
    const double blocks = double((nkb + pl.S - 1) / pl.S);
    const bool apart = columns && a->sb_stride_n != 1;
    const double item = pair_item_us(columns, blocks) + (apart ? apart_us(true, 256, false, true, nkb) * blocks : 0.0);
    double us = 4.3 + double(waves) * (columns ? std::max(item, 2.08) : item);        // (two blocks: the stores)
    if (pl.S > 1) us += 3.5 + double(4 * pl.S + 2) * double(a->M) * double(a->N) / 8.0e6;
    if (apart) {
      const int64_t tiles = ((a->M + BM - 1) / BM) * ((a->N + pl.bn - 1) / pl.bn) * pl.S;
      best += double((tiles + sms - 1) / sms) * blocks * apart_us(false, pl.bn, pl.S > 1, blocks >= 12, nkb);
    }
    const bool short_even = nkb == 1 && !columns && pl.bn == 256 && waves <= 5;
    pl.pair = us < best && (nkb >= 8 || (waves >= 3 && (nkb >= 3 || (nkb == 2 && columns) || short_even)));
    if (pl.pair) pl.bn = 256;
    best = std::min(best, us);
  }
  pl.us = best;
  // Column scales through gemm_ring.cu's ring, where the contraction is long enough for its later start (the measurement is there).
  // A range of a cut problem is worth it from 15 blocks on, as its float32 tile takes longer to leave (weight gradient of 12026 tokens, 384 x 256, 8 x
  // 12 blocks 10.4 / 10.6 us, 15047 tokens 2176 x 256, 4 x 30 20.0 / 18.2), but where the scales lie apart (19200 x 6656 -> 128, 4 x 13 65.5 / 53.4).
  // Cut problems of 192-column tiles stay: their float32 tiles leave in three steps there (0.95-1.08 times as fast).
  const int64_t ring_from = pl.S > 1 && a->sb_stride_n == 1 ? 15 : 12;
  pl.ring = !pl.pair && columns && (nkb + pl.S - 1) / pl.S >= ring_from && (pl.bn == 128 || (pl.bn == 192 && (pl.S == 1 && a->out_dtype == TG_OUT_BF16)));
  return pl;
}

}  // namespace tg

using namespace tg;

static int validate_gemm(const tg_gemm_args* a) {
  if (a == nullptr) return TG_ERR_SHAPE;
  if (a->M < 0 || a->N < 0 || a->K < 0) return TG_ERR_SHAPE;
  if (a->M > INT32_MAX || a->N > INT32_MAX || a->K > INT32_MAX) return TG_ERR_TOO_LARGE;
  if ((a->a_major != TG_MAJOR_K && a->a_major != TG_MAJOR_MN) || (a->b_major != TG_MAJOR_K && a->b_major != TG_MAJOR_MN))
    return TG_ERR_SHAPE;
  if (a->sb_gran_n != 1 && a->sb_gran_n != 128) return TG_ERR_SHAPE;
  if (a->out_dtype != TG_OUT_BF16 && a->out_dtype != TG_OUT_F32) return TG_ERR_SHAPE;
  if (a->N % 8 != 0 || a->ldd % 8 != 0 || a->ldd < a->N) return TG_ERR_SHAPE;
  if (a->lda % 16 != 0 || a->ldb % 16 != 0) return TG_ERR_SHAPE;
  const int64_t a_inner = a->a_major == TG_MAJOR_K ? a->K : a->M;
  const int64_t b_inner = a->b_major == TG_MAJOR_K ? a->K : a->N;
  if (a->lda < a_inner || a->ldb < b_inner) return TG_ERR_SHAPE;
  return TG_OK;
}

extern "C" int64_t tg_gemm_workspace_bytes(const tg_gemm_args* a) {
  if (validate_gemm(a) != TG_OK || a->M == 0 || a->N == 0 || a->K == 0) return 0;
  if (skinny_takes(a)) return skinny_workspace_bytes(a);
  return plan_gemm(a).bytes;
}

extern "C" int tgh_gemm_plan(const tg_gemm_args* a, int* tile_columns, int* ranges) {
  if (int rc = validate_gemm(a)) return rc;
  if (a->M == 0 || a->N == 0 || a->K == 0 || skinny_takes(a)) return TG_ERR_TOO_LARGE;
  const GemmPlan pl = plan_gemm(a);
  *tile_columns = pl.bn;
  *ranges = pl.S;
  return TG_OK;
}

extern "C" int tgh_gemm_kernel(const tg_gemm_args* a, int* kernel) {
  if (int rc = validate_gemm(a)) return rc;
  if (a->M == 0 || a->N == 0 || a->K == 0 || skinny_takes(a)) return TG_ERR_TOO_LARGE;
  const GemmPlan pl = plan_gemm(a);
  *kernel = pl.pair ? 2 : pl.ring ? 1 : 0;
  return TG_OK;
}

static int check_scales(const tg_gemm_args* a) {
  // the kernels walk the scale arrays with 32-bit element offsets
  const int64_t nkb_all = (a->K + BK - 1) / BK;
  const int64_t n_sb = a->sb_gran_n == 1 ? a->N : (a->N + 127) / 128;
  if (a->sa_stride_m < 0 || a->sa_stride_kb < 0 || a->sb_stride_n < 0 || a->sb_stride_kb < 0) return TG_ERR_SHAPE;
  if (a->M * a->sa_stride_m + nkb_all * a->sa_stride_kb > INT32_MAX || n_sb * a->sb_stride_n + nkb_all * a->sb_stride_kb > INT32_MAX)
    return TG_ERR_TOO_LARGE;
  return TG_OK;
}

static GemmParams params_of(const tg_gemm_args* a) {
  GemmParams p;
  p.sa = a->sa; p.sa_sm = a->sa_stride_m; p.sa_sk = a->sa_stride_kb;
  p.sb = a->sb; p.sb_sn = a->sb_stride_n; p.sb_sk = a->sb_stride_kb;
  p.d = a->d; p.ldd = a->ldd;
  p.M = int(a->M); p.N = int(a->N); p.nkb = int((a->K + BK - 1) / BK);
  p.nkb_rem = 0;
  p.a_mn = a->a_major == TG_MAJOR_MN; p.b_mn = a->b_major == TG_MAJOR_MN;
  p.tiles_m = p.tiles_n = 0;
  p.band = 1;
  p.ksplit = 1;
  p.slice_elems = 0;
  p.status = a->status;
  return p;
}

static bool cut_fits(const tg_gemm_args* a, const GemmPlan& pl) {
  return pl.S > 1 && a->workspace != nullptr && a->workspace_bytes >= pl.bytes && aligned16(a->workspace);
}
static void cut_params(const tg_gemm_args* a, int S, GemmParams& p) {
  p.ksplit = S;
  p.nkb_rem = p.nkb % S;
  p.nkb /= S;
  p.slice_elems = a->M * a->N;
  p.d = a->workspace;
  p.ldd = a->N;
}
static int reduce_ranges(const tg_gemm_args* a, int S, cudaStream_t st) {
  const long long quads = a->M * (a->N / 4);
  const int blocks = int(quads / 256 + 1 < 4096 ? quads / 256 + 1 : 4096);
  TG_CUDA_CHECK(launch_if_short(blocks <= 8 * gemm_sms(), a->out_dtype == TG_OUT_F32 ? splitk_reduce_kernel<true> : splitk_reduce_kernel<false>,
                                dim3(unsigned(blocks)), 256, 0, st, static_cast<const float*>(a->workspace), a->d, int(a->M), int(a->N),
                                static_cast<long long>(a->ldd), S, static_cast<long long>(a->M * a->N)));
  return TG_OK;
}

// A problem that passed all checks and is not the few-token kernel's, as planned.
static int run_tiled(const tg_gemm_args* a, const GemmPlan& pl, cudaStream_t st) {
  GemmParams p = params_of(a);
  const bool g1 = a->sb_gran_n == 1, f32 = a->out_dtype == TG_OUT_F32;
  const int bn = pl.bn;
  if (cut_fits(a, pl)) {
    cut_params(a, pl.S, p);
    int rc;
    if (pl.pair || pl.ring) rc = ring_run(a, p, pl.pair, bn, true, st);
    else if (bn == 256) rc = launch_gemm<256, 128, true>(a, p, st);
    else if (bn == 192) rc = launch_gemm<192, 1, true>(a, p, st);
    else rc = g1 ? launch_gemm<128, 1, true>(a, p, st) : launch_gemm<128, 128, true>(a, p, st);
    if (rc != TG_OK) return rc;
    return reduce_ranges(a, pl.S, st);
  }
  if (pl.pair || pl.ring) return ring_run(a, p, pl.pair, bn, f32, st);
  if (bn == 256) return f32 ? launch_gemm<256, 128, true>(a, p, st) : launch_gemm<256, 128, false>(a, p, st);
  if (bn == 192) return f32 ? launch_gemm<192, 1, true>(a, p, st) : launch_gemm<192, 1, false>(a, p, st);
  if (g1) return f32 ? launch_gemm<128, 1, true>(a, p, st) : launch_gemm<128, 1, false>(a, p, st);
  return f32 ? launch_gemm<128, 128, true>(a, p, st) : launch_gemm<128, 128, false>(a, p, st);
}

extern "C" int tg_gemm_fp8_blockscaled(const tg_gemm_args* a, void* stream) {
  if (int rc = validate_gemm(a)) return rc;
  if (a->M == 0 || a->N == 0) return TG_OK;
  if (!aligned16(a->a) || !aligned16(a->b) || !aligned16(a->d)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (a->K == 0) {
    const size_t esz = a->out_dtype == TG_OUT_F32 ? 4 : 2;
    TG_CUDA_CHECK(cudaMemset2DAsync(a->d, size_t(a->ldd) * esz, 0, size_t(a->N) * esz, size_t(a->M), st));
    return TG_OK;
  }
  if (int rc = check_scales(a)) return rc;
  if (skinny_takes(a)) {
    const int64_t need = skinny_workspace_bytes(a);
    if (need == 0 || (a->workspace != nullptr && a->workspace_bytes >= need && aligned16(a->workspace))) return skinny_run(a, st);
  }
  return run_tiled(a, plan_gemm(a), st);
}

// Whether a problem passes all checks of the public call and is a tiled kernel's.
static bool ready(const tg_gemm_args* a) {
  if (validate_gemm(a) != TG_OK || a->M == 0 || a->N == 0 || a->K == 0 || skinny_takes(a)) return false;
  return aligned16(a->a) && aligned16(a->b) && aligned16(a->d) && check_scales(a) == TG_OK;
}

// Modelled time of a (column scales) in S ranges and then b (block scales), both on pairs in one launch.
static double pairs_together_us(const tg_gemm_args* a, int S, const tg_gemm_args* b, int& rounds) {
  auto tiles = [](const tg_gemm_args* x) { return ((x->M + 255) / 256) * ((x->N + 255) / 256); };
  auto blocks = [](const tg_gemm_args* x, int n) { return double(((x->K + BK - 1) / BK + n - 1) / n); };
  double us = 4.3 + two_problems_us(tiles(a) * S, pair_item_us(true, blocks(a, S)), tiles(b), pair_item_us(false, blocks(b, 1)),
                                    std::max(1, gemm_pairs()), rounds);
  if (S > 1) us += 3.5 + double(4 * S + 2) * double(a->M) * double(a->N) / 8.0e6;
  return us;
}

// How two products run: each by itself (`planned`: as a and b say), in one wave of n1 + n2 tiles, or both on pairs.
struct TwoPlan {
  int joint;         // TGH_TWO_*
  bool planned;
  GemmPlan a, b;
  int n1, n2;        // one wave: the tiles of a and of b
  bool cut;          // on pairs: b in ranges
  int rounds;        // on pairs: of a's items on the pairs that b's last round leaves idle
};

static TwoPlan plan_two(const tg_gemm_args* a, const tg_gemm_args* b) {
  TwoPlan t = {};
  t.joint = TGH_TWO_APART;
  t.planned = ready(a) && ready(b);
  if (!t.planned) return t;
  t.a = plan_gemm(a);
  t.b = plan_gemm(b);
  // Together they are one wave, uncut, of 128-column tiles in bf16 by this file's kernel.  (One wave is also what an early launch asks for:
  // gemm_fp8_blockscaled_kernel's rule.)
  auto wave_tiles = [](const tg_gemm_args* x, const GemmPlan& pl) -> int64_t {
    if (x->out_dtype != TG_OUT_BF16 || pl.pair || pl.ring || pl.bn != 128 || pl.S != 1 || (x->K + BK - 1) / BK > 32) return 0;
    return ((x->M + 127) / 128) * ((x->N + 127) / 128);
  };
  const int64_t n1 = wave_tiles(a, t.a), n2 = wave_tiles(b, t.b);
  if (n1 > 0 && n2 > 0 && n1 + n2 <= gemm_sms() && (a->sb_gran_n == 128 || b->sb_gran_n == 1)) {
    t.joint = TGH_TWO_WAVE;
    t.n1 = int(n1);
    t.n2 = int(n2);
    return t;
  }
  // Both on pairs of SMs, where one launch fills the last rounds (gemm_ring_two_kernel).  The modelled saving is 4 to 8 % too high (four
  // linears of 32768 tokens: 6-8 % modelled, -0.1 to 3 % measured in short runs, -1 to 2 % at the power cap); from a twelfth on large
  // problems gain (2-20 %, 700 x 4096 -> 4096 54.1 / 47.2 us with the quantisers).  Two short kernels launched early one after the other hide some
  // of each other's ramps, which the model counts twice: below 2.1 us and 15 % of modelled saving 8466 x 384 -> 256 had 15.7 apart / 17.4, 512 x 1024 -> 1920 13.2 / 13.9
  // (with 2 us but 20 %, 444 x 8064 -> 256 12.0 / 11.5); of 89 joint problems two with more still lose (211 x 3072 -> 2432 17.5 / 18.8).  A data gradient with a scale per
  // column stays apart: 12000 x 768 -> 3072 115 / 123 us, 4096 x 768 -> 3072 49.5 / 60, though 24576 x 1024 -> 1024 110 / 92.
  // (a is uncut: the callers hand both the same workspace, which only b may use in a joint launch.)
  auto wide = [](const tg_gemm_args* x) { return x->M > 128 && x->N > 128; };
  if (a->sb_gran_n == 128 && b->sb_gran_n == 1 && a->out_dtype == TG_OUT_BF16 && wide(a) && wide(b) && gemm_pairs() > 0 && t.a.S == 1) {
    t.cut = cut_fits(b, t.b);
    if (t.cut || b->out_dtype == TG_OUT_BF16) {
      const double apart_us = t.a.us + t.b.us, together_us = pairs_together_us(b, t.cut ? t.b.S : 1, a, t.rounds);
      if (together_us < (11.0 / 12.0) * apart_us && (together_us < apart_us - 2.1 || together_us < 0.85 * apart_us)) t.joint = TGH_TWO_PAIRS;
    }
  }
  return t;
}

template <int GRAN1, int GRAN2>
static int launch_two(const tg_gemm_args* a, const tg_gemm_args* b, int n1, int n2, cudaStream_t st) {
  GemmProblem one, two;
  one.p = params_of(a);
  two.p = params_of(b);
  if (int rc = prepare_gemm<128, GRAN1, false>(a, one.p, one.a, one.b, one.d)) return rc;
  if (int rc = prepare_gemm<128, GRAN2, false>(b, two.p, two.a, two.b, two.d)) return rc;
  auto kern = gemm_two_kernel<GRAN1, GRAN2>;
  constexpr int smem = std::max(Cfg<128, GRAN1, false>::smem_bytes, Cfg<128, GRAN2, false>::smem_bytes);
  static std::atomic<bool> attr_set[64];
  int dev = 0;
  TG_CUDA_CHECK(cudaGetDevice(&dev));
  if (!attr_set[dev & 63].load(std::memory_order_acquire)) {
    TG_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attr_set[dev & 63].store(true, std::memory_order_release);
  }
  TG_CUDA_CHECK(launch_early(kern, n1 + n2, Cfg<128, GRAN1, false>::threads, smem, st, one, two, n1));
  return TG_OK;
}

extern "C" int tgh_gemm_two_plan(const tg_gemm_args* a, const tg_gemm_args* b, int* rounds) {
  const TwoPlan t = plan_two(a, b);
  *rounds = t.joint == TGH_TWO_PAIRS ? t.rounds : 0;
  return t.joint;
}

extern "C" int tgh_gemm_two(const tg_gemm_args* a, const tg_gemm_args* b, void* stream) {
  const TwoPlan t = plan_two(a, b);
  if (!t.planned) {
    if (int rc = tg_gemm_fp8_blockscaled(a, stream)) return rc;
    return tg_gemm_fp8_blockscaled(b, stream);
  }
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (t.joint == TGH_TWO_WAVE) {
    if (a->sb_gran_n == 1) return launch_two<1, 1>(a, b, t.n1, t.n2, st);
    return b->sb_gran_n == 1 ? launch_two<128, 1>(a, b, t.n1, t.n2, st) : launch_two<128, 128>(a, b, t.n1, t.n2, st);
  }
  if (t.joint == TGH_TWO_PAIRS) {
    GemmParams p = params_of(b);
    if (t.cut) cut_params(b, t.b.S, p);
    if (int rc = ring_pair_two(b, p, t.cut, a, params_of(a), st)) return rc;
    return t.cut ? reduce_ranges(b, t.b.S, st) : TG_OK;
  }
  if (int rc = run_tiled(a, t.a, st)) return rc;
  return run_tiled(b, t.b, st);
}
