// Block-scaled e4m3 GEMM for few tokens (M <= 128) against a wide weight: D[m][n] = sum_kb SX(m,kb) SW(n,kb) X[m] . W[n].
//
// One pass over the weight is the work: at 16 x 8192 x 8192 it is 67 MB (10.2 us at the measured copy rate) against 0.7 us of
// tensor-core time.  What the tiled kernel (gemm_fp8.cu) does badly there, and what is done instead:
//   * the weight's N dimension takes the MMA's 128 rows and the tokens its columns (16, 32, 64 or 128 of them): no dead
//     rows, and a stage of the pipeline is 16 KB of weight plus as little as 2 KB of tokens.  Seven of them in flight per SM: with
//     twelve, or with an L2 prefetch of the first ones while the kernel before runs, the SMs read from more places of the
//     weight at once and 16 x 8192 x 8192 takes 14.7 instead of 14.0 us;
//   * the (tile, contraction block) units are numbered tile by tile and every block of the grid takes as many consecutive ones; it
//     leaves each tile's part of float32 sums in a slot of the workspace.  Preferably a whole number of blocks shares a tile:
//     all tiles are then at the same contraction rows at the same time, and what the SMs read together is whole rows of
//     the weight, not 128-byte pieces of rows 8 KB apart (8192 x 8192: 5.0 against 4.5 TB/s);
//   * scales arrive with the stage they belong to (see the producer warp);
//   * a thread holds one weight row's sums over the tokens, so a slot is written 128 consecutive bytes per warp and token, and
//     the reduce kernel, which adds a tile's slots in order, reads and writes along N: nothing is transposed;
//   * where a tile is shared by at most four blocks (32 tiles and more), these form a thread-block cluster, the slots are
//     their shared memories and the blocks add them up themselves: one launch, no workspace, the same order of additions;
//   * programmatic dependent launch: barriers and tensor memory are set up while the kernel before runs, and the reduce kernel is
//     resident when the last sums arrive.
// Bound by the weight's bytes plus about 4 us of ramps; 128 tokens by the L2's, 32 KB per block of contraction.  Microseconds per
// GEMM in a chain of them: split contraction and transposing reduce -> scales fetched by the promotion warps -> now:
// 16 x 8192 x 8192 24.8 -> 15.1 -> 14.0, 64 x 8192 x 8192 18.8 -> 16.9, 128 x 8192 x 8192 26.8 -> 21.5,
// 16 x 2048 x 6144 13.5 -> 6.8 -> 5.9.
#include "umma.cuh"

namespace tg {

// From 129 tokens on the tokens fill 128 MMA rows themselves, a token scale is a thread's own number instead of a column's,
// and the tiled kernel is the faster one: 200 tokens, tiled / this kernel with 256 columns, a scale per 128 weight columns (per
// column): 2048 x 8192 8.6 / 14.1 us (10.1 / 13.7), 4096 x 4096 12.0 / 16.2 (14.1 / 15.7), 8192 x 8192 25.0 / 40.4 (37.4 / 37.3).
// Below, both sides with the weight from memory, this kernel / tiled, K x N, a scale per 128 weight columns unless said (with a scale per column
// the tiled side takes up to a tenth longer, this one the same):
//   1 to 32 tokens.  Weights of more than 512 columns stay here (16 tokens 1024 x 1024 4.7 / 5.0, 1024 x 4096 5.1 / 5.7, 8192 x 8192 13.4 / 16.9).
//     Narrower ones are a few tiles, and the tiled kernel has them all in flight once it cuts the contraction three times or more, from K = 3072
//     on: 16 x 2560 x 512 7.1 / 8.1, 3072 x 512 7.3 / 6.7, 4096 x 512 8.6 / 7.3, 8192 x 512 9.1 / 7.8, 8192 x 256 12.5 / 7.5; it makes eight ranges at most, so from
//     4 M weights on it falls behind again: 12288 x 512 8.7 / 8.9, 16384 x 512 9.0 / 10.0, 32768 x 256 12.2 / 14.3.  One token against 2048 x 256 with a
//     scale per column 5.0 / 7.4.  In between lies 32 x 3584 x 512 with 6.2 / 7.4.  512 x 512: 32 tokens 4.0 / 3.8, 8 tokens 3.6 / 3.7.
//   33 to 64 tokens.  Short contractions are the tiled kernel's: 48 x 512 x 512 4.8 / 3.9, 640 x 7680 6.1 / 5.3, 1024 x 1024 5.7 / 5.1, 1024 x 4096 6.3 / 5.7; 2048 x 6144
//     7.9 / 8.0, 8192 x 8192 15.9 / 17.6.  Narrow weights of long contractions stay here: 64 x 2048 x 512 5.8 / 7.1, though 48 x 4096 x 256 8.7 / 7.2.
//   65 to 128 tokens.  With a scale per column only short contractions are tiled (100 x 1024 x 4096 7.5 / 6.2, 8192 x 8192 20.3 / 21.6, though 2048 x 8192
//     9.8 / 8.9).  With one per 128 columns nearly all (100 x 1024 x 4096 7.5 / 5.8, 4096 x 4096 10.8 / 10.1, 8192 x 8192 20.1 / 18.6); not up to 2048 columns of
//     1152 to 4608 (2048 x 2048 7.5 / 7.9), with fewer than 128 tokens up to 2560 of about 2048 (65 x 2048 x 2176 7.0 / 7.8), nor 27 to 34 M weights (8192 x 4096 14.4 / 14.9, 5504 x
//     5120 13.2 / 13.7), and with 128 tokens, whose contraction ranges are fixed, 20 to 34 M (8192 x 3072 13.1 / 14.4, 5504 x 4096 12.6 / 14.3; but 4096 x
//     6144 13.9 / 13.5).
// 1092 problems of these ranges: the kernel taken is more than 5 % slower than the other in 40 of them.
constexpr int kSkinnyMaxTokens = 128;

template <int BN_>
struct SkinnyCfg {
  static constexpr int BN = BN_;                                    // tokens
  // at most 32 columns of sums per warp (with 64 a warp's own chain of loads was longer than a unit: M = 64 21 us)
  static constexpr int promo_warps = BN == 16 ? 4 : BN == 128 ? 16 : 8;
  static constexpr int cols = BN / (promo_warps / 4);
  static constexpr int producer_warp = promo_warps, issuer_warp = promo_warps + 1;
  // two issuers take alternate units: a thread gets a tcgen05 instruction out every ~80 cycles whatever its size, and a unit's
  // five would hold an SM to 16 KB per 330 ns
  static constexpr int issuers = 2;
  static constexpr int threads = 32 * (promo_warps + 1 + issuers);
  static constexpr int bufs = 4;                                    // accumulator buffers in tensor memory
  static constexpr int tmem_cols = BN * bufs < 32 ? 32 : BN * bufs;
  static constexpr int stage_bytes = kTileBytes + BN * 128;
  // a stage's scales: a factor per token, then one per weight row (or one for all of them)
  static constexpr int stage_scales = BN + 128;
  static constexpr int stages_fit = (kSmemLimit - 1024) / (stage_bytes + 4 * stage_scales);
  static constexpr int stages = stages_fit > 7 ? 7 : stages_fit;
  static constexpr int scale_bytes = stages * 4 * stage_scales;
  static constexpr int smem_bytes = stages * stage_bytes + scale_bytes;
  static constexpr int n_bars = 2 * stages + 2 * bufs + 1;
  static_assert(n_bars <= 40, "control block too small");
};

struct SkinnyParams {
  const float* sx;               // token scales, [m * sx_m + kb * sx_k]
  const float* sw;               // weight scales, [n * sw_n + kb * sw_k], n in rows or in blocks of 128 (W_ROWS or not)
  unsigned sx_m, sx_k, sw_n, sw_k;
  float* ws;                     // slots of [M][128] sums
  int M, N, nkb;
  int units, w_mn;               // units = tiles * nkb; w_mn: the weight is stored [K][N]
  int share;                     // > 0: the `share` blocks of a tile are a cluster and finish the tile themselves
  void* d;                       // (share > 0) the result
  long long ldd;
  int d_f32;
  unsigned* status;
};

// Block c of g takes units [c * units / g, (c + 1) * units / g); unit u belongs to block ((u + 1) g - 1) / units.  The part that
// block c does of tile t has slot c + t: each step along the units enters a new block, a new tile, or both.
__host__ __device__ __forceinline__ int skinny_first(int c, int g, int units) { return int((long long)c * units / g); }
__host__ __device__ __forceinline__ int skinny_block_of(int u, int g, int units) { return int(((long long)(u + 1) * g - 1) / units); }

__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// arrive on `bar` (one of the arrivals it counts) when this thread's cp.async so far are done
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// Barrier over all threads of the cluster (a cluster of one where the launch has none); it ends because every path above does.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// four floats at shared-memory address `addr` of the cluster's block `rank`
__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr, int rank) {
  float4 v;
  asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"(rank) : "memory");
  return v;
}

// W_ROWS: a weight scale per row (128 x 1 tiles), else one per 128 rows
template <int BN_, bool W_ROWS>
__global__ void __launch_bounds__((SkinnyCfg<BN_>::threads), 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const SkinnyParams p) {
  using C = SkinnyCfg<BN_>;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(16) uint64_t ctl_bars[40];
  __shared__ uint32_t ctl_tmem_ptr;
  __shared__ int ctl_abort;
  const uint32_t sbase = smem_u32(smem), bar0 = smem_u32(ctl_bars);
  const uint32_t full0 = bar0, empty0 = bar0 + 8u * C::stages, tfull0 = bar0 + 16u * C::stages, tempty0 = tfull0 + 8u * C::bufs;
  const uint32_t drain_bar = tempty0 + 8u * C::bufs;
  volatile int* abort_flag = &ctl_abort;
  if ((sbase & 1023u) != 0) {
    if (threadIdx.x == 0 && p.status != nullptr) atomicCAS(p.status, 0u, 6u);
    return;
  }
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int u0 = skinny_first(int(blockIdx.x), int(gridDim.x), p.units), u1 = skinny_first(int(blockIdx.x) + 1, int(gridDim.x), p.units);
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::stages; ++s) {
      mbar_init(full0 + 8u * s, 1 + 32);           // the boxes, and each producer lane's scales
      mbar_init(empty0 + 8u * s, C::promo_warps);
    }
    for (int b = 0; b < C::bufs; ++b) {
      mbar_init(tfull0 + 8u * b, 1);
      mbar_init(tempty0 + 8u * b, C::promo_warps);
    }
    mbar_init(drain_bar, C::issuers);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == C::producer_warp && elect_one()) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_w)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_x)) : "memory");
  }
  if (warp == C::issuer_warp) {
    tmem_alloc(smem_u32(&ctl_tmem_ptr), C::tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *static_cast<volatile uint32_t*>(&ctl_tmem_ptr);
  grid_wait();            // what the kernels before wrote is visible from here on, and what they read may be overwritten
  grid_trigger();

  if (warp == C::producer_warp) {
    // Scales come with the stage they belong to: cp.async by all lanes, which arrive on its barrier as the boxes do.  (The
    // promotion warps fetched their own, eight units ahead: with the staging in shared memory that was most of a
    // unit's 330 ns at 16 tokens and 630 at 128, weight from the L2.)
    constexpr int kPer = (BN_ + 31) / 32;
    uint32_t s = 0, ph = 1;
    bool ok = true;
    int kb = u0 % p.nkb, tile = u0 / p.nkb;
    unsigned sx_off[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) sx_off[i] = unsigned(min(lane + 32 * i, p.M - 1)) * p.sx_m;      // past M: a valid scale, unused sums
    for (int u = u0; u < u1; ++u) {
      ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8u * s, ph, abort_flag, p.status, 1u));
      if (!ok) break;
      const uint32_t fb = full0 + 8u * s;
      if (elect_one()) {
        const uint32_t dst = sbase + s * C::stage_bytes;
        const int k0 = kb * BK, n0 = tile * BM;
        mbar_expect_tx(fb, C::stage_bytes);
        tma_load_2d(dst, &tmap_w, fb, p.w_mn ? n0 : k0, p.w_mn ? k0 : n0);
        tma_load_2d(dst + kTileBytes, &tmap_x, fb, k0, 0);
      }
      __syncwarp();
      const uint32_t sc = sbase + uint32_t(C::stages * C::stage_bytes) + s * uint32_t(4 * C::stage_scales) + 4u * uint32_t(lane);
#pragma unroll
      for (int i = 0; i < kPer; ++i)
        if (BN_ % 32 == 0 || lane < BN_) cp_async4(sc + 128u * i, p.sx + sx_off[i] + unsigned(kb) * p.sx_k);
      if (W_ROWS) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          cp_async4(sc + 4u * BN_ + 128u * i, p.sw + unsigned(min(tile * BM + lane + 32 * i, p.N - 1)) * p.sw_n + unsigned(kb) * p.sw_k);
      } else if (lane == 0) {
        cp_async4(sc + 4u * BN_, p.sw + unsigned(tile) * p.sw_n + unsigned(kb) * p.sw_k);
      }
      cp_async_arrive(fb);
      if (++s == C::stages) { s = 0; ph ^= 1u; }
      if (++kb == p.nkb) { kb = 0; ++tile; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp >= C::issuer_warp) {
    // columns of the MMA: the tokens there are, in sixteens
    const uint32_t n_mma = uint32_t((p.M + 15) / 16 * 16);
    const uint32_t idesc = (1u << 4) | (uint32_t(p.w_mn) << 15) | ((n_mma >> 3) << 17) | (uint32_t(BM >> 4) << 24);
    const uint32_t a_step = p.w_mn ? (UMMA_K * 128) >> 4 : UMMA_K >> 4, b_step = UMMA_K >> 4;
    const uint64_t desc_a0 = make_smem_desc(sbase), desc_b0 = make_smem_desc(sbase + kTileBytes);
    const uint32_t desc_hi = uint32_t(desc_a0 >> 32), a_lo0 = uint32_t(desc_a0), b_lo0 = uint32_t(desc_b0);
    const bool stage_lane = lane >= 16;
    uint32_t s = uint32_t(warp - C::issuer_warp), sph = 0, buf = s, bph = 1;
    bool ok = true;
    for (int u = u0 + int(s); u < u1; u += C::issuers) {
      const uint32_t bar = stage_lane ? full0 + 8u * s : tempty0 + 8u * buf;
      ok = __all_sync(0xffffffffu, mbar_wait(bar, stage_lane ? sph : bph, abort_flag, p.status, stage_lane ? 3u : 2u));
      if (!ok) break;
      __syncwarp();                  // (the vote is no memory barrier, and the elected lane has seen one of the two only)
      tc_fence_after();
      if (elect_one()) {
        const uint32_t d_tmem = tmem_base + buf * uint32_t(BN_), soff = s * uint32_t(C::stage_bytes >> 4);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_f8(d_tmem, (uint64_t(desc_hi) << 32) | (a_lo0 + soff + k * a_step), (uint64_t(desc_hi) << 32) | (b_lo0 + soff + k * b_step),
                  idesc, k > 0 ? 1u : 0u);
        umma_commit(tfull0 + 8u * buf);      // (the promotion warps, which see this, free the stage)
      }
      __syncwarp();
      if ((s += C::issuers) >= uint32_t(C::stages)) { s -= C::stages; sph ^= 1u; }
      if ((buf += C::issuers) >= uint32_t(C::bufs)) { buf -= C::bufs; bph ^= 1u; }
    }
    if (elect_one()) {
      umma_commit(drain_bar);
      mbar_wait(drain_bar, 0u, abort_flag, p.status, 4u);
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3, c0 = (warp >> 2) * C::cols, r = quarter * 32 + lane;
    const float* scales0 = reinterpret_cast<const float*>(smem + C::stages * C::stage_bytes);
    const uint32_t tcol0 = tmem_base + (uint32_t(quarter * 32) << 16) + uint32_t(c0);
    int kb = u0 % p.nkb, tile = u0 / p.nkb;
    float2 acc[C::cols / 2];
#pragma unroll
    for (int j = 0; j < C::cols / 2; ++j) acc[j] = make_float2(0.f, 0.f);
    uint32_t buf = 0, bph = 0, stage_s = 0, sph = 0;
    bool ok = true;
    for (int u = u0; u < u1; ++u) {
      const bool ends = kb + 1 == p.nkb || u + 1 == u1;              // the last block of this tile here
      const int tile_now = tile;
      if (++kb == p.nkb) { kb = 0; ++tile; }
      // the stage's scales (its barrier was complete before the MMAs were issued: the first probe succeeds)
      ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8u * stage_s, sph, abort_flag, p.status, 5u));
      if (!ok) break;
      const float* in = scales0 + stage_s * C::stage_scales;
      const float sw = in[BN_ + (W_ROWS ? r : 0)];
      const float2 sw2 = make_float2(sw, sw);
      // token factors of sixteen columns, times the weight's where that is one number
      float2 f[8];
      auto factors = [&](int q) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 sc = *reinterpret_cast<const float4*>(in + c0 + 16 * q + 4 * j);
          f[2 * j] = make_float2(sc.x, sc.y);
          f[2 * j + 1] = make_float2(sc.z, sc.w);
        }
        if (!W_ROWS) {
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = __fmul2_rn(f[j], sw2);
        }
      };
      factors(0);
      ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8u * buf, bph, abort_flag, p.status, 5u));
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tcol0 + buf * uint32_t(BN_);
#pragma unroll
      for (int q = 0; q < C::cols / 16; ++q) {
        uint32_t v[16];
        tmem_ld16(taddr + 16 * q, v);
        tmem_wait_ld16(v);
        if (q > 0) factors(q);
        if (q == C::cols / 16 - 1) {                                 // every sum of the buffer and every scale is in registers: hand both back
          tc_fence_before();
          __syncwarp();
          mbar_arrive_if(tempty0 + 8u * buf, lane == 0);
          mbar_arrive_if(empty0 + 8u * stage_s, lane == 0);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 pj = make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
          float2& a = acc[8 * q + j];
          a = W_ROWS ? __ffma2_rn(__fmul2_rn(pj, f[j]), sw2, a) : __ffma2_rn(pj, f[j], a);
        }
      }
      if (++stage_s == uint32_t(C::stages)) { stage_s = 0; sph ^= 1u; }
      if (++buf == C::bufs) { buf = 0; bph ^= 1u; }
      if (ends) {
        // (share > 0: this is the block's last unit, every stage has been read; the pipeline's shared memory becomes the slot)
        float* out = (p.share > 0 ? reinterpret_cast<float*>(smem) : p.ws + size_t(int(blockIdx.x) + tile_now) * size_t(p.M) * BM) + r;
        const bool row_ok = tile_now * BM + r < p.N;
#pragma unroll
        for (int j = 0; j < C::cols; ++j)
          if (row_ok && c0 + j < p.M) out[size_t(c0 + j) * BM] = (j & 1) ? acc[j / 2].y : acc[j / 2].x;
#pragma unroll
        for (int j = 0; j < C::cols / 2; ++j) acc[j] = make_float2(0.f, 0.f);
      }
    }
  }

  if (p.share > 0) {
    __syncwarp();
    cluster_sync();                      // every block's slot is written
    const int tile = int(blockIdx.x) / p.share, rank = int(blockIdx.x) - tile * p.share;
    const uint32_t base = smem_u32(smem);
    for (int i = rank * C::threads + int(threadIdx.x); i < p.M * (BM / 4); i += p.share * C::threads) {
      const int m = i / (BM / 4), n = tile * BM + (i % (BM / 4)) * 4;
      if (n >= p.N) continue;
      float4 a = ld_cluster_f32x4(base + uint32_t(i) * 16u, 0);
      for (int k = 1; k < p.share; ++k) {
        const float4 b = ld_cluster_f32x4(base + uint32_t(i) * 16u, k);
        a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
      }
      if (p.d_f32) *reinterpret_cast<float4*>(static_cast<float*>(p.d) + m * p.ldd + n) = a;
      else *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.d) + m * p.ldd + n) = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
    }
    cluster_sync();                      // nobody reads this block's shared memory any more
  }

  tc_fence_before();
  __syncthreads();
  if (warp == C::issuer_warp) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, C::tmem_cols);
  }
}

// D[m][n] = the sum of a tile's slots, in block order.  A thread makes four consecutive n of one token.
template <bool OUT_F32>
__global__ void __launch_bounds__(256)
skinny_reduce_kernel(const float* __restrict__ ws, void* __restrict__ d, int M, int N, long long ldd, int nkb, int units, int g) {
  const int i = int(blockIdx.x) * 256 + int(threadIdx.x), quads = (N + 3) / 4, m = i / quads, n = (i - m * quads) * 4;
  grid_trigger();
  grid_wait();
  ws = loads_below(ws);
  if (m >= M) return;
  const int tile = n / BM;
  const int c0 = skinny_block_of(tile * nkb, g, units), c1 = skinny_block_of(tile * nkb + nkb - 1, g, units);
  const float* src = ws + (size_t(c0 + tile) * M + m) * BM + (n - tile * BM);
  float4 a = __ldcg(reinterpret_cast<const float4*>(src));
  for (int c = c0 + 1; c <= c1; ++c) {
    src += size_t(M) * BM;
    const float4 b = __ldcg(reinterpret_cast<const float4*>(src));
    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
  }
  if (OUT_F32) *reinterpret_cast<float4*>(static_cast<float*>(d) + m * ldd + n) = a;
  else *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(d) + m * ldd + n) = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
}

// ---- host --------------------------------------------------------------------------------

// The activation must be [M][K] (it becomes the K-major B operand).  Below 512 of contraction or 256 of width the weight is
// nothing to stream and the tiled kernel's single launch is the shorter way.
bool skinny_takes(const tg_gemm_args* a) {
  if (a->M <= 0 || a->M > kSkinnyMaxTokens || a->a_major != TG_MAJOR_K || a->K % BK != 0 || a->K < 512 || a->N < 256 || a->N > (1 << 22) ||
      a->K > (1 << 22))
    return false;
  const bool columns = a->sb_gran_n == 1;
  const int64_t weights = a->K * a->N;
  if (a->M <= 32) {
    if (a->N > 512) return true;
    if (a->K < 3072) return a->K > 512 || a->M <= 16;
    return weights > 4 << 20 || (a->M > 20 && a->N > 448 && a->K > 3072 && a->K <= 4096);
  }
  if (a->N <= 512 && a->K <= 1024) return false;
  if (a->M <= 64) return a->K > (columns || a->N < 4096 ? 768 : 1024);
  if (a->K <= 1024 || columns) return a->K > 1024;
  if (a->N <= 2048 ? a->K <= 4608 : a->N <= 2560 && a->K > 1536 && a->K < 3072 && a->M < 128) return true;
  return weights > (a->M == 128 ? 19 << 20 : 26 << 20) && weights <= 32 << 20;
}

struct SkinnyPlan {
  int tiles, nkb, units, grid, share;
};

// Clusters of `size` blocks of this kernel that fit on the device together (an SM holds one block; GPCs are not multiples of
// every size).
static int clusters_that_fit(int size) {
  static std::atomic<int> known[64][5];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = known[dev][size].load(std::memory_order_relaxed);
  if (n == 0) {
    using C = SkinnyCfg<16>;
    auto kern = gemm_skinny_kernel<16, false>;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = unsigned(size);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(size) * 64u);
    cfg.blockDim = dim3(C::threads);
    cfg.dynamicSmemBytes = C::smem_bytes;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem_bytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = -1;
    }
    known[dev][size].store(n, std::memory_order_relaxed);
  }
  return n < 0 ? 0 : n;
}
static SkinnyPlan plan(const tg_gemm_args* a) {
  SkinnyPlan p;
  p.tiles = int((a->N + BM - 1) / BM);
  p.nkb = int(a->K / BK);
  p.units = p.tiles * p.nkb;
  const int sms = gemm_sms();
  p.grid = p.units < sms ? p.units : sms;
  // Ranges that end where tiles end (tiles * s blocks, s to a tile) read whole rows together and leave fewer slots; all SMs
  // (ranges that end anywhere) is the better balance.  In microseconds: 0.33 per unit on one SM (16 KB at 50 GB/s; 0.41 with
  // 128 tokens beside it), all units at the measured 5.0 / 4.5 TB/s, a slot written and read at ~6 TB/s.
  const double slot = double(a->M) * BM * 8 / 6.0e6, unit = a->M <= 64 ? 0.33 : 0.41;
  auto cost = [&](int g, int slots, double rate) {
    const double sm = unit * ((p.units + g - 1) / g), hbm = double(p.units) * kTileBytes / rate;
    return (sm > hbm ? sm : hbm) + slot * slots;
  };
  const int most = p.grid;
  double best = cost(most, most + p.tiles, 4.5e6);
  for (int s = 1; p.tiles * s <= most; ++s) {
    const double c = cost(p.tiles * s, p.tiles * s, 5.0e6);
    if (c < best) { best = c; p.grid = p.tiles * s; }
  }
  // A cluster per tile saves the second launch (about 2.5 us) and its slots' way through memory.
  p.share = 0;
  if (p.tiles >= 32) {
    best += 2.5;
    for (int s = 1; s <= 4 && s <= p.nkb && p.tiles * s <= most; ++s) {
      const double c = cost(p.tiles * s, 0, 5.0e6);
      if (c < best && (s == 1 || clusters_that_fit(s) >= p.tiles)) { best = c; p.grid = p.tiles * s; p.share = s; }
    }
  }
  return p;
}

int64_t skinny_workspace_bytes(const tg_gemm_args* a) {
  const SkinnyPlan p = plan(a);
  if (p.share > 0) return 0;
  return int64_t(p.grid + p.tiles) * a->M * BM * int64_t(sizeof(float));
}

template <int BN_, bool W_ROWS>
static int launch(const tg_gemm_args* a, const SkinnyPlan& pl, SkinnyParams p, cudaStream_t st) {
  using C = SkinnyCfg<BN_>;
  auto kern = gemm_skinny_kernel<BN_, W_ROWS>;
  CUtensorMap tw, tx;
  const int64_t w_inner = p.w_mn ? a->N : a->K, w_outer = p.w_mn ? a->K : a->N;
  if (int rc = make_tmap(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->b, w_inner, w_outer, a->ldb, 128, 128)) return rc;
  if (int rc = make_tmap(&tx, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a->a, a->K, a->M, a->lda, 128, BN_)) return rc;
  static std::atomic<bool> attr_set[64];
  int dev = 0;
  TG_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return TG_ERR_SHAPE;
  if (!attr_set[dev].load(std::memory_order_acquire)) {
    TG_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem_bytes));
    attr_set[dev].store(true, std::memory_order_release);
  }
  TG_CUDA_CHECK(launch_early_clusters(kern, pl.share > 1 ? pl.share : 1, pl.grid, C::threads, C::smem_bytes, st, tw, tx, p));
  return TG_OK;
}

int skinny_run(const tg_gemm_args* a, cudaStream_t st) {
  const SkinnyPlan pl = plan(a);
  SkinnyParams p;
  p.sx = a->sa; p.sx_m = unsigned(a->sa_stride_m); p.sx_k = unsigned(a->sa_stride_kb);
  p.sw = a->sb; p.sw_n = unsigned(a->sb_stride_n); p.sw_k = unsigned(a->sb_stride_kb);
  p.ws = static_cast<float*>(a->workspace);
  p.M = int(a->M); p.N = int(a->N); p.nkb = pl.nkb;
  p.units = pl.units;
  p.w_mn = a->b_major == TG_MAJOR_MN;
  p.share = pl.share;
  p.d = a->d; p.ldd = static_cast<long long>(a->ldd); p.d_f32 = a->out_dtype == TG_OUT_F32;
  p.status = a->status;
  const bool rows = a->sb_gran_n == 1;
  int rc;
  if (a->M <= 16) rc = rows ? launch<16, true>(a, pl, p, st) : launch<16, false>(a, pl, p, st);
  else if (a->M <= 32) rc = rows ? launch<32, true>(a, pl, p, st) : launch<32, false>(a, pl, p, st);
  else if (a->M <= 64) rc = rows ? launch<64, true>(a, pl, p, st) : launch<64, false>(a, pl, p, st);
  else rc = rows ? launch<128, true>(a, pl, p, st) : launch<128, false>(a, pl, p, st);
  if (rc != TG_OK || pl.share > 0) return rc;
  const int64_t threads = a->M * ((a->N + 3) / 4);
  const int blocks = int((threads + 255) / 256);
  if (a->out_dtype == TG_OUT_F32)
    TG_CUDA_CHECK(launch_early(skinny_reduce_kernel<true>, blocks, 256, 0, st, static_cast<const float*>(p.ws), a->d, p.M, p.N,
                               static_cast<long long>(a->ldd), p.nkb, p.units, pl.grid));
  else
    TG_CUDA_CHECK(launch_early(skinny_reduce_kernel<false>, blocks, 256, 0, st, static_cast<const float*>(p.ws), a->d, p.M, p.N,
                               static_cast<long long>(a->ldd), p.nkb, p.units, pl.grid));
  return TG_OK;
}

}  // namespace tg
