// RMSNorm forward (optionally fused with the 1x128 e4m3 quantiser) and backward.
//
// Reference semantics: train-gpt kernels.py:44-53 (+ the variance pass at :66) for the
// fused single-rounding norm, kernels.py:30-33 for the "pure" three-rounding norm,
// kernels.py:104-118 for the backward, fp8.py:39-47 + :66 for the quantiser that consumes
// the norm's bf16 output.
//
// Layout: a row is split over WPR warps (norm_geom, bwd_geom); each warp owns
// NCHUNK chunks of 256 columns and each lane 8 consecutive columns (one 128-bit load) per chunk, so a half-warp owns
// exactly one 128-column quantisation tile.  The row stays on the SM (registers or shared memory) between the
// sum-of-squares pass and the normalise/quantise pass: x is read from HBM once.
#include <cstdlib>

#include <atomic>

#include <algorithm>

#include "common.cuh"
#include "host_api.h"

namespace tg {

constexpr int kNormWarps = 8;  // warps per thread block


// Sum of squares of the 8 bf16 values in w, as a balanced tree (keeps the rounding error of
// a row's variance at a few 2^-24 regardless of outliers).
__device__ __forceinline__ float sumsq8(const uint4& w) {
  const float2 v0 = bf16x2_unpack(w.x), v1 = bf16x2_unpack(w.y), v2 = bf16x2_unpack(w.z), v3 = bf16x2_unpack(w.w);
  const float2 t = __fadd2_rn(__ffma2_rn(v2, v2, __fmul2_rn(v0, v0)), __ffma2_rn(v3, v3, __fmul2_rn(v1, v1)));
  return t.x + t.y;
}

template <int N>
__device__ __forceinline__ float tree_sum(float (&v)[N]) {
#pragma unroll
  for (int stride = 1; stride < N; stride *= 2)
#pragma unroll
    for (int i = 0; i + stride < N; i += 2 * stride) v[i] += v[i + stride];
  return v[0];
}

// Sum over the lanes of a warp and, where a row has several, over its WPR warps in order.  `red` holds one float per warp of
// the block and alternates between two buffers from row to row: a warp writes one only after its group's barrier of the row
// before, which every warp of the group reaches after reading the other.
template <int WPR>
__device__ __forceinline__ float row_sum(float v, float* red, int warp, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if constexpr (WPR > 1) {
    if (lane == 0) red[warp] = v;
    asm volatile("bar.sync %0, %1;" ::"r"(1 + warp / WPR), "n"(WPR * 32) : "memory");   // this row's warps only
    const int g0 = (warp / WPR) * WPR;
    v = red[g0];
#pragma unroll
    for (int i = 1; i < WPR; ++i) v += red[g0 + i];
  }
  return v;
}

// Plain norm of rows that one warp holds in registers.
template <int NCHUNK, bool PURE>
__global__ void __launch_bounds__(kNormWarps * 32, 3)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma,
                   float eps, __nv_bfloat16* __restrict__ y, float* __restrict__ rnorm_out, int64_t rows, int cols) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col_base = lane * 8;

  // gamma lives in shared memory, already widened to float (one conversion per block
  // instead of one per row), not in registers, so that more blocks fit on an SM
  extern __shared__ float4 s_gamma[];
  for (int i = threadIdx.x; i < cols / 8; i += blockDim.x) {
    const uint4 gq = reinterpret_cast<const uint4*>(gamma)[i];
    s_gamma[2 * i] = make_float4(bf16lo(gq.x), bf16hi(gq.x), bf16lo(gq.y), bf16hi(gq.y));
    s_gamma[2 * i + 1] = make_float4(bf16lo(gq.z), bf16hi(gq.z), bf16lo(gq.w), bf16hi(gq.w));
  }
  __syncthreads();

  for (int64_t row = int64_t(blockIdx.x) * kNormWarps + warp; row < rows; row += int64_t(gridDim.x) * kNormWarps) {
    uint4 w[NCHUNK];
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      const int col = col_base + c * 256;
      w[c] = col < cols ? ld_stream_v4(x + row * cols + col) : make_uint4(0, 0, 0, 0);
    }
    float part[NCHUNK];
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) part[c] = sumsq8(w[c]);
    const float ss = row_sum<1>(tree_sum(part), nullptr, warp, lane);
    const float rn = __frsqrt_rn(__fdiv_rn(ss, float(cols)) + eps);
    if (rnorm_out != nullptr && lane == 0) rnorm_out[row] = rn;
    const float rn_b = __bfloat162float(__float2bfloat16_rn(rn));  // kernels.py:32 `.astype(x.dtype)`
    const float2 rn2 = PURE ? make_float2(rn_b, rn_b) : make_float2(rn, rn);
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      const int col = col_base + c * 256;
      if (col >= cols) continue;
      const uint32_t xi[4] = {w[c].x, w[c].y, w[c].z, w[c].w};
      const float4 g0 = s_gamma[col >> 2], g1 = s_gamma[(col >> 2) + 1];
      const float2 gf[4] = {make_float2(g0.x, g0.y), make_float2(g0.z, g0.w), make_float2(g1.x, g1.y), make_float2(g1.z, g1.w)};
      uint4 yo;
      uint32_t* yp = &yo.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 t = __fmul2_rn(bf16x2_unpack(xi[j]), rn2);
        if (PURE) t = bf16x2_unpack(pack_bf16x2(t.x, t.y));   // kernels.py:32 rounds before the gamma multiply
        t = __fmul2_rn(t, gf[j]);
        yp[j] = pack_bf16x2(t.x, t.y);
      }
      *reinterpret_cast<uint4*>(y + row * cols + col) = yo;
    }
  }
}

// ---------------------------------------------------------------------------------------
// Norm (+ quantise) staged through shared memory: fused forms, and every form of rows wider than 2048 columns.  A
// register-resident kernel needs ~120 registers at 2048 columns per warp, so only
// 16 warps fit on an SM and every warp idles while its next row's loads are in flight.  Here
// each warp owns two slots of shared memory for its part of a row: cp.async fetches row i+1 into one
// slot while the warp makes its passes (sum of squares; normalise + amax; divide + store) over row i in the other.  A lane
// only ever touches the 16-byte pieces it fetched itself, so cp.async.wait_group is the only
// synchronisation within a warp; the warps of a wide row meet once, at the sum.
// Wide rows, register-resident -> staged, microseconds (DRAM floor): 3001 x 4096 plain 12.2 -> 9.0 (7.5), quantised 14.6 -> 10.9
// (5.7); 4096 x 8192 29.7 -> 22.3 (20.5), 32.3 -> 24.6 (15.5); 16384 x 8192 quantised 110.7 -> 84.7 (62).  Eight warps per row of
// four chunks, or gamma in registers and a third slot, were no better (3001 x 4096 10.5, 4096 x 8192 25.4 and 29.7).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

constexpr int staged_blocks(int wpr) { return wpr == 1 ? 3 : 2; }      // per SM: 72 KB each up to 2048 columns, 80-96 beyond
constexpr int pow2_at_least(int n) { return n <= 1 ? 1 : 2 * pow2_at_least((n + 1) / 2); }

// ADD: the row that is normalised is bf16(x + res) -- the residual add of model.py:68 / :72 folded into
// the norm that follows it -- and is also written to `sum_out` (the new residual stream); `res` rows
// are staged beside the x rows and the sum replaces the x row in shared memory before the first pass.
// q may be NULL: then only y is produced (the plain norm, or with ADD the final norm, which has no quantised consumer).
template <int NCHUNK, bool PURE, bool FULL, bool ADD = false, int WPR = 1>
__global__ void __launch_bounds__(kNormWarps * 32, staged_blocks(WPR))
rmsnorm_quant_staged_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma,
                            float eps, uint8_t* __restrict__ q, float* __restrict__ scales,
                            __nv_bfloat16* __restrict__ y, float* __restrict__ rnorm_out, int64_t rows,
                            int cols, const __nv_bfloat16* __restrict__ res = nullptr,
                            __nv_bfloat16* __restrict__ sum_out = nullptr) {
  constexpr int RPB = kNormWarps / WPR;  // rows in work per block
  __shared__ float s_red[2][kNormWarps];
  constexpr int kRowBytes = NCHUNK * 512;
  constexpr int kSlotBytes = ADD ? 2 * kRowBytes : kRowBytes;     // x row (then: the sum), res row
  extern __shared__ float4 s_gamma[];   // [cols] floats, then [warps][2][slot] bf16
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col_base = (warp % WPR) * (NCHUNK * 256) + lane * 8;
  const uint32_t slot0 = uint32_t(__cvta_generic_to_shared(s_gamma)) + uint32_t(cols) * 4u +
                         uint32_t(warp) * 2u * kSlotBytes + uint32_t(lane) * 16u;

  // gamma widened to float in two planes (columns 8i..8i+3 of every 8-column piece, then columns
  // 8i+4..8i+7): a warp's 16-byte reads of either plane are contiguous, hence conflict-free
  const int pieces = cols / 8;
  grid_trigger();
  grid_wait();
  gamma = loads_below(gamma);
  for (int i = threadIdx.x; i < pieces; i += blockDim.x) {
    const uint4 gq = reinterpret_cast<const uint4*>(gamma)[i];
    s_gamma[i] = make_float4(bf16lo(gq.x), bf16hi(gq.x), bf16lo(gq.y), bf16hi(gq.y));
    s_gamma[pieces + i] = make_float4(bf16lo(gq.z), bf16hi(gq.z), bf16lo(gq.w), bf16hi(gq.w));
  }
  __syncthreads();

  const int64_t stride = int64_t(gridDim.x) * RPB;
  int64_t row = int64_t(blockIdx.x) * RPB + warp / WPR;
  auto prefetch = [&](int64_t r, int slot) {
    if (r < rows) {
#pragma unroll
      for (int c = 0; c < NCHUNK; ++c) {
        const int col = col_base + c * 256;
        if (FULL || col < cols) {
          cp_async16(slot0 + slot * kSlotBytes + c * 512, x + r * cols + col);
          if (ADD) cp_async16(slot0 + slot * kSlotBytes + kRowBytes + c * 512, res + r * cols + col);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");   // an empty group keeps the wait count uniform
  };
  prefetch(row, 0);
  for (int it = 0; row < rows; row += stride, ++it) {
    const uint32_t base = slot0 + (it & 1) * kSlotBytes;
    prefetch(row + stride, (it & 1) ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");

    if (ADD) {
      // the residual add, one rounding to bf16 as the elementwise add it replaces
#pragma unroll
      for (int c = 0; c < NCHUNK; ++c) {
        const int col = col_base + c * 256;
        if (FULL || col < cols) {
          const uint4 a = lds128(base + c * 512), b = lds128(base + kRowBytes + c * 512);
          const uint32_t ai[4] = {a.x, a.y, a.z, a.w}, bi[4] = {b.x, b.y, b.z, b.w};
          uint4 o;
          uint32_t* op = &o.x;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 t = __fadd2_rn(bf16x2_unpack(ai[j]), bf16x2_unpack(bi[j]));
            op[j] = pack_bf16x2(t.x, t.y);
          }
          sts128(base + c * 512, o);
          *reinterpret_cast<uint4*>(sum_out + row * cols + col) = o;
        }
      }
    }

    // pass 1: sum of squares
    float part[NCHUNK];
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) part[c] = (FULL || col_base + c * 256 < cols) ? sumsq8(lds128(base + c * 512)) : 0.f;
    const float ss = row_sum<WPR>(tree_sum(part), s_red[it & 1], warp, lane);
    const float var = __fdiv_rn(ss, float(cols));
    const float rn = __frsqrt_rn(var + eps);
    if (rnorm_out != nullptr && lane == 0 && warp % WPR == 0) rnorm_out[row] = rn;
    const float rn_b = __bfloat162float(__float2bfloat16_rn(rn));  // kernels.py:32 `.astype(x.dtype)`

    // pass 2: normalise, round to bf16 (the value the reference's norm returns), per-tile amax; one exchange brings lane j
    // of each half the amax of chunk j % G, that lane computes the tile's scale and
    // reciprocal, shuffles hand them to the lanes that need them; divide and store.
    const float2 rn2 = PURE ? make_float2(rn_b, rn_b) : make_float2(rn, rn);
    constexpr int G = pow2_at_least(NCHUNK);     // (the exchange wants a power of two; chunks past NCHUNK are constant zeros)
    uint4 yo[NCHUNK];
    uint32_t amax_bits[G];
#pragma unroll
    for (int u = NCHUNK; u < G; ++u) amax_bits[u] = 0u;
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      const int col = col_base + c * 256;
      amax_bits[c] = 0u;
      yo[c] = make_uint4(0u, 0u, 0u, 0u);
      if (FULL || col < cols) {
        const uint4 xv = lds128(base + c * 512);
        const uint32_t xi[4] = {xv.x, xv.y, xv.z, xv.w};
        const float4 g0 = s_gamma[col >> 3], g1 = s_gamma[pieces + (col >> 3)];
        const float2 gf[4] = {make_float2(g0.x, g0.y), make_float2(g0.z, g0.w), make_float2(g1.x, g1.y), make_float2(g1.z, g1.w)};
        uint32_t* yp = &yo[c].x;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 t = __fmul2_rn(bf16x2_unpack(xi[j]), rn2);
          if (PURE) t = bf16x2_unpack(pack_bf16x2(t.x, t.y));   // kernels.py:32 rounds before the gamma multiply
          t = __fmul2_rn(t, gf[j]);
          yp[j] = pack_bf16x2(t.x, t.y);
        }
        if (y != nullptr) *reinterpret_cast<uint4*>(y + row * cols + col) = yo[c];
        amax_bits[c] = absmax8_h(yo[c]);
      }
    }
    if (q == nullptr) continue;
    float s[G], r[G], s_mine;
    bool fin;
    tile_scales_own<G>(exchange_tile_amax<G>(amax_bits), s, r, s_mine, fin);
    {
      const int j = lane & 15;
      const int col = col_base - lane * 8 + j * 256 + (lane & 16) * 8;     // first column of the tile this lane computed
      if (j < NCHUNK && (FULL || col < cols)) scales[row * (cols / kTile) + col / kTile] = s_mine;
    }
    uint8_t* qp = q + row * cols + col_base;
    if (fin) {   // one branch: a NaN or Inf in any of the warp's tiles is the rare case
#pragma unroll
      for (int c = 0; c < NCHUNK; ++c)
        if (FULL || col_base + c * 256 < cols) *reinterpret_cast<uint2*>(qp + c * 256) = quantize8_sr(yo[c], s[c], r[c]);
    } else {
#pragma unroll
      for (int c = 0; c < NCHUNK; ++c)
        if (FULL || col_base + c * 256 < cols) *reinterpret_cast<uint2*>(qp + c * 256) = quantize8(yo[c], s[c]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---------------------------------------------------------------------------------------
// Backward.  Per row: S1 = sum x^2, rnorm = rsqrt(S1/D + eps), normed = x*rnorm,
// gs = g*gamma, dot = mean(gs*normed), dx = rnorm*(gs - normed*dot); per column:
// dgamma = sum_rows g*normed, accumulated per lane in registers over all rows the block
// visits, combined across the block's warps in shared memory, written as one float32 row
// of `partial` per block and reduced over blocks (in block order) by a second kernel.
//
// Staged through shared memory: register-resident it kept x, g and 8 column sums per 16-byte piece live at
// once (246 registers at 2048 columns per warp: one block of eight warps per SM, each idle while its
// next row is in flight; 55 % of the copy bandwidth).  Here each warp owns SLOTS
// pairs of slots for its part of a row and cp.async keeps SLOTS - 1 rows of x and g in flight
// while one is processed: x goes to registers once, g is read from shared memory in the column-sum pass and again in
// the dx pass, gamma sits in shared memory widened to float.  Every lane reads only the
// 16-byte pieces it fetched itself, so cp.async.wait_group is the only synchronisation within a warp; the warps of a wide row
// meet at its two sums.  Wide rows, register-resident -> staged, microseconds (DRAM floor): 3001 x 4096 33.1 -> 19.6 (11.2),
// 16384 x 8192 232.6 -> 135.9 (122.8), 4096 x 2304 35.0 -> 17.0 (8.6), 8192 x 6144 111.8 -> 56.8 (46).
// ---------------------------------------------------------------------------------------
// ADD: dx = bf16(addend + the norm's input gradient) -- the gradient fan-in at a residual junction (the
// skip path's gradient plus the branch's) folded into the kernel, one rounding instead of two.
template <int NCHUNK, int WARPS, int SLOTS, bool FULL, bool ADD = false, int WPR = 1>
__global__ void __launch_bounds__(WARPS * 32, 1)
rmsnorm_bwd_staged_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma,
                          const __nv_bfloat16* __restrict__ g, float eps, __nv_bfloat16* __restrict__ dx,
                          float* __restrict__ partial, int64_t rows, int cols,
                          const __nv_bfloat16* __restrict__ addend = nullptr) {
  constexpr int kRowBytes = NCHUNK * 512, RPB = WARPS / WPR;      // a warp's part of a row; rows in work per block
  __shared__ float s_red[2][2][WARPS];
  extern __shared__ float4 s_gamma[];   // [cols] floats in two planes, then [warps][SLOTS][x row | g row] bf16
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col_base = (warp % WPR) * (NCHUNK * 256) + lane * 8;
  const uint32_t stage0 = uint32_t(__cvta_generic_to_shared(s_gamma)) + uint32_t(cols) * 4u;
  const uint32_t slot0 = stage0 + uint32_t(warp) * uint32_t(SLOTS * 2 * kRowBytes) + uint32_t(lane) * 16u;
  const float inv_d = __fdiv_rn(1.0f, float(cols));

  const int pieces = cols / 8;
  grid_wait();
  gamma = loads_below(gamma);
  for (int i = threadIdx.x; i < pieces; i += blockDim.x) {
    const uint4 gq = reinterpret_cast<const uint4*>(gamma)[i];
    s_gamma[i] = make_float4(bf16lo(gq.x), bf16hi(gq.x), bf16lo(gq.y), bf16hi(gq.y));
    s_gamma[pieces + i] = make_float4(bf16lo(gq.z), bf16hi(gq.z), bf16lo(gq.w), bf16hi(gq.w));
  }
  __syncthreads();

  float2 acc[NCHUNK][4];
#pragma unroll
  for (int c = 0; c < NCHUNK; ++c)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[c][j] = make_float2(0.f, 0.f);

  const int64_t stride = int64_t(gridDim.x) * RPB;
  int64_t row = int64_t(blockIdx.x) * RPB + warp / WPR;
  // the addend's row, for which shared memory has no room, comes as far as the L2 (GB/s at 32768 rows without -> with it: 2048
  // columns 5860 -> 6000, 1280 5390 -> 5520, 512 4570 -> 4650; 1024 5480 -> 5400)
  constexpr bool kFetchAddend = ADD && NCHUNK != 4;
  auto prefetch = [&](int64_t r, int slot) {
    if (r < rows) {
      const uint32_t dst = slot0 + uint32_t(slot) * 2u * kRowBytes;
#pragma unroll
      for (int c = 0; c < NCHUNK; ++c) {
        const int col = col_base + c * 256;
        if (FULL || col < cols) {
          cp_async16(dst + c * 512, x + r * cols + col);
          cp_async16(dst + kRowBytes + c * 512, g + r * cols + col);
        }
      }
      if (kFetchAddend) {
        const int col = col_base + lane * 56;                            // a line of 128 bytes per lane
        if (lane < NCHUNK * 4 && col < cols) asm volatile("prefetch.global.L2 [%0];" ::"l"(addend + r * cols + col) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");   // an empty group keeps the wait count uniform
  };
  // SLOTS - 1 rows are in flight while one is processed
#pragma unroll
  for (int d = 0; d < SLOTS - 1; ++d) prefetch(row + d * stride, d);
  int slot = 0, slot_in = SLOTS - 1;
  for (int it = 0; row < rows; row += stride, ++it) {
    const uint32_t xs = slot0 + uint32_t(slot) * 2u * kRowBytes, gs = xs + kRowBytes;
    prefetch(row + (SLOTS - 1) * stride, slot_in);    // into the slot the previous iteration finished with
    asm volatile("cp.async.wait_group %0;" ::"n"(SLOTS - 1) : "memory");
    slot_in = slot;
    if (++slot == SLOTS) slot = 0;

    uint4 w[NCHUNK];
    float part[NCHUNK];
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      w[c] = (FULL || col_base + c * 256 < cols) ? lds128(xs + c * 512) : make_uint4(0, 0, 0, 0);
      part[c] = sumsq8(w[c]);
    }
    const float ss = row_sum<WPR>(tree_sum(part), s_red[it & 1][0], warp, lane);
    const float rn = __frsqrt_rn(__fdiv_rn(ss, float(cols)) + eps);
    const float2 rn2 = make_float2(rn, rn);

    // (ADD) the addend's first pieces are fetched here, ahead of the pass that uses them, as many as there are registers for;
    // the rest that many pieces ahead of their use, and always before a store: dx may alias the addend, so a load that
    // follows a store in the program waits its turn (32768 x 2048: 90 us, and 165 with each piece fetched where it is used)
    constexpr int kAhead = !ADD ? 1 : NCHUNK < 4 ? NCHUNK : 4;
    uint4 ad[kAhead];
    auto fetch_addend = [&](int c) {
      return FULL || col_base + c * 256 < cols ? ld_stream_v4(addend + row * cols + col_base + c * 256) : make_uint4(0, 0, 0, 0);
    };
    if constexpr (ADD) {
#pragma unroll
      for (int c = 0; c < kAhead; ++c) ad[c] = fetch_addend(c);
    }

    // column sums of g * normed, and gs * normed summed over the row
    float dpart[NCHUNK];
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      float dsum = 0.f;
      const int col = col_base + c * 256;
      if (FULL || col < cols) {
        const uint4 gv = lds128(gs + c * 512);
        const float4 m0 = s_gamma[col >> 3], m1 = s_gamma[pieces + (col >> 3)];
        const float2 mf[4] = {make_float2(m0.x, m0.y), make_float2(m0.z, m0.w), make_float2(m1.x, m1.y), make_float2(m1.z, m1.w)};
        const uint32_t xi[4] = {w[c].x, w[c].y, w[c].z, w[c].w};
        const uint32_t gi[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 n2 = __fmul2_rn(bf16x2_unpack(xi[j]), rn2), g2 = bf16x2_unpack(gi[j]);
          acc[c][j] = __ffma2_rn(g2, n2, acc[c][j]);
          const float2 gm = __fmul2_rn(g2, mf[j]);
          dsum = fmaf(gm.x, n2.x, dsum);
          dsum = fmaf(gm.y, n2.y, dsum);
        }
      }
      dpart[c] = dsum;
    }
    const float dsum = row_sum<WPR>(tree_sum(dpart), s_red[it & 1][1], warp, lane);
    const float dot = __fmul_rn(dsum, inv_d);
    const float2 ndot2 = make_float2(-dot, -dot);

    // (no instruction: stops the compiler from keeping the 8 * NCHUNK normalised values of the pass
    // above alive for the pass below, which costs more registers than recomputing them)
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) asm volatile("" : "+r"(w[c].x), "+r"(w[c].y), "+r"(w[c].z), "+r"(w[c].w));
#pragma unroll
    for (int c = 0; c < NCHUNK; ++c) {
      const int col = col_base + c * 256;
      if (!(FULL || col < cols)) continue;
      const uint4 gv = lds128(gs + c * 512);
      const float4 m0 = s_gamma[col >> 3], m1 = s_gamma[pieces + (col >> 3)];
      const float2 mf[4] = {make_float2(m0.x, m0.y), make_float2(m0.z, m0.w), make_float2(m1.x, m1.y), make_float2(m1.z, m1.w)};
      const uint32_t xi[4] = {w[c].x, w[c].y, w[c].z, w[c].w};
      const uint32_t gi[4] = {gv.x, gv.y, gv.z, gv.w};
      uint4 av = make_uint4(0, 0, 0, 0);
      if constexpr (ADD) {
        av = ad[c % kAhead];
        if (c + kAhead < NCHUNK) ad[c % kAhead] = fetch_addend(c + kAhead);
      }
      const uint32_t ai[4] = {av.x, av.y, av.z, av.w};
      uint4 o;
      uint32_t* op = &o.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 n2 = __fmul2_rn(bf16x2_unpack(xi[j]), rn2), gm = __fmul2_rn(bf16x2_unpack(gi[j]), mf[j]);
        // rnorm * (gs - normed*dot), the subtraction fused as kernels.py:114 allows XLA to
        float2 d = __fmul2_rn(rn2, __ffma2_rn(n2, ndot2, gm));
        // (scalar: a packed add of a packed product is contracted into one fma, which rounds the sum once instead of
        // twice -- another last bit, that the e4m3 roundings further down a backward pass amplify)
        if constexpr (ADD) {
          const float2 a2 = bf16x2_unpack(ai[j]);
          d = make_float2(__fadd_rn(d.x, a2.x), __fadd_rn(d.y, a2.y));
        }
        op[j] = pack_bf16x2(d.x, d.y);
      }
      *reinterpret_cast<uint4*>(dx + row * cols + col) = o;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");

  grid_trigger();          // the reduction's blocks may take the places of this kernel's as they leave
  // combine the block's rows in order over the (now idle) staging area, then publish the
  // block's row of partial column sums
  __syncthreads();
  float* s_sum = reinterpret_cast<float*>(s_gamma) + cols;
  for (int i = threadIdx.x; i < cols; i += blockDim.x) s_sum[i] = 0.f;
  __syncthreads();
  for (int turn = 0; turn < RPB; ++turn) {
    if (warp / WPR == turn) {
#pragma unroll
      for (int c = 0; c < NCHUNK; ++c) {
        const int col = col_base + c * 256;
        if (FULL || col < cols) {
          float4* dst = reinterpret_cast<float4*>(s_sum + col);
          float4 a = dst[0], b = dst[1];
          a.x += acc[c][0].x; a.y += acc[c][0].y; a.z += acc[c][1].x; a.w += acc[c][1].y;
          b.x += acc[c][2].x; b.y += acc[c][2].y; b.z += acc[c][3].x; b.w += acc[c][3].y;
          dst[0] = a; dst[1] = b;
        }
      }
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < cols; i += blockDim.x) partial[int64_t(blockIdx.x) * cols + i] = s_sum[i];
}

// Column sums of the per-block partials.  A thread block owns 32 columns.  The order of additions is fixed by (n_blocks, cols)
// alone: row class w = b mod 8 has four sums, the i-th over b = w + 8 i, w + 8 i + 32, ..., the rows left over when a class's
// groups of four are complete go to its first; the four are added in pairs, the eight classes in order.  Warp w + 8 i keeps the i-th
// sum of class w and has all of its (at most seven) loads in flight at once: with eight warps of four sums each the kernel was
// a chain of five L2 round trips, 5.2 us at 2048 columns.
// The norms of a step can be finished together (row y of the grid is job y): alone each is a launch of 2 us, 49 of them in a step
// of 24 layers.
// A launch hands over one job or room for 64: the kilobyte of parameters is 0.3 to 0.7 us of host time, for which a norm by itself has
// no use (64 x 2048 forward and backward, a loop of calls: 14.2 to 14.6 us with it, 13.9 without).
constexpr int kDgammaJobs = 64;
template <int N>
struct DgammaJobs {
  tgh_dgamma_job job[N];
};
template <int N>
__global__ void __launch_bounds__(1024) rmsnorm_dgamma_reduce_kernel(const __grid_constant__ DgammaJobs<N> jobs, int n_blocks, int cols) {
  __shared__ float s_part[32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + lane;
  const float* partial = static_cast<const float*>(jobs.job[blockIdx.y].partial);
  __nv_bfloat16* dgamma = static_cast<__nv_bfloat16*>(jobs.job[blockIdx.y].dgamma);
  grid_wait();
  float t = 0.f;
  if (col < cols) {
    const int w = warp & 7;
    const int groups = n_blocks >= w + 25 ? (n_blocks - w - 25) / 32 + 1 : 0;      // complete groups of four rows of class w
    const float* p = partial + int64_t(warp) * cols + col;
    const int b = w + 32 * groups;                                                  // at most three rows are left
    float v[4], u[3];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = i < groups ? __ldcg(p + int64_t(i) * 32 * cols) : 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) u[i] = warp < 8 && b + 8 * i < n_blocks ? __ldcg(partial + int64_t(b + 8 * i) * cols + col) : 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) t += v[i];                                          // (x + 0 is x)
    for (int k = 4; k < groups; ++k) t += __ldcg(p + int64_t(k) * 32 * cols);       // (a GPU of more than 160 SMs)
#pragma unroll
    for (int i = 0; i < 3; ++i) t += u[i];
  }
  s_part[warp][lane] = t;
  __syncthreads();
  if (warp == 0 && col < cols) {
    t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const float u = (s_part[w][lane] + s_part[w + 8][lane]) + (s_part[w + 16][lane] + s_part[w + 24][lane]);
      t = w == 0 ? u : t + u;
    }
    dgamma[col] = __float2bfloat16_rn(t);
  }
}

// ---------------------------------------------------------------------------------------
// Forward for few rows (a decode batch): one thread block per row, one 16-byte piece per thread.  The kernels above give a row
// to one to four warps, which is right when there are rows to fill the GPU with; for a few the time is one warp's chain of
// loads and passes over 8 KB and more of row, plus widening gamma into shared memory.  16 x 8192: 5.0 -> 2.5 us, 1 x 2048: 3.1 -> 1.5.
// The sum of squares is added in the order of those kernels (a lane's pieces of every 256 columns as a tree, eight of them to
// a warp, then the lanes, then the warps), so which of them runs does not show in the result.
// Launched early (see common.cuh): in a decode loop the kernel before it is the last GEMM's reduction.
// ---------------------------------------------------------------------------------------
// chunk: pieces of 256 columns in a warp's tree (a power of two), groups: warps per row in the kernels above
template <bool QUANT, bool PURE>
__global__ void __launch_bounds__(1024)
rmsnorm_row_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gamma, float eps, uint8_t* __restrict__ q,
                   float* __restrict__ scales, __nv_bfloat16* __restrict__ y, float* __restrict__ rnorm_out, int cols, int chunks, int groups) {
  __shared__ float s_part[32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col = int(threadIdx.x) * 8;
  const int64_t row = blockIdx.x;
  grid_trigger();
  grid_wait();
  gamma = loads_below(gamma);              // (in a training step the optimiser's kernel, not far ahead, writes it)
  const bool ok = col < cols;
  const uint4 w = ok ? ld_stream_v4(x + row * cols + col) : make_uint4(0, 0, 0, 0);
  const uint4 gq = ok ? *reinterpret_cast<const uint4*>(gamma + col) : make_uint4(0, 0, 0, 0);
  s_part[warp][lane] = sumsq8(w);
  __syncthreads();
  const int warps = int(blockDim.x >> 5);
  auto group_sum = [&](int g) {
    float v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = c < chunks && g * chunks + c < warps ? s_part[g * chunks + c][lane] : 0.f;
    float s = tree_sum(v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
  };
  // One group: every warp adds it up for itself.  Two to four: a warp each, and one more barrier (all warps through all groups were
  // 1024 shared-memory reads of an 8192-wide row: 16 x 8192 3.4 us, now 2.5).
  float ss;
  if (groups == 1) {
    ss = group_sum(0);
  } else {
    __shared__ float s_group[4];
    if (warp < groups) {
      const float s = group_sum(warp);
      if (lane == 0) s_group[warp] = s;
    }
    __syncthreads();
    ss = s_group[0];
    for (int g = 1; g < groups; ++g) ss += s_group[g];
  }
  const float rn = __frsqrt_rn(__fdiv_rn(ss, float(cols)) + eps);
  if (rnorm_out != nullptr && threadIdx.x == 0) rnorm_out[row] = rn;
  const float rn_b = __bfloat162float(__float2bfloat16_rn(rn));  // kernels.py:32 `.astype(x.dtype)`
  const float2 rn2 = PURE ? make_float2(rn_b, rn_b) : make_float2(rn, rn);
  const uint32_t xi[4] = {w.x, w.y, w.z, w.w}, gi[4] = {gq.x, gq.y, gq.z, gq.w};
  uint4 yo;
  uint32_t* yp = &yo.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 t = __fmul2_rn(bf16x2_unpack(xi[j]), rn2);
    if (PURE) t = bf16x2_unpack(pack_bf16x2(t.x, t.y));   // kernels.py:32 rounds before the gamma multiply
    t = __fmul2_rn(t, bf16x2_unpack(gi[j]));
    yp[j] = pack_bf16x2(t.x, t.y);
  }
  if (y != nullptr && ok) *reinterpret_cast<uint4*>(y + row * cols + col) = yo;
  if constexpr (QUANT) {
    uint32_t m = absmax8(yo);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) m = __vmaxu2(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float s = scale_from_amax(absmax_to_float(m));
    if (ok) {
      *reinterpret_cast<uint2*>(q + row * cols + col) = quantize8(yo, s);
      if ((lane & 15) == 0) scales[row * (cols / kTile) + col / kTile] = s;
    }
  }
}
// Where the two meet (graph replays, microseconds with the quantiser, this kernel / the ones above): 1023 x 1024 3.0 / 3.8, 2047 x 1024 3.8 / 3.9
// but without the quantiser 3.3 / 2.9; 1023 x 2048 3.8 / 5.2, 1447 x 2048 4.6 / 5.8, 2047 x 2048 5.9 / 6.0; 681 x 3072 3.6 / 4.3, 964 x 3072
// 4.7 / 4.4; 511 x 4096 3.7 / 4.7, 723 x 4096 4.6 / 4.8 and 3.5 / 4.4; 255 x 8192 3.9 / 5.1, 361 x 8192 5.5 / 5.3; narrower rows fill warps of their own
// (2895 x 512 4.0 / 3.0).  Beyond 4096 columns an SM holds three blocks or two, and a second round of them is the slower way: 444 x 4608 0.85 times as
// long, 455 1.08; 296 x 6144 0.92, 341 x 6144 5.2 / 4.6.
static bool few_rows(int64_t rows, int64_t cols) {
  if (cols <= 4096) return rows * cols <= (cols < 1536 ? 1 << 20 : cols <= 2048 ? 3 << 20 : 1 << 21);
  const int64_t threads = (cols / 8 + 31) / 32 * 32;
  return rows <= 2048 / threads * sm_count() && rows * cols <= 1 << 21;
}

struct NormGeom {
  int nchunk, wpr;
};

// Forward.  Rows of up to 2048 columns: one warp, 1, 2, 4 or 8 chunks.  Wider ones: two or four warps with 5 to 8 chunks each, as
// many as the row needs (rounded up to eight, 2304 columns would be 2048 in one warp and 256 in the other).
static bool norm_geom(int64_t cols, NormGeom* g) {
  if (cols <= 0 || cols > 8192) return false;
  const int chunks = int((cols + 255) / 256);
  g->wpr = chunks <= 8 ? 1 : chunks <= 16 ? 2 : 4;
  g->nchunk = g->wpr == 1 ? pow2_at_least(chunks) : (chunks + g->wpr - 1) / g->wpr;
  return true;
}
// Backward.  Sixteen warps of 3 or 4 chunks where a row fits them evenly: more warps hide the row's two sums better than eight of
// twice the width (32768 x 1296: 51.8 us against 58.4).  Rows of 7 and 8 chunks stay with one warp (74 us at 32768 x 2048
// either way); above 6144 columns eight warps per row of four chunks spill (16384 x 8192 173 us), so four of 7 or 8.
static bool bwd_geom(int64_t cols, NormGeom* g) {
  if (cols <= 0 || cols > 8192) return false;
  const int chunks = int((cols + 255) / 256);
  g->wpr = chunks <= 4 ? 1 : chunks <= 6 ? 2 : chunks <= 8 ? 1 : chunks <= 16 ? 4 : chunks <= 24 ? 8 : 4;
  g->nchunk = g->wpr == 1 ? pow2_at_least(chunks) : (chunks + g->wpr - 1) / g->wpr;
  return true;
}

static int norm_blocks(int64_t rows, int wpr, int per_sm) {
  const int rpb = kNormWarps / wpr;
  int64_t need = (rows + rpb - 1) / rpb;
  const int64_t cap = int64_t(sm_count()) * per_sm;
  return int(need < cap ? need : cap);
}

// Dynamic shared memory of `bytes` for `kern`, once per device.
template <typename K>
static int allow_smem(K kern, int bytes, std::atomic<bool> (&done)[64]) {
  int dev = 0;
  TG_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return TG_ERR_SHAPE;
  if (!done[dev].load(std::memory_order_acquire)) {
    TG_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    done[dev].store(true, std::memory_order_release);
  }
  return TG_OK;
}

struct NormFwd {
  const __nv_bfloat16 *x, *gamma, *res;
  float eps;
  uint8_t* q;
  float* scales;
  __nv_bfloat16* y;
  float* rnorm;
  int64_t rows;
  int cols;
  __nv_bfloat16* sum_out;
};

template <int NC, bool PURE, bool FULL, bool ADD, int WPR>
static int launch_staged(const NormFwd& a, cudaStream_t st) {
  static std::atomic<bool> done[64];
  auto kern = rmsnorm_quant_staged_kernel<NC, PURE, FULL, ADD, WPR>;
  constexpr int slots = kNormWarps * 2 * NC * 512 * (ADD ? 2 : 1);
  if (int rc = allow_smem(kern, WPR * NC * 1024 + slots, done)) return rc;
  // early at every size: one wave of blocks, whose set-up then hides (32768 x 2048, forward and backward: 116.8 -> 113.8 us)
  TG_CUDA_CHECK(launch_early(kern, norm_blocks(a.rows, WPR, staged_blocks(WPR)), kNormWarps * 32, a.cols * 4 + slots, st, a.x, a.gamma, a.eps, a.q, a.scales,
                             a.y, a.rnorm, a.rows, a.cols, a.res, a.sum_out));
  return TG_OK;
}
template <bool ADD>
static int launch_staged(const NormGeom& g, bool pure, const NormFwd& a, cudaStream_t st) {
  const bool full = a.cols == g.wpr * g.nchunk * 256;   // no ragged chunk: the column guards compile away
#define TG_STAGED_CASE(NC, W)                                                                                  \
  if (g.nchunk == NC && g.wpr == W)                                                                            \
    return pure ? (full ? launch_staged<NC, true, true, ADD, W>(a, st) : launch_staged<NC, true, false, ADD, W>(a, st)) \
                : (full ? launch_staged<NC, false, true, ADD, W>(a, st) : launch_staged<NC, false, false, ADD, W>(a, st));
  TG_STAGED_CASE(1, 1) TG_STAGED_CASE(2, 1) TG_STAGED_CASE(4, 1) TG_STAGED_CASE(8, 1)
  if constexpr (!ADD) {
    TG_STAGED_CASE(5, 2) TG_STAGED_CASE(6, 2) TG_STAGED_CASE(7, 2) TG_STAGED_CASE(8, 2)
    TG_STAGED_CASE(5, 4) TG_STAGED_CASE(6, 4) TG_STAGED_CASE(7, 4) TG_STAGED_CASE(8, 4)
  }
#undef TG_STAGED_CASE
  return TG_ERR_SHAPE;
}

template <bool QUANT>
static int launch_fwd(const void* x, const void* gamma, float eps, void* q, float* scales, void* y,
                      float* rnorm, int64_t rows, int64_t cols, int mode, cudaStream_t st) {
  NormGeom g;
  if (!norm_geom(cols, &g)) return cols > 8192 ? TG_ERR_TOO_LARGE : TG_ERR_SHAPE;
  if (few_rows(rows, cols)) {
    auto kern = mode == TG_NORM_PURE ? rmsnorm_row_kernel<QUANT, true> : rmsnorm_row_kernel<QUANT, false>;
    TG_CUDA_CHECK(launch_early(kern, int(rows), int((cols / 8 + 31) / 32 * 32), 0, st, static_cast<const __nv_bfloat16*>(x),
                               static_cast<const __nv_bfloat16*>(gamma), eps, static_cast<uint8_t*>(q), scales,
                               static_cast<__nv_bfloat16*>(y), rnorm, int(cols), g.nchunk, g.wpr));
    return TG_OK;
  }
  const NormFwd a = {static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(gamma), nullptr, eps, static_cast<uint8_t*>(q),
                     scales, static_cast<__nv_bfloat16*>(y), rnorm, rows, int(cols), nullptr};
  if (QUANT || g.wpr > 1) return launch_staged<false>(g, mode == TG_NORM_PURE, a, st);
  const int blocks = norm_blocks(rows, 1, 16);
#define TG_FWD_CASE(NC)                                                                                       \
  if (g.nchunk == NC) {                                                                                       \
    auto kern = mode == TG_NORM_PURE ? rmsnorm_fwd_kernel<NC, true> : rmsnorm_fwd_kernel<NC, false>;          \
    kern<<<blocks, kNormWarps * 32, size_t(cols) * 4, st>>>(a.x, a.gamma, eps, a.y, rnorm, rows, int(cols)); \
  } else
  TG_FWD_CASE(1) TG_FWD_CASE(2) TG_FWD_CASE(4) TG_FWD_CASE(8) { return TG_ERR_SHAPE; }
#undef TG_FWD_CASE
  TG_CUDA_CHECK(cudaGetLastError());
  return TG_OK;
}

// One block per SM with up to 192 KB of slots.
constexpr int bwd_warps(int nchunk, int wpr) { return nchunk > 4 ? 8 : nchunk == 4 && wpr == 1 ? 12 : 16; }
constexpr int bwd_slots(int nchunk, int wpr) { return nchunk > 4 || (nchunk == 4 && wpr > 1) ? 3 : 4; }

static int bwd_blocks(int64_t rows, const NormGeom& g) {
  const int rpb = bwd_warps(g.nchunk, g.wpr) / g.wpr;
  const int64_t need = (rows + rpb - 1) / rpb, cap = sm_count();
  return int(need < cap ? need : cap);
}

struct NormBwd {
  const __nv_bfloat16 *x, *gamma, *g, *addend;
  float eps;
  __nv_bfloat16* dx;
  float* partial;
  int64_t rows;
  int cols, blocks;
};
template <int NC, bool FULL, bool ADD, int WPR>
static int launch_bwd(const NormBwd& a, cudaStream_t st) {
  static std::atomic<bool> done[64];
  constexpr int warps = bwd_warps(NC, WPR), slots = bwd_slots(NC, WPR), stage = warps * slots * 2 * NC * 512;
  static_assert(WPR * NC * 1024 + stage + 256 <= 227 * 1024, "row slots exceed shared memory");
  auto kern = rmsnorm_bwd_staged_kernel<NC, warps, slots, FULL, ADD, WPR>;
  if (int rc = allow_smem(kern, WPR * NC * 1024 + stage, done)) return rc;
  TG_CUDA_CHECK(launch_early(kern, a.blocks, warps * 32, a.cols * 4 + stage, st, a.x, a.gamma, a.g, a.eps, a.dx, a.partial, a.rows, a.cols,
                             a.addend));
  return TG_OK;
}
static int launch_bwd(const NormGeom& g, const NormBwd& a, cudaStream_t st) {
  const bool full = a.cols == g.wpr * g.nchunk * 256, add = a.addend != nullptr;
#define TG_BWD_CASE(NC, W)                                                                          \
  if (g.nchunk == NC && g.wpr == W) {                                                               \
    if constexpr (W <= 2) {                                                                         \
      if (add) return full ? launch_bwd<NC, true, true, W>(a, st) : launch_bwd<NC, false, true, W>(a, st); \
    }                                                                                               \
    return full ? launch_bwd<NC, true, false, W>(a, st) : launch_bwd<NC, false, false, W>(a, st);   \
  }
  TG_BWD_CASE(1, 1) TG_BWD_CASE(2, 1) TG_BWD_CASE(4, 1) TG_BWD_CASE(8, 1) TG_BWD_CASE(3, 2)
  TG_BWD_CASE(3, 4) TG_BWD_CASE(4, 4) TG_BWD_CASE(3, 8) TG_BWD_CASE(7, 4) TG_BWD_CASE(8, 4)
#undef TG_BWD_CASE
  return TG_ERR_SHAPE;
}

}  // namespace tg

using namespace tg;

extern "C" int tg_rmsnorm_fwd(const void* x, const void* gamma, float eps, void* y, float* rnorm,
                              int64_t rows, int64_t cols, int mode, void* stream) {
  if (rows < 0 || cols <= 0 || cols % 8 != 0 || (mode != TG_NORM_FUSED && mode != TG_NORM_PURE)) return TG_ERR_SHAPE;
  if (rows == 0) return TG_OK;
  if (!aligned16(x) || !aligned16(gamma) || !aligned16(y)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  return launch_fwd<false>(x, gamma, eps, nullptr, nullptr, y, rnorm, rows, cols, mode,
                           static_cast<cudaStream_t>(stream));
}

extern "C" int tg_rmsnorm_quant_fwd(const void* x, const void* gamma, float eps, void* q,
                                    float* scales, void* y, float* rnorm, int64_t rows,
                                    int64_t cols, int mode, void* stream) {
  if (rows < 0 || cols <= 0 || cols % kTile != 0 || (mode != TG_NORM_FUSED && mode != TG_NORM_PURE)) return TG_ERR_SHAPE;
  if (rows == 0) return TG_OK;
  if (!aligned16(x) || !aligned16(gamma) || !aligned16(q) || !aligned16(y)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  return launch_fwd<true>(x, gamma, eps, q, scales, y, rnorm, rows, cols, mode,
                          static_cast<cudaStream_t>(stream));
}

extern "C" int tg_add_rmsnorm_quant_fwd(const void* x, const void* res, const void* gamma, float eps, void* sum_out,
                                        void* q, float* scales, void* y, float* rnorm, int64_t rows, int64_t cols,
                                        int mode, void* stream) {
  if (rows < 0 || cols <= 0 || cols % kTile != 0 || (mode != TG_NORM_FUSED && mode != TG_NORM_PURE)) return TG_ERR_SHAPE;
  if (x == nullptr || res == nullptr || sum_out == nullptr || (q == nullptr) != (scales == nullptr)) return TG_ERR_SHAPE;
  if (q == nullptr && y == nullptr) return TG_ERR_SHAPE;
  if (rows == 0) return TG_OK;
  if (!aligned16(x) || !aligned16(res) || !aligned16(gamma) || !aligned16(q) || !aligned16(y) || !aligned16(sum_out)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  NormGeom g;
  if (!norm_geom(cols, &g)) return cols > 8192 ? TG_ERR_TOO_LARGE : TG_ERR_SHAPE;
  if (g.wpr != 1) return TG_ERR_TOO_LARGE;      // rows one warp holds (cols <= 2048): the staged kernel
  const NormFwd a = {static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(gamma), static_cast<const __nv_bfloat16*>(res), eps,
                     static_cast<uint8_t*>(q), scales, static_cast<__nv_bfloat16*>(y), rnorm, rows, int(cols),
                     static_cast<__nv_bfloat16*>(sum_out)};
  return launch_staged<true>(g, mode == TG_NORM_PURE, a, static_cast<cudaStream_t>(stream));
}

extern "C" int64_t tg_rmsnorm_bwd_scratch_bytes(int64_t rows, int64_t cols) {
  NormGeom g;
  if (rows <= 0 || !bwd_geom(cols, &g)) return 0;
  return int64_t(bwd_blocks(rows, g)) * cols * int64_t(sizeof(float));
}

template <int N>
static int reduce_dgamma_up_to(const tgh_dgamma_job* jobs, int n, int blocks, int cols, cudaStream_t st) {
  DgammaJobs<N> a = {};
  std::copy(jobs, jobs + n, a.job);
  TG_CUDA_CHECK(launch_if_short(true, rmsnorm_dgamma_reduce_kernel<N>, dim3(unsigned((cols + 31) / 32), unsigned(n)), 1024, 0, st, a, blocks, cols));
  return TG_OK;
}
static int reduce_dgamma(const tgh_dgamma_job* jobs, int n, int blocks, int cols, cudaStream_t st) {
  if (n == 1) return reduce_dgamma_up_to<1>(jobs, 1, blocks, cols, st);
  for (int i = 0; i < n; i += kDgammaJobs)
    if (int rc = reduce_dgamma_up_to<kDgammaJobs>(jobs + i, std::min(n - i, kDgammaJobs), blocks, cols, st)) return rc;
  return TG_OK;
}

// (dgamma NULL: up to the partial sums; the public calls below refuse it)
static int rmsnorm_bwd_impl(const void* x, const void* gamma, const void* g, const void* addend, float eps, void* dx,
                            void* dgamma, void* scratch, int64_t rows, int64_t cols, void* stream) {
  if (rows < 0 || cols <= 0 || cols % 8 != 0) return TG_ERR_SHAPE;
  NormGeom geo;
  if (!bwd_geom(cols, &geo)) return cols > 8192 ? TG_ERR_TOO_LARGE : TG_ERR_SHAPE;
  if (addend != nullptr && cols > 2048) return TG_ERR_TOO_LARGE;   // the fused add exists for rows one warp holds
  if (!aligned16(x) || !aligned16(gamma) || !aligned16(g) || !aligned16(dx) || !aligned16(scratch) || !aligned16(addend))
    return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (rows == 0) {
    if (dgamma != nullptr) TG_CUDA_CHECK(cudaMemsetAsync(dgamma, 0, size_t(cols) * 2, st));
    return TG_OK;
  }
  const int blocks = bwd_blocks(rows, geo);
  const NormBwd a = {static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(gamma), static_cast<const __nv_bfloat16*>(g),
                     static_cast<const __nv_bfloat16*>(addend), eps, static_cast<__nv_bfloat16*>(dx), static_cast<float*>(scratch), rows,
                     int(cols), blocks};
  if (int rc = launch_bwd(geo, a, st)) return rc;
  if (dgamma == nullptr) return TG_OK;
  const tgh_dgamma_job job = {scratch, dgamma};
  return reduce_dgamma(&job, 1, blocks, int(cols), st);
}

extern "C" int tg_rmsnorm_bwd(const void* x, const void* gamma, const void* g, float eps, void* dx,
                              void* dgamma, void* scratch, int64_t rows, int64_t cols, void* stream) {
  if (dgamma == nullptr) return TG_ERR_SHAPE;
  return rmsnorm_bwd_impl(x, gamma, g, nullptr, eps, dx, dgamma, scratch, rows, cols, stream);
}

extern "C" int tg_rmsnorm_bwd_add(const void* x, const void* gamma, const void* g, const void* addend, float eps,
                                  void* dx, void* dgamma, void* scratch, int64_t rows, int64_t cols, void* stream) {
  if (addend == nullptr || dgamma == nullptr) return TG_ERR_SHAPE;
  return rmsnorm_bwd_impl(x, gamma, g, addend, eps, dx, dgamma, scratch, rows, cols, stream);
}

extern "C" int tgh_rmsnorm_bwd_parts(const void* x, const void* gamma, const void* g, const void* addend, float eps, void* dx, void* partial,
                                     int64_t rows, int64_t cols, void* stream) {
  return rmsnorm_bwd_impl(x, gamma, g, addend, eps, dx, nullptr, partial, rows, cols, stream);
}

extern "C" int tgh_norm_few_rows(int64_t rows, int64_t cols) { return few_rows(rows, cols); }

extern "C" int tgh_dgamma_reduce(const tgh_dgamma_job* jobs, int n, int64_t rows, int64_t cols, void* stream) {
  NormGeom g;
  if (rows <= 0 || cols <= 0 || !bwd_geom(cols, &g)) return TG_ERR_SHAPE;
  if (int rc = check_arch()) return rc;
  return reduce_dgamma(jobs, n, bwd_blocks(rows, g), int(cols), static_cast<cudaStream_t>(stream));
}

// ---------------------------------------------------------------------------------------
// Norm backward for callers that may not allocate device memory.
//
// tg_rmsnorm_bwd wants a scratch buffer from its caller.  Some hosts of this library have
// nowhere to get one: an XLA custom-call handler receives only the buffers the compiler
// planned for it, and the reference's launchers hand XLA 90 % of the device up front
// (XLA_PYTHON_CLIENT_MEM_FRACTION=0.9, train-gpt bench_fp8_norm.py:64), so a cudaMalloc
// from inside the handler can fail outright or stall the stream it synchronises with.
// For them the partial column sums live in a fixed array inside the library image.  Every
// GPU that loads the library carries these 4 MiB until the process exits.
// ---------------------------------------------------------------------------------------
namespace tg {
constexpr int64_t kStaticBwdScratchBytes = 4ll << 20;
static __device__ __align__(256) unsigned char g_bwd_scratch[kStaticBwdScratchBytes];
}  // namespace tg

extern "C" int64_t tg_rmsnorm_bwd_static_max_scratch_bytes(void) { return tg::kStaticBwdScratchBytes; }

extern "C" int tg_rmsnorm_bwd_static(const void* x, const void* gamma, const void* g, float eps,
                                     void* dx, void* dgamma, int64_t rows, int64_t cols, void* stream) {
  // In host code `g_bwd_scratch` is only a handle for the runtime, not an address a kernel
  // can use; the device address is looked up once per device, with that device current.
  static std::atomic<void*> dev_ptr[64] = {};   // written once per device; host threads may race to be first
  if (rows < 0 || cols <= 0 || cols % 8 != 0 || dgamma == nullptr) return TG_ERR_SHAPE;
  const int64_t need = tg_rmsnorm_bwd_scratch_bytes(rows, cols);
  if (need > tg::kStaticBwdScratchBytes) {
    // message for tg_last_cuda_error(): the size limit is the caller's to handle
    tg::record_cuda_error(cudaErrorInvalidValue,
                          "tg_rmsnorm_bwd_static: rows x cols needs more than the 4 MiB built-in scratch; "
                          "use tg_rmsnorm_bwd with a caller-owned buffer");
    return TG_ERR_TOO_LARGE;
  }
  int dev = 0;
  TG_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return TG_ERR_SHAPE;
  void* scratch = dev_ptr[dev].load(std::memory_order_acquire);
  if (scratch == nullptr) {
    TG_CUDA_CHECK(cudaGetSymbolAddress(&scratch, tg::g_bwd_scratch));
    dev_ptr[dev].store(scratch, std::memory_order_release);  // racing first calls on one device store the same value
  }
  return tg_rmsnorm_bwd(x, gamma, g, eps, dx, dgamma, scratch, rows, cols, stream);
}
