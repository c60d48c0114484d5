// e4m3 quantisers with float32 amax/448 scales (train-gpt fp8.py:39-47), three tile
// shapes.  All are HBM-bound streaming kernels: 2 bytes in, 1 byte + 4/128 byte out per
// element, every input byte read once with 128-bit loads and kept in registers between
// the amax pass and the divide pass.
#include "common.cuh"
#include "host_api.h"

namespace tg {

// ---------------------------------------------------------------------------------------
// 1 x 128 tiles.  cols % 128 == 0, so tile t is the 256 contiguous bytes at x + 256 t and
// its scale is scales[t].  Sixteen lanes own a tile (16 B = 8 values each); each thread
// keeps kUnroll independent tiles in flight.
// ---------------------------------------------------------------------------------------
constexpr int kRowUnroll = 4;
constexpr int kRowThreads = 256;

__global__ void __launch_bounds__(kRowThreads)
quantize_rowwise_kernel(const uint4* __restrict__ x, uint2* __restrict__ q,
                        float* __restrict__ scales, int64_t n_tiles) {
  const int lane16 = threadIdx.x & 15;
  const int64_t group = (int64_t(blockIdx.x) * kRowThreads + threadIdx.x) >> 4;  // half-warp id
  const int64_t n_groups = (int64_t(gridDim.x) * kRowThreads) >> 4;
  for (int64_t t0 = group * kRowUnroll; t0 < n_tiles; t0 += n_groups * kRowUnroll) {
    uint4 w[kRowUnroll];
#pragma unroll
    for (int u = 0; u < kRowUnroll; ++u) {
      const int64_t t = t0 + u;
      w[u] = (t < n_tiles) ? ld_stream_v4(x + t * 16 + lane16) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < kRowUnroll; ++u) {
      float m = amax8(w[u]);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) m = max_nan(m, __shfl_xor_sync(0xffffffffu, m, o));
      const float s = scale_from_amax(m);
      const int64_t t = t0 + u;
      if (t < n_tiles) {
        q[t * 16 + lane16] = quantize8(w[u], s);
        if (lane16 == 0) scales[t] = s;
      }
    }
  }
}

// ---------------------------------------------------------------------------------------
// Panels: what needs a scale per column per 128 rows (128 x 1 tiles), per 128 x 128 tile, or the 1 x 128 form beside
// either.  A thread block owns a 128-row x 128-column panel: a half-warp spans the 128 columns (16 lanes x 8
// columns), so each of the 16 half-warps owns every 16th row (8 rows per thread, kept in registers).
// Column maxima are combined across the warps through shared memory (one thread per column
// finishes the reduction and the reciprocal), then the same registers are divided and stored.
// 64 registers: four blocks per SM, so one block's loads overlap the others' arithmetic.
// ---------------------------------------------------------------------------------------
constexpr int kColPanelCols = 128;
constexpr int kColThreads = 256;
constexpr int kColHalfWarps = kColThreads / 16;           // 16
constexpr int kColRowsPerThread = kTile / kColHalfWarps;  // 8

// Activation folded into the load (ACT != TG_ACT_NONE): the tile that is quantised is
//   relu2      bf16( max(x,0)^2 )                         model.py:72, `jax.nn.relu(h) ** 2`
//   gelu       bf16( x/2 (1 + erf(x/sqrt 2)) )            the activation the benchmark's training configuration names
//   relu2_bwd  bf16( gate * 2 max(x,0) )                  the cotangent of relu2 for upstream gradient `gate`
//   gelu_bwd   bf16( gate * (Phi(x) + x phi(x)) )
// each computed in float32 from the bf16 input(s) and rounded to bf16 ONCE, which is what the
// unfused composition (an elementwise bf16 kernel, then the quantiser) would have handed over.
// The MLP's activation and its gradient are then never written to memory.
// erf(x / sqrt 2) as sign(x) (1 - 2^P(|x|)): P is the degree-9 polynomial (no constant term) fitted to
// log2 erfc(a / sqrt 2) on a in [0, 6.08] with weight erfc, so that the ABSOLUTE error of erfc is 2e-9
// everywhere -- which is what the float32 forms below can see: they add the result to 1.  One
// special-function instruction and ten multiply-adds, against libdevice erff's two branches of that
// size.  Rounded to bf16, x/2 (1 + erf) from this routine and from a correctly rounded erff agree for
// every finite bf16 x in exact float32 arithmetic; the approximate ex2 flips a bf16 ulp on about one
// element in ten thousand.
__device__ __forceinline__ float erf_of_x_over_sqrt2(float x) {
  const float a = fminf(fabsf(x), 6.081118f);       // erfc is 1.2e-9 there: 1 - that is 1
  float p = 5.117859700476401e-07f;
  p = fmaf(p, a, -9.538196536595933e-06f);
  p = fmaf(p, a, 7.480611384380609e-05f);
  p = fmaf(p, a, -0.0002837043721228838f);
  p = fmaf(p, a, 1.3612322618428152e-05f);
  p = fmaf(p, a, 0.006932816002517939f);
  p = fmaf(p, a, -0.05243593826889992f);
  p = fmaf(p, a, -0.4592210352420807f);
  p = fmaf(p, a, -1.1511043310165405f);
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(p * a));
  return copysignf(1.0f - e, x);
}

template <int ACT>
__device__ __forceinline__ float act_value(float x, float gate) {
  if (ACT == TG_ACT_RELU2) { const float r = fmaxf(x, 0.f); return r * r; }
  if (ACT == TG_ACT_RELU2_BWD) return gate * (2.f * fmaxf(x, 0.f));
  if (ACT == TG_ACT_GELU) return x * 0.5f * (1.f + erf_of_x_over_sqrt2(x));
  if (ACT == TG_ACT_GELU_BWD) {
    const float cdf = 0.5f * (1.f + erf_of_x_over_sqrt2(x));
    const float pdf = expf(-0.5f * x * x) * 0.39894228040143267794f;
    return gate * (cdf + x * pdf);
  }
  return x;
}
// The same erf for two arguments at once in packed f32x2 instructions (the kernel is bound by instruction
// issue, and the polynomial is most of the activation's instructions); same operations in the same order
// as the scalar routine, so the same bits.  (Forward form 0.201 -> 0.184 ms at 32768 x 4096; backward form, with the density as a
// packed product and two ex2 instead of two expf, 0.268 -> 0.234 ms.)
__device__ __forceinline__ float2 erf_of_x_over_sqrt2_pair(float2 x) {
  const float2 a = make_float2(fminf(fabsf(x.x), 6.081118f), fminf(fabsf(x.y), 6.081118f));
  auto c2 = [](float c) { return make_float2(c, c); };
  float2 p = c2(5.117859700476401e-07f);
  p = __ffma2_rn(p, a, c2(-9.538196536595933e-06f));
  p = __ffma2_rn(p, a, c2(7.480611384380609e-05f));
  p = __ffma2_rn(p, a, c2(-0.0002837043721228838f));
  p = __ffma2_rn(p, a, c2(1.3612322618428152e-05f));
  p = __ffma2_rn(p, a, c2(0.006932816002517939f));
  p = __ffma2_rn(p, a, c2(-0.05243593826889992f));
  p = __ffma2_rn(p, a, c2(-0.4592210352420807f));
  p = __ffma2_rn(p, a, c2(-1.1511043310165405f));
  const float2 t = __fmul2_rn(p, a);
  float2 e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(t.x));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(t.y));
  const float2 r = __ffma2_rn(e, c2(-1.0f), c2(1.0f));       // 1 - e, exact product
  return make_float2(copysignf(r.x, x.x), copysignf(r.y, x.y));
}

template <int ACT>
__device__ __forceinline__ uint32_t act_pair(uint32_t x2, uint32_t g2) {
  if constexpr (ACT == TG_ACT_GELU) {
    const float2 x = bf16x2_unpack(x2);
    const float2 one_plus = __fadd2_rn(make_float2(1.f, 1.f), erf_of_x_over_sqrt2_pair(x));
    const float2 y = __fmul2_rn(__fmul2_rn(x, make_float2(0.5f, 0.5f)), one_plus);
    return pack_bf16x2(y.x, y.y);
  } else if constexpr (ACT == TG_ACT_GELU_BWD) {
    const float2 x = bf16x2_unpack(x2), gate = bf16x2_unpack(g2);
    const float2 cdf = __fmul2_rn(make_float2(0.5f, 0.5f), __fadd2_rn(make_float2(1.f, 1.f), erf_of_x_over_sqrt2_pair(x)));
    // the density: 2^(-x^2 log2(e) / 2) / sqrt(2 pi); x^2 is exact (a bf16 squared), the product is rounded once
    const float2 t = __fmul2_rn(__fmul2_rn(x, x), make_float2(-0.72134752044448170f, -0.72134752044448170f));
    float2 pdf;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(pdf.x) : "f"(t.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(pdf.y) : "f"(t.y));
    pdf = __fmul2_rn(pdf, make_float2(0.39894228040143267794f, 0.39894228040143267794f));
    const float2 y = __fmul2_rn(gate, __ffma2_rn(x, pdf, cdf));
    return pack_bf16x2(y.x, y.y);
  } else {
    return pack_bf16x2(act_value<ACT>(bf16lo(x2), bf16lo(g2)), act_value<ACT>(bf16hi(x2), bf16hi(g2)));
  }
}
template <int ACT>
__device__ __forceinline__ uint4 act_apply(uint4 x, uint4 g) {
  return make_uint4(act_pair<ACT>(x.x, g.x), act_pair<ACT>(x.y, g.y), act_pair<ACT>(x.z, g.z), act_pair<ACT>(x.w, g.w));
}

// The second form of a panel beside (or instead of) its 1 x 128 one.
enum PanelForm { kNoForm = 0, kColForm = 1, kBlockForm = 2 };

struct PanelJob {
  const __nv_bfloat16* x;      // rows x cols, pitch ld
  const __nv_bfloat16* gate;   // same layout; read by the *_BWD activations only
  uint8_t* q_row;              // 1 x 128 form, or NULL
  float* s_row;
  uint8_t* q;                  // column or block form
  float* s;
  int64_t ld, q_row_ld, s_row_ld, q_ld, s_ld;
  int rows, cols;
  int out_cols;                // columns of the column form: >= cols, a multiple of 8; the extra ones are zeros
  int tiles_x;                 // panels across
  int first;                   // number of the job's first thread block
  int form;                    // PanelForm
};

struct PanelSmem {
  float max[kColThreads / 32][kColPanelCols];
  __align__(16) float scale[kColPanelCols];
  __align__(16) float rcp[kColPanelCols];
};

// Eight consecutive values of a row of which the first `valid` exist, at any alignment.
__device__ __forceinline__ uint4 load8_ragged(const __nv_bfloat16* p, int valid) {
  uint32_t v[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (j < valid) v[j >> 1] |= uint32_t(reinterpret_cast<const unsigned short*>(p)[j]) << (16 * (j & 1));
  return make_uint4(v[0], v[1], v[2], v[3]);
}

// FULL: the panel lies wholly inside the tensor (all 128 rows, all 128 columns, rows at 16-byte boundaries), the case of
// every block of a launch whose sizes are multiples of 128: no bounds predicate is evaluated and row addresses are
// one 64-bit add apart.  (The kernel is bound by instruction issue; the per-opcode counters showed the
// address arithmetic and the bounds branches of the general form to be a third of its instructions.)
// RAGGED: rows at any alignment, any number of columns (column form only).
template <bool ROW, int FORM, int ACT, bool FULL, bool RAGGED = false>
__device__ __forceinline__ void panel(const PanelJob& a, int bx, int by, PanelSmem& sm) {
  const int cx = threadIdx.x & 15, hw = threadIdx.x >> 4;
  const int col0 = bx * kColPanelCols + cx * 8;
  const int64_t row0 = int64_t(by) * kTile + hw;     // this thread's rows: row0 + 16 r
  const int64_t rows = a.rows;

  uint4 w[kColRowsPerThread];
  {
    const __nv_bfloat16* xp = a.x + row0 * a.ld + col0;
    const __nv_bfloat16* gp = a.gate + row0 * a.ld + col0;     // only dereferenced by the *_BWD variants
    const int64_t step = int64_t(kColHalfWarps) * a.ld;
#pragma unroll
    for (int r = 0; r < kColRowsPerThread; ++r, xp += step, gp += step) {
      const bool ok = FULL || row0 + r * kColHalfWarps < rows;
      if constexpr (RAGGED) w[r] = load8_ragged(xp, ok ? a.cols - col0 : 0);
      else w[r] = FULL || (ok && col0 < a.cols) ? ld_stream_v4(xp) : make_uint4(0, 0, 0, 0);
      if constexpr (ACT != TG_ACT_NONE) {
        uint4 g = make_uint4(0, 0, 0, 0);
        if constexpr (ACT == TG_ACT_RELU2_BWD || ACT == TG_ACT_GELU_BWD)
          if (ok) g = ld_stream_v4(gp);
        w[r] = act_apply<ACT>(w[r], g);   // rows past the end stay zero: every variant maps (0, 0) to 0
      }
    }
  }
  if constexpr (ROW) {   // cols % 128 == 0 here: every lane holds real columns
    // the 8 row tiles of a half-warp: one exchange leaves lane j with the amax of row j % 8
    uint32_t mr[kColRowsPerThread];
#pragma unroll
    for (int r = 0; r < kColRowsPerThread; ++r) mr[r] = absmax8_h(w[r]);
    float sr[kColRowsPerThread], rr[kColRowsPerThread], s_mine;
    bool fin;
    tile_scales_own<kColRowsPerThread>(exchange_tile_amax<kColRowsPerThread>(mr), sr, rr, s_mine, fin);
    {
      const int64_t row = row0 + int64_t(cx & 7) * kColHalfWarps;   // lane j of the half computed row r = j % 8
      if (cx < kColRowsPerThread && (FULL || row < rows)) a.s_row[row * a.s_row_ld + bx] = s_mine;
    }
    uint8_t* qp = a.q_row + row0 * a.q_row_ld + col0;
    const int64_t step = int64_t(kColHalfWarps) * a.q_row_ld;
    // one branch around the whole loop, not one per row: a NaN or Inf anywhere in the warp's tiles is the rare case
    if (fin) {
#pragma unroll
      for (int r = 0; r < kColRowsPerThread; ++r, qp += step)
        if (FULL || row0 + r * kColHalfWarps < rows) *reinterpret_cast<uint2*>(qp) = quantize8_sr(w[r], sr[r], rr[r]);
    } else {
#pragma unroll
      for (int r = 0; r < kColRowsPerThread; ++r, qp += step)
        if (FULL || row0 + r * kColHalfWarps < rows) *reinterpret_cast<uint2*>(qp) = quantize8(w[r], sr[r]);
    }
  }
  if constexpr (FORM == kNoForm) return;
  uint32_t m2[4];  // packed |.|-maxima of column pairs (0,1) (2,3) (4,5) (6,7) over this thread's rows
  static_assert(kColRowsPerThread == 8, "the tree below takes 8 rows");
  m2[0] = absmax2_tree8(w[0].x, w[1].x, w[2].x, w[3].x, w[4].x, w[5].x, w[6].x, w[7].x);
  m2[1] = absmax2_tree8(w[0].y, w[1].y, w[2].y, w[3].y, w[4].y, w[5].y, w[6].y, w[7].y);
  m2[2] = absmax2_tree8(w[0].z, w[1].z, w[2].z, w[3].z, w[4].z, w[5].z, w[6].z, w[7].z);
  m2[3] = absmax2_tree8(w[0].w, w[1].w, w[2].w, w[3].w, w[4].w, w[5].w, w[6].w, w[7].w);
  const int wp = threadIdx.x >> 5;
  uint8_t* qp = a.q + row0 * a.q_ld + col0;
  const int64_t step = int64_t(kColHalfWarps) * a.q_ld;
  if constexpr (FORM == kBlockForm) {
    uint32_t mb = __vmaxu2(__vmaxu2(m2[0], m2[1]), __vmaxu2(m2[2], m2[3]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mb = __vmaxu2(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    if ((threadIdx.x & 31) == 0) sm.scale[wp] = absmax_to_float(mb);
    __syncthreads();
    float m = sm.scale[0];
#pragma unroll
    for (int wv = 1; wv < kColThreads / 32; ++wv) m = max_nan(m, sm.scale[wv]);
    const float sc = scale_from_amax(m);
    if (threadIdx.x == 0) a.s[int64_t(by) * a.s_ld + bx] = sc;
#pragma unroll
    for (int r = 0; r < kColRowsPerThread; ++r, qp += step)
      if (FULL || row0 + r * kColHalfWarps < rows) *reinterpret_cast<uint2*>(qp) = quantize8(w[r], sc);
    return;
  }
  // the two half-warps of a warp hold the same columns: combine them in registers first
#pragma unroll
  for (int j = 0; j < 4; ++j) m2[j] = __vmaxu2(m2[j], __shfl_xor_sync(0xffffffffu, m2[j], 16));
  if ((threadIdx.x & 16) == 0) {
    float4* dst = reinterpret_cast<float4*>(&sm.max[wp][cx * 8]);
    dst[0] = make_float4(__uint_as_float(m2[0] << 16), __uint_as_float(m2[0] & 0xffff0000u),
                         __uint_as_float(m2[1] << 16), __uint_as_float(m2[1] & 0xffff0000u));
    dst[1] = make_float4(__uint_as_float(m2[2] << 16), __uint_as_float(m2[2] & 0xffff0000u),
                         __uint_as_float(m2[3] << 16), __uint_as_float(m2[3] & 0xffff0000u));
  }
  __syncthreads();
  // one thread per column finishes the maximum, derives scale and reciprocal once, and
  // publishes both (conflict-free: consecutive threads, consecutive words)
  if (threadIdx.x < kColPanelCols) {
    float v = sm.max[0][threadIdx.x];
#pragma unroll
    for (int h = 1; h < kColThreads / 32; ++h) v = max_nan(v, sm.max[h][threadIdx.x]);
    const float sc = scale_from_amax(v);
    sm.scale[threadIdx.x] = sc;
    sm.rcp[threadIdx.x] = __frcp_rn(sc);
    const int col = bx * kColPanelCols + threadIdx.x;
    if (FULL || col < a.out_cols) a.s[int64_t(by) * a.s_ld + col] = sc;
  }
  __syncthreads();
  if (!FULL && col0 >= a.out_cols) return;    // out_cols % 8 == 0
  float s[8], rc[8];
  {
    const float4 a0 = *reinterpret_cast<const float4*>(&sm.scale[cx * 8]), a1 = *reinterpret_cast<const float4*>(&sm.scale[cx * 8 + 4]);
    const float4 b0 = *reinterpret_cast<const float4*>(&sm.rcp[cx * 8]), b1 = *reinterpret_cast<const float4*>(&sm.rcp[cx * 8 + 4]);
    s[0] = a0.x; s[1] = a0.y; s[2] = a0.z; s[3] = a0.w; s[4] = a1.x; s[5] = a1.y; s[6] = a1.z; s[7] = a1.w;
    rc[0] = b0.x; rc[1] = b0.y; rc[2] = b0.z; rc[3] = b0.w; rc[4] = b1.x; rc[5] = b1.y; rc[6] = b1.z; rc[7] = b1.w;
  }
  bool all_finite = true;
#pragma unroll
  for (int j = 0; j < 8; ++j) all_finite = all_finite && (fabsf(s[j]) <= 3.402823466e38f);
  // this thread's four column pairs: scale and negated reciprocal as packed operands (see quantize2_sr)
  float2 s2[4], nr2[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    s2[j] = make_float2(s[2 * j], s[2 * j + 1]);
    nr2[j] = make_float2(-rc[2 * j], -rc[2 * j + 1]);
  }
  if (all_finite) {
#pragma unroll
    for (int r = 0; r < kColRowsPerThread; ++r, qp += step) {
      if (!FULL && row0 + r * kColHalfWarps >= rows) break;
      const uint4 v = w[r];
      *reinterpret_cast<uint2*>(qp) =
          make_uint2(cvt_e4m3x4(quotient2_sr(v.x, s2[0], nr2[0]), quotient2_sr(v.y, s2[1], nr2[1])),
                     cvt_e4m3x4(quotient2_sr(v.z, s2[2], nr2[2]), quotient2_sr(v.w, s2[3], nr2[3])));
    }
  } else {
#pragma unroll
    for (int r = 0; r < kColRowsPerThread; ++r, qp += step) {
      if (!FULL && row0 + r * kColHalfWarps >= rows) break;
      const uint4 v = w[r];
      const uint32_t b0 = cvt_e4m3x2(__fdiv_rn(bf16lo(v.x), s[0]), __fdiv_rn(bf16hi(v.x), s[1]));
      const uint32_t b1 = cvt_e4m3x2(__fdiv_rn(bf16lo(v.y), s[2]), __fdiv_rn(bf16hi(v.y), s[3]));
      const uint32_t b2 = cvt_e4m3x2(__fdiv_rn(bf16lo(v.z), s[4]), __fdiv_rn(bf16hi(v.z), s[5]));
      const uint32_t b3 = cvt_e4m3x2(__fdiv_rn(bf16lo(v.w), s[6]), __fdiv_rn(bf16hi(v.w), s[7]));
      *reinterpret_cast<uint2*>(qp) = make_uint2(__byte_perm(b0, b1, 0x5410), __byte_perm(b2, b3, 0x5410));
    }
  }
}

__host__ __device__ __forceinline__ bool is_ragged(const PanelJob& a) {
  return ((a.ld | a.cols) & 7) != 0 || (reinterpret_cast<uintptr_t>(a.x) & 15u) != 0;
}

template <bool ROW, int FORM, int ACT>
__device__ __forceinline__ void panel_any(const PanelJob& a, int bx, int by, PanelSmem& sm) {
  const bool full = (by + 1) * kTile <= a.rows && (bx + 1) * kColPanelCols <= a.cols;
  if (full) panel<ROW, FORM, ACT, true>(a, bx, by, sm);
  else panel<ROW, FORM, ACT, false>(a, bx, by, sm);
}

// One tensor.  Blocks per SM: four at 64 registers, without a spill (8-14 % faster than three: the top stall is the wait for
// the panel's loads, and a fourth block is a third more of them in flight).
template <bool ROW, int FORM, bool RAGGED = false>
__global__ void __launch_bounds__(kColThreads, 4) quantize_panel_kernel(const __grid_constant__ PanelJob a) {
  __shared__ PanelSmem sm;
  grid_trigger();
  grid_wait();
  const int by = int(blockIdx.x) / a.tiles_x, bx = int(blockIdx.x) - by * a.tiles_x;
  if constexpr (RAGGED) panel<ROW, FORM, TG_ACT_NONE, false, true>(a, bx, by, sm);
  else panel_any<ROW, FORM, TG_ACT_NONE>(a, bx, by, sm);
}

// Several tensors in ONE launch: a linear's activation (both its forms from one read) and its weight, or the weights of a
// layer.  The small ones do not fill the GPU by themselves and every launch costs 2-3 us: at 4096 x 768 -> 3072 the three
// launches (row form, column form, weight) took 14.3 us, as two jobs of one launch 10.3.  With every form's code in one kernel
// the compiler spills a few registers (7 % at 32768 x 8192), so past kJointPanels panels -- about 25 us of work, beside
// which a launch no longer counts -- each tensor takes the kernel of its own.
constexpr int kMaxJobs = 6;
constexpr int64_t kJointPanels = 2048;
template <int MAX>
struct PanelJobList {
  PanelJob job[MAX];
  int n;
};
using PanelJobs = PanelJobList<kMaxJobs>;
template <int MAX>
__device__ __forceinline__ int job_of_block(const PanelJobList<MAX>& jobs) {
  int j = 0;
  for (int i = 1; i < jobs.n; ++i)
    if (int(blockIdx.x) >= jobs.job[i].first) j = i;
  return j;
}
__global__ void __launch_bounds__(kColThreads, 4) quantize_panels_kernel(const __grid_constant__ PanelJobs jobs) {
  __shared__ PanelSmem sm;
  grid_trigger();
  grid_wait();
  const int j = job_of_block(jobs);
  const PanelJob& a = jobs.job[j];
  const int t = int(blockIdx.x) - a.first, by = t / a.tiles_x, bx = t - by * a.tiles_x;
  if (a.q_row != nullptr) {
    if (a.form == kColForm) panel_any<true, kColForm, TG_ACT_NONE>(a, bx, by, sm);
    else if (a.form == kBlockForm) panel_any<true, kBlockForm, TG_ACT_NONE>(a, bx, by, sm);
    else panel_any<true, kNoForm, TG_ACT_NONE>(a, bx, by, sm);
  } else {
    if (a.form == kBlockForm) panel_any<false, kBlockForm, TG_ACT_NONE>(a, bx, by, sm);
    else if (is_ragged(a)) panel<false, kColForm, TG_ACT_NONE, false, true>(a, bx, by, sm);
    else panel_any<false, kColForm, TG_ACT_NONE>(a, bx, by, sm);
  }
}

// Weights in 128 x 128 tiles, many in one launch (a launch per weight is 96 in a 24-layer model's step, 5 us each at
// 1024 x 4096).
constexpr int kMaxBlockJobs = 24;
using BlockJobs = PanelJobList<kMaxBlockJobs>;
__global__ void __launch_bounds__(kColThreads, 4) quantize_weights_kernel(const __grid_constant__ BlockJobs jobs) {
  __shared__ PanelSmem sm;
  grid_trigger();
  grid_wait();
  const PanelJob& a = jobs.job[job_of_block(jobs)];
  const int t = int(blockIdx.x) - a.first, by = t / a.tiles_x, bx = t - by * a.tiles_x;
  panel_any<false, kBlockForm, TG_ACT_NONE>(a, bx, by, sm);
}

// Both forms of an activation computed on the fly.  The activation variants take 80 registers and three blocks; the GELU
// cotangent variant, the one with the most live values, runs 2 % faster with 128 registers and two blocks than with
// 80 and three, spilling.
template <int ACT>
__global__ void __launch_bounds__(kColThreads, ACT == TG_ACT_GELU_BWD ? 2 : 3)
quantize_act_kernel(const __grid_constant__ PanelJob a) {
  __shared__ PanelSmem sm;
  grid_trigger();
  grid_wait();
  panel_any<true, kColForm, ACT>(a, blockIdx.x, blockIdx.y, sm);
}

static PanelJob make_job(const void* x, int64_t rows, int64_t cols, int64_t ld) {
  PanelJob a = {};
  a.x = static_cast<const __nv_bfloat16*>(x);
  a.ld = ld;
  a.rows = int(rows);
  a.cols = a.out_cols = int(cols);
  a.tiles_x = int((cols + kColPanelCols - 1) / kColPanelCols);
  return a;
}
static void with_row(PanelJob& a, void* q, int64_t q_ld, float* s, int64_t s_ld) {
  a.q_row = static_cast<uint8_t*>(q); a.q_row_ld = q_ld; a.s_row = s; a.s_row_ld = s_ld;
}
static void with_form(PanelJob& a, int form, void* q, int64_t q_ld, float* s, int64_t s_ld) {
  a.form = form; a.q = static_cast<uint8_t*>(q); a.q_ld = q_ld; a.s = s; a.s_ld = s_ld;
}

static int64_t panels_of(const PanelJob& a) { return int64_t(a.tiles_x) * ((a.rows + kTile - 1) / kTile); }

// up to eight panels per SM.  (Early at every size, the 24-layer step and a wide layer are 1 to 2 % slower.)
static bool is_short(int64_t panels) { return panels <= 8 * sm_count(); }

static int launch_panel(const PanelJob& a, cudaStream_t st) {
  const int64_t blocks = panels_of(a);
  if (blocks > INT32_MAX) return TG_ERR_TOO_LARGE;
  auto kern = a.q_row != nullptr ? (a.form == kColForm     ? quantize_panel_kernel<true, kColForm>
                                    : a.form == kBlockForm ? quantize_panel_kernel<true, kBlockForm>
                                                           : quantize_panel_kernel<true, kNoForm>)
              : a.form != kColForm ? quantize_panel_kernel<false, kBlockForm>
              : is_ragged(a)       ? quantize_panel_kernel<false, kColForm, true>
                                   : quantize_panel_kernel<false, kColForm>;
  TG_CUDA_CHECK(launch_if_short(is_short(blocks), kern, dim3(unsigned(blocks)), kColThreads, 0, st, a));
  return TG_OK;
}

// numbers the jobs' thread blocks; returns how many there are, or -1
template <int MAX>
static int64_t number_blocks(PanelJobList<MAX>& jobs) {
  int64_t blocks = 0;
  for (int i = 0; i < jobs.n; ++i) {
    jobs.job[i].first = int(blocks);
    blocks += panels_of(jobs.job[i]);
    if (blocks > INT32_MAX) return -1;
  }
  return blocks;
}

}  // namespace tg

using namespace tg;

extern "C" int tg_quantize_rowwise(const void* x, void* q, float* scales, int64_t rows,
                                   int64_t cols, void* stream) {
  if (rows < 0 || cols < 0 || cols % kTile != 0) return TG_ERR_SHAPE;
  if (rows == 0 || cols == 0) return TG_OK;
  if (!aligned16(x) || !aligned16(q) || (reinterpret_cast<uintptr_t>(scales) & 3u)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  const int64_t n_tiles = rows * (cols / kTile);
  const int64_t tiles_per_block = (kRowThreads / 16) * kRowUnroll;
  int64_t blocks = (n_tiles + tiles_per_block - 1) / tiles_per_block;
  const int64_t cap = int64_t(sm_count()) * 8 * 4;  // 8 resident blocks per SM, 4 waves
  if (blocks > cap) blocks = cap;
  quantize_rowwise_kernel<<<dim3(unsigned(blocks)), kRowThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint4*>(x), static_cast<uint2*>(q), scales, n_tiles);
  TG_CUDA_CHECK(cudaGetLastError());
  return TG_OK;
}

static bool too_large(int64_t rows, int64_t cols) { return rows > INT32_MAX - 256 || cols > INT32_MAX - 256; }

extern "C" int tg_quantize_colwise(const void* x, void* q, float* scales, int64_t rows,
                                   int64_t cols, void* stream) {
  if (rows < 0 || cols < 0 || cols % 8 != 0) return TG_ERR_SHAPE;
  if (rows == 0 || cols == 0) return TG_OK;
  if (!aligned16(x) || !aligned16(q) || !aligned16(scales)) return TG_ERR_ALIGN;
  if (too_large(rows, cols)) return TG_ERR_TOO_LARGE;
  if (int rc = check_arch()) return rc;
  PanelJob a = make_job(x, rows, cols, cols);
  with_form(a, kColForm, q, cols, scales, cols);
  return launch_panel(a, static_cast<cudaStream_t>(stream));
}

extern "C" int tg_quantize_rowcol_ld(const void* x, void* q_row, int64_t q_row_ld, float* s_row, int64_t s_row_ld,
                                     void* q_col, int64_t q_col_ld, float* s_col, int64_t s_col_ld, int64_t rows,
                                     int64_t cols, void* stream) {
  if (rows < 0 || cols < 0 || cols % kTile != 0) return TG_ERR_SHAPE;
  if (q_row_ld < cols || q_row_ld % 16 != 0 || s_row_ld < cols / kTile) return TG_ERR_SHAPE;
  if (q_col_ld < cols || q_col_ld % 16 != 0 || s_col_ld < cols) return TG_ERR_SHAPE;
  if (rows == 0 || cols == 0) return TG_OK;
  if (!aligned16(x) || (reinterpret_cast<uintptr_t>(q_row) & 7u) || (reinterpret_cast<uintptr_t>(q_col) & 7u) ||
      (reinterpret_cast<uintptr_t>(s_col) & 3u) || (reinterpret_cast<uintptr_t>(s_row) & 3u))
    return TG_ERR_ALIGN;
  if (too_large(rows, cols)) return TG_ERR_TOO_LARGE;
  if (int rc = check_arch()) return rc;
  PanelJob a = make_job(x, rows, cols, cols);
  with_row(a, q_row, q_row_ld, s_row, s_row_ld);
  with_form(a, kColForm, q_col, q_col_ld, s_col, s_col_ld);
  return launch_panel(a, static_cast<cudaStream_t>(stream));
}

extern "C" int tg_quantize_rowcol(const void* x, void* q_row, float* s_row, void* q_col, float* s_col,
                                  int64_t rows, int64_t cols, void* stream) {
  if (cols > 0 && (!aligned16(q_row) || !aligned16(q_col) || !aligned16(s_col))) return TG_ERR_ALIGN;
  const int64_t ld = cols < 16 ? 16 : cols;
  return tg_quantize_rowcol_ld(x, q_row, ld, s_row, cols / kTile, q_col, ld, s_col, cols, rows, cols, stream);
}

extern "C" int tg_act_quantize_rowcol(const void* x, const void* gate, int act, void* q_row, float* s_row, void* q_col,
                                      float* s_col, int64_t rows, int64_t cols, void* stream) {
  if (rows < 0 || cols < 0 || cols % kTile != 0) return TG_ERR_SHAPE;
  const bool bwd = act == TG_ACT_RELU2_BWD || act == TG_ACT_GELU_BWD;
  if (act != TG_ACT_RELU2 && act != TG_ACT_GELU && !bwd) return TG_ERR_SHAPE;
  if (rows == 0 || cols == 0) return TG_OK;
  if (bwd && gate == nullptr) return TG_ERR_SHAPE;
  if (!aligned16(x) || (bwd && !aligned16(gate)) || !aligned16(q_row) || !aligned16(q_col) || !aligned16(s_col) ||
      (reinterpret_cast<uintptr_t>(s_row) & 3u))
    return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  const int64_t gx = cols / kColPanelCols, gy = (rows + kTile - 1) / kTile;
  if (gy > 65535 || too_large(rows, cols)) return TG_ERR_TOO_LARGE;
  const dim3 grid{unsigned(gx), unsigned(gy)};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  PanelJob a = make_job(x, rows, cols, cols);
  a.gate = static_cast<const __nv_bfloat16*>(gate);
  with_row(a, q_row, cols, s_row, cols / kTile);
  with_form(a, kColForm, q_col, cols, s_col, cols);
  auto kern = act == TG_ACT_RELU2       ? quantize_act_kernel<TG_ACT_RELU2>
              : act == TG_ACT_GELU       ? quantize_act_kernel<TG_ACT_GELU>
              : act == TG_ACT_RELU2_BWD  ? quantize_act_kernel<TG_ACT_RELU2_BWD>
                                         : quantize_act_kernel<TG_ACT_GELU_BWD>;
  TG_CUDA_CHECK(launch_if_short(is_short(gx * gy), kern, grid, kColThreads, 0, st, a));
  return TG_OK;
}

extern "C" int tg_quantize_block128(const void* x, void* q, float* scales, int64_t rows,
                                    int64_t cols, void* stream) {
  if (rows < 0 || cols < 0 || cols % kTile != 0) return TG_ERR_SHAPE;
  if (rows == 0 || cols == 0) return TG_OK;
  if (!aligned16(x) || !aligned16(q) || (reinterpret_cast<uintptr_t>(scales) & 3u)) return TG_ERR_ALIGN;
  if (too_large(rows, cols)) return TG_ERR_TOO_LARGE;
  if (int rc = check_arch()) return rc;
  PanelJob a = make_job(x, rows, cols, cols);
  with_form(a, kBlockForm, q, cols, scales, cols / kTile);
  return launch_panel(a, static_cast<cudaStream_t>(stream));
}

static int make_job(const tgh_quantize_job& b, PanelJob* out) {
  const bool col = b.form == TGH_FORM_COLUMNS, block = b.form == TGH_FORM_BLOCKS;
  if (b.rows < 0 || b.cols < 0 || (b.q_row == nullptr && !col && !block)) return TG_ERR_SHAPE;
  if ((b.q_row != nullptr || block) && b.cols % kTile != 0) return TG_ERR_SHAPE;
  if (b.ld < b.cols || (b.q_row != nullptr && b.q_row_ld % 16 != 0) || (b.q != nullptr && (b.q_ld % 16 != 0 || b.q_ld < b.cols)))
    return TG_ERR_SHAPE;
  const bool col_only = col && b.q_row == nullptr;      // reads rows at any alignment
  if ((!col_only && (b.ld % 8 != 0 || !aligned16(b.x))) || (reinterpret_cast<uintptr_t>(b.x) & 1u) ||
      (reinterpret_cast<uintptr_t>(b.q_row) & 7u) || (reinterpret_cast<uintptr_t>(b.q) & 7u))
    return TG_ERR_ALIGN;
  if (too_large(b.rows, b.cols)) return TG_ERR_TOO_LARGE;
  PanelJob a = make_job(b.x, b.rows, b.cols, b.ld);
  if (b.q_row != nullptr) with_row(a, b.q_row, b.q_row_ld, b.s_row, b.s_row_ld);
  if (col) {
    with_form(a, kColForm, b.q, b.q_ld, b.s, b.s_ld);
    if (b.cols % 8 != 0) {                       // ragged columns: zeros up to the pitch of the output
      a.out_cols = int(b.q_ld);
      if (b.s_ld < b.q_ld || b.q_ld - b.cols >= 128) return TG_ERR_SHAPE;
      a.tiles_x = (a.out_cols + kColPanelCols - 1) / kColPanelCols;
    }
  }
  if (block) with_form(a, kBlockForm, b.q, b.q_ld, b.s, b.s_ld);
  *out = a;
  return TG_OK;
}

extern "C" int tgh_quantize_jobs(const tgh_quantize_job* in, int n, void* stream) {
  if (n < 0) return TG_ERR_SHAPE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  bool weights = n > 1;
  int64_t panels = 0;
  for (int i = 0; i < n; ++i) {
    PanelJob a;
    if (in[i].rows == 0 || in[i].cols == 0) continue;
    if (int rc = make_job(in[i], &a)) return rc;
    weights = weights && a.q_row == nullptr && a.form == kBlockForm;
    panels += panels_of(a);
  }
  if (panels == 0) return TG_OK;
  if (int rc = check_arch()) return rc;
  auto joint = [&](auto& jobs, auto kernel, int from, int to) -> int {
    jobs.n = 0;
    for (int i = from; i < to; ++i)
      if (in[i].rows != 0 && in[i].cols != 0) make_job(in[i], &jobs.job[jobs.n++]);
    const int64_t blocks = number_blocks(jobs);
    if (blocks < 0) return TG_ERR_TOO_LARGE;
    if (blocks == 0) return TG_OK;
    TG_CUDA_CHECK(launch_if_short(is_short(blocks), kernel, dim3(unsigned(blocks)), kColThreads, 0, st, jobs));
    return TG_OK;
  };
  if (weights) {
    BlockJobs jobs;
    for (int i = 0; i < n; i += kMaxBlockJobs)
      if (int rc = joint(jobs, quantize_weights_kernel, i, i + kMaxBlockJobs < n ? i + kMaxBlockJobs : n)) return rc;
    return TG_OK;
  }
  if (n > 1 && n <= kMaxJobs && panels <= kJointPanels) {
    PanelJobs jobs;
    return joint(jobs, quantize_panels_kernel, 0, n);
  }
  for (int i = 0; i < n; ++i) {
    if (in[i].rows == 0 || in[i].cols == 0) continue;
    PanelJob a;
    make_job(in[i], &a);
    if (int rc = launch_panel(a, st)) return rc;
  }
  return TG_OK;
}
