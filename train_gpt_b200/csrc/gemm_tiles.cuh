// What the two tiled block-scaled GEMM kernels (gemm_fp8.cu, gemm_ring.cu) share: their parameters, the numbering of the work items,
// the promotion of a piece of an accumulator, the epilogue's staging stores.
#pragma once

#include "umma.cuh"

namespace tg {

struct GemmParams {
  const float* sa;
  long long sa_sm, sa_sk;
  const float* sb;
  long long sb_sn, sb_sk;
  void* d;              // output, row pitch ldd elements
  long long ldd;
  int M, N, nkb;        // nkb = contraction blocks per work item (all of them unless the contraction is split)
  int nkb_rem;          // ... plus one for the first nkb_rem ranges of a split contraction (ranges need not be equal)
  int a_mn, b_mn;       // 1 = MN-major storage
  int tiles_m, tiles_n;
  int band;             // tile rows per band of the tile numbering
  // ceil(2^40 / d) for the three divisors of the item -> tile arithmetic (tiles per contraction range,
  // tiles per band, rows of the last band), 0 = divide the slow way (the exactness bound x * d < 2^40
  // does not hold); rows of a full band = `band`, its reciprocal in mg_band
  unsigned long long mg_tiles, mg_per_band, mg_band, mg_last;
  int ksplit;           // the contraction is cut into this many ranges; range s of a tile is its own
                        // work item and writes its float32 partial sums to d + s * slice_elems
  long long slice_elems;
  unsigned* status;
};

// Staging stores of the epilogue, address = (base + OFF) ^ flip with OFF a compile-time constant.
// The address is formed inside the asm block so that the compiler cannot hoist one register per
// store out of the unrolled loops: the accumulators leave no room for that (it spilled loop
// invariants of the mainloop instead).  `base` has bits 4-6 clear or small enough that adding OFF
// never carries past bit 6, so the xor is the 128-byte swizzle of the 16-byte chunk index.
template <int OFF>
__device__ __forceinline__ void sts_swz_b32(uint32_t base, uint32_t flip, uint32_t x) {
  asm volatile("{\n\t.reg .b32 t;\n\tadd.u32 t, %0, %1;\n\txor.b32 t, t, %2;\n\tst.shared.b32 [t], %3;\n\t}"
               ::"r"(base), "n"(OFF), "r"(flip), "r"(x) : "memory");
}
// (float operands are passed as floats: routing accumulator halves through integer registers kept
// ptxas from leaving them in their packed pairs and cost ~25 spilled registers)
template <int OFF>
__device__ __forceinline__ void sts_swz_f32x2(uint32_t base, uint32_t flip, float2 v) {
  asm volatile("{\n\t.reg .b32 t;\n\tadd.u32 t, %0, %1;\n\txor.b32 t, t, %2;\n\tst.shared.v2.f32 [t], {%3, %4};\n\t}"
               ::"r"(base), "n"(OFF), "r"(flip), "f"(v.x), "f"(v.y) : "memory");
}
template <int OFF>
__device__ __forceinline__ void sts_swz_f32x4(uint32_t base, uint32_t flip, float2 v, float2 w) {
  asm volatile("{\n\t.reg .b32 t;\n\tadd.u32 t, %0, %1;\n\txor.b32 t, t, %2;\n\tst.shared.v4.f32 [t], {%3, %4, %5, %6};\n\t}"
               ::"r"(base), "n"(OFF), "r"(flip), "f"(v.x), "f"(v.y), "f"(w.x), "f"(w.y) : "memory");
}
template <int OFF>
__device__ __forceinline__ void sts_swz_v4(uint32_t base, uint32_t flip, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("{\n\t.reg .b32 t;\n\tadd.u32 t, %0, %1;\n\txor.b32 t, t, %2;\n\tst.shared.v4.b32 [t], {%3, %4, %5, %6};\n\t}"
               ::"r"(base), "n"(OFF), "r"(flip), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// which accumulator buffer a block uses: a constant, or the value of the carried counter
template <int B> struct StaticBuf { __device__ static constexpr uint32_t get(uint32_t) { return uint32_t(B); } };
struct DynBuf { __device__ static uint32_t get(uint32_t b) { return b; } };

// f(integral_constant<int, 0>) ... f(integral_constant<int, N-1>): a loop whose index is a constant
// expression inside the body (template arguments, "n" asm operands)
template <int I> struct IntC { static constexpr int value = I; };
template <int N, int I = 0, typename F>
__device__ __forceinline__ void static_loop(F&& f) {
  if constexpr (I < N) {
    f(IntC<I>{});
    static_loop<N, I + 1>(f);
  }
}

// acc[j] += scale * v[2j..2j+1] for NC TMEM columns; SB_GRAN == 1 multiplies by the per-column
// scales staged in shared memory first.
template <int SB_GRAN, int NC>
__device__ __forceinline__ void promote(float2* acc, const uint32_t (&v)[NC], const float* stage, float sa_v, float s_scalar) {
  if (SB_GRAN == 1) {
    const float2 sa2 = make_float2(sa_v, sa_v);
#pragma unroll
    for (int j = 0; j < NC / 4; ++j) {
      const float4 sb4 = *reinterpret_cast<const float4*>(stage + 4 * j);
      const float2 p0 = make_float2(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]));
      const float2 p1 = make_float2(__uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
      acc[2 * j] = __ffma2_rn(__fmul2_rn(p0, make_float2(sb4.x, sb4.y)), sa2, acc[2 * j]);
      acc[2 * j + 1] = __ffma2_rn(__fmul2_rn(p1, make_float2(sb4.z, sb4.w)), sa2, acc[2 * j + 1]);
    }
  } else {
    const float2 s2 = make_float2(s_scalar, s_scalar);
#pragma unroll
    for (int j = 0; j < NC / 2; ++j) {
      const float2 pv = make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
      acc[j] = __ffma2_rn(pv, s2, acc[j]);
    }
  }
}

// Work item -> tile coordinates.  Tiles are numbered in bands of `band` tile rows; inside a band
// the numbering runs down the rows first, then across the columns, so that the CTAs of a wave
// (consecutive numbers) cover a near-square patch of the output: the A and B panels they fetch
// together are as few as possible, which is what keeps the operands' L2 lines alive between the
// CTAs that share them.  (Row-major numbering made a 148-CTA wave touch every B panel of a
// 24-tile-wide problem plus 7 A panels; in bands of 16 it touches 16 + 10.)
// x / d through a multiplication by mg = ceil(2^40 / d): exact while x * d < 2^40 (the host checks
// and passes 0 otherwise).  A 32-bit division by a run-time value costs ~20 dependent instructions,
// and every role does three of them at each tile boundary.
__device__ __forceinline__ int fast_div(int x, int d, unsigned long long mg) {
  return mg != 0 ? int((static_cast<unsigned long long>(static_cast<unsigned>(x)) * mg) >> 40) : x / d;
}
__device__ __forceinline__ void tile_coords(const GemmParams& p, int tile, int& tm, int& tn) {
  const int per_band = p.band * p.tiles_n;
  const int b = fast_div(tile, per_band, p.mg_per_band), w = tile - b * per_band;
  const int left = p.tiles_m - b * p.band;
  const bool full = left >= p.band;
  const int rows = full ? p.band : left;
  tn = fast_div(w, rows, full ? p.mg_band : p.mg_last);
  tm = b * p.band + (w - tn * rows);
}
// work item -> (contraction range, tile)
__device__ __forceinline__ void item_split(const GemmParams& p, int item, int n_tiles, int& ks, int& tile) {
  ks = fast_div(item, n_tiles, p.mg_tiles);
  tile = item - ks * n_tiles;
}
// contraction range -> its first block and its number of blocks
__device__ __forceinline__ int range_blocks(const GemmParams& p, int ks) { return p.nkb + (ks < p.nkb_rem ? 1 : 0); }
__device__ __forceinline__ int range_first(const GemmParams& p, int ks) { return ks * p.nkb + min(ks, p.nkb_rem); }

// ---- host --------------------------------------------------------------------------------

// output map: [contraction slice][row][column]; a launch that is not cut has one slice.  A box is 32 rows of box_cols columns
// (span = box_cols elements: 32, 64 or 128 bytes, swizzled).
inline int make_output_map(CUtensorMap* map, bool f32, const tg_gemm_args* a, const GemmParams& p, int box_cols, int span) {
  EncodeTiledFn enc;
  if (int rc = get_encode_fn(&enc)) return rc;
  const int esz = f32 ? 4 : 2;
  cuuint64_t dims[3] = {cuuint64_t(a->N), cuuint64_t(a->M), cuuint64_t(p.ksplit)};
  cuuint64_t strides[2] = {cuuint64_t(p.ldd) * esz, cuuint64_t(p.ksplit > 1 ? p.slice_elems : a->M * p.ldd) * esz};
  cuuint32_t box[3] = {cuuint32_t(box_cols), 32u, 1u};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, p.d, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE,
                   span == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : span == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? TG_OK : record_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled (output)");
}

// The reciprocals of the item -> tile arithmetic, from tiles_m, tiles_n, band and ksplit:
// q = (x * ceil(2^40 / d)) >> 40 is x / d for every x <= x_max when x_max * d < 2^40.
inline int set_reciprocals(GemmParams& p) {
  auto magic = [](int64_t x_max, int64_t d) -> unsigned long long {
    if (d <= 0 || x_max >= (int64_t(1) << 31) || x_max * d >= (int64_t(1) << 40)) return 0ull;
    return ((1ull << 40) + uint64_t(d) - 1) / uint64_t(d);
  };
  const int64_t n_tiles = int64_t(p.tiles_m) * p.tiles_n, n_items = n_tiles * p.ksplit, per_band = int64_t(p.band) * p.tiles_n;
  const int64_t last_rows = p.tiles_m % p.band;
  p.mg_tiles = magic(n_items, n_tiles);
  p.mg_per_band = magic(n_tiles, per_band);
  p.mg_band = magic(per_band, p.band);
  p.mg_last = last_rows > 0 ? magic(per_band, last_rows) : 0ull;
  return n_items > INT32_MAX || n_items * (p.nkb + 1) > INT32_MAX ? TG_ERR_TOO_LARGE : TG_OK;
}

// The kernel of gemm_ring.cu: on pairs of SMs, or 128 x bn tiles with a scale per column.
int ring_run(const tg_gemm_args* a, const GemmParams& p, bool pair, int bn, bool f32, cudaStream_t st);
// Problem a (column scales; f32: cut into ranges, p.d the slices), then problem b (block scales, bf16, uncut), both on pairs in one launch.
int ring_pair_two(const tg_gemm_args* a, const GemmParams& pa, bool f32, const tg_gemm_args* b, const GemmParams& pb, cudaStream_t st);

// Microseconds of one 256 x 256 item of so many blocks on a pair, as the plans count them.
inline double pair_item_us(bool columns, double blocks) { return (columns ? 0.54 : 0.42) * blocks + 0.86; }

// Two problems of n1 items of t1 and n2 of t2 microseconds on `units` units: the units that the first one's last round leaves idle begin
// with the second, for `rounds` rounds, and then all take what is left of it.  Returns the time of the best such order.
inline double two_problems_us(int64_t n1, double t1, int64_t n2, double t2, int64_t units, int& rounds) {
  const int64_t busy = n1 % units, idle = units - busy;
  rounds = 0;
  if (busy == 0) return double(n1 / units) * t1 + double((n2 + units - 1) / units) * t2;
  double best = 0.0;
  for (int e = 0; e <= int(t1 / t2) + 1; ++e) {
    const int64_t rest = std::max<int64_t>(0, n2 - e * idle), each = rest / units, more = rest % units;
    const double us = std::max(t1 + t2 * double(each + (more > idle)), t2 * double(e + each + (more > 0)));
    if (e == 0 || us < best) {
      best = us;
      rounds = e;
    }
  }
  return double(n1 / units) * t1 + best;
}

}  // namespace tg
