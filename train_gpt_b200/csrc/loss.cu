// Capped-logit cross-entropy, forward and backward, one pass over the logits each.
//
// Reference semantics: train-gpt model.py:97 (`cap * tanh(logits / cap)` on the bf16 output of
// the unembedding GEMM, every op rounding to bf16, the Python-float cap weakly typed = bf16)
// followed by losses.py:9-12 (cast to float32, log_softmax over the vocabulary, gather the
// target's log-probability, mean over tokens).  Done op by op that is five elementwise passes
// and two softmax passes over a (tokens x vocab) tensor (3.3 GB in bf16 at 32768 x 50304, twice
// that in float32); here the forward reads the logits once and writes the bf16 tanh values,
// and the backward turns those into the logits' gradient in place.
//
// Layout: one thread block per token row; each thread walks the row in 16-byte pieces (8 bf16)
// and keeps a running (max, sum of exp) pair; the block combines the pairs.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "host_api.h"
#include "mbarrier.cuh"

namespace tg {

constexpr int kLossThreads = 256;

// RN_bf16(v) as a float
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

struct Softcap {
  float c, r;   // the cap rounded to bf16, and RN(1/c)
  __device__ __forceinline__ explicit Softcap(float cap) {
    c = round_bf16(cap);
    r = __frcp_rn(c);
  }
  __device__ __forceinline__ float z_of_tanh(float t) const { return round_bf16(__fmul_rn(c, t)); }
  // bf16(x / c) as a float: the division is q0 = x*r, q = fma(-fma(q0, c, -x), r, q0), which is
  // the correctly rounded quotient when r is the correctly rounded reciprocal (Markstein); the
  // residual is taken as q0*c - x and subtracted so that x = -0 stays -0
  __device__ __forceinline__ float quotient(float x) const {
    const float q0 = __fmul_rn(x, r);
    return round_bf16(__fmaf_rn(-__fmaf_rn(q0, c, -x), r, q0));
  }
};

// bf16(tanh(a)) for a bf16 argument needs no evaluation outside 2^-6 <= |a| < 4: below, tanh(a)
// differs from a by less than a^2/3 <= 2^-13.6 relative, far inside half a bf16 ulp (>= 2^-10), so
// the result is a itself; from 4 on, 1 - tanh(a) <= 6.8e-4 < 2^-9, so it rounds to +-1.  The 1024
// arguments in between (8 binades x 128 mantissas) are evaluated with tanhf.  A thread block keeps
// the result for EVERY magnitude (32768 two-byte entries, index = the bf16 bits without the sign; a
// NaN maps to itself) in shared memory, so that the per-element work is one load and a sign merge, with no
// range tests; blocks are persistent (each walks many rows), so the fill is paid once per block.
constexpr uint32_t kTanhLo = (127u - 6u) << 7;   // bf16 magnitude bits of 2^-6
constexpr uint32_t kTanhHi = (127u + 2u) << 7;   // ... of 4.0
constexpr int kTanhEntries = 32768;
constexpr int kTanhBytes = kTanhEntries * 2;

__device__ __forceinline__ uint32_t tanh_bits_of_magnitude(uint32_t mag) {
  if (mag < kTanhLo || mag > 0x7f80u) return mag;                 // tiny (or NaN): tanh(a) rounds to a
  if (mag >= kTanhHi) return 0x3f80u;                             // 1
  return __float_as_uint(round_bf16(tanhf(__uint_as_float(mag << 16)))) >> 16;
}
__device__ __forceinline__ void tanh_table_fill(uint16_t* table) {
  for (int i = threadIdx.x; i < kTanhEntries; i += blockDim.x) table[i] = uint16_t(tanh_bits_of_magnitude(uint32_t(i)));
}
// a: a bf16 value held in a float (the scalar form: the target's own logit, once per row)
__device__ __forceinline__ float tanh_bf16(float a) {
  const uint32_t bits = __float_as_uint(a);
  return __uint_as_float((bits & 0x80000000u) | (tanh_bits_of_magnitude((bits >> 16) & 0x7fffu) << 16));
}

// (m, s) <- combine with (m2, s2): s counts exp(z - m)
__device__ __forceinline__ void lse_merge(float& m, float& s, float m2, float s2) {
  const float mn = fmaxf(m, m2);
  s = s * __expf(m - mn) + s2 * __expf(m2 - mn);
  m = mn;
}

// The forward is bound by instruction issue, not by DRAM, so the element work is written in packed
// f32x2 operations on the two halves of each loaded word: the exact quotient x / c (one reciprocal multiply and one
// correction step, as in the quantisers), one rounding to a bf16 pair, two table loads, the cap multiply and its
// rounding, and the online softmax.
// 512 threads, three blocks per SM (the table is 64 KB): 1.57 ms at 32768 x 50304 (1.50 with the prefetch below); 256 / 384 / 768
// threads measured 1.98 / 1.66 / 1.65
constexpr int kLossFwdThreads = 512;

__global__ void __launch_bounds__(kLossFwdThreads)
softcap_ce_fwd_kernel(const __nv_bfloat16* __restrict__ logits, const int32_t* __restrict__ targets, float cap,
                      __nv_bfloat16* __restrict__ tanh_out, float* __restrict__ lse_out, float* __restrict__ nll_out,
                      int rows, int vocab, int64_t ld, int64_t ld_t) {
  __shared__ float s_m[kLossFwdThreads / 32], s_s[kLossFwdThreads / 32];
  extern __shared__ __align__(16) uint16_t s_tanh[];
  tanh_table_fill(s_tanh);
  __syncthreads();
  const Softcap sc(cap);
  const float2 c2 = make_float2(sc.c, sc.c), nr2 = make_float2(-sc.r, -sc.r);
  const float2 l2e = make_float2(1.4426950408889634f, 1.4426950408889634f);
  for (int64_t row = blockIdx.x; row < rows; row += gridDim.x) {
    const __nv_bfloat16* p = logits + row * ld;
    float m = -3.0e38f, s = 0.f;
    // the next piece is loaded before this one is worked on: the kernel's top stall was the wait for its
    // one 16-byte load per thread
    uint4 w_next = threadIdx.x * 8 < vocab ? ld_stream_v4(p + threadIdx.x * 8) : make_uint4(0u, 0u, 0u, 0u);
    for (int i = threadIdx.x * 8; i < vocab; i += kLossFwdThreads * 8) {
      const uint4 w = w_next;
      if (i + kLossFwdThreads * 8 < vocab) w_next = ld_stream_v4(p + i + kLossFwdThreads * 8);
      const uint32_t xi[4] = {w.x, w.y, w.z, w.w};
      float2 z[4];
      uint4 to;
      uint32_t* tp = &to.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        // bf16(x / c) for both halves: q0 = x r, q = fma(-fma(q0, c, -x), r, q0) with the negations folded into
        // the operands (nx = -x, nr = -r), the correctly rounded quotient since r is the correctly rounded reciprocal
        const float2 nx = bf16x2_unpack_neg(xi[j]);
        const float2 q0 = __fmul2_rn(nx, nr2);
        const float2 q = __ffma2_rn(__ffma2_rn(q0, c2, nx), nr2, q0);
        const uint32_t a2 = pack_bf16x2(q.x, q.y);
        // bf16(tanh(.)) of both: table by magnitude, signs put back
        const uint32_t t_lo = s_tanh[a2 & 0x7fffu], t_hi = s_tanh[(a2 >> 16) & 0x7fffu];
        const uint32_t t2 = __byte_perm(t_lo, t_hi, 0x5410) | (a2 & 0x80008000u);
        tp[j] = t2;
        // z = bf16(c tanh)
        const float2 zf = __fmul2_rn(c2, bf16x2_unpack(t2));
        z[j] = bf16x2_unpack(pack_bf16x2(zf.x, zf.y));
      }
      const int valid = vocab - i;        // < 8 only in the last piece of a vocabulary that is not a multiple of 8
      if (valid < 8) {
        // the piece was read whole (the row pitch is a multiple of 8 elements); columns past the
        // vocabulary take no part in the softmax and are not written
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (2 * j >= valid) z[j].x = -INFINITY;
          if (2 * j + 1 >= valid) z[j].y = -INFINITY;
        }
        if (tanh_out != nullptr) {
          const __nv_bfloat16* tv = reinterpret_cast<const __nv_bfloat16*>(&to);
          for (int j = 0; j < valid; ++j) tanh_out[row * ld_t + i + j] = tv[j];
        }
      } else if (tanh_out != nullptr) {
        *reinterpret_cast<uint4*>(tanh_out + row * ld_t + i) = to;
      }
      const float mx = fmaxf(fmaxf(fmaxf(z[0].x, z[0].y), fmaxf(z[1].x, z[1].y)), fmaxf(fmaxf(z[2].x, z[2].y), fmaxf(z[3].x, z[3].y)));
      const float mn = fmaxf(m, mx);
      const float2 nmn = make_float2(-mn, -mn);
      float2 acc = make_float2(s * __expf(m - mn), 0.f);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 d = __fmul2_rn(__fadd2_rn(z[j], nmn), l2e);     // (z - max) log2 e: the difference is exact
        float2 e;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(d.x));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(d.y));
        acc = __fadd2_rn(acc, e);
      }
      s = acc.x + acc.y;
      m = mn;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lse_merge(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();                       // the previous row's partials have been read
    if (lane == 0) { s_m[warp] = m; s_s[warp] = s; }
    __syncthreads();
    if (threadIdx.x == 0) {
      m = s_m[0]; s = s_s[0];
#pragma unroll
      for (int wi = 1; wi < kLossFwdThreads / 32; ++wi) lse_merge(m, s, s_m[wi], s_s[wi]);
      const float lse = m + logf(s);
      int t = targets[row];
      t = t < 0 ? 0 : (t >= vocab ? vocab - 1 : t);   // out-of-range targets clamp, as jnp.take_along_axis does
      const float zt = sc.z_of_tanh(tanh_bf16(sc.quotient(__bfloat162float(p[t]))));
      lse_out[row] = lse;
      nll_out[row] = lse - zt;
    }
  }
}

// dlogits = gscale / rows * (exp(z - lse) - [col == target]) * (1 - tanh^2), rounded to bf16.
// `d` may be the buffer `tanh_in` lives in: every element is read and then written by one thread.
__global__ void __launch_bounds__(kLossThreads)
softcap_ce_bwd_kernel(const __nv_bfloat16* tanh_in, const int32_t* __restrict__ targets,
                      const float* __restrict__ lse, const float* __restrict__ gscale, float cap, float inv_rows,
                      __nv_bfloat16* d, int vocab, int64_t ld_t, int64_t ld_d) {
  const int64_t row = blockIdx.x;
  const Softcap sc(cap);
  const float l = lse[row];
  const float g = (gscale != nullptr ? *gscale : 1.0f) * inv_rows;
  int t = targets[row];
  t = t < 0 ? 0 : (t >= vocab ? vocab - 1 : t);
  const __nv_bfloat16* p = tanh_in + row * ld_t;
  for (int i = threadIdx.x * 8; i < vocab; i += kLossThreads * 8) {
    const uint4 w = *reinterpret_cast<const uint4*>(p + i);
    const uint32_t ti[4] = {w.x, w.y, w.z, w.w};
    uint4 o;
    uint32_t* op = &o.x;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float t0 = bf16lo(ti[j]), t1 = bf16hi(ti[j]);
      float p0 = __expf(sc.z_of_tanh(t0) - l), p1 = __expf(sc.z_of_tanh(t1) - l);
      if (i + 2 * j == t) p0 -= 1.0f;
      if (i + 2 * j + 1 == t) p1 -= 1.0f;
      op[j] = pack_bf16x2(p0 * g * __fmaf_rn(-t0, t0, 1.0f), p1 * g * __fmaf_rn(-t1, t1, 1.0f));
    }
    const int valid = vocab - i;
    if (valid < 8) {                     // ragged last piece: nothing is stored past the vocabulary
      const __nv_bfloat16* ov = reinterpret_cast<const __nv_bfloat16*>(&o);
      for (int j = 0; j < valid; ++j) d[row * ld_d + i + j] = ov[j];
    } else {
      *reinterpret_cast<uint4*>(d + row * ld_d + i) = o;
    }
  }
}

// ---------------------------------------------------------------------------------------
// Loss and gradient from ONE read of the logits.  The pair of kernels above moves 8 bytes per logit (read, tanh
// out; tanh in, gradient out) and wants rows of a 16-byte pitch, which costs a vocabulary like 50257 a padding copy
// in and a compacting one out: 1.8 of 2.5 ms at 8192 x 50257.  Here a row's tanh values stay in shared memory
// between the softmax sum and the gradient, so a logit is read once (2 bytes) and its gradient written once (2).
//
// Rows of any alignment: a row is cut at the 16-byte boundaries of MEMORY, not of the row (its first and last
// piece may belong to two rows and go element by element), and the gradient, laid out like the logits, is cut alike.
//
// bf16(tanh(bf16(x / c))) by table over the bits of x.  From 4 c on it is +-1.  Below `lo`, a power of two at most
// c / 128, the quotient is below 2^-6 and tanh is the identity after rounding, so t(x) is the rounded quotient and the
// quotients of one binade are those of the next with another exponent: bits(t(x)) = bits(t(x')) + bits(x) - bits(x')
// for the x' of the `lo` binade with x's mantissa.  In between: at most 11 binades x 128 mantissas, 2.8 KB.
// (The 64 KB table of the forward kernel leaves no room for a row; with this one two blocks fit on an SM even
// at 50304 columns, so that one block's stores overlap the other's loads.)  Magnitudes below 2^-111 are taken as 2^-111:
// their capped value is far below half an ulp of anything it meets.  A NaN would look up 1: a row's largest
// magnitude is tracked and a NaN in it makes the row's sum, and with it the loss and the gradient, NaN.
//
// The sum of exp(z), two ways.  Rows that are whole pieces (the vocabulary a multiple of 8) sum exactly as softcap_ce_fwd_kernel
// does -- running maximum, 512 threads, the same order -- so that the log-sum and with it every bit of the gradient equal those
// of the pair of kernels: a last bit there, amplified by the e4m3 roundings of a deep backward pass, is another trajectory.
// Ragged rows, which that kernel could only sum after a copy, skip the running maximum (|z| <= c <= 64: the sum neither
// overflows nor loses its terms) and take as many threads as fill their last pass.
//
// One thread block per row (one warp for rows up to 2048 columns); a thread meets the same pieces in both passes and has places of its own
// for them, counted from the row's first whole piece, so the only synchronisation is the reduction of the sum.  (Counted from the row's first
// boundary, a place changes hands where a ragged row is followed by an even one: a warp a row ahead overwrote what its neighbour was still to read.)
// Bound by instruction issue and the ALU pipe (49 warp instructions per 64 logits, two of them ex2 in each pass), no longer by
// memory.  8192 x 50257: 699 us for the two kernels, 2507 with the copies -> 415 us (DRAM floor 251); 8192 x 50304: 704 -> 462.
// ---------------------------------------------------------------------------------------
constexpr int kCeMaxThreads = 640;
constexpr int kCeWarpCols = 2048;                 // rows up to this wide take one warp
constexpr int kCeSmemLimit = 226 * 1024;
constexpr int kCeTableMax = 11 * 128 + 2;
constexpr int kCeTableBytes = (kCeTableMax * 2 + 15) / 16 * 16;
constexpr uint32_t kCeFloor2 = 0x08000800u;
constexpr float kLog2e = 1.4426950408889634f;

struct CeArgs {
  const __nv_bfloat16* logits;
  const void* targets;
  int targets_64;
  float cap;
  __nv_bfloat16* d;
  const float* gscale;
  int only_if_scaled;
  float* nll;
  int rows, vocab;
  int64_t ld;
};

__device__ __forceinline__ float ex2(float v) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(v));
  return e;
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}

template <bool WARP, bool WHOLE>
__global__ void __launch_bounds__(WARP ? 256 : WHOLE ? kLossFwdThreads : kCeMaxThreads, WARP ? 4 : 2) softcap_ce_kernel(const CeArgs p) {
  grid_trigger();
  if (p.only_if_scaled) {
    grid_wait();
    if (*p.gscale == 1.0f) return;
  }
  extern __shared__ __align__(16) uint8_t s_ce[];
  __shared__ float s_sum[2][kCeMaxThreads / 32];
  __shared__ float s_lse;
  const Softcap sc(p.cap);
  // the power-of-two edges of the table as bf16 bits: 2^floor(log2 c) is c with its mantissa cleared
  const uint32_t c_pow = (__float_as_uint(sc.c) >> 16) & 0x7f80u;
  const uint32_t lo = c_pow - (7u << 7), hi = c_pow + (3u << 7);      // c / 256 < lo <= c / 128; 4 c < hi <= 8 c
  uint16_t* table = reinterpret_cast<uint16_t*>(s_ce);
  for (uint32_t i = threadIdx.x; i <= hi - lo; i += blockDim.x)
    table[i] = uint16_t(__float_as_uint(tanh_bf16(sc.quotient(__uint_as_float((lo + i) << 16)))) >> 16);
  __syncthreads();
  grid_wait();            // (the table comes from the cap alone)

  const uint32_t lo2 = lo * 0x10001u, hi2 = hi * 0x10001u;
  // (address of entry 0) - 2 lo, once per half: the sum with a pair of doubled indexes is two 16-bit addresses
  // (shared addresses of the table are far below 2^16, and a 32-bit sum of the two halves is exact)
  const uint32_t tab = uint32_t(__cvta_generic_to_shared(s_ce)) - 2u * lo, tab2 = tab + (tab << 16);
  const int nt = WARP ? 32 : int(blockDim.x), tid = WARP ? int(threadIdx.x & 31) : int(threadIdx.x);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slots = (p.vocab + 14) / 8;                               // 16-byte pieces a row can touch
  uint4* row_t = reinterpret_cast<uint4*>(s_ce + kCeTableBytes) + (WARP ? warp * slots : 0);
  const float gs = (p.gscale != nullptr ? *p.gscale : 1.0f) * (1.0f / float(p.rows));
  const float2 l2e = make_float2(kLog2e, kLog2e), gs2 = make_float2(gs, gs);
  const float2 one = make_float2(1.f, 1.f), minus1 = make_float2(-1.f, -1.f);
  const __nv_bfloat162 c2 = __float2bfloat162_rn(sc.c);
  const int step = WARP ? int(gridDim.x) * 8 : int(gridDim.x);
  int row = WARP ? int(blockIdx.x) * 8 + warp : int(blockIdx.x);

  struct Row {
    const __nv_bfloat16* base;     // the row's first 16-byte boundary at or below its start
    int off;                       // elements of that piece which belong to the row before
    int first, last;               // the whole pieces [first, last): at most one ragged piece before and one after
  };
  auto row_of = [&](int r) {
    Row q;
    const __nv_bfloat16* s = p.logits + int64_t(r) * p.ld;
    q.off = int((reinterpret_cast<uintptr_t>(s) & 15u) >> 1);
    q.base = s - q.off;
    q.first = q.off != 0;
    q.last = (q.off + p.vocab) >> 3;
    return q;
  };
  auto load = [&](const Row& q, int i) -> uint4 { return i < q.last ? ld_stream_v4(q.base + i * 8) : make_uint4(0u, 0u, 0u, 0u); };
  // the tanh values of a pair of logits
  auto tanh_pair = [&](uint32_t w, uint32_t mag) {
    const uint32_t m = __vmaxu2(mag, kCeFloor2);
    const uint32_t at = __vmaxu2(mag, (mag & 0x007f007fu) + lo2);
    const uint32_t addr = (__vminu2(at, hi2) << 1) + tab2;
    const uint32_t t_lo = lds_u16(addr & 0xffffu), t_hi = lds_u16(addr >> 16);
    // (no carry crosses the halves: t + m <= 0xffff, and t + m >= at by construction)
    return (__byte_perm(t_lo, t_hi, 0x5410) + m - at) | (w & 0x80008000u);
  };
  // bf16(c t) of a pair: the product of two bf16 values rounded once, as the float product rounded to bf16 is
  auto capped = [&](uint32_t t2) {
    const __nv_bfloat162 z = __hmul2(c2, *reinterpret_cast<const __nv_bfloat162*>(&t2));
    return bf16x2_unpack(*reinterpret_cast<const uint32_t*>(&z));
  };
  // the ragged pieces of a row, an element per lane of the last warp: lanes 0..7 the piece before the whole ones, lanes
  // 8..15 the piece after them.  (One thread per piece, element after element, held every row up by 8 %.)
  auto edge_of = [&](const Row& q) {
    const int end = q.off + p.vocab;
    if (!WARP && warp != nt / 32 - 1) return -1;
    if (lane < 8) return q.off != 0 && lane >= q.off && lane < end ? lane : -1;
    const int e = q.last * 8 + lane - 8;
    return lane < 16 && q.last >= q.first && e < end ? e : -1;
  };
  auto grad1 = [&](float t, float z, float lse, bool hit) {
    const float pr = ex2(__fmul_rn(z - lse, kLog2e)) - (hit ? 1.0f : 0.0f);
    return __float2bfloat16_rn(__fmul_rn(__fmul_rn(pr, gs), __fmaf_rn(__fmul_rn(t, t), -1.0f, 1.0f)));
  };

  if (row >= p.rows) return;
  Row q = row_of(row);
  uint4 w0 = load(q, q.first + tid), w1 = load(q, q.first + tid + nt);
  for (int it = 0; row < p.rows; row += step, ++it) {
    // ---- tanh values and the sum of exp(z)
    float2 acc = make_float2(0.f, 0.f);
    float m_run = -3.0e38f, s_run = 0.f;          // WHOLE: running maximum and sum (of a lane of one of the row's warps)
    float m_row = -3.0e38f, s_row = 0.f;          // WARP && WHOLE: what the warps before this pass have found
    uint32_t top = 0u;
    auto warp_lse = [&] {                         // the sum over a warp's lanes, in lane 0's order
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        lse_merge(m_run, s_run, __shfl_xor_sync(0xffffffffu, m_run, o), __shfl_xor_sync(0xffffffffu, s_run, o));
    };
    // (one warp per row takes the part of warp 0, 1, ... of a block in turn: its passes are full up to the last, so that the
    // shuffles meet every lane)
    const int end = WARP && WHOLE ? (q.last + 31) & ~31 : q.last;
    for (int i = q.first + tid; i < end; i += nt) {
      const uint4 w = w0;
      w0 = w1;
      w1 = load(q, i + 2 * nt);
      const uint32_t wi[4] = {w.x, w.y, w.z, w.w};
      uint4 to;
      uint32_t* tp = &to.x;
      float2 z[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t mag = wi[j] & 0x7fff7fffu;
        top = __vmaxu2(top, mag);
        tp[j] = tanh_pair(wi[j], mag);
        z[j] = capped(tp[j]);
      }
      if (!(WARP && WHOLE) || i < q.last) row_t[i - q.first] = to;
      if constexpr (WHOLE) {
        if (!WARP || i < q.last) {
          const float mx = fmaxf(fmaxf(fmaxf(z[0].x, z[0].y), fmaxf(z[1].x, z[1].y)), fmaxf(fmaxf(z[2].x, z[2].y), fmaxf(z[3].x, z[3].y)));
          const float mn = fmaxf(m_run, mx);
          const float2 nmn = make_float2(-mn, -mn);
          float2 a2 = make_float2(s_run * __expf(m_run - mn), 0.f);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 dz = __fmul2_rn(__fadd2_rn(z[j], nmn), l2e);
            a2 = __fadd2_rn(a2, make_float2(ex2(dz.x), ex2(dz.y)));
          }
          s_run = a2.x + a2.y;
          m_run = mn;
        }
        if constexpr (WARP) {
          warp_lse();
          lse_merge(m_row, s_row, m_run, s_run);
          m_run = -3.0e38f;
          s_run = 0.f;
        }
      } else {
        float2 e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 zl = __fmul2_rn(z[j], l2e);
          e[j] = make_float2(ex2(zl.x), ex2(zl.y));
        }
        acc = __fadd2_rn(acc, __fadd2_rn(__fadd2_rn(e[0], e[1]), __fadd2_rn(e[2], e[3])));
      }
    }
    const int e_mine = WHOLE ? -1 : edge_of(q);
    uint32_t t_edge = 0u;
    if (!WHOLE && e_mine >= 0) {
      const uint32_t w = reinterpret_cast<const unsigned short*>(q.base)[e_mine];
      t_edge = tanh_pair(w, w & 0x7fffu) & 0xffffu;
      top = __vmaxu2(top, w & 0x7fffu);
      acc.x += ex2(__fmul_rn(capped(t_edge).x, kLog2e));
    }
    // the next row's first pieces are on their way while this one is finished
    const Row now = q;
    if (row + step < p.rows) {
      q = row_of(row + step);
      w0 = load(q, q.first + tid);
      w1 = load(q, q.first + tid + nt);
    }
    const bool nan = (top & 0xffffu) > 0x7f80u || (top >> 16) > 0x7f80u;
    float lse;
    if constexpr (WHOLE && WARP) {
      lse = __shfl_sync(0xffffffffu, m_row + logf(s_row), 0);
      if (__any_sync(0xffffffffu, nan)) lse = __int_as_float(0x7fffffff);
    } else if constexpr (WHOLE) {
      if (nan) s_run = __int_as_float(0x7fffffff);
      warp_lse();
      if (lane == 0) {
        s_sum[0][warp] = m_run;
        s_sum[1][warp] = s_run;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        m_run = s_sum[0][0];
        s_run = s_sum[1][0];
#pragma unroll
        for (int wi = 1; wi < kLossFwdThreads / 32; ++wi) lse_merge(m_run, s_run, s_sum[0][wi], s_sum[1][wi]);
        s_lse = m_run + logf(s_run);
      }
      __syncthreads();
      lse = s_lse;
    } else {
      float s = nan ? __int_as_float(0x7fffffff) : acc.x + acc.y;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (!WARP) {
        if (lane == 0) s_sum[it & 1][warp] = s;
        __syncthreads();
        s = lane < nt / 32 ? s_sum[it & 1][lane] : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      }
      lse = logf(s);
    }
    const float2 nl2 = make_float2(-lse, -lse);
    int64_t t = p.targets_64 ? static_cast<const int64_t*>(p.targets)[row] : static_cast<const int32_t*>(p.targets)[row];
    t = t < 0 ? 0 : (t >= p.vocab ? p.vocab - 1 : t);                 // clamped, as jnp.take_along_axis does
    const int at = int(t) + now.off, piece = at >> 3;                 // the target's place in the row's pieces
    const bool own = piece >= now.first && piece < now.last && (piece - now.first) % nt == tid;
    const uint16_t* row_e = reinterpret_cast<const uint16_t*>(row_t - now.first);
    // ---- the gradient: gscale / rows * (exp(z - lse) - [target]) * (1 - t^2)
    if (p.d != nullptr) {
      __nv_bfloat16* dp = p.d + (now.base - p.logits);
      for (int i = now.first + tid; i < now.last; i += nt) {
        const uint4 tw = row_t[i - now.first];
        const uint32_t ti[4] = {tw.x, tw.y, tw.z, tw.w};
        uint4 o;
        uint32_t* op = &o.x;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 tf = bf16x2_unpack(ti[j]);
          const float2 zl = __fmul2_rn(__fadd2_rn(capped(ti[j]), nl2), l2e);
          const float2 pr = __fmul2_rn(make_float2(ex2(zl.x), ex2(zl.y)), gs2);
          const float2 r = __fmul2_rn(pr, __ffma2_rn(__fmul2_rn(tf, tf), minus1, one));   // t^2 is exact
          op[j] = pack_bf16x2(r.x, r.y);
        }
        *reinterpret_cast<uint4*>(dp + i * 8) = o;
      }
      if (e_mine >= 0) dp[e_mine] = grad1(bf16lo(t_edge), capped(t_edge).x, lse, e_mine == at);
      if (own) {                                                      // the target's own element again, now with its -1
        const uint32_t t2 = row_e[at];
        dp[at] = grad1(bf16lo(t2), capped(t2).x, lse, true);
      }
    }
    // ---- the target's log-probability, by the thread that holds it
    if (p.nll != nullptr) {
      if (own) p.nll[row] = lse - capped(row_e[at]).x;
      if (e_mine == at) p.nll[row] = lse - capped(t_edge).x;
    }
  }
}

// ---------------------------------------------------------------------------------------
// The same for ragged rows of a large problem, with the exponentials taken once.  softcap_ce_kernel keeps the tanh values of a row and takes
// exp(z) again for the gradient; here the first pass leaves g = exp(z) (1 - t^2) behind in float32, and the second is a scaling,
//     gradient = g / sum * gscale / rows      (the target's element is computed by itself, with its -1),
// a load, two packed multiplications and a conversion per pair.  A row of 50257 such values is 201 KB: eight pieces of each thread go to
// tensor memory, which nothing else here uses (a group of 512 threads has 128 KB of it), the others to shared memory, so that TWO rows
// are in flight on an SM, one in its first pass while the other is in its second.  One thread block per SM, so there is
// room for tanh of every bf16 magnitude (64 KB) as well: a look-up is then an address and a load, with no range tests and no
// bookkeeping for NaN.
//
// 37 warp instructions per 64 logits instead of 49.  What bounds it: three fifths of the peak of instruction issue and of the shared-memory
// pipe each (a look-up of 32 random entries takes 3.5 cycles) and three quarters of the copy rate.  The loads come through the L2: one
// thread fetches its row's pieces four passes ahead with a bulk prefetch (without: 383 us at 8192 x 50257, with whole rows ahead 398, so 336).
//
// The exponent's argument is z log2 e instead of (z - lse) log2 e: smaller, so its rounding costs the gradient less (the sum's order
// and the last bits of the gradient are other ones than softcap_ce_kernel's).
//
// 8192 x 50257 406 -> 336 us (4.9 TB/s), 8192 x 25001 226 -> 179, 2048 x 50257 105 -> 93, 4096 x 9001 60 -> 51.  The rule (softcap_ce_kernel / this one, with
// a gradient; without one in brackets):
//   columns   8201 leave a third pass nearly empty (3000 rows 39.4 / 40.8, 30.8 / 35.3), 8929 no longer (3952 rows 55.9 / 51.7, 44.2 / 43.4), 9001 (45.5 / 41.2, 35.6 / 35.6).
//   rounds    two rows per SM at a time, 296 in all, and the table's 64 KB to begin with.  A last round of a few rows costs as much as a full one here,
//             there a row alone on its SM is faster: 620 x 50257 38.8 / 42.5 (27.3 / 30.9), 700 x 32003 28.4 / 30.7, 920 x 25001 31.2 / 32.6 (22.6 / 25.6), but 722 x 34425
//             36.8 / 32.6 (27.5 / 24.9), 1251 x 22492 38.6 / 35.5 (29.6 / 28.9), 1248 x 20001 33.8 / 33.0 (25.2 / 26.8), 1248 x 15441 28.1 / 28.7 (21.0 / 23.5), 1600 x 12301 33.2 / 31.0 (25.1 / 25.6).  So with six
//             rounds and more, or a last one of more than two fifths, from 18 M logits on (1184 x 15441 25.6 / 25.3 (19.4 / 20.4)); five with a shorter one from 24 M.
//             One rule for both, so that a loss has the same bits with and without a gradient; it goes by the gradient's time, and without one is up to 7 %
//             slower than softcap_ce_kernel at the smallest of these (800 x 25001 20.2 / 21.7), faster from 30 M on.
// ---------------------------------------------------------------------------------------
constexpr int kCgMinCols = 8704;
constexpr int kCgThreads = 512, kCgGroups = 2;
constexpr int kCgAhead = 4;                                  // pieces of a thread that are on their way to the L2
constexpr int kCgTmemSlots = 8;                              // pieces of a thread in tensor memory
constexpr int kCgSlotBytes = kCgThreads * 32;                // a piece of every thread: eight floats each
constexpr int kCgSmemSlots = (kCeSmemLimit - kTanhBytes) / (kCgGroups * kCgSlotBytes);
constexpr int kCgMaxCols = (kCgTmemSlots + kCgSmemSlots) * kCgThreads * 8;

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float2 (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "f"(v[0].x), "f"(v[0].y), "f"(v[1].x), "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x), "f"(v[3].y) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float2 (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[2].x), "=f"(v[2].y), "=f"(v[3].x), "=f"(v[3].y)
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld8(float2 (&v)[4]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(v[0].x), "+f"(v[0].y), "+f"(v[1].x), "+f"(v[1].y), "+f"(v[2].x), "+f"(v[2].y), "+f"(v[3].x), "+f"(v[3].y)::"memory");
}

__global__ void __launch_bounds__(kCgThreads * kCgGroups, 1) softcap_ce_groups_kernel(const CeArgs p, int smem_slots) {
  if (p.only_if_scaled) {
    grid_wait();
    if (*p.gscale == 1.0f) return;
  }
  extern __shared__ __align__(16) uint8_t s_cg[];
  __shared__ float s_sum[kCgGroups][2][kCgThreads / 32];
  __shared__ uint32_t s_tmem;
  const Softcap sc(p.cap);
  const uint32_t lane = threadIdx.x & 31;
  const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0);
  const int group = warp / (kCgThreads / 32), gw = warp % (kCgThreads / 32), tid = int(threadIdx.x) % kCgThreads;
  if (warp == 0) {
    tmem_alloc(smem_u32(&s_tmem), 512);
    tmem_relinquish();
  }
  {
    // bf16(tanh(bf16(x / c))) by the magnitude of x.  From 4 c on it is 1, for infinity too; a NaN stays one.
    const uint32_t one_from = ((__float_as_uint(sc.c) >> 16) & 0x7f80u) + (3u << 7);
    uint16_t* table = reinterpret_cast<uint16_t*>(s_cg);
    for (uint32_t i = threadIdx.x; i < uint32_t(kTanhEntries); i += blockDim.x)
      table[i] = i > 0x7f80u ? uint16_t(0x7fffu) : i >= one_from ? uint16_t(0x3f80u)
                 : uint16_t(__float_as_uint(tanh_bf16(sc.quotient(__uint_as_float(i << 16)))) >> 16);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_trigger();         // (not before the tensor memory is there: a kernel that started early could take it and wait for this one)
  grid_wait();            // (the table comes from the cap alone)

  // a warp reads and writes the lanes 32 (warp % 4).. of tensor memory; the four warps of a group that share them have 64 columns each
  const uint32_t taddr0 = *reinterpret_cast<volatile uint32_t*>(&s_tmem) + (uint32_t(warp & 3) << 21) + uint32_t(group * 256 + (gw >> 2) * 64);
  float4* spill = reinterpret_cast<float4*>(s_cg + kTanhBytes) + group * smem_slots * (kCgSlotBytes / 16) + tid;
  const uint32_t tab = smem_u32(s_cg);
  const float gs = (p.gscale != nullptr ? *p.gscale : 1.0f) * (1.0f / float(p.rows));
  const float2 l2e = make_float2(kLog2e, kLog2e), one = make_float2(1.f, 1.f), minus1 = make_float2(-1.f, -1.f);
  const __nv_bfloat162 c2 = __float2bfloat162_rn(sc.c);
  const int step = int(gridDim.x) * kCgGroups;
  int row = int(blockIdx.x) * kCgGroups + group;

  struct Row {
    const __nv_bfloat16* base;     // the row's first 16-byte boundary at or below its start
    int off;                       // elements of that piece which belong to the row before
    int first, last;               // the whole pieces [first, last): at most one ragged piece before and one after
  };
  auto row_of = [&](int r) {
    Row q;
    const __nv_bfloat16* s = p.logits + int64_t(r) * p.ld;
    q.off = int((reinterpret_cast<uintptr_t>(s) & 15u) >> 1);
    q.base = s - q.off;
    q.first = q.off != 0;
    q.last = (q.off + p.vocab) >> 3;
    return q;
  };
  auto target_of = [&](int r) {
    const int64_t t = p.targets_64 ? static_cast<const int64_t*>(p.targets)[r] : static_cast<const int32_t*>(p.targets)[r];
    return int(t < 0 ? 0 : (t >= p.vocab ? p.vocab - 1 : t));         // clamped, as jnp.take_along_axis does
  };
  // (past the end: the last piece again, whose values are then not used)
  auto load = [&](const Row& q, int i) -> uint4 { return ld_stream_v4(q.base + min(i, q.last - 1) * 8); };
  // n pieces of a row, from its whole piece `at` on, into the L2
  auto prefetch = [&](const Row& q, int at, int n) {
    n = min(n, q.last - q.first - at);
    if (n > 0) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(q.base + (q.first + at) * 8), "r"(n * 16) : "memory");
  };
  auto tanh_pair = [&](uint32_t w) {
    const uint32_t lo = lds_u16(tab + ((w << 1) & 0xfffeu)), hi = lds_u16(tab + ((w >> 15) & 0xfffeu));
    return __byte_perm(lo, hi, 0x5410) | (w & 0x80008000u);
  };
  // bf16(c t) of a pair: the product of two bf16 values rounded once, as the float product rounded to bf16 is
  auto capped = [&](uint32_t t2) {
    const __nv_bfloat162 z = __hmul2(c2, *reinterpret_cast<const __nv_bfloat162*>(&t2));
    return bf16x2_unpack(*reinterpret_cast<const uint32_t*>(&z));
  };
  // the ragged pieces, an element per lane of the group's last warp: lanes 0..7 the piece before the whole ones, 8..15 the one after
  auto edge_of = [&](const Row& q) {
    const int end = q.off + p.vocab;
    if (gw != kCgThreads / 32 - 1) return -1;
    if (lane < 8) return q.off != 0 && int(lane) >= q.off && int(lane) < end ? int(lane) : -1;
    const int e = q.last * 8 + int(lane) - 8;
    return lane < 16 && q.last >= q.first && e < end ? e : -1;
  };
  auto grad1 = [&](float t, float z, float lse, bool hit) {
    const float pr = ex2(__fmul_rn(z - lse, kLog2e)) - (hit ? 1.0f : 0.0f);
    return __float2bfloat16_rn(__fmul_rn(__fmul_rn(pr, gs), __fmaf_rn(__fmul_rn(t, t), -1.0f, 1.0f)));
  };

  if (row < p.rows) {
    Row q = row_of(row);
    int target = target_of(row);
    uint4 w0 = load(q, q.first + tid), w1 = load(q, q.first + tid + kCgThreads);
    for (int it = 0; row < p.rows; row += step, ++it) {
      const int at = target + q.off;                                  // the target's place in the row's pieces
      const uint32_t x_at = reinterpret_cast<const unsigned short*>(q.base)[at];
      if (row + step < p.rows) target = target_of(row + step);
      // ---- the sum of exp(z), and g of every element.  (Whole warps: a store to tensor memory is the warp's.)
      float2 acc = make_float2(0.f, 0.f);
      const int mine = q.first + tid, n_k = (q.last - q.first - gw * 32 + kCgThreads - 1) / kCgThreads;
      auto first_pass = [&](const uint4& w, int k, float2 (&g)[4]) {
        const uint32_t wi[4] = {w.x, w.y, w.z, w.w};
        float2 e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t t2 = tanh_pair(wi[j]);
          const float2 tf = bf16x2_unpack(t2), zl = __fmul2_rn(capped(t2), l2e);
          e[j] = make_float2(ex2(zl.x), ex2(zl.y));
          g[j] = __fmul2_rn(e[j], __ffma2_rn(__fmul2_rn(tf, tf), minus1, one));   // t^2 is exact
        }
        const float2 sum = __fadd2_rn(__fadd2_rn(e[0], e[1]), __fadd2_rn(e[2], e[3]));
        if (mine + k * kCgThreads < q.last) acc = __fadd2_rn(acc, sum);
      };
      auto keep = [&](int k, const float2 (&g)[4]) {
        if (k < kCgTmemSlots) {
          tmem_st8(taddr0 + 8 * k, g);
          return;
        }
        float4* d = spill + (k - kCgTmemSlots) * (2 * kCgThreads);
        d[0] = make_float4(g[0].x, g[0].y, g[1].x, g[1].y);
        d[kCgThreads] = make_float4(g[2].x, g[2].y, g[3].x, g[3].y);
      };
#pragma unroll 1
      for (int k = 0; k < n_k; k += 2) {
        float2 g[4];
        if (tid == 0) prefetch(q, (k + kCgAhead) * kCgThreads, 2 * kCgThreads);
        first_pass(w0, k, g);
        w0 = load(q, mine + (k + 2) * kCgThreads);
        if (p.d != nullptr) keep(k, g);
        if (k + 1 < n_k) {
          first_pass(w1, k + 1, g);
          w1 = load(q, mine + (k + 3) * kCgThreads);
          if (p.d != nullptr) keep(k + 1, g);
        }
      }
      const int e_mine = edge_of(q);
      uint32_t t_edge = 0u;
      if (e_mine >= 0) {
        t_edge = tanh_pair(reinterpret_cast<const unsigned short*>(q.base)[e_mine]) & 0xffffu;
        acc.x += ex2(__fmul_rn(capped(t_edge).x, kLog2e));
      }
      // the next row's first pieces are on their way while this one is finished
      const Row now = q;
      if (row + step < p.rows) {
        q = row_of(row + step);
        if (tid == 0) prefetch(q, 2 * kCgThreads, (kCgAhead - 2) * kCgThreads);
        w0 = load(q, q.first + tid);
        w1 = load(q, q.first + tid + kCgThreads);
      }
      float s = acc.x + acc.y;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) s_sum[group][it & 1][gw] = s;
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kCgThreads) : "memory");
      s = lane < kCgThreads / 32 ? s_sum[group][it & 1][lane] : 0.f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const float lse = logf(s), inv = __frcp_rn(s);
      const int piece = at >> 3;
      const bool own = piece >= now.first && piece < now.last && (piece - now.first) % kCgThreads == tid;
      const uint32_t t_at = tanh_pair(x_at) & 0xffffu;
      // ---- the gradient: g, 1 / sum and gscale / rows multiplied
      if (p.d != nullptr) {
        __nv_bfloat16* dp = p.d + (now.base - p.logits);
        // by the product of the last two.  Where that is no normal number (its product with g still may be one) gscale goes in 2^64 times as
        // large and g 2^64 times as small, both exact where the result is no zero: a gradient scaled by a power of two has the same digits.
        const bool direct = !(fabsf(__fmul_rn(inv, gs)) < 1.2e-38f);
        const float factor = __fmul_rn(inv, direct ? gs : gs * 0x1p64f);
        const float2 f2 = make_float2(factor, factor), down = make_float2(0x1p-64f, 0x1p-64f);
        auto second_pass = [&](float2 (&g)[4], int i) {
          uint4 o;
          uint32_t* op = &o.x;
          if (!direct) {
#pragma unroll
            for (int j = 0; j < 4; ++j) g[j] = __fmul2_rn(g[j], down);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 r = __fmul2_rn(g[j], f2);
            op[j] = pack_bf16x2(r.x, r.y);
          }
          if (i < now.last) *reinterpret_cast<uint4*>(dp + i * 8) = o;
        };
#pragma unroll 2
        for (int k = 0; k < min(n_k, kCgTmemSlots); ++k) {
          float2 g[4];
          tmem_ld8(taddr0 + 8 * k, g);
          tmem_wait_ld8(g);
          second_pass(g, mine + k * kCgThreads);
        }
#pragma unroll 2
        for (int k = kCgTmemSlots; k < n_k; ++k) {
          const float4* d = spill + (k - kCgTmemSlots) * (2 * kCgThreads);
          const float4 a = d[0], b = d[kCgThreads];
          float2 g[4] = {make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y), make_float2(b.z, b.w)};
          second_pass(g, mine + k * kCgThreads);
        }
        if (e_mine >= 0) dp[e_mine] = grad1(bf16lo(t_edge), capped(t_edge).x, lse, e_mine == at);
        if (own) dp[at] = grad1(bf16lo(t_at), capped(t_at).x, lse, true);      // the target's own element again, now with its -1
      }
      // ---- the target's log-probability
      if (p.nll != nullptr && (own || e_mine == at)) p.nll[row] = lse - capped(t_at).x;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(*reinterpret_cast<volatile uint32_t*>(&s_tmem), 512);
  }
}

// Mean of n floats, to the bit what torch's mean of a contiguous vector gives (measured up to 65536 values): T threads, T the largest
// power of two in n / 4 but at most 512; thread j adds the 16-byte pieces j, j + T, ... value by value, the first thread's values also those
// after the last whole piece, one per thread; the four sums in order, then halves of T.  Below 128 values T is the largest power of
// two in n and thread j has v[j] + v[j + T].  One block launched early; torch's own goes through the dispatcher and waits for the
// kernel before it, which a step of the small model, bound by its host time, shows (352 us without, 363 with it and the parameters'
// check in Python, 347 with neither).
constexpr int kMeanThreads = 512;
constexpr int64_t kMeanMax = 65536;
__global__ void __launch_bounds__(kMeanThreads) mean_kernel(const float* __restrict__ v, int n, int threads, float factor, float* __restrict__ out) {
  __shared__ float s_sum[kMeanThreads];
  const int j = int(threadIdx.x);
  grid_trigger();
  grid_wait();
  v = loads_below(v);
  float t = 0.f;
  if (n < 128) {
    if (j < threads) t = j + threads < n ? v[j] + v[j + threads] : v[j];
  } else if (j < threads) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    const int pieces = n / 4;
#pragma unroll 4
    for (int i = j; i < pieces; i += threads) {
      const float4 w = reinterpret_cast<const float4*>(v)[i];
      a.x += w.x; a.y += w.y; a.z += w.z; a.w += w.w;
    }
    if (pieces * 4 + j < n) a.x += v[pieces * 4 + j];
    t = ((a.x + a.y) + a.z) + a.w;
  }
  s_sum[j] = t;
  for (int h = threads / 2; h >= 32; h >>= 1) {
    __syncthreads();
    if (j < h) s_sum[j] = t = t + s_sum[j + h];
  }
  if (j < 32) {
    const int top = threads / 2 < 16 ? threads / 2 : 16;
    for (int h = top; h > 0; h >>= 1) t += __shfl_down_sync(0xffffffffu, t, h);
    if (j == 0) *out = t * factor;
  }
}

// (`sms`: the row's rounds are counted for so many)
static bool ce_in_groups(int64_t rows, int64_t vocab, int64_t sms) {
  if (vocab < kCgMinCols || vocab > kCgMaxCols) return false;
  const int64_t at_once = kCgGroups * sms, rounds = (rows + at_once - 1) / at_once, logits = rows * vocab;
  const bool filled = 5 * (rows - (rounds - 1) * at_once) > 2 * at_once;
  if (rounds >= 6 || filled) return logits >= 18'000'000;
  return rounds == 5 && logits >= 24'000'000;
}

constexpr int kCeSmemMax = kCeSmemLimit;
static int64_t ce_smem(int64_t vocab) {
  const int64_t row = (vocab + 14) / 8 * 16;
  return kCeTableBytes + (vocab <= kCeWarpCols ? 8 * row : row);
}

}  // namespace tg

using namespace tg;

extern "C" int tgh_mean(const float* v, int64_t n, float* out, void* stream) {
  if (n <= 0 || v == nullptr || out == nullptr) return TG_ERR_SHAPE;
  if (n > kMeanMax) return TG_ERR_TOO_LARGE;
  if (!aligned16(v)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  const int64_t most = n < 128 ? n : n / 4;
  int threads = 1;
  while (2 * threads <= most && threads < kMeanThreads) threads *= 2;
  TG_CUDA_CHECK(launch_early(mean_kernel, 1, kMeanThreads, 0, static_cast<cudaStream_t>(stream), v, int(n), threads, 1.0f / float(n), out));
  return TG_OK;
}

extern "C" int tgh_softcap_ce_fits(float cap, int64_t rows, int64_t vocab) {
  // the cap: exp(cap) and the table's exponents stay in range (see softcap_ce_kernel)
  return cap >= 0x1p-10f && cap <= 64.0f && rows <= INT32_MAX && vocab > 0 && vocab < (1 << 24) && ce_smem(vocab) <= kCeSmemMax;
}

extern "C" int tgh_softcap_ce_in_groups(int64_t rows, int64_t vocab) { return ce_in_groups(rows, vocab, sm_count()); }

extern "C" int tgh_softcap_ce(const void* logits, const void* targets, int targets_64, float cap, void* dlogits, const float* gscale,
                              int only_if_scaled, float* nll, int64_t rows, int64_t vocab, int64_t ld, void* stream) {
  if (rows < 0 || vocab <= 0 || ld < vocab || (only_if_scaled && gscale == nullptr))
    return TG_ERR_SHAPE;
  if (!tgh_softcap_ce_fits(cap, rows, vocab)) return TG_ERR_TOO_LARGE;
  if (!aligned16(logits) || !aligned16(dlogits)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CeArgs a = {static_cast<const __nv_bfloat16*>(logits), targets, targets_64, cap, static_cast<__nv_bfloat16*>(dlogits), gscale,
              only_if_scaled, nll, int(rows), int(vocab), ld};
  if (rows > 0) {
    static std::atomic<bool> attr_set[64];
    int dev = 0;
    TG_CUDA_CHECK(cudaGetDevice(&dev));
    if (!attr_set[dev & 63].load(std::memory_order_acquire)) {
      for (auto kern : {softcap_ce_kernel<false, false>, softcap_ce_kernel<false, true>, softcap_ce_kernel<true, false>, softcap_ce_kernel<true, true>})
        TG_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kCeSmemMax));
      TG_CUDA_CHECK(cudaFuncSetAttribute(softcap_ce_groups_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCeSmemMax));
      attr_set[dev & 63].store(true, std::memory_order_release);
    }
    const size_t smem = size_t(ce_smem(vocab));
    const int64_t per_sm_smem = std::max<int64_t>(1, (227 * 1024) / int64_t(smem + 1024));
    const bool whole = vocab % 8 == 0 && ld % 8 == 0, is_short = rows * vocab <= 1 << 20;
    if (vocab <= kCeWarpCols) {
      const int64_t cap_blocks = int64_t(sm_count()) * std::min<int64_t>(per_sm_smem, 4);
      const int blocks = int(std::min<int64_t>((rows + 7) / 8, cap_blocks));
      TG_CUDA_CHECK(launch_if_short(is_short, whole ? softcap_ce_kernel<true, true> : softcap_ce_kernel<true, false>, dim3(unsigned(blocks)), 256,
                                    smem, st, a));
    } else if (whole) {
      const int64_t cap_blocks = int64_t(sm_count()) * std::min<int64_t>(per_sm_smem, 2);
      TG_CUDA_CHECK(launch_if_short(is_short, softcap_ce_kernel<false, true>, dim3(unsigned(std::min<int64_t>(rows, cap_blocks))), kLossFwdThreads,
                                    smem, st, a));
    } else if (ce_in_groups(rows, vocab, sm_count())) {
      const int slots = int(std::max<int64_t>(0, (vocab / 8 + kCgThreads - 1) / kCgThreads - kCgTmemSlots));
      const int blocks = int(std::min<int64_t>((rows + kCgGroups - 1) / kCgGroups, sm_count()));
      TG_CUDA_CHECK(launch_if_short(is_short, softcap_ce_groups_kernel, dim3(unsigned(blocks)), kCgThreads * kCgGroups,
                                    size_t(kTanhBytes + kCgGroups * slots * kCgSlotBytes), st, a, slots));
    } else {
      // as many threads as make the last pass over the row nearly full (of at most 640: two blocks an SM at 48 registers)
      const int64_t pieces = (vocab + 7) / 8;
      int nt = kCeMaxThreads;
      double best = 0.0;
      for (int n = kCeMaxThreads; n >= 256; n -= 32) {
        const double full = double(pieces) / double((pieces + n - 1) / n * n);
        if (full > best + 0.02) { best = full; nt = n; }
      }
      const int64_t cap_blocks = int64_t(sm_count()) * std::min<int64_t>(per_sm_smem, 1280 / nt);
      TG_CUDA_CHECK(launch_if_short(is_short, softcap_ce_kernel<false, false>, dim3(unsigned(std::min<int64_t>(rows, cap_blocks))), nt, smem, st, a));
    }
  }
  return TG_OK;
}

extern "C" int tg_softcap_ce_fwd(const void* logits, const int32_t* targets, float cap, void* tanh_out, float* lse,
                                 float* nll, int64_t rows, int64_t vocab, int64_t ld, int64_t ld_tanh, void* stream) {
  if (rows < 0 || vocab <= 0 || ld % 8 != 0 || ld < vocab || vocab > INT32_MAX) return TG_ERR_SHAPE;
  if (tanh_out != nullptr && (ld_tanh % 8 != 0 || ld_tanh < vocab)) return TG_ERR_SHAPE;
  if (!(cap > 0.0f)) return TG_ERR_SHAPE;
  if (rows > INT32_MAX) return TG_ERR_TOO_LARGE;
  if (rows == 0) return TG_OK;
  if (!aligned16(logits) || !aligned16(tanh_out)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  // persistent blocks, as many as fit (the 64 KB table allows three per SM)
  static int per_sm_of[64] = {0};          // per device: the attribute below is a per-device setting
  int dev = 0;
  TG_CUDA_CHECK(cudaGetDevice(&dev));
  int& per_sm = per_sm_of[dev & 63];
  if (per_sm == 0) {
    TG_CUDA_CHECK(cudaFuncSetAttribute(softcap_ce_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTanhBytes));
    int n = 0;
    TG_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, softcap_ce_fwd_kernel, kLossFwdThreads, kTanhBytes));
    per_sm = n > 0 ? n : 1;
  }
  const int64_t blocks = std::min<int64_t>(rows, int64_t(sm_count()) * per_sm);
  softcap_ce_fwd_kernel<<<int(blocks), kLossFwdThreads, kTanhBytes, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(logits), targets, cap, static_cast<__nv_bfloat16*>(tanh_out), lse, nll,
      int(rows), int(vocab), ld, ld_tanh);
  TG_CUDA_CHECK(cudaGetLastError());
  return TG_OK;
}

extern "C" int tg_softcap_ce_bwd(const void* tanh_in, const int32_t* targets, const float* lse, const float* gscale,
                                 float cap, void* dlogits, int64_t rows, int64_t vocab, int64_t ld_tanh, int64_t ld_d,
                                 void* stream) {
  if (rows < 0 || vocab <= 0 || ld_tanh % 8 != 0 || ld_d % 8 != 0 || ld_tanh < vocab || ld_d < vocab ||
      vocab > INT32_MAX)
    return TG_ERR_SHAPE;
  if (!(cap > 0.0f)) return TG_ERR_SHAPE;
  if (rows > INT32_MAX) return TG_ERR_TOO_LARGE;
  if (rows == 0) return TG_OK;
  if (!aligned16(tanh_in) || !aligned16(dlogits)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  softcap_ce_bwd_kernel<<<int(rows), kLossThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(tanh_in), targets, lse, gscale, cap, 1.0f / float(rows),
      static_cast<__nv_bfloat16*>(dlogits), int(vocab), ld_tanh, ld_d);
  TG_CUDA_CHECK(cudaGetLastError());
  return TG_OK;
}
