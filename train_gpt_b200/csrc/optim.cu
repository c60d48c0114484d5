// Global gradient norm, clip and AdamW for bf16 parameters: the optimiser half of the
// reference's train step (train-gpt train.py:114-123,132-134: optax.chain(clip_by_global_norm,
// adamw) with bf16 parameters, hence bf16 moments).  Bandwidth-bound: the update reads p, g, m,
// v and writes p, m, v once (14 bytes per parameter); the clip factor is applied to the
// gradient on the fly instead of in a pass of its own.
#include "common.cuh"
#include "host_api.h"

namespace tg {

constexpr int kOptThreads = 256;
constexpr int kSumsqBlocks = 1024;   // partial sums of tg_sumsq_bf16 (caller scratch: this many floats)

__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__device__ __forceinline__ float sumsq8(const uint4& w) {
  const float2 a = bf16x2_unpack(w.x), b = bf16x2_unpack(w.y), c = bf16x2_unpack(w.z), d = bf16x2_unpack(w.w);
  const float2 t = __fadd2_rn(__ffma2_rn(c, c, __fmul2_rn(a, a)), __ffma2_rn(d, d, __fmul2_rn(b, b)));
  return t.x + t.y;
}

__global__ void __launch_bounds__(kOptThreads)
sumsq_partial_kernel(const __nv_bfloat16* __restrict__ x, long long n, float* __restrict__ partial) {
  __shared__ float s_w[kOptThreads / 32];
  float acc = 0.f;
  const long long vecs = n / 8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < vecs; i += (long long)gridDim.x * blockDim.x) {
    acc += sumsq8(ld_stream_v4(x + 8 * i));
  }
  if (blockIdx.x == 0)   // ragged tail (n % 8 elements)
    for (long long i = vecs * 8 + threadIdx.x; i < n; i += blockDim.x) {
      const float f = __bfloat162float(x[i]);
      acc = fmaf(f, f, acc);
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = s_w[0];
#pragma unroll
    for (int i = 1; i < kOptThreads / 32; ++i) t += s_w[i];
    partial[blockIdx.x] = t;
  }
}

// out[0] = sum of the partials, in index order (deterministic), by one warp
__global__ void sumsq_final_kernel(const float* __restrict__ partial, int count, float* __restrict__ out) {
  float acc = 0.f;
  for (int i = threadIdx.x; i < count; i += 32) acc += partial[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (threadIdx.x == 0) out[0] = acc;
}

struct AdamwArgs {
  float lr, b1, b2, eps, wd;
};

// One AdamW element.  Rounding points follow optax with bf16 moments: the
// clipped gradient, the stored moments and the stored parameter are bf16 values; everything
// between two stores is float32.
struct AdamwElement {
  AdamwArgs a;
  float inv_bc1, inv_bc2, gs;
  __device__ __forceinline__ AdamwElement(const AdamwArgs& args, float t, float scale) : a(args), gs(scale) {
    inv_bc1 = 1.0f / (1.0f - powf(a.b1, t));
    inv_bc2 = 1.0f / (1.0f - powf(a.b2, t));
  }
  __device__ __forceinline__ float operator()(float pf, float gf, float& mf, float& vf) const {
    const float gc = bf16_round(gf * gs);                               // optax.clip_by_global_norm
    mf = bf16_round(a.b1 * mf + (1.0f - a.b1) * gc);                     // scale_by_adam: mu
    vf = bf16_round(a.b2 * vf + (1.0f - a.b2) * gc * gc);                //                nu
    const float u = (mf * inv_bc1) / (sqrtf(vf * inv_bc2) + a.eps) + a.wd * pf;   // + add_decayed_weights
    return bf16_round(pf - a.lr * u);                                   // apply_updates
  }
};

struct AdamwSpan {
  __nv_bfloat16* p;
  const __nv_bfloat16* g;
  __nv_bfloat16 *m, *v;
  long long n;
};
struct AdamwPiece {
  uint4 p, g, m, v;
  __device__ __forceinline__ void load(const AdamwSpan& s, long long i) {
    p = *reinterpret_cast<const uint4*>(s.p + 8 * i);
    g = ld_stream_v4(s.g + 8 * i);
    m = *reinterpret_cast<const uint4*>(s.m + 8 * i);
    v = *reinterpret_cast<const uint4*>(s.v + 8 * i);
  }
  __device__ __forceinline__ void update_and_store(const AdamwSpan& s, long long i, const AdamwElement& one) {
    uint32_t *pp = &p.x, *mp = &m.x, *vp = &v.x;
    const uint32_t* gp = &g.x;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float m0 = bf16lo(mp[j]), m1 = bf16hi(mp[j]), v0 = bf16lo(vp[j]), v1 = bf16hi(vp[j]);
      const float p0 = one(bf16lo(pp[j]), bf16lo(gp[j]), m0, v0);
      const float p1 = one(bf16hi(pp[j]), bf16hi(gp[j]), m1, v1);
      pp[j] = pack_bf16x2(p0, p1);
      mp[j] = pack_bf16x2(m0, m1);
      vp[j] = pack_bf16x2(v0, v1);
    }
    *reinterpret_cast<uint4*>(s.p + 8 * i) = p;
    *reinterpret_cast<uint4*>(s.m + 8 * i) = m;
    *reinterpret_cast<uint4*>(s.v + 8 * i) = v;
  }
};
__device__ __forceinline__ void adamw_piece(const AdamwSpan& s, long long i, const AdamwElement& one) {
  if (8 * i + 8 <= s.n) {
    AdamwPiece w;
    w.load(s, i);
    w.update_and_store(s, i, one);
    return;
  }
  for (long long e = 8 * i; e < s.n; ++e) {       // ragged tail
    float mf = __bfloat162float(s.m[e]), vf = __bfloat162float(s.v[e]);
    s.p[e] = __float2bfloat16_rn(one(__bfloat162float(s.p[e]), __bfloat162float(s.g[e]), mf, vf));
    s.m[e] = __float2bfloat16_rn(mf);
    s.v[e] = __float2bfloat16_rn(vf);
  }
}

// One AdamW step on n bf16 parameters.
__global__ void __launch_bounds__(kOptThreads)
adamw_kernel(AdamwSpan s, AdamwArgs a, const int* __restrict__ step, const float* __restrict__ gscale) {
  const AdamwElement one(a, float(*step), gscale != nullptr ? *gscale : 1.0f);
  const long long pieces = (s.n + 7) / 8;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < pieces; i += (long long)gridDim.x * blockDim.x)
    adamw_piece(s, i, one);
}

// ---------------------------------------------------------------------------------------
// The whole optimiser step of a model in two launches: the global norm over every gradient tensor, then the clipped update of
// every parameter tensor.  Tensor by tensor it was two launches per norm term and one per update (104 at 26 buckets)
// and five elementwise torch kernels for the clip factor and the step count: 215 us of launches beside the 1.3 ms of memory
// traffic at 406 M parameters, and nothing but launches for a small model.
//
// The update's work is handed out in chunks of kChunk elements numbered through all tensors; a block's chunk numbers only grow, so it
// walks the table of tensors once.  It waits for memory: with two pieces (eight 16-byte loads) in flight per thread instead of one
// the update of 406 M elements takes 966 us (1031; 5.9 TB/s).
// ---------------------------------------------------------------------------------------
constexpr int kMaxSpans = 64;
constexpr int kPieces = 4;                   // of 8 elements per thread and chunk
constexpr int kChunk = kOptThreads * 8 * kPieces;

struct Spans {
  AdamwSpan s[kMaxSpans];
  int first[kMaxSpans + 1];                  // number of the tensor's first chunk (norm: of its first thread block)
  int n;
};
// Over this block's chunks: whole(span, first piece of this thread) for a chunk that lies inside its tensor -- the thread's
// kPieces pieces, kOptThreads apart, can then be loaded together -- else part(span, piece) for each piece there is (the last
// possibly ragged).
template <typename W, typename P>
__device__ __forceinline__ void for_chunks(const Spans& t, W&& whole, P&& part) {
  int k = 0;
  for (int c = blockIdx.x; c < t.first[t.n]; c += gridDim.x) {
    while (c >= t.first[k + 1]) ++k;
    const AdamwSpan& s = t.s[k];
    const long long i0 = (long long)(c - t.first[k]) * (kChunk / 8) + threadIdx.x, pieces = (s.n + 7) / 8;
    if ((long long)(c - t.first[k] + 1) * kChunk <= s.n) {
      whole(s, i0);
    } else {
#pragma unroll 1
      for (int u = 0; u < kPieces; ++u)
        if (i0 + u * kOptThreads < pieces) part(s, i0 + u * kOptThreads);
    }
  }
}

// The norm's sums have the order of tg_sumsq_bf16 on each tensor -- as many thread blocks, each thread's pieces, lanes, warps and
// blocks added alike -- and of a halving tree over the tensors' sums (see below), so the bits are those of one
// launch per tensor and a torch sum of up to 127 of them.  They matter: the clip factor multiplies every gradient, and the e4m3 roundings of the
// steps that follow amplify its last bit.
//
// The block of a tensor that finishes last adds its blocks' sums, the last of these the tensors'; both reset their tickets.  Where
// the grid is small (`few`), the last block of all does both, which saves a round through a ticket: the small model's
// 0.5 M elements 4.8 us, 6.3 without.  406 M elements: 122 us (6.7 TB/s).
// Scratch: the ticket of the tensors in 16 bytes, then per tensor a ticket, a sum and kSumsqBlocks partial sums.
struct NormScratch {
  unsigned* done;
  unsigned* ticket;          // [n]
  float* sum;                // [n]
  float* partial;            // [n][kSumsqBlocks]
};
__host__ __device__ __forceinline__ NormScratch norm_scratch(void* p, int n) {
  NormScratch s;
  s.done = static_cast<unsigned*>(p);
  s.ticket = s.done + 4;
  s.sum = reinterpret_cast<float*>(s.ticket + n);
  s.partial = s.sum + n;
  return s;
}
static int64_t sumsq_blocks(int64_t n) {
  const int64_t want = (n / 8 + kOptThreads - 1) / kOptThreads;
  return want < 1 ? 1 : want > kSumsqBlocks ? kSumsqBlocks : want;
}

__global__ void __launch_bounds__(kOptThreads)
global_norm_kernel(const __grid_constant__ Spans t, void* scratch, int from, int n, int few, float* __restrict__ norm, const float* __restrict__ loss_in,
                   const unsigned* __restrict__ status, float* __restrict__ loss_out) {
  __shared__ float s_w[kOptThreads / 32];
  __shared__ int s_last, s_very_last;
  constexpr int kTree = 2 * kOptThreads;
  __shared__ float s_tree[kTree];
  grid_trigger();
  grid_wait();
  loss_in = loads_below(loss_in);
  status = loads_below(status);
  const NormScratch sc = norm_scratch(scratch, n);
  int k = 0;                                             // this block's tensor: the last whose first block is not above it
#pragma unroll
  for (int step = kMaxSpans / 2; step > 0; step >>= 1)
    if (k + step < t.n && t.first[k + step] <= int(blockIdx.x)) k += step;
  const int block = int(blockIdx.x) - t.first[k], blocks = t.first[k + 1] - t.first[k], lane = threadIdx.x & 31;
  const AdamwSpan& s = t.s[k];
  k += from;
  const long long vecs = s.n / 8, stride = (long long)blocks * kOptThreads;
  float acc = 0.f;
  for (long long i = (long long)block * kOptThreads + threadIdx.x; i < vecs; i += kPieces * stride) {
    uint4 w[kPieces];
#pragma unroll
    for (int u = 0; u < kPieces; ++u) w[u] = i + u * stride < vecs ? ld_stream_v4(s.g + 8 * (i + u * stride)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < kPieces; ++u) acc += sumsq8(w[u]);          // (what does not exist adds +0: no change)
  }
  if (block == 0)
    for (long long i = vecs * 8 + threadIdx.x; i < s.n; i += kOptThreads) {
      const float f = __bfloat162float(s.g[i]);
      acc = fmaf(f, f, acc);
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) s_w[threadIdx.x >> 5] = acc;
  __syncthreads();
  float* partial = sc.partial + (long long)k * kSumsqBlocks;
  if (threadIdx.x == 0) {
    acc = s_w[0];
#pragma unroll
    for (int i = 1; i < kOptThreads / 32; ++i) acc += s_w[i];
    partial[block] = acc;
    __threadfence();
    s_last = few ? atomicAdd(sc.done, 1u) == gridDim.x - 1u : atomicAdd(sc.ticket + k, 1u) == unsigned(blocks) - 1u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // a tensor's sum over its blocks, by one warp
  auto tensor_sum = [&](const float* part, int count) {
    float v = 0.f;
    for (int i = lane; i < count; i += 32 * 8) {
      float w[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) w[u] = i + 32 * u < count ? __ldcg(part + i + 32 * u) : 0.f;
#pragma unroll
      for (int u = 0; u < 8; ++u) v += w[u];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  const bool here = n <= kTree;
  if (few) {
    for (int j = threadIdx.x >> 5; j < n; j += kOptThreads / 32) {
      const float v = tensor_sum(sc.partial + (long long)j * kSumsqBlocks, t.first[j + 1] - t.first[j]);
      if (lane == 0) s_tree[j] = v;
    }
  } else {
    if (threadIdx.x < 32) {
      const float v = tensor_sum(partial, blocks);
      if (lane == 0) {
        __stcg(sc.sum + k, v);
        sc.ticket[k] = 0u;
        __threadfence();
        s_very_last = atomicAdd(sc.done, 1u) == unsigned(n) - 1u;
      }
    }
    __syncthreads();
    if (!s_very_last) return;
    __threadfence();
    if (here)
      for (int i = threadIdx.x; i < n; i += kOptThreads) s_tree[i] = __ldcg(sc.sum + i);
  }
  __syncthreads();
  // the tensors' sums as torch.sum adds a short vector: with p the largest power of two in n, v[i] + v[i + p], then halves of p
  int p = 1;
  while (2 * p <= n) p *= 2;
  auto at = [&](int i) { return here ? s_tree[i] : __ldcg(sc.sum + i); };
  for (int h = p; h > 0; h >>= 1) {
    for (int i = threadIdx.x; i < h && i + h < n; i += kOptThreads) {
      const float v = at(i) + at(i + h);
      if (here) s_tree[i] = v;
      else __stcg(sc.sum + i, v);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *sc.done = 0u;
    *norm = __fsqrt_rn(at(0));
    if (loss_out != nullptr) *loss_out = *status != 0u ? __int_as_float(0x7fffffff) : *loss_in;
  }
}

// clip (optax.clip_by_global_norm: the reciprocal of the norm times clip where the norm is not below clip) and update; the last
// launch's last block counts the step
__global__ void __launch_bounds__(kOptThreads)
adamw_spans_kernel(const __grid_constant__ Spans t, AdamwArgs a, const float* __restrict__ norm, float clip, int* step, int count) {
  __shared__ bool s_last;
  grid_trigger();
  grid_wait();
  norm = loads_below(norm);
  const float n = *norm;
  const AdamwElement one(a, float(step[0] + 1), n < clip ? 1.0f : __fmul_rn(__frcp_rn(n), clip));
  for_chunks(
      t,
      [&](const AdamwSpan& s, long long i) {
#pragma unroll
        for (int u = 0; u < kPieces; u += 2) {                  // two pieces in flight per thread
          AdamwPiece w0, w1;
          w0.load(s, i + u * kOptThreads);
          w1.load(s, i + (u + 1) * kOptThreads);
          w0.update_and_store(s, i + u * kOptThreads, one);
          w1.update_and_store(s, i + (u + 1) * kOptThreads, one);
        }
      },
      [&](const AdamwSpan& s, long long i) { adamw_piece(s, i, one); });
  if (!count) return;
  __syncthreads();                                       // every thread of the block has read the step count
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(reinterpret_cast<unsigned*>(step + 1), 1u) == gridDim.x - 1) {
      step[1] = 0;
      step[0] += 1;
    }
  }
}

// Token and position embeddings of a step: one 16-byte piece per thread.  The embedding gradient's memory is cleared here, where that is no
// launch of its own (as two fills they were 6 us of a small step's host time).
__global__ void __launch_bounds__(kOptThreads)
embed_kernel(const int64_t* __restrict__ ids, const __nv_bfloat16* __restrict__ embed, const __nv_bfloat16* __restrict__ pos,
             __nv_bfloat16* __restrict__ x, long long tokens, int seq, int d, int64_t vocab, unsigned* status, uint2* table, uint4* g_embed) {
  const int per_row = d / 8;
  grid_trigger();
  grid_wait();
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  for (long long i = first; i < vocab; i += step) table[i] = make_uint2(0u, 0u);
  for (long long i = first; i < vocab * per_row; i += step) g_embed[i] = make_uint4(0u, 0u, 0u, 0u);
  ids = loads_below(ids);
  embed = loads_below(embed);
  pos = loads_below(pos);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tokens * per_row; i += (long long)gridDim.x * blockDim.x) {
    const long long tok = i / per_row;
    const int c = int(i - tok * per_row) * 8;
    int64_t id = ids[tok];
    if (id < 0) id += vocab;
    uint4 o = make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
    if (id >= 0 && id < vocab) {
      const uint4 e = *reinterpret_cast<const uint4*>(embed + id * d + c), q = *reinterpret_cast<const uint4*>(pos + (tok % seq) * d + c);
      const uint32_t ei[4] = {e.x, e.y, e.z, e.w}, qi[4] = {q.x, q.y, q.z, q.w};
      uint32_t* op = &o.x;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 t = __fadd2_rn(bf16x2_unpack(ei[j]), bf16x2_unpack(qi[j]));
        op[j] = pack_bf16x2(t.x, t.y);
      }
    } else if (c == 0) {
      atomicCAS(status, 0u, unsigned(TGH_STATUS_TOKEN));
    }
    *reinterpret_cast<uint4*>(x + tok * d + c) = o;
  }
}

// The token embedding's gradient without a sort (torch's accumulating index_put sorts the ids: ten launches).  The rows of
// an id are added in token order.  token_count_kernel leaves the first token and the number of tokens of every id in a table, and the
// tokens of an id that has few, in any order, in the id's own row of the (zeroed) gradient, which is only written at the end.  Then one
// warp per token and 256 columns: that of an id's first token and first columns puts a short list in order and adds the rows, all columns
// of them; a frequent id has a warp for each 256 columns, which finds its tokens by scanning on from the first one, eight loads of ids
// in flight, most of what it meets being hits.  (Scanning for every id that occurs twice was L2 traffic: 32768 tokens of
// 50304 ids, d 1024, 474 us against 89 now and 250 for index_put; 8192 tokens 88 against 48 and 183; one id in ten tokens the
// same, 8192 tokens, 292 against 265 and 1122.)
constexpr int kListed = 32;                  // tokens in a list, where a row holds as many

__device__ __forceinline__ int listed_tokens(int d) { return d / 2 < kListed ? d / 2 : kListed; }

__global__ void __launch_bounds__(kOptThreads)
token_count_kernel(const int64_t* __restrict__ ids, int tokens, int d, int64_t vocab, uint2* __restrict__ table, __nv_bfloat16* __restrict__ g_embed) {
  const int t = int(blockIdx.x) * kOptThreads + int(threadIdx.x);
  grid_trigger();
  grid_wait();
  ids = loads_below(ids);
  if (t >= tokens) return;
  int64_t id = ids[t];
  if (id < 0) id += vocab;
  if (id < 0 || id >= vocab) return;
  atomicMax(&table[id].x, unsigned(tokens - t));            // zero-filled: the largest is the first token
  const unsigned at = atomicAdd(&table[id].y, 1u);
  if (at < unsigned(listed_tokens(d))) reinterpret_cast<int*>(g_embed + id * d)[at] = t;
}

// acc = bf16(acc + w), eight values
__device__ __forceinline__ void add8(uint4& acc, const uint4& w) {
  uint32_t* ap = &acc.x;
  const uint32_t wi[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __fadd2_rn(bf16x2_unpack(ap[j]), bf16x2_unpack(wi[j]));
    ap[j] = pack_bf16x2(t.x, t.y);
  }
}

__global__ void __launch_bounds__(kOptThreads)
embed_bwd_kernel(const int64_t* __restrict__ ids, const __nv_bfloat16* __restrict__ dx, __nv_bfloat16* g_embed,
                 const uint2* __restrict__ table, int tokens, int d, int64_t vocab) {
  const int chunks = (d + 255) / 256, lane = threadIdx.x & 31;
  const long long unit = (long long)blockIdx.x * (kOptThreads / 32) + (threadIdx.x >> 5);
  const int first = int(unit / chunks), chunk = int(unit - (long long)first * chunks);
  grid_trigger();
  grid_wait();
  ids = loads_below(ids);
  table = loads_below(table);
  if (first >= tokens) return;
  int64_t id = ids[first];
  if (id < 0) id += vocab;
  if (id < 0 || id >= vocab) return;
  const uint2 entry = table[id];
  if (int(entry.x) != tokens - first) return;               // not the id's first token
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  const int count = int(entry.y);
  __nv_bfloat16* out = g_embed + id * d;
  if (count <= listed_tokens(d)) {
    if (chunk != 0) return;
    const int mine = lane < count ? __ldcg(reinterpret_cast<const int*>(out) + lane) : INT32_MAX;
    int rank = 0;
    for (int j = 0; j < count; ++j) rank += __shfl_sync(0xffffffffu, mine, j) < mine;
    __syncwarp();                                           // the list is read: the row may be written
    for (int col0 = 0; col0 < d; col0 += 256) {
      const int col = col0 + lane * 8;
      const bool ok = col < d;
      uint4 acc = zero;
      for (int r = 0; r < count; r += 4) {
        uint4 w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned holder = __ballot_sync(0xffffffffu, lane < count && rank == r + i);
          const int t = __shfl_sync(0xffffffffu, mine, holder != 0u ? __ffs(holder) - 1 : 0);
          w[i] = holder != 0u && ok ? ld_stream_v4(dx + (long long)t * d + col) : zero;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (r + i < count) add8(acc, w[i]);
      }
      if (ok) *reinterpret_cast<uint4*>(out + col) = acc;
    }
    return;
  }
  const int col = chunk * 256 + lane * 8;
  const bool ok = col < d;
  constexpr int kIds = 8;
  uint4 acc = zero;
  int left = count;
  for (int t0 = first; left > 0 && t0 < tokens; t0 += 32 * kIds) {
    int64_t other[kIds];
#pragma unroll
    for (int u = 0; u < kIds; ++u) {
      const int t = t0 + 32 * u + lane;
      other[u] = t < tokens ? ids[t] : vocab;
    }
#pragma unroll
    for (int u = 0; u < kIds; ++u) {
      unsigned hits = __ballot_sync(0xffffffffu, (other[u] < 0 ? other[u] + vocab : other[u]) == id);
      left -= __popc(hits);
      while (hits != 0u) {
        uint4 w[4];
        int n = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int at = __ffs(hits) - 1;
          w[i] = at >= 0 && ok ? ld_stream_v4(dx + (long long)(t0 + 32 * u + at) * d + col) : zero;
          n += at >= 0;
          hits &= hits - 1u;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < n) add8(acc, w[i]);
      }
    }
  }
  if (ok) *reinterpret_cast<uint4*>(out + col) = acc;
}

// at most a chunk per SM: a few microseconds
static bool is_short(int64_t chunks) { return chunks <= sm_count(); }

// numbers the tensors' chunks (blocks: the thread blocks that the norm takes) through; returns how many there are, or -1
static int64_t number_chunks(Spans& t, const tgh_span* in, int n, bool blocks) {
  int64_t c = 0;
  t.n = n;
  for (int i = 0; i < n; ++i) {
    t.s[i] = {static_cast<__nv_bfloat16*>(in[i].p), static_cast<const __nv_bfloat16*>(in[i].g), static_cast<__nv_bfloat16*>(in[i].m),
              static_cast<__nv_bfloat16*>(in[i].v), static_cast<long long>(in[i].n)};
    t.first[i] = int(c);
    c += blocks ? sumsq_blocks(in[i].n) : (in[i].n + kChunk - 1) / kChunk;
    if (c > INT32_MAX) return -1;
  }
  t.first[n] = int(c);
  return c;
}

}  // namespace tg

using namespace tg;

extern "C" int64_t tg_sumsq_scratch_bytes(void) { return int64_t(kSumsqBlocks) * int64_t(sizeof(float)); }

extern "C" int tg_sumsq_bf16(const void* x, int64_t n, float* out, void* scratch, void* stream) {
  if (n < 0 || out == nullptr || scratch == nullptr) return TG_ERR_SHAPE;
  if (!aligned16(x) || !aligned16(scratch)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int blocks = int(sumsq_blocks(n));
  sumsq_partial_kernel<<<blocks, kOptThreads, 0, st>>>(static_cast<const __nv_bfloat16*>(x), n, static_cast<float*>(scratch));
  TG_CUDA_CHECK(cudaGetLastError());
  sumsq_final_kernel<<<1, 32, 0, st>>>(static_cast<const float*>(scratch), blocks, out);
  TG_CUDA_CHECK(cudaGetLastError());
  return TG_OK;
}

extern "C" int tg_adamw_bf16(void* p, const void* g, void* m, void* v, int64_t n, float lr, float b1, float b2,
                             float eps, float weight_decay, const int32_t* step, const float* gscale, void* stream) {
  if (n < 0 || step == nullptr) return TG_ERR_SHAPE;
  if (!(b1 >= 0.f && b1 < 1.f && b2 >= 0.f && b2 < 1.f)) return TG_ERR_SHAPE;
  if (n == 0) return TG_OK;
  if (!aligned16(p) || !aligned16(g) || !aligned16(m) || !aligned16(v)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  int64_t want = (n / 8 + kOptThreads - 1) / kOptThreads;
  const int64_t cap = int64_t(sm_count()) * 8;
  const int blocks = int(want < 1 ? 1 : (want > cap ? cap : want));
  const AdamwArgs a = {lr, b1, b2, eps, weight_decay};
  const AdamwSpan one = {static_cast<__nv_bfloat16*>(p), static_cast<const __nv_bfloat16*>(g), static_cast<__nv_bfloat16*>(m),
                         static_cast<__nv_bfloat16*>(v), static_cast<long long>(n)};
  adamw_kernel<<<blocks, kOptThreads, 0, static_cast<cudaStream_t>(stream)>>>(one, a, step, gscale);
  TG_CUDA_CHECK(cudaGetLastError());
  return TG_OK;
}

extern "C" int64_t tgh_global_norm_scratch_bytes(int n) { return 16 + int64_t(n) * (8 + int64_t(sizeof(float)) * kSumsqBlocks); }

extern "C" int tgh_global_norm(const tgh_span* spans, int n, void* scratch, float* norm, const float* loss_in, const unsigned* status,
                               float* loss_out, void* stream) {
  if (n <= 0 || scratch == nullptr || norm == nullptr || (loss_out != nullptr && (loss_in == nullptr || status == nullptr)))
    return TG_ERR_SHAPE;
  for (int i = 0; i < n; ++i) {
    if (spans[i].n < 0) return TG_ERR_SHAPE;
    if (!aligned16(spans[i].g)) return TG_ERR_ALIGN;
  }
  if (!aligned16(scratch)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  for (int i = 0; i < n; i += kMaxSpans) {
    Spans t;
    const int64_t blocks = number_chunks(t, spans + i, n - i < kMaxSpans ? n - i : kMaxSpans, true);
    if (blocks < 0) return TG_ERR_TOO_LARGE;
    const bool few = blocks <= int64_t(kPieces) * sm_count();         // at most a chunk's worth per SM
    TG_CUDA_CHECK(launch_if_short(few, global_norm_kernel, dim3(unsigned(blocks)), kOptThreads, 0, static_cast<cudaStream_t>(stream), t, scratch,
                                  i, n, int(few && n <= kMaxSpans), norm, loss_in, status, loss_out));
  }
  return TG_OK;
}

extern "C" int tgh_adamw(const tgh_span* spans, int n, float lr, float b1, float b2, float eps, float weight_decay, const float* norm,
                         float clip, int32_t* step, void* stream) {
  if (n <= 0 || step == nullptr || norm == nullptr || !(b1 >= 0.f && b1 < 1.f && b2 >= 0.f && b2 < 1.f)) return TG_ERR_SHAPE;
  for (int i = 0; i < n; ++i) {
    if (spans[i].n < 0) return TG_ERR_SHAPE;
    if (!aligned16(spans[i].p) || !aligned16(spans[i].g) || !aligned16(spans[i].m) || !aligned16(spans[i].v)) return TG_ERR_ALIGN;
  }
  if (int rc = check_arch()) return rc;
  const AdamwArgs a = {lr, b1, b2, eps, weight_decay};
  for (int i = 0; i < n; i += kMaxSpans) {
    Spans t;
    const int64_t chunks = number_chunks(t, spans + i, n - i < kMaxSpans ? n - i : kMaxSpans, false);
    if (chunks < 0) return TG_ERR_TOO_LARGE;
    const int64_t cap = int64_t(sm_count()) * 8;
    const int blocks = int(chunks < 1 ? 1 : chunks < cap ? chunks : cap);
    TG_CUDA_CHECK(launch_if_short(is_short(chunks), adamw_spans_kernel, dim3(unsigned(blocks)), kOptThreads, 0, static_cast<cudaStream_t>(stream), t, a,
                                  norm, clip, step, int(i + kMaxSpans >= n)));
  }
  return TG_OK;
}

extern "C" int tgh_embed(const int64_t* ids, const void* embed, const void* pos, void* x, int64_t batch, int64_t seq, int64_t d,
                         int64_t vocab, unsigned* status, void* table, void* g_embed, void* stream) {
  if (batch < 0 || seq < 0 || d <= 0 || d % 8 != 0 || d > INT32_MAX || seq > INT32_MAX || status == nullptr) return TG_ERR_SHAPE;
  if (batch == 0 || seq == 0) return TG_OK;
  if (!aligned16(embed) || !aligned16(pos) || !aligned16(x) || !aligned16(table) || !aligned16(g_embed)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  const int64_t pieces = std::max(batch * seq, vocab) * (d / 8);
  const int64_t blocks = (pieces + kOptThreads - 1) / kOptThreads, cap = int64_t(sm_count()) * 16;
  TG_CUDA_CHECK(launch_if_short(pieces <= 1 << 17, embed_kernel, dim3(unsigned(blocks < cap ? blocks : cap)), kOptThreads, 0,
                                static_cast<cudaStream_t>(stream), ids, static_cast<const __nv_bfloat16*>(embed),
                                static_cast<const __nv_bfloat16*>(pos), static_cast<__nv_bfloat16*>(x), static_cast<long long>(batch * seq),
                                int(seq), int(d), vocab, status, static_cast<uint2*>(table), static_cast<uint4*>(g_embed)));
  return TG_OK;
}

static int embed_bwd(const int64_t* ids, const void* dx, void* g_embed, void* table, int64_t tokens, int64_t d, int64_t vocab, bool clear, void* stream) {
  if (tokens <= 0 || d <= 0 || d % 8 != 0 || vocab <= 0) return TG_ERR_SHAPE;
  if (d > INT32_MAX || tokens > INT32_MAX) return TG_ERR_TOO_LARGE;
  if (!aligned16(dx) || !aligned16(g_embed) || !aligned16(table)) return TG_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (clear) {
    TG_CUDA_CHECK(cudaMemsetAsync(table, 0, size_t(vocab) * sizeof(uint2), st));
    TG_CUDA_CHECK(cudaMemsetAsync(g_embed, 0, size_t(vocab) * size_t(d) * 2, st));
  }
  TG_CUDA_CHECK(launch_early(token_count_kernel, int((tokens + kOptThreads - 1) / kOptThreads), kOptThreads, 0, st, ids, int(tokens), int(d), vocab,
                             static_cast<uint2*>(table), static_cast<__nv_bfloat16*>(g_embed)));
  const int64_t per_block = kOptThreads / 32, blocks = (tokens * ((d + 255) / 256) + per_block - 1) / per_block;
  if (blocks > INT32_MAX) return TG_ERR_TOO_LARGE;
  TG_CUDA_CHECK(launch_early(embed_bwd_kernel, int(blocks), kOptThreads, 0, st, ids, static_cast<const __nv_bfloat16*>(dx),
                             static_cast<__nv_bfloat16*>(g_embed), static_cast<const uint2*>(table), int(tokens), int(d), vocab));
  return TG_OK;
}

extern "C" int tgh_embed_bwd(const int64_t* ids, const void* dx, void* g_embed, void* table, int64_t tokens, int64_t d, int64_t vocab,
                             void* stream) {
  return embed_bwd(ids, dx, g_embed, table, tokens, d, vocab, true, stream);
}
extern "C" int tgh_embed_bwd_cleared(const int64_t* ids, const void* dx, void* g_embed, void* table, int64_t tokens, int64_t d, int64_t vocab,
                                     void* stream) {
  return embed_bwd(ids, dx, g_embed, table, tokens, d, vocab, false, stream);
}
