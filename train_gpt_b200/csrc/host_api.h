// Entry points of the library that only its own host path (host.cpp) calls.  Same conventions as the public C ABI
// (device pointers, a stream, an int status, nothing allocates, no exceptions), but no promise: they change with the
// host path.  A status of TG_ERR_TOO_LARGE means "not this way": the caller takes the general entry points instead.
#ifndef TRAIN_GPT_B200_HOST_API_H_
#define TRAIN_GPT_B200_HOST_API_H_

#include <stdint.h>

#include "../../include/train_gpt_b200.h"

#ifdef __cplusplus
extern "C" {
#endif

/* One tensor to quantise: bf16 [rows, cols] of pitch ld in its 1 x 128 form (q_row / s_row, or NULL), and / or a second form
 * (q / s): a scale per column per 128 rows, or one per 128 x 128 tile.  Pitches of the e4m3 outputs are multiples of 16.
 * Any number of columns for the column form (also rows that do not start at 16-byte boundaries, where ld is no multiple
 * of 8); with cols % 8 != 0 its q and s get q_ld columns, the extra ones quantised zeros. */
enum { TGH_FORM_NONE = 0, TGH_FORM_COLUMNS = 1, TGH_FORM_BLOCKS = 2 };
typedef struct {
  const void* x;
  int64_t rows, cols, ld;
  void* q_row; float* s_row; int64_t q_row_ld, s_row_ld;
  int form;
  void* q; float* s; int64_t q_ld, s_ld;
} tgh_quantize_job;
/* Any number of them: in one launch where they are of block form only (24 a launch) or small and at most six. */
int tgh_quantize_jobs(const tgh_quantize_job* jobs, int n, void* stream);

/* Columns of the output tiles, and ranges that the contraction is cut into, for a problem that the tiled GEMM takes (TG_ERR_TOO_LARGE:
 * the few-token kernel does).  Needs no GPU. */
int tgh_gemm_plan(const tg_gemm_args* args, int* tile_columns, int* ranges);
/* Which tiled kernel a problem goes to: 0 gemm_fp8.cu, 1 gemm_ring.cu on single SMs, 2 the same on pairs of SMs.  Needs no GPU. */
int tgh_gemm_kernel(const tg_gemm_args* args, int* kernel);
/* Pairs of SMs that a launch on pairs uses at most. */
int tgh_gemm_pairs(void);
/* Two products that do not depend on one another: in one launch where that is faster, else a and then b.  They may share a workspace: what runs
 * apart runs in stream order, and of a joint launch only b is ever cut. */
int tgh_gemm_two(const tg_gemm_args* a, const tg_gemm_args* b, void* stream);
/* How it runs them: apart, in one wave of 128-column tiles, or b and then a on pairs of SMs, with `rounds` rounds of a's items on the pairs
 * that b's last round leaves idle.  Needs no GPU. */
enum { TGH_TWO_APART = 0, TGH_TWO_WAVE = 1, TGH_TWO_PAIRS = 2 };
int tgh_gemm_two_plan(const tg_gemm_args* a, const tg_gemm_args* b, int* rounds);

/* Whether a norm's forward takes a thread block per row.  Needs no GPU. */
int tgh_norm_few_rows(int64_t rows, int64_t cols);

/* tg_rmsnorm_bwd (addend NULL) or tg_rmsnorm_bwd_add up to the partial sums of the weight's gradient, tg_rmsnorm_bwd_scratch_bytes(rows, cols)
 * of them, and the weight gradients of any number of norms of one size from those. */
typedef struct { const void* partial; void* dgamma; } tgh_dgamma_job;
int tgh_rmsnorm_bwd_parts(const void* x, const void* gamma, const void* g, const void* addend, float eps, void* dx, void* partial, int64_t rows,
                          int64_t cols, void* stream);
int tgh_dgamma_reduce(const tgh_dgamma_job* jobs, int n, int64_t rows, int64_t cols, void* stream);

/* Whether tgh_softcap_ce takes this problem (a row and its cap fit the one-pass kernel). */
int tgh_softcap_ce_fits(float cap, int64_t rows, int64_t vocab);
/* Whether it runs ragged rows (of 16-byte pieces) in groups of 512 threads with a row in tensor memory.  Needs no GPU. */
int tgh_softcap_ce_in_groups(int64_t rows, int64_t vocab);
/* Capped cross-entropy of each row AND the gradient of their mean from one read of the logits.
 *   logits    bf16 [rows, ld], row r starting at logits + r * ld (any alignment; the base 16-byte aligned)
 *   targets   int64 [rows], or int32 if !targets_64
 *   dlogits   bf16 [rows, ld] (base 16-byte aligned) or NULL: gscale / rows * d(sum nll)/dlogits
 *   gscale    device float or NULL for 1;  only_if_scaled: the launch does nothing where *gscale is 1
 *   nll       float [rows] or NULL */
int tgh_softcap_ce(const void* logits, const void* targets, int targets_64, float cap, void* dlogits, const float* gscale,
                   int only_if_scaled, float* nll, int64_t rows, int64_t vocab, int64_t ld, void* stream);

/* The mean of n floats (16-byte aligned) with the bits of torch's; n up to 65536, TG_ERR_TOO_LARGE beyond. */
int tgh_mean(const float* v, int64_t n, float* out, void* stream);

/* x[b, t, :] = bf16(embed[ids[b, t]] + pos[t]) (train-gpt model.py:83).  Negative ids count from the end; one outside the
 * vocabulary stores TGH_STATUS_TOKEN in *status and makes its row NaN.  Also clears tgh_embed_bwd's table and the
 * gradient [vocab, d]. */
enum { TGH_STATUS_TOKEN = 16 };
int tgh_embed(const int64_t* ids, const void* embed, const void* pos, void* x, int64_t batch, int64_t seq, int64_t d, int64_t vocab,
              unsigned* status, void* table, void* g_embed, void* stream);

/* The gradient of embed: the rows of dx [tokens, d] added up by token id in token order, rounded to bf16 after every addition (as
 * an accumulating index_put does); zeros for ids that do not occur.  table: vocab * 8 bytes of scratch.  (_cleared: both are all zero already.) */
int tgh_embed_bwd(const int64_t* ids, const void* dx, void* g_embed, void* table, int64_t tokens, int64_t d, int64_t vocab, void* stream);
int tgh_embed_bwd_cleared(const int64_t* ids, const void* dx, void* g_embed, void* table, int64_t tokens, int64_t d, int64_t vocab, void* stream);

/* A parameter tensor with its gradient and moments: n contiguous bf16 values each, 16-byte aligned. */
typedef struct { void* p; const void* g; void* m; void* v; int64_t n; } tgh_span;
/* norm = sqrt of the sum of squares of every span's g: the spans' sums as tg_sumsq_bf16 gives them, added as a halving tree.
 * scratch: tgh_global_norm_scratch_bytes(n) bytes for this n, all zero before the first use; calls that share one are ordered by
 * one stream.  loss_out, if not NULL: *loss_in, or NaN where *status is not 0. */
int64_t tgh_global_norm_scratch_bytes(int n);
int tgh_global_norm(const tgh_span* spans, int n, void* scratch, float* norm, const float* loss_in, const unsigned* status,
                    float* loss_out, void* stream);
/* Clip by *norm (factor clip / norm where norm >= clip) and AdamW step number step[0] + 1 on every span, then ++step[0].
 * step[1] is 0 before and after. */
int tgh_adamw(const tgh_span* spans, int n, float lr, float b1, float b2, float eps, float weight_decay, const float* norm,
              float clip, int32_t* step, void* stream);

#ifdef __cplusplus
}
#endif
#endif
