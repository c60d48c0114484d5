// Entry points of the library that only its own host path (host.cpp) calls.  Same conventions as the public C ABI
// (device pointers, a stream, an int status, nothing allocates, no exceptions), but no promise: they change with the
// host path.  A status of TG_ERR_TOO_LARGE means "not this way": the caller takes the general entry points instead.
#ifndef TRAIN_GPT_B200_HOST_API_H_
#define TRAIN_GPT_B200_HOST_API_H_

#include <stdint.h>

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
/* Up to six of them in one launch. */
int tgh_quantize_jobs(const tgh_quantize_job* jobs, int n, void* stream);

/* Whether tgh_softcap_ce takes this problem (a row and its cap fit the one-pass kernel). */
int tgh_softcap_ce_fits(float cap, int64_t rows, int64_t vocab);
/* Mean capped cross-entropy AND its gradient from one read of the logits.
 *   logits    bf16 [rows, ld], row r starting at logits + r * ld (any alignment; the base 16-byte aligned)
 *   targets   int64 [rows], or int32 if !targets_64
 *   dlogits   bf16 [rows, ld] (base 16-byte aligned) or NULL: gscale / rows * d(sum nll)/dlogits
 *   gscale    device float or NULL for 1;  only_if_scaled: the launch does nothing where *gscale is 1
 *   nll       float [rows] or NULL;  loss: float scalar, mean of nll, or NULL */
int tgh_softcap_ce(const void* logits, const void* targets, int targets_64, float cap, void* dlogits, const float* gscale,
                   int only_if_scaled, float* nll, float* loss, int64_t rows, int64_t vocab, int64_t ld, void* stream);

#ifdef __cplusplus
}
#endif
#endif
