// Entry points of the library that only its own host path (host.cpp) calls.  Same conventions as the public C ABI
// (device pointers, a stream, an int status, nothing allocates, no exceptions), but no promise: they change with the
// host path.  A status of TG_ERR_TOO_LARGE means "not this way": the caller takes the general entry points instead.
#ifndef TRAIN_GPT_B200_HOST_API_H_
#define TRAIN_GPT_B200_HOST_API_H_

#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

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
