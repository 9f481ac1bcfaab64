/* Testing aids of libmolla_sample_testing.so: the same library compiled with
 * -DMOLLA_SAMPLE_TESTING. None of them has a counterpart in the reference, and none exists in
 * libmolla_sample.so: the production kernels carry no profiling stamps and take no experiment
 * switches. The switches are process-wide and not thread-safe: set, call, reset. */
#ifndef MOLLA_SAMPLE_TESTING_H
#define MOLLA_SAMPLE_TESTING_H

#include "molla_sample.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Experiment switches of the row kernels. The ordinary entry points: bit 32 sends all rows through the tile
 * kernels, bit 64 all rows that fit a thread-block cluster (V <= 307200) through the cluster kernel. Whole rows' logprobs:
 * bit 128 pretends that the device takes no clusters of sixteen. Streaming kernel: bit 1 no last-use hint on the second
 * pass over a row, bit 2 no keep hint on list traffic. All of them: bit 4 pretends, after the row has arrived, that one warp's bounded wait ran out
 * (nothing is withheld and nothing is left waiting): the row must come back with
 * MOLLA_ROW_LOAD_TIMEOUT, token -1 and its sampler state untouched. 0 = production behaviour. */
void molla_sample_debug_knobs(int32_t knobs);

/* When given a device buffer of B x 32 int64, later calls record clock64() stamps at the phase
 * boundaries of each row (NULL switches it off again). */
void molla_sample_debug_profile(void *d_stamps);

/* When given a device buffer of B x cap int32, later calls write, for every row sampled with
 * 1 < top_k < 128, the ids that survive top-k (`_top_k`, sample.mojo:485-490) in descending
 * probability, padded with -1 (NULL switches it off again). */
void molla_sample_debug_topk(void *d_ids, int32_t cap);

/* How often the ordinary entry points launched the cluster kernel (counts[0]) and the tile kernels
 * (counts[1]) since the last call of this function. */
void molla_sample_debug_launches(int64_t *counts);

/* The final-logit softcap as the row kernels evaluate it, four logits at a time, of n values at d_x into d_out
 * (device memory, the legacy default stream). Returns when it is done. */
void molla_sample_debug_softcap(const float *d_x, int64_t n, float cap, float *d_out);

/* For how many floats e from 0 to 1 its quotient (1 - e) / (1 + e), by a reciprocal, is not the division's
 * (-1: the kernel could not be run). */
int64_t molla_sample_debug_softcap_quotients(void);

#ifdef __cplusplus
}
#endif
#endif /* MOLLA_SAMPLE_TESTING_H */
