// Logprobs of rows that are long enough to be cut into tiles (molla_logprob.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

// Whether rows of V logits go this way; shorter ones are one block's work.
bool molla_logprob_tiled(int V, int top_n);
size_t molla_logprob_workspace_bytes(int B, int V);

// The chosen tokens' and the top N's logprobs (workspace of molla_logprob_workspace_bytes; `early`: the kernel before on
// the stream neither uses that memory nor began before the logits were there, and the pass over the tiles may run beside it),
// or with `full_out` [B x V] whole rows' (no workspace; rows = batch rows, no softcap; `wide`: in clusters of sixteen where
// the device takes them).
cudaError_t molla_logprob_launch(const float *logits, long long row_stride, int B, int V, const int *tokens, int top_n, float *chosen,
                                 int *top_ids, float *top_lps, const int *rows, int n_logit_rows, float softcap, void *workspace, bool early,
                                 float *full_out, bool wide, cudaStream_t st);
