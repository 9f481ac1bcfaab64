// The launch of the one-row-per-cluster kernel (molla_cluster.cu), called by the entry points
// in molla_sample.cu.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

struct BatchArgs;

// Whether B rows of V logits, of a call of `call_B`, are better off there than in the tile kernels.
bool molla_cluster_better(int V, int B, int call_B);

// Whether the clusters of all B rows, of a call of `call_B`, are on the device at the same time, or need not be (`capped`: the
// logits have a softcap).
bool molla_cluster_resident(int V, int B, int call_B, bool capped);

// Whether a row of V logits fits one thread block.
bool molla_cluster_is_block(int V);

// Enqueues the sampling of `a.B` rows, for which molla_cluster_better holds, on `st`. Returns MOLLA_OK or
// a MOLLA_ERR_* code with its message in `err`.
int molla_cluster_launch(const BatchArgs &a, cudaStream_t st, char *err, size_t errlen);
