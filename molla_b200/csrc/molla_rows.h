// The launch of the ordinary entry points' kernels (molla_rows.cu), called by molla_sample.cu.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

struct BatchArgs;

// Device bytes the kernels need for a batch of this shape.
size_t molla_rows_workspace_bytes(int B, int V);

// Enqueues the sampling of `a.B` rows on `st`. Returns MOLLA_OK or a MOLLA_ERR_* code with its message in `err`.
// With `spare`, a kernel that is launched next as a programmatic dependent begins when the last of these has begun, and
// *spare is workspace memory of 16 bytes per 1024 logits of every row that this last one does not use (or nullptr).
int molla_rows_launch(const BatchArgs &a, void *d_workspace, cudaStream_t st, char *err, size_t errlen, float **spare);
