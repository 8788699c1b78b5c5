// List-builder entry points used by the C ABI layer.
#pragma once
#include <cuda_runtime.h>

#include "bnb_internal.h"

namespace bnb {
// Full list rebuild (bin, sort, blocks, AABBs, cull at rcull, masks, work items).
// Returns the number of kernels launched.
int rebuild_list(const Dev &d, const int *colRep, const float *pos, float rcull, cudaStream_t s);
// Per-step packing of coordinates into block slots plus AABBs.
void pack_positions(const Dev &d, const float *pos, cudaStream_t s);
}  // namespace bnb
