// braid.cuh -- host interface of the steady-ant braid multiplication kernels.
#pragma once

#include "slcs_internal.cuh"

namespace slcs {

// Device workspace of one product (a multiple of 256 bytes).
slcs_status braid_workspace_bytes(int p, int q, int k, int cutoff, size_t *bytes);

// One product: staggered_multiply<row_glue>(P, Q, k) of full permutations
// (row->col device arrays); out receives p + q - k entries.
struct BraidJob {
    const int32_t *P;
    int p;
    const int32_t *Q;
    int q;
    int32_t *out;
};
constexpr int BRAID_MANY = 16;
// Up to BRAID_MANY products of one overlap k, side by side in the same
// launches, each with ws_bytes of workspace (that of the largest) one after
// another.  Nodes of at most `cutoff` entries (0, or more than a block takes:
// 1200) are finished by one block.  A product with an input that is not a
// permutation raises DEV_ERR_INPUT.
slcs_status launch_braids(const BraidJob *jobs, int count, int k, bool row_glue, int cutoff, void *ws, size_t ws_bytes,
                          cudaStream_t st);

} // namespace slcs
