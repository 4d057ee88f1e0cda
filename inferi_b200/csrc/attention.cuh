// Decode attention: a launch's arguments and the split of its positions.
//
// Semantics follow `run_cpu` of crates/inferi-shaders/src/fused_attention.rs:191-245: score = q.k / sqrt(head_size),
// softmax over positions 0..=pos, weighted sum of V.  Cache rows are [position, kv_dim] (fused_attention.rs:107-108).
#pragma once

#include "common.cuh"

#include <math.h>

namespace ib {

constexpr int ATTN_WARPS = 4;

struct AttnArgs {
    ib_attn_params p;
    const uint32_t *pos_ptr;
    const float *q;
    const void *kc, *vc;
    float *out, *scratch;
    unsigned int *counters;
    uint32_t max_splits;
    uint32_t pdl;       // programmatic dependent launch: 0 no, 1 the predecessor writes only q and the newest cache row, 2 it may write anything
    uint32_t cluster;   // CTAs per thread-block cluster along the slices of a kv head; 0: no clusters
};

__device__ __forceinline__ float merge_weight(float m, float mx) { return (m == -INFINITY) ? 0.f : expf(m - mx); }

// The split of `total` positions: number of non-empty slices and positions per slice.
// The slices stop multiplying at `knee` until each holds `knee_per` positions: the merge reads every
// slice's partial, so more slices have to shorten the row loop by more than they lengthen the merge.
__host__ __device__ __forceinline__ void attn_split_plan(uint32_t total, uint32_t max_splits, uint32_t &nsplit, uint32_t &per,
                                                         uint32_t min_per_split, uint32_t knee, uint32_t knee_per) {
    nsplit = (total + min_per_split - 1) / min_per_split;
    if (nsplit > knee) {
        const uint32_t by_len = (total + knee_per - 1) / knee_per;
        nsplit = by_len > knee ? by_len : knee;
    }
    if (nsplit > max_splits) nsplit = max_splits;
    per = (total + nsplit - 1) / nsplit;
    nsplit = (total + per - 1) / per;  // every remaining split is non-empty
}

}  // namespace ib
