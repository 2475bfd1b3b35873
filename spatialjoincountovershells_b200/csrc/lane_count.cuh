// Grid count with one lane per halo (lane_count.cu).
#pragma once

#include "count_common.cuh"

namespace sjcs {

// Whether q's radius table and flags can take the lane count on an index of
// this size (any schedule: the counts are the same).
bool lane_count_applies(const sjcs_query* q, const count::CountParams& p);
// Count q against the p.nidx indexes of p (mpts, mcs, mn) on stream s.
int launch_lane_count(sjcs_ctx* ctx, const sjcs_query* q, const count::CountParams& p, cudaStream_t s);

}  // namespace sjcs
