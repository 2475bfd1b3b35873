// Grid count with one lane per halo (lane_count.cu).
#pragma once

#include "count_common.cuh"

namespace sjcs {

// Whether q's radius table and flags can take the lane count on an index of
// this size (any schedule: the counts are the same).
bool lane_count_applies(const sjcs_query* q, const count::CountParams& p);
// Item list of a count, when the caller provides it: kLaneCtlWords zeroed
// control words and room for cap items, eight per halo (one per image) or more.
constexpr int kLaneCtlWords = count::kListWords;
struct LaneScratch {
    uint32_t* ctl;
    uint2* list;
    uint32_t cap;
};
// Count q against the p.nidx indexes of p (mpts, mcs, mn) on stream s.
int launch_lane_count(sjcs_ctx* ctx, const sjcs_query* q, const count::CountParams& p, cudaStream_t s,
                      const LaneScratch* given = nullptr);
// The same over a Morton index (p.nidx == 1, p.g its cells per axis, mcs[0] its
// offset table); with a model, ranks come from it.
struct LearnedLeaf;
struct LearnedRoot;
struct LaneModel {
    const LearnedLeaf* leaves;
    const LearnedRoot* root;
    int key_shift;  // 63 - 3 * level
};
int launch_lane_count_cells(sjcs_ctx* ctx, const sjcs_query* q, const count::CountParams& p, cudaStream_t s,
                            const LaneModel* model);
// Whether a warp to a halo is done sooner than a lane to a halo; the list that
// its count leaves heavy images to (the query's own, or `given`; under capture
// memory of the stream); and the count of what was listed.
enum class RangesOf { Rows, Cells };
bool warps_count_sooner(sjcs_ctx* ctx, const count::CountParams& p);
int list_for_warps(sjcs_ctx* ctx, const sjcs_query* q, count::CountParams* p, RangesOf ranges, StreamScratch& scr,
                   cudaStream_t s, const LaneScratch* given);
int launch_listed_images(sjcs_ctx* ctx, const sjcs_query* q, const count::CountParams& p, RangesOf ranges,
                         cudaStream_t s, const LaneScratch* given, const LaneModel* model);
// launch_shell_count under the static schedule without allocating.
int launch_shell_count_noalloc(sjcs_ctx* ctx, const sjcs_query* q, const sjcs_index* idx, const LaneScratch& scratch,
                               cudaStream_t s);

}  // namespace sjcs
