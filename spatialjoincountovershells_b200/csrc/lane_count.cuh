// Grid count with one lane per halo (lane_count.cu).
#pragma once

#include "count_common.cuh"

namespace sjcs {

// Whether q's radius table and flags can take the lane count on an index of
// this size (any schedule: the counts are the same).
bool lane_count_applies(const sjcs_query* q, const count::CountParams& p);
// Item list of a count, when the caller provides it: kLaneCtlWords zeroed
// control words and room for cap items, eight per halo (one per image) or more.
constexpr int kLaneCtlWords = count::kListWords + 2;
struct LaneScratch {
    uint32_t* ctl;
    uint2* list;
    uint32_t cap;
};
// Count q against the p.nidx indexes of p (mpts, mcs, mn) on stream s.
// With `warps`, the launch of a count that gives a warp to each halo, a sample of
// the halos decides on the device which of the two counts.
class Warps {
    int (*call_)(const void*, const count::CountParams&) = nullptr;
    const void* f_ = nullptr;

  public:
    Warps() = default;
    template <class F>
    explicit Warps(const F& f)  // f outlives the call it is passed to
        : call_([](const void* o, const count::CountParams& p) { return (*static_cast<const F*>(o))(p); }), f_(&f) {}
    explicit operator bool() const { return call_ != nullptr; }
    int operator()(const count::CountParams& p) const { return call_(f_, p); }
};
int launch_lane_count(sjcs_ctx* ctx, const sjcs_query* q, const count::CountParams& p, cudaStream_t s,
                      const LaneScratch* given = nullptr, const Warps& warps = {});
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
                            const LaneModel* model, const Warps& warps = {});
// Whether a lane or a warp to each halo is done sooner, or a sample of the halos
// has to tell; the list that the warps leave heavy images to (the query's own, or
// `given`; under capture memory of the stream); and the count of what was listed.
enum class RangesOf { Rows, Cells, Model };
enum class Counter { Lanes, Warps, Sampled };
Counter who_counts(sjcs_ctx* ctx, const count::CountParams& p, RangesOf ranges, bool sorted = true);
int list_for_warps(sjcs_ctx* ctx, const sjcs_query* q, count::CountParams* p, RangesOf ranges, StreamScratch& scr,
                   cudaStream_t s, const LaneScratch* given);
int launch_listed_images(sjcs_ctx* ctx, const sjcs_query* q, const count::CountParams& p, RangesOf ranges,
                         cudaStream_t s, const LaneScratch* given, const LaneModel* model);
// launch_shell_count under the static schedule without allocating.
int launch_shell_count_noalloc(sjcs_ctx* ctx, const sjcs_query* q, const sjcs_index* idx, const LaneScratch& scratch,
                               cudaStream_t s);

}  // namespace sjcs
