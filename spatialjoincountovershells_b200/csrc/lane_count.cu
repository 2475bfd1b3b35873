// Periodic multi-shell count with one lane per halo, over grid indexes (whose
// candidate ranges are rows of cells) and Morton indexes (quads of cells, their
// ranks from the offset table or the learned model); for more than five batches
// of 32 halos per SM.  With fewer a warp takes a halo (shell_count.cu,
// morton_count.cu) and only the list is counted here.
//
// k_lane_count   32 halos of the Morton order per warp, one per lane.  A lane
//                plans its box's rows of cells, up to 25 at a time, clips each
//                in x to the sphere, fetches the rows' slot ranges and then
//                walks its own candidates one by one; its counts go to a private
//                column of 16-bit counters in shared memory and
//                from there to the halo's row.  Shifted periodic images wait
//                in a per-warp list until there are 32 of them and are then
//                walked the same way.
// k_listed_count what does not suit a lane: images of more than 400 rows, and
//                lanes with so many candidates that the rest of the warp
//                would wait.  k_lane_count (or the kernels that give a warp to
//                each halo) lists them; here a warp takes two
//                neighbouring items (or a part of them), reads the rows that
//                reach either sphere in windows of 32 slots, tests a loaded
//                candidate against both centres and counts in 16-bit columns,
//                one per lane and halo.  Two halos of one clump share nearly
//                all candidates, so the loads and the row bookkeeping are
//                paid once for both.
// k_left_count   when the list had no room for all items: a warp takes the
//                marked images of 64 halos one by one.  (Single lanes counting
//                them in k_lane_count took 7.6 ms for 20000 uniform halos on
//                1e6 particles at R = 100 and 66 ms for 10000 on 5e4 at R =
//                600; 0.34 and 1.1 since.)
//
// A candidate costs one float4 load, the eight fp32 operations of the
// reference's distance, one lookup and one counter update; the box test and
// the compare with r2max are gone from the loop.  The lookup word of the
// distance's bit pattern (sjcs_query::LaneTable) carries into the shell index
// exactly when the distance has reached the slot's threshold, everything from
// safe2 on lands in one spare counter, and below safe2 the box test cannot
// fail.  The few candidates between safe2 and r2max (about 0.4 % of halos at
// R = 5 meet one) are tested literally: the walk keeps the least key -
// zone0, and a halo that met the zone is listed again for it alone.
//
// Why lanes walk their own rows: mapping 32 lanes onto one halo's ~21 rows of
// ~5 candidates cost a five-step shuffle search per window and shared-memory
// atomics on the few shells that hold most of the volume, 484-559 warp
// instructions per halo and file; this form takes about 235 (at 7 % of halos
// near a face).  The price is a
// gather of 32 addresses per load, but an L1 gather of 32 x 16 bytes takes
// 11.0 cycles per SM against 5.2 coalesced and 9.2 from shared memory (random
// slots, measured), so staging the candidates would not pay.  What bounds it:
// the L1/shared data pipe (75 % of its peak, 51 % issue active).
//
// k_listed_count runs at 54 % of the data pipe's and 56 % of issue's peak (1e6
// clustered halos on 2e7 particles, R = 20; 53 and 54 on 5e7): between them a
// warp waits for its rows' loads.
//
// Measured (B200, count kernels of one call, warp-per-halo kernel -> this one):
// 1e7 uniform halos on 1e8 particles, R = 5, 40 shells 6.66 -> 4.00 ms; 1e6 on
// 1e7 0.42 -> 0.20; 1e6 clustered halos on 3e7 clustered particles 9.2 (static
// schedule) and 7.1 (queue) -> 3.43, one item at a time 4.28; 1e6 on 5e7, R =
// 20, 64 shells 55 and 40.8 -> 18.5, one item at a time 24.3; 1e5 on 2e7, R =
// 10 2.14 and 1.45 -> 0.75, one at a time 0.90.  Morton forms, 1e7 uniform
// halos on 1e8 particles: offset table 14.2 -> 8.0, learned 25.3 -> 17.2; 5e5
// clustered ones on 2e7: 4.87 -> 2.19 and 4.65 (queue) -> 2.86 by single cells,
// quads a few per cent less.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "grid_rows.cuh"
#include "lane_count.cuh"
#include "morton.cuh"

namespace sjcs {
namespace {

using namespace count;

// One block of 16 warps per SM: its warps take neighbouring batches and share
// their particle lines in L1 (4.00 ms at 1e8 x 1e7; 18 warps 4.31, 20 4.05, 24
// with spills 4.80; in smaller blocks the same warps took 8 to 17 % longer).
constexpr int LN_WARPS = 16;
constexpr int LN_ROWS = 25;       // rows of cells a lane walks
constexpr uint32_t LN_PEND = 96;  // shifted images waiting per warp
constexpr int LN_DEPTH = 4;       // candidates in flight per lane (3: 1 % longer, 2: 2 %, 6: 1 %)
// Listed items: 20 blocks of one warp per SM (96 registers; five blocks of four
// warps take 2 % longer, 16 warps without spills 11 %).
constexpr int HV_WARPS = 1, HV_THREADS = HV_WARPS * 32, HV_BLOCKS = 20;
// The allocation-free count takes 16: no local memory, which the driver may
// have to set aside at a launch.
constexpr int HV_BLOCKS_NOALLOC = 16;
constexpr uint32_t kSpan = 1u << 20;  // candidates between two looks at what the 16-bit counters hold
// Items above this many candidates (in the box's rows) are split into 8 to 64
// parts: one warp would need longer than the rest of the pass (16384 and 32768
// took 8 and 3 % longer on clustered data, R = 20).  When there are fewer
// halos than a few per warp, items are split from kHugeFew on.
constexpr uint32_t kHuge = 65536, kHugeFew = 2048;
constexpr int kCtlLeft = 6;  // control word: something was marked in LaneParams::left; the next one, claims of it
constexpr int kCtlGate = 8;  // LaneParams::gate
constexpr uint32_t kGallop = 15;  // first step of the search for a cell's end
constexpr uint32_t kEndSlot = 0xfffeffffu;  // no index has this many particles on this path
// Work in cycles of the data pipe, to decide which lanes are listed and how: a
// lane's step for its whole warp; a listed item for every 32 rows of its box;
// one of its rows; and a candidate, in 1/32 cycles, when rows are read one by
// one and when they are flattened first.  Fitted to 9e5 halos of about 550
// candidates in rows of 8 (2.5 ms walked, 5 flattened, 8 row by row) and to
// rows of 40, where row by row and flattened meet.
constexpr uint32_t kStepCost = 36, kItemCost = 370;  // and those of count_common.cuh
constexpr uint32_t kMaxWalkRows = 400;  // rows of a box that lanes walk
// 16-bit counters and range lengths: a lane's candidates are at most this many,
// or 8/5 of it in a chunked box, whose ranges are summed before the sphere
// leaves out any of them.
constexpr uint32_t kWalkMax = 30000;

struct LaneParams {
    const uint32_t* __restrict__ slots;  // the fields of sjcs_query::LaneTable
    int nslots, kbase, shift, ncol;
    float safe2, cmax;
    uint32_t walk_max;     // most candidates a lane walks, at most kWalkMax
    uint32_t huge;         // candidates from which an item is split
    int khi;               // last key of the slots less kbase
    uint32_t zone0, zone;  // bit pattern of safe2; that of r2max less it
    // Items: the huge ones from the front of the list, the others from its end.
    uint2* __restrict__ list;  // (halo, flags)
    uint32_t cap, cap_huge, cap_other;  // its room, and that of either kind when warps counted
    uint32_t* __restrict__ gate;        // 1: warps count instead of lanes (null: lanes)
    uint32_t* __restrict__ ctl;   // [0] items asked for, [1] huge, [2] others, [3-5] claims by phase, kCtlLeft
    uint32_t* __restrict__ left;  // marks of what did not fit the list (null: the list holds every item)
    // learned index: its model (leaves null: the other kinds)
    const LearnedLeaf* __restrict__ leaves;
    const LearnedRoot* __restrict__ root;
    const uint32_t* __restrict__ wpref;  // &pts[0].w (stride 4 words)
    int key_shift;                       // cell code -> first key of the cell
};

// Up to this many batches of 32 halos per SM a warp takes a halo at a time:
// lanes would plan for a few warps only and leave most of it to the list.  Count
// alone, lanes -> warps: 5000 uniform halos on 1e6 particles at R = 5 37 -> 30
// us, 20000 on 1e7 at R = 10 92 -> 62, 10500 clustered ones on 5e6 at R = 7 140
// -> 113; learned index, 1500 on 1e6 77 -> 30.  35000 halos on 5e6, R = 7:
// uniform 62 -> 55, clustered 151 -> 152; on 1e7, R = 10 98 -> 77 and 283 -> 325.
constexpr uint64_t kFewBatches = 5;
// Candidates per row and per quad of a box up to which a warp to a halo is ahead
// of the listed count (uniform halos, nothing walked; 2e5 on 1e7 particles: R =
// 20 and 30, 8 and 22 to a row, 575 us against 1048 and 1319 against 1683, R =
// 50, 102 to a row, 5121 against 2793; quads of 94 at R = 20 893 against 991, of
// 705 at R = 30 3140 against 1664).
constexpr double kLongRow = 37.0, kLongQuad = 200.0;
// Halos sampled to see whether they lie in clumps, and how many of them may.
constexpr int kSample = 256, kSampleDense = 32;

// What a candidate range is: a row of grid cells clipped in x; or four Morton
// cells that follow each other in the curve (x and y even and the next ones),
// from the first to the last of them that can reach, its ends from the offset
// table or from the learned model.  A quad has two ends where single cells
// have eight, for a tenth more candidates (learned, 1e8 x 1e7 uniform: 23.7 ms
// by cells, 21.7 by pairs in x, 17.3 by quads; by the table 8.47, 8.59, 8.03).
enum Ranges { RANGE_ROWS = 0, RANGE_CELLS = 1, RANGE_MODEL = 2 };

// Ranges of an image's box (2^31 when there are more).
template <int R>
__device__ __forceinline__ uint32_t box_ranges(const Image& im) {
    if (R == RANGE_ROWS) return im.nrows;
    const uint64_t n = (uint64_t)((im.x1 >> 1) - (im.x0 >> 1) + 1) * (uint64_t)((im.y1 >> 1) - (im.y0 >> 1) + 1) *
                       (uint64_t)im.nz;
    return n > 0x80000000ull ? 0x80000000u : (uint32_t)n;
}

__device__ __forceinline__ uint2 table_range(const uint32_t* __restrict__ cs, uint32_t a, uint32_t e) {
    return make_uint2(__ldg(cs + a), __ldg(cs + e));
}

// Two quads' first reaching cells and the cells past their last (the same:
// none); and the ranges of slots.
struct Quads {
    uint32_t a[2], e[2];
};

// The slots of two quads from the model (the table if the judge found it
// wrong), for a lane that has more of them to fetch.  The first cell's start is
// searched for in the model's window, the end from there on, by steps that
// double: some twenty particles on (a few probes in the same lines), where the
// window of a second lookup has some hundreds (about nine probes in as many
// sectors, and four reads to find the leaf).  Steps from 7 or 15 on are alike;
// from 3 on take 3 % longer.  Out of line: see below.
__device__ __noinline__ Quads model_ranges(const LaneParams& q, const uint32_t* __restrict__ cs, Quads c) {
    constexpr int N = 2;
    const LearnedRoot rt = *q.root;
    Quads s;
    bool open[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        s.a[j] = s.e[j] = 0u;
        open[j] = c.a[j] != c.e[j];
    }
    if (rt.mismatches != 0ull) {
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (open[j]) {
                s.a[j] = __ldg(cs + c.a[j]);
                s.e[j] = __ldg(cs + c.e[j]);
            }
        return s;
    }
    uint64_t key[N];
#pragma unroll
    for (int j = 0; j < N; ++j) key[j] = (uint64_t)c.a[j] << q.key_shift;
    learned_rank_n<N>(rt, q.leaves, q.wpref, key, open, s.a);
    uint32_t end[N], hi[N], v[N];
    bool any = false;
#pragma unroll
    for (int j = 0; j < N; ++j) {
        end[j] = (uint32_t)(((uint64_t)c.e[j] << q.key_shift) >> 33);
        s.e[j] = hi[j] = s.a[j];
        any |= open[j];
    }
    for (uint32_t step = kGallop; any; step = step < 0x40000000u ? 2u * step + 2u : step) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            v[j] = 0xffffffffu;
            if (open[j]) {
                hi[j] = rt.n - s.e[j] > step ? s.e[j] + step : rt.n;
                if (hi[j] < rt.n) v[j] = __ldg(q.wpref + 4ull * hi[j]);
            }
        }
        any = false;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            open[j] = v[j] < end[j];
            if (open[j]) s.e[j] = hi[j] + 1u;
            any |= open[j];
        }
    }
    lower_bound_n<N>(q.wpref, end, s.e, hi);
    return s;
}

// One quad's, both ends searched for together: a lane that waits for one range
// waits for one chain of probes (the two in turn took 6 % longer).
__device__ __noinline__ uint2 model_ends(const LaneParams& q, const uint32_t* __restrict__ cs, uint32_t a, uint32_t e) {
    if (a == e) return make_uint2(0u, 0u);
    const LearnedRoot rt = *q.root;
    if (rt.mismatches != 0ull) return table_range(cs, a, e);
    const uint64_t key[2] = {(uint64_t)a << q.key_shift, (uint64_t)e << q.key_shift};
    const bool act[2] = {true, true};
    uint32_t s[2];
    learned_rank_n<2>(rt, q.leaves, q.wpref, key, act, s);
    return make_uint2(s[0], s[1]);
}

// The cells of quad (x, y) that lie in the box: bit 0 (x, y), 1 (x + 1, y),
// 2 (x, y + 1), 3 (x + 1, y + 1) -- the order of their codes.
__device__ __forceinline__ uint32_t quad_mask(const Image& im, int x, int y) {
    return ((x >= im.x0 ? 5u : 0u) | (x < im.x1 ? 10u : 0u)) & ((y >= im.y0 ? 3u : 0u) | (y < im.y1 ? 12u : 0u));
}
// Its first marked cell, and the one past its last (the same: none marked).
__device__ __forceinline__ void quad_cells(uint32_t mask, int x, int y, int z, uint32_t* a, uint32_t* e) {
    const uint32_t code = morton_cell((uint32_t)x, (uint32_t)y, (uint32_t)z);
    *a = *e = 0u;
    if (mask) {
        *a = code + (uint32_t)__ffs((int)mask) - 1u;
        *e = code + 32u - (uint32_t)__clz((int)mask);
    }
}

// An item's flags: bits 0-2 the shifted axes, bits 3-4 the index to count.
constexpr uint32_t kItemZone = 1u << 7;  // only distances from safe2 on
constexpr uint32_t kItemFar = 1u << 8;   // centre beyond cmax: literal test throughout

__device__ __forceinline__ uint32_t listed_cost(uint32_t T, uint32_t rows, uint32_t box_rows) {
    return min(kFlatCand * T >> 5, (kRowCand * T >> 5) + kRowCost * rows) + kItemCost * ((box_rows + 31u) >> 5);
}

// Shared memory of one warp beside its counters.
template <bool PACK>
struct LaneRows;
template <>
struct LaneRows<false> {
    uint32_t s0[LN_ROWS + 2][32];   // first slot of a lane's range
    uint16_t len[LN_ROWS + 2][32];  // its candidates
    uint32_t pend[LN_PEND];         // halo | shifted axes << 29
};
template <>
struct LaneRows<true> {
    uint32_t row[LN_ROWS + 2][32];  // first slot less the lane's first one << 8 | candidates (<= 255)
    uint32_t pend[LN_PEND];
};
constexpr uint32_t kPackSpan = 1u << 24, kPackLen = 255;

// A coordinate's periodic image: lo < 0 takes precedence (MultiRangeCount.c:38-43).
__device__ __forceinline__ float shifted(float v, float half) {
    return (__fsub_rn(v, half) < kBoxLow) ? __fadd_rn(v, kBoxUpp) : __fsub_rn(v, kBoxUpp);
}

// A centre for which safe2 is not proved.
__device__ __forceinline__ bool beyond(const LaneParams& q, const float4 c) {
    return !(fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)), fabsf(c.z)) <= q.cmax);
}

// Axes on which the halo's box crosses a face.
__device__ __forceinline__ uint32_t oob_flags(const CountParams& p, const float4 c) {
    return ((__fsub_rn(c.x, p.half) < kBoxLow) | (__fadd_rn(c.x, p.half) > kBoxUpp) ? 1u : 0u) |
           ((__fsub_rn(c.y, p.half) < kBoxLow) | (__fadd_rn(c.y, p.half) > kBoxUpp) ? 2u : 0u) |
           ((__fsub_rn(c.z, p.half) < kBoxLow) | (__fadd_rn(c.z, p.half) > kBoxUpp) ? 4u : 0u);
}

// Lanes with `push` add an item (h, flags) to the list.  What a full list does
// not take is marked in `left` instead: 16 bits per index and halo, one per
// image of the halo and one per image of which only the zone is wanted;
// k_left_count takes those.  Out of line: inlined at its four uses it left the
// walk 96 registers instead of 106 and the kernel slower (5.6 ms instead of 4.0
// for 1e7 halos on 1e8 particles).
__device__ __noinline__ void push_items(const CountParams& p, const LaneParams& q, bool push, bool huge, uint32_t h,
                                           uint32_t flags, int lane) {
    const uint32_t all = __ballot_sync(0xffffffffu, push);
    if (!all) return;
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t base = q.cap;
    // a full list is not counted on: no wrap, however many items come
    if (lane == 0 && *const_cast<volatile uint32_t*>(q.ctl) < q.cap) base = atomicAdd(q.ctl, (uint32_t)__popc(all));
    base = __shfl_sync(0xffffffffu, base, 0);
    const bool fits = push && base < q.cap && (uint32_t)__popc(all & lt) < q.cap - base;
    const uint32_t hb = __ballot_sync(0xffffffffu, fits && huge), ob = __ballot_sync(0xffffffffu, fits && !huge);
    uint32_t at = 0;
    if (lane < 2) {
        const uint32_t k = (uint32_t)__popc(lane == 0 ? hb : ob);
        if (k) at = atomicAdd(q.ctl + 1 + lane, k);
    }
    const uint32_t ah = __shfl_sync(0xffffffffu, at, 0), ao = __shfl_sync(0xffffffffu, at, 1);
    if (fits) {
        const uint32_t i = huge ? ah + (uint32_t)__popc(hb & lt) : q.cap - 1u - (ao + (uint32_t)__popc(ob & lt));
        q.list[i] = make_uint2(h, flags);
    } else if (push && q.left) {
        const uint64_t at16 = (uint64_t)((flags >> 3) & 3u) * p.nhalos + h;
        const uint32_t bit = (flags & 7u) + ((flags & kItemZone) ? 8u : 0u);
        atomicOr(q.left + (at16 >> 1), 1u << (bit + 16u * (uint32_t)(at16 & 1u)));
        q.ctl[kCtlLeft] = 1u;
    }
}

template <int R, bool PACK>
__global__ void __launch_bounds__(LN_WARPS * 32, 1)
k_lane_count(const __grid_constant__ CountParams p, const __grid_constant__ LaneParams q) {
    extern __shared__ uint32_t smem[];
    if (q.gate && *q.gate != 0u) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    LaneRows<PACK>* rows = reinterpret_cast<LaneRows<PACK>*>(smem) + warp;
    const int nwarps = (int)(blockDim.x >> 5);
    uint32_t* cols32 = reinterpret_cast<uint32_t*>(reinterpret_cast<LaneRows<PACK>*>(smem) + nwarps);
    const int colwords = (q.ncol + 1) * 16;
    uint32_t* slots = cols32 + nwarps * colwords;
    cols32 += warp * colwords;
    // two lanes' 16-bit counters to a word
    unsigned char* mycol = reinterpret_cast<unsigned char*>(cols32) + 4 * (lane >> 1);
    const uint32_t one = (lane & 1) ? 65536u : 1u;
    for (int i = tid; i < q.nslots; i += (int)blockDim.x) slots[i] = q.slots[i];
    for (int i = lane; i < colwords; i += 32) cols32[i] = 0u;
    __syncthreads();
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t nbatch = (uint32_t)((p.nhalos + 31) / 32);
    const uint32_t W = gridDim.x * (uint32_t)nwarps;
    [[maybe_unused]] const float hmx = 0.5f * p.h[0] + 3e-3f;
    const float hmy = 0.5f * p.h[1] + 3e-3f, hmz = 0.5f * p.h[2] + 3e-3f;
    const uint32_t plane_cells = (uint32_t)p.g.G[1] * (uint32_t)p.g.G[0];
    // One index after the other: a batch counted on all of them at once held
    // their particle lines in L1 together (14.3 against 13.0 ms for 1e7 halos
    // on three files of 1e8).
    for (int f = 0; f < p.nidx; ++f) {
        const float4* __restrict__ pts = p.mpts[f];
        const uint32_t* __restrict__ cs = p.mcs[f];
        const uint32_t np = p.mn[f], file = (uint32_t)f << 3;
        uint32_t b = blockIdx.x * (uint32_t)nwarps + (uint32_t)warp, npend = 0;
        for (;;) {
            float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
            uint32_t h = 0, S = 0;
            bool valid;
            if (npend >= 32u || (b >= nbatch && npend)) {
                // a batch of shifted images
                const uint32_t take = min(npend, 32u);
                npend -= take;
                valid = (uint32_t)lane < take;
                if (valid) {
                    const uint32_t it = rows->pend[npend + lane];
                    h = it & 0x1fffffffu;
                    S = it >> 29;
                    c = p.halos[h];
                    if (S & 1u) c.x = shifted(c.x, p.half);
                    if (S & 2u) c.y = shifted(c.y, p.half);
                    if (S & 4u) c.z = shifted(c.z, p.half);
                }
                __syncwarp();
            } else if (b < nbatch) {
                h = b * 32u + (uint32_t)lane;
                b += W;
                valid = h < p.nhalos;
                if (valid) c = p.halos[h];
                if (p.periodic) {
                    uint32_t F = valid ? oob_flags(p, c) : 0u;
                    uint32_t T = F;
                    for (;;) {
                        const uint32_t bal = __ballot_sync(0xffffffffu, T != 0u);
                        if (!bal) break;
                        if (npend + (uint32_t)__popc(bal) <= LN_PEND) {
                            if (T) rows->pend[npend + __popc(bal & lt)] = h | (T << 29);
                            npend += __popc(bal);
                        } else {
                            push_items(p, q, T != 0u, false, h, T | file, lane);
                        }
                        T = T ? (T - 1u) & F : 0u;
                    }
                    __syncwarp();
                }
            } else {
                break;
            }
            // a centre that is not finite has no finite distance: nothing to count
            const bool fin = (c.x - c.x == 0.0f) & (c.y - c.y == 0.0f) & (c.z - c.z == 0.0f);
            const bool far = beyond(q, c);
            const Image im = make_image(p, c.x, c.y, c.z);
            const uint32_t nranges = box_ranges<R>(im);
            const bool cand = valid & fin & !far & (R != RANGE_ROWS || im.ny <= LN_ROWS) & (nranges <= kMaxWalkRows);
            bool mine = cand;
            const bool chunked = __any_sync(
                0xffffffffu, cand && (R == RANGE_ROWS ? im.ny > 5 || im.nz > 5 : nranges > (uint32_t)LN_ROWS));
            if (chunked || __any_sync(0xffffffffu, valid & fin & !cand)) {
                // Boxes of more than 25 ranges are walked a few planes (of quads:
                // 25) at a time.
                // What is listed instead is decided on the candidates of the
                // whole box: long rows, more than the 16-bit counters hold, and
                // lanes that would keep the others waiting.
                uint32_t box = 0;
                [[maybe_unused]] uint32_t first = 0, last = 0, longest = 0;
                if (R == RANGE_ROWS && cand) {
                    // eight rows' loads in flight at a time
                    const uint32_t gx = (uint32_t)p.g.G[0], xl = (uint32_t)im.x0, xh = (uint32_t)im.x1 + 1u;
                    uint32_t rc = ((uint32_t)im.z0 * (uint32_t)p.g.G[1] + (uint32_t)im.y0) * gx;
                    int yi = 0;
                    for (uint32_t r = 0; r < im.nrows; r += 8u) {
                        uint32_t lo[8], hi[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            lo[u] = hi[u] = 0u;
                            if (r + u < im.nrows) {
                                lo[u] = __ldg(cs + (rc + xl));
                                hi[u] = __ldg(cs + (rc + xh));
                            }
                            rc += gx;
                            if (++yi == im.ny) {
                                yi = 0;
                                rc += plane_cells - (uint32_t)im.ny * gx;
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            box += hi[u] - lo[u];
                            if (PACK) {
                                longest = max(longest, hi[u] - lo[u]);
                                last = max(last, hi[u]);
                            }
                        }
                        if (PACK && r == 0u) first = lo[0];
                    }
                } else if (cand) {
                    // What the quads' ranges hold, from the first cell of the box in a
                    // quad to its last: cells between them that lie outside the box are
                    // walked too.  From the table; the model would answer the same.
                    int qx = 0, qy = 0, qz = 0;
                    for (uint32_t r = 0; r < nranges; r += 4u) {
                        uint2 r4[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            uint32_t a = 0u, e = 0u;
                            if (r + u < nranges) {
                                const int xx = 2 * ((im.x0 >> 1) + qx), yy = 2 * ((im.y0 >> 1) + qy);
                                quad_cells(quad_mask(im, xx, yy), xx, yy, im.z0 + qz, &a, &e);
                            }
                            r4[u] = a != e ? table_range(cs, a, e) : make_uint2(0u, 0u);
                            if (++qx > (im.x1 >> 1) - (im.x0 >> 1)) {
                                qx = 0;
                                if (++qy > (im.y1 >> 1) - (im.y0 >> 1)) {
                                    qy = 0;
                                    ++qz;
                                }
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) box += r4[u].y - r4[u].x;
                    }
                } else if (valid & fin) {
                    box = q.huge + 1u;
                }
                __syncwarp();
                // about what the sphere leaves of the box
                const uint32_t est = box - (box >> 2) - (box >> 3), rows_est = nranges - (nranges >> 2);
                if (chunked) {
                    mine = cand && est <= q.walk_max && (!PACK || (longest <= kPackLen && last - first < kPackSpan));
                    const uint32_t mxT = __reduce_max_sync(0xffffffffu, mine ? est : 0u);
                    const uint32_t hc = listed_cost(est, rows_est, nranges);
                    uint32_t best = kStepCost * mxT, tau = mxT;
#pragma unroll
                    for (int k = 1; k < 5; ++k) {
                        const uint32_t t = k == 4 ? 0u : mxT >> k;
                        const bool over = mine && est > t;
                        const uint32_t st = __reduce_max_sync(0xffffffffu, (mine && !over) ? est : 0u);
                        const uint32_t cost = __reduce_add_sync(0xffffffffu, over ? hc : 0u) + kStepCost * st;
                        if (cost < best) {
                            best = cost;
                            tau = t;
                        }
                    }
                    mine &= est <= tau;
                }
                push_items(p, q, valid & fin & !mine, box > q.huge, h,
                           file | S | (far ? kItemFar : 0u) | (short_rows(est, rows_est) ? kItemShort : 0u), lane);
            }
            const int ny = mine ? im.ny : 0, nz = mine ? im.nz : 0;
            const int nymax = __reduce_max_sync(0xffffffffu, ny), nzmax = __reduce_max_sync(0xffffffffu, nz);
            // steps over the box: planes of rows, or runs of quads
            const int planes = R != RANGE_ROWS ? LN_ROWS : chunked ? LN_ROWS / max(nymax, 1) : 5;  // per walk
            const int ncell = R != RANGE_ROWS && mine ? (int)nranges : 0;
            const int zend = R != RANGE_ROWS ? __reduce_max_sync(0xffffffffu, ncell) : nzmax;
            [[maybe_unused]] int cxi = 0, cyi = 0, czi = 0;  // the next quad
            // Row gaps as max(0, |cell middle - centre| - half a cell - margin), the
            // centre clamped into the box (edge cells also hold what lies outside
            // it).  The margin of 3e-3 is that of cell_gap at the far face.
            [[maybe_unused]] const float xbase =
                ((float)im.x0 + 0.5f) * p.h[0] - fminf(fmaxf(c.x, 0.0f), kBoxUpp);
            const float ccy = fminf(fmaxf(c.y, 0.0f), kBoxUpp), ccz = fminf(fmaxf(c.z, 0.0f), kBoxUpp);
            const float ybase = ((float)im.y0 + 0.5f) * p.h[1] - ccy, zbase = ((float)im.z0 + 0.5f) * p.h[2] - ccz;
            constexpr int kMagicI = 0x4b400000;  // bits of 1.5 * 2^23: adding it rounds to an integer in the low bits
            constexpr float kMagic = 12582912.0f;
            const int ra = im.x0 + kMagicI, rz = im.x1 + kMagicI;
            const float r2q = p.r2p + p.r2slack;
            const float cxh = c.x - 0.5f * p.h[0];  // half a cell lower: rounding to nearest gives the end point's cell
            const float xpad = 1e-3f + 1e-6f * fabsf(c.x);
            const uint32_t rowc0 = ((uint32_t)im.z0 * (uint32_t)p.g.G[1] + (uint32_t)im.y0) * (uint32_t)p.g.G[0] - (uint32_t)kMagicI;
            uint32_t z = 0xffffffffu;  // least key - zone0 met
            bool walked = false;
            for (int zb = 0; zb < zend; zb += planes) {
                uint32_t m = 0, T = 0;
                [[maybe_unused]] uint32_t base = 0;
                [[maybe_unused]] bool wide = false;
                auto keep = [&](uint32_t a, uint32_t e) {
                    const uint32_t l = e - a;
                    if (l) {
                        if constexpr (PACK) {
                            if (m == 0u) base = a;
                            wide |= (l > kPackLen) | (a - base >= kPackSpan);
                            rows->row[m][lane] = ((a - base) << 8) | l;
                        } else {
                            rows->s0[m][lane] = a;
                            rows->len[m][lane] = (uint16_t)l;
                        }
                        ++m;
                        T += l;
                    }
                };
                if constexpr (R == RANGE_ROWS) {
                    for (int zi = zb; zi < min(zb + planes, nzmax); ++zi) {
                        const float gz = fmaxf(fabsf(__fmaf_rn((float)zi, p.h[2], zbase)) - hmz, 0.0f);
                        const float rz2 = r2q - gz * gz;
                        const uint32_t rowz = rowc0 + (uint32_t)zi * plane_cells;
                        for (int y5 = 0; y5 < nymax; y5 += 5) {
                            uint32_t a[5], e[5];
#pragma unroll
                            for (int u = 0; u < 5; ++u) {
                                const float gy = fmaxf(fabsf(__fmaf_rn((float)(y5 + u), p.h[1], ybase)) - hmy, 0.0f);
                                const float rem = rz2 - gy * gy;
                                a[u] = e[u] = 0u;
                                if (rem >= 0.0f && y5 + u < ny && zi < nz) {
                                    // approximate square root: its error (< 1e-6 relative) is far inside the margin
                                    const float sq = rem * rsqrtf(fmaxf(rem, 1e-35f));
                                    const float xr = __fmaf_rn(sq, 1.0f + 2e-6f, xpad);
                                    const int xa = min(max(__float_as_int(__fmaf_rn(cxh - xr, p.g.inv_h[0], kMagic)), ra), rz);
                                    const int xb = min(max(__float_as_int(__fmaf_rn(cxh + xr, p.g.inv_h[0], kMagic)), ra), rz);
                                    const uint32_t row = rowz + (uint32_t)(y5 + u) * (uint32_t)p.g.G[0];
                                    a[u] = __ldg(cs + (row + (uint32_t)xa));
                                    e[u] = __ldg(cs + (row + (uint32_t)xb + 1u));
                                }
                            }
#pragma unroll
                            for (int u = 0; u < 5; ++u) keep(a[u], e[u]);
                        }
                    }
                } else {
                    const int left = min(zend - zb, planes);
                    for (int k4 = 0; k4 < left; k4 += 4) {
                        uint32_t ca[4], ce[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            ca[u] = ce[u] = 0u;
                            if (k4 + u < left && zb + k4 + u < ncell) {
                                const int dx = cxi * 2 - (im.x0 & 1), dy = cyi * 2 - (im.y0 & 1);  // from x0, y0 on
                                const float ga = fmaxf(fabsf(__fmaf_rn((float)dx, p.h[0], xbase)) - hmx, 0.0f);
                                const float gb = fmaxf(fabsf(__fmaf_rn((float)(dx + 1), p.h[0], xbase)) - hmx, 0.0f);
                                const float ya = fmaxf(fabsf(__fmaf_rn((float)dy, p.h[1], ybase)) - hmy, 0.0f);
                                const float yb = fmaxf(fabsf(__fmaf_rn((float)(dy + 1), p.h[1], ybase)) - hmy, 0.0f);
                                const float gz = fmaxf(fabsf(__fmaf_rn((float)czi, p.h[2], zbase)) - hmz, 0.0f);
                                const float rz = r2q - gz * gz, rya = rz - ya * ya, ryb = rz - yb * yb;
                                // no particle of a cell can be within R otherwise
                                const uint32_t mask = quad_mask(im, im.x0 + dx, im.y0 + dy) &
                                                      ((rya - ga * ga >= 0.0f ? 1u : 0u) | (rya - gb * gb >= 0.0f ? 2u : 0u) |
                                                       (ryb - ga * ga >= 0.0f ? 4u : 0u) | (ryb - gb * gb >= 0.0f ? 8u : 0u));
                                quad_cells(mask, im.x0 + dx, im.y0 + dy, im.z0 + czi, &ca[u], &ce[u]);
                                if (++cxi > (im.x1 >> 1) - (im.x0 >> 1)) {
                                    cxi = 0;
                                    if (++cyi > (im.y1 >> 1) - (im.y0 >> 1)) {
                                        cyi = 0;
                                        ++czi;
                                    }
                                }
                            }
                        }
                        if constexpr (R == RANGE_CELLS) {
                            uint2 r4[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u)
                                r4[u] = ca[u] != ce[u] ? table_range(cs, ca[u], ce[u]) : make_uint2(0u, 0u);
#pragma unroll
                            for (int u = 0; u < 4; ++u) keep(r4[u].x, r4[u].y);
                        } else {
#pragma unroll
                            for (int u = 0; u < 4; u += 2) {
                                const Quads r = model_ranges(q, cs, {{ca[u], ca[u + 1]}, {ce[u], ce[u + 1]}});
                                keep(r.a[0], r.e[0]);
                                keep(r.a[1], r.e[1]);
                            }
                        }
                    }
                }
                // which lanes walk their own rows: the threshold with the least work
                bool coop = !chunked && (T > q.walk_max || (PACK && wide));
                uint32_t steps = __reduce_max_sync(0xffffffffu, coop ? 0u : T);
                if (!chunked && steps > 160u) {
                    const uint32_t mxT = steps;
                    const uint32_t hc = listed_cost(T, m, 25u);
                    uint32_t best = kStepCost * mxT, tau = mxT;
#pragma unroll
                    for (int k = 1; k < 5; ++k) {
                        const uint32_t t = k == 4 ? 0u : mxT >> k;
                        const bool over = !coop && T > t;
                        const uint32_t st = __reduce_max_sync(0xffffffffu, (!coop && !over) ? T : 0u);
                        const uint32_t cost = __reduce_add_sync(0xffffffffu, over ? hc : 0u) + kStepCost * st;
                        if (cost < best) {
                            best = cost;
                            tau = t;
                            steps = st;
                        }
                    }
                    coop |= T > tau;
                }
                if (__any_sync(0xffffffffu, coop)) push_items(p, q, coop, T > q.huge, h, file | S | (short_rows(T, m) ? kItemShort : 0u), lane);
                if (steps) {
                    uint32_t j, e;
                    float4 buf[LN_DEPTH];
                    // The lane's next candidate; past its last one nothing is loaded.
                    // Packed ranges: one lookup per range, and 27 KB an SM less for
                    // the lists, which L1 has instead (4.24 -> 4.00 ms at 1e8 x 1e7).
                    [[maybe_unused]] uint32_t left = coop ? 0u : T, nw = 0;
                    [[maybe_unused]] const uint32_t *rs = nullptr, *rw = nullptr;
                    [[maybe_unused]] const uint16_t* rl = nullptr;
                    [[maybe_unused]] uint32_t ns = 0, nl = 0;
                    if constexpr (PACK) {
                        const uint32_t w = left ? rows->row[0][lane] : 0u;
                        j = base + (w >> 8);
                        e = j + (w & 255u);
                        rw = &rows->row[1][lane];
                        nw = *rw;
                    } else {
                        // the list ends in a range of slots past the particles
                        const uint32_t mm = coop ? 0u : m;
                        rows->s0[mm][lane] = kEndSlot;
                        rows->len[mm][lane] = 0xffffu;
                        j = rows->s0[0][lane];
                        e = j + rows->len[0][lane];
                        rs = &rows->s0[1][lane];
                        rl = &rows->len[1][lane];
                        ns = *rs;
                        nl = *rl;
                    }
                    auto next = [&](float4& v) {
                        v.x = INFINITY;
                        if constexpr (PACK) {
                            const bool more = left != 0u;
                            if (more) v = __ldg(pts + j);
                            ++j;
                            left -= more ? 1u : 0u;
                            if (more && j == e) {
                                j = base + (nw >> 8);
                                e = j + (nw & 255u);
                                rw += 32;
                                nw = *rw;
                            }
                        } else {
                            if (j < np) v = __ldg(pts + j);
                            ++j;
                            if (j == e) {
                                j = ns;
                                e = ns + nl;
                                rs += 32;
                                rl += 32;
                                ns = *rs;
                                nl = *rl;
                            }
                        }
                    };
                    auto find = [&](const float4& v) {
                        const float dx = __fsub_rn(v.x, c.x), dy = __fsub_rn(v.y, c.y), dz = __fsub_rn(v.z, c.z);
                        const float dist = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                        const uint32_t key = __float_as_uint(dist);
                        z = __viaddmin_u32(key, 0u - q.zone0, z);
                        const uint32_t t = (uint32_t)__viaddmin_s32_relu((int)key, -q.kbase, q.khi);
                        return ((slots[t >> q.shift] + t) >> q.shift) * 64u;
                    };
#pragma unroll
                    for (int u = 0; u < LN_DEPTH; ++u) next(buf[u]);
                    for (uint32_t it = 0; it < steps; it += LN_DEPTH) {
                        uint32_t at[LN_DEPTH];
#pragma unroll
                        for (int u = 0; u < LN_DEPTH; ++u) at[u] = find(buf[u]);
#pragma unroll
                        for (int u = 0; u < LN_DEPTH; ++u) next(buf[u]);
#pragma unroll
                        for (int u = 0; u < LN_DEPTH; ++u) {
                            atomicAdd(reinterpret_cast<uint32_t*>(mycol + at[u]), one);
                        }
                    }
                    walked = true;
                }
            }
            if (__any_sync(0xffffffffu, z < q.zone)) push_items(p, q, z < q.zone, false, h, file | S | kItemZone, lane);
            // the lanes' counters to their halos' rows
            if (walked) {
                uint32_t* row = p.counts + (uint64_t)__float_as_uint(c.w) * (uint64_t)p.nrads;
#pragma unroll 4
                for (int sh = 0; sh < q.ncol; ++sh) {
                    const uint32_t v = *reinterpret_cast<uint16_t*>(mycol + 2 * (lane & 1) + sh * 64);
                    if (v) atomicAdd(row + sh, v);
                }
                __syncwarp();
                for (int i = lane; i < colwords; i += 32) cols32[i] = 0u;
                __syncwarp();
            }
        }
    }
}

// The centre an item counts.
__device__ __forceinline__ float4 item_centre(const CountParams& p, const uint2 it) {
    float4 c = p.halos[it.x];
    if (it.y & 1u) c.x = shifted(c.x, p.half);
    if (it.y & 2u) c.y = shifted(c.y, p.half);
    if (it.y & 4u) c.z = shifted(c.z, p.half);
    return c;
}

// The rare parts of a listed count stay out of line: inlined at every use they
// made the kernel larger than the instruction cache (11 of 17 stall cycles
// per issue were instruction fetches).

// Each lane's candidate (slot j, or none: ~0) against one centre, counted
// literally if its distance lies in the zone.
__device__ __noinline__ void zone_count(const CountParams& p, const float4* __restrict__ pts, uint32_t j, float4 c,
                                        float safe2) {
    if (j == 0xffffffffu) return;
    Image im;
    im.cx = c.x;
    im.cy = c.y;
    im.cz = c.z;
    im.lox = __fsub_rn(c.x, p.half);
    im.hix = __fadd_rn(c.x, p.half);
    im.loy = __fsub_rn(c.y, p.half);
    im.hiy = __fadd_rn(c.y, p.half);
    im.loz = __fsub_rn(c.z, p.half);
    im.hiz = __fadd_rn(c.z, p.half);
    test_candidate<BIN_BSEARCH, true, true>(p, im, __ldg(pts + j), true,
                                            p.counts + (uint64_t)__float_as_uint(c.w) * (uint64_t)p.nrads, p.r2, p.lut,
                                            safe2);
}

// A warp's counters of one halo ([shell][lane], 16 bits each) to the halo's row.
__device__ __noinline__ void flush_columns(uint32_t* __restrict__ cols, int ncol, uint32_t* __restrict__ row, int lane) {
    __syncwarp();
    for (int s = lane; s < ncol; s += 32) {
        uint32_t sum = 0;
        const uint32_t* r = cols + s * 16;
#pragma unroll 4
        for (int j = 0; j < 16; ++j) {
            const uint32_t w = r[(j + lane) & 15];
            sum += (w & 0xffffu) + (w >> 16);
        }
        if (sum) atomicAdd(row + s, sum);
    }
    __syncwarp();
    for (int i = lane; i < (ncol + 1) * 16; i += 32) cols[i] = 0u;
    __syncwarp();
}

// The first cell of quad r of an image's box of Morton cells, x fastest.
__device__ __forceinline__ void quad_xyz(const Image& im, uint32_t r, int* x, int* y, int* z) {
    const uint32_t nx = (uint32_t)((im.x1 >> 1) - (im.x0 >> 1) + 1), ny = (uint32_t)((im.y1 >> 1) - (im.y0 >> 1) + 1);
    const uint32_t t = r / nx, u = t / ny;
    *x = 2 * ((im.x0 >> 1) + (int)(r - t * nx));
    *y = 2 * ((im.y0 >> 1) + (int)(t - u * ny));
    *z = im.z0 + (int)u;
}

// Lane r's range: row or cell rb + r of the box, if it can reach any of the H
// spheres (a row clipped in x to them); empty otherwise.
template <int R, int H>
__device__ __forceinline__ uint2 lane_range(const CountParams& p, const LaneParams& q, const uint32_t* __restrict__ cs,
                                            const Image& im, const float4 (&c)[H], uint32_t r, uint32_t n) {
    uint2 s = make_uint2(0u, 0u);
    if constexpr (R == RANGE_ROWS) {
        if (r >= n) return s;
        int yy, zz, xa = im.x1 + 1, xb = im.x0 - 1;
        row_yz(im, r, &yy, &zz);
#pragma unroll
        for (int k = 0; k < H; ++k) {
            const float gy = cell_gap(c[k].y, yy, p.h[1], p.g.G[1]), gz = cell_gap(c[k].z, zz, p.h[2], p.g.G[2]);
            const float rem = __fadd_rn(__fsub_rn(__fsub_rn(p.r2p, __fmul_rn(gy, gy)), __fmul_rn(gz, gz)), p.r2slack);
            if (rem >= 0.0f) {
                // approximate square root: its error (< 1e-6 relative) is far inside the margin
                float xr = rem > 0.0f ? __fmul_rn(rem, rsqrtf(rem)) : 0.0f;
                xr = __fadd_rn(xr, 1e-3f + 1e-6f * (fabsf(c[k].x) + xr));
                xa = min(xa, cell_of(__fsub_rn(c[k].x, xr), p.g.inv_h[0], p.g.G[0]));
                xb = max(xb, cell_of(__fadd_rn(c[k].x, xr), p.g.inv_h[0], p.g.G[0]));
            }
        }
        xa = max(xa, im.x0);
        xb = min(xb, im.x1);
        if (xa <= xb) {
            const uint64_t rc = ((uint64_t)zz * (uint64_t)p.g.G[1] + (uint64_t)yy) * (uint64_t)p.g.G[0];
            s = make_uint2(__ldg(cs + rc + xa), __ldg(cs + rc + xb + 1));
        }
    } else {
        uint32_t ca = 0u, ce = 0u;
        if (r < n) {
            int xx, yy, zz;
            uint32_t mask = 0u;
            quad_xyz(im, r, &xx, &yy, &zz);
#pragma unroll
            for (int k = 0; k < H; ++k) {
                const float gz = cell_gap(c[k].z, zz, p.h[2], p.g.G[2]);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float gx = cell_gap(c[k].x, xx + (u & 1), p.h[0], p.g.G[0]),
                                gy = cell_gap(c[k].y, yy + (u >> 1), p.h[1], p.g.G[1]);
                    const float rem =
                        __fadd_rn(__fsub_rn(__fsub_rn(__fsub_rn(p.r2p, __fmul_rn(gx, gx)), __fmul_rn(gy, gy)),
                                            __fmul_rn(gz, gz)),
                                  p.r2slack);
                    mask |= (rem >= 0.0f ? 1u : 0u) << u;
                }
            }
            quad_cells(mask & quad_mask(im, xx, yy), xx, yy, zz, &ca, &ce);
        }
        if constexpr (R == RANGE_CELLS) {
            if (ca != ce) s = table_range(cs, ca, ce);
        } else {
            s = model_ends(q, cs, ca, ce);
        }
    }
    return s;
}

// Zone and far items: the literal test, straight into the count row.
template <int R>
__device__ __noinline__ void count_literal(const CountParams& p, const LaneParams& q, const uint2 it, uint32_t part,
                                           uint32_t nparts, int lane) {
    const float4 c[1] = {item_centre(p, it)};
    uint32_t* row = p.counts + (uint64_t)__float_as_uint(c[0].w) * (uint64_t)p.nrads;
    const Image im = make_image(p, c[0].x, c[0].y, c[0].z);
    const uint32_t n = box_ranges<R>(im);
    CountParams pf = p;
    pf.pts = p.mpts[(it.y >> 3) & 3u];
    const uint32_t* __restrict__ cs = p.mcs[(it.y >> 3) & 3u];
    for (uint32_t rb = 0; rb < n; rb += 32u) {
        const uint2 s = lane_range<R, 1>(p, q, cs, im, c, rb + (uint32_t)lane, n);
        if (it.y & kItemZone)
            run_rows_part<BIN_BSEARCH, true, true>(pf, im, s.x, s.y, row, p.r2, p.lut, lane, part, nparts, q.safe2);
        else
            run_rows_part<BIN_BSEARCH, true>(pf, im, s.x, s.y, row, p.r2, p.lut, lane, part, nparts);
    }
}

// Part `part` of `nparts` of H listed items of one index, counted together:
// the rows are those that reach any of the H spheres, and a candidate once
// loaded is tested against every centre.  Starts with the box's range rb.
template <int R, int H, bool SHORT>
__device__ __forceinline__ void count_items(const CountParams& p, const LaneParams& q, const uint2* it, uint32_t part,
                                            uint32_t nparts, uint32_t* __restrict__ cols,
                                            const uint32_t* __restrict__ slots, int lane, uint32_t rb = 0) {
    float4 c[H];
    Image im;
#pragma unroll
    for (int k = 0; k < H; ++k) {
        c[k] = item_centre(p, it[k]);
        const Image ik = make_image(p, c[k].x, c[k].y, c[k].z);
        if (k == 0) {
            im = ik;
        } else {
            im.x0 = min(im.x0, ik.x0);
            im.x1 = max(im.x1, ik.x1);
            im.y0 = min(im.y0, ik.y0);
            im.y1 = max(im.y1, ik.y1);
            im.z0 = min(im.z0, ik.z0);
            im.z1 = max(im.z1, ik.z1);
        }
    }
    im.ny = im.y1 - im.y0 + 1;
    im.nz = im.z1 - im.z0 + 1;
    const uint64_t nr = (uint64_t)im.ny * (uint64_t)im.nz;
    im.nrows = nr > 0x80000000ull ? 0x80000000u : (uint32_t)nr;
    const uint32_t f = (it[0].y >> 3) & 3u;
    const float4* __restrict__ pts = p.mpts[f];
    const uint32_t* __restrict__ cs = p.mcs[f];
    const uint32_t colwords = (uint32_t)(q.ncol + 1) * 16u;
    unsigned char* mycol = reinterpret_cast<unsigned char*>(cols) + 4 * (lane >> 1);
    const uint32_t one = (lane & 1) ? 65536u : 1u;
    uint32_t held = 0;  // bound of any 16-bit counter
    const uint32_t nranges = box_ranges<R>(im);
    for (; rb < nranges; rb += 32u) {
        const uint2 range = lane_range<R, H>(p, q, cs, im, c, rb + (uint32_t)lane, nranges);
        const uint32_t a = range.x, e = range.y;
        // this warp's share of the rows' candidates, [tb, te) of the flattened sequence
        const uint32_t len = e - a;
        uint32_t incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t tb = 0, te = total;
        if (nparts > 1) {
            tb = (uint32_t)(((uint64_t)total * part) / nparts);
            te = (uint32_t)(((uint64_t)total * (part + 1u)) / nparts);
        }
        uint32_t z = 0xffffffffu;
        // a candidate's counter offset per centre; the lookups of several
        // candidates are in flight before their counters are touched
        auto find = [&](const float4& v, uint32_t* at) {
#pragma unroll
            for (int k = 0; k < H; ++k) {
                const float dx = __fsub_rn(v.x, c[k].x), dy = __fsub_rn(v.y, c[k].y), dz = __fsub_rn(v.z, c[k].z);
                const float dist = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                const uint32_t key = __float_as_uint(dist);
                z = __viaddmin_u32(key, 0u - q.zone0, z);
                const uint32_t t = (uint32_t)__viaddmin_s32_relu((int)key, -q.kbase, q.khi);
                at[k] = ((slots[t >> q.shift] + t) >> q.shift) * 64u;
            }
        };
        auto add = [&](const uint32_t* at) {
#pragma unroll
            for (int k = 0; k < H; ++k)
                atomicAdd(reinterpret_cast<uint32_t*>(mycol + at[k]) + k * colwords, one);
        };
        // distances from safe2 on, which the slots leave out
        auto zone_at = [&](uint32_t j) {
#pragma unroll
            for (int k = 0; k < H; ++k) zone_count(p, pts, j, c[k], q.safe2);
        };
        const uint32_t excl = incl - len;
        // at most 2^20 candidates at a time: 2^15 windows and 64 partial ones
        for (uint32_t t0 = tb, t1; t0 < te; t0 = t1) {
            t1 = te - t0 > kSpan ? t0 + kSpan : te;
            const uint32_t lo = max(excl, t0), hi = min(incl, t1);
            if constexpr (!SHORT) {
                // each row in windows of 32 slots
                uint32_t bal = __ballot_sync(0xffffffffu, lo < hi);
                const uint32_t rs = a + (lo - excl), re = a + (hi - excl);
                while (bal) {
                    const int j = __ffs(bal) - 1;
                    bal &= bal - 1;
                    const uint32_t s0 = __shfl_sync(0xffffffffu, rs, j), s1 = __shfl_sync(0xffffffffu, re, j);
                    uint32_t w = s0 + (uint32_t)lane;  // the lane's slot
                    const float4* src = pts + w;
                    uint32_t left = s1 - s0;
                    for (; left >= 128u; left -= 128u, src += 128, w += 128u) {
                        const float4 v0 = __ldg(src), v1 = __ldg(src + 32), v2 = __ldg(src + 64), v3 = __ldg(src + 96);
                        uint32_t at[4][H];
                        find(v0, at[0]);
                        find(v1, at[1]);
                        find(v2, at[2]);
                        find(v3, at[3]);
#pragma unroll
                        for (int u = 0; u < 4; ++u) add(at[u]);
                        if (__any_sync(0xffffffffu, z < q.zone)) {
#pragma unroll 1
                            for (uint32_t u = 0; u < 128u; u += 32u) zone_at(w + u);
                            z = 0xffffffffu;
                        }
                    }
                    if (left) {
                        float4 v[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            v[u].x = INFINITY;
                            if ((uint32_t)lane + 32u * (uint32_t)u < left) v[u] = __ldg(src + 32 * u);
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (32u * (uint32_t)u < left) {
                                uint32_t at[H];
                                find(v[u], at);
                                add(at);
                            }
                        if (__any_sync(0xffffffffu, z < q.zone)) {
#pragma unroll 1
                            for (uint32_t u = 0; u < 128u; u += 32u) zone_at(w + u < s1 ? w + u : 0xffffffffu);
                            z = 0xffffffffu;
                        }
                    }
                }
            } else {
                // windows over the flattened sequence
                const uint32_t off = a - excl;
                for (uint32_t wb = t0; wb < t1; wb += 64) {
                    const uint32_t u0 = wb + (uint32_t)lane, u1 = u0 + 32u;
                    int r0 = 0, r1 = 0;
#pragma unroll
                    for (int k = 16; k >= 1; k >>= 1) {
                        const uint32_t v0 = __shfl_sync(0xffffffffu, incl, r0 + k - 1);
                        const uint32_t v1 = __shfl_sync(0xffffffffu, incl, r1 + k - 1);
                        r0 += (v0 <= u0) ? k : 0;
                        r1 += (v1 <= u1) ? k : 0;
                    }
                    const uint32_t o0 = __shfl_sync(0xffffffffu, off, r0);
                    const uint32_t o1 = __shfl_sync(0xffffffffu, off, r1);
                    float4 v0, v1;
                    v0.x = v1.x = INFINITY;
                    if (u0 < t1) v0 = __ldg(pts + (u0 + o0));
                    if (u1 < t1) v1 = __ldg(pts + (u1 + o1));
                    uint32_t at0[H], at1[H];
                    find(v0, at0);
                    find(v1, at1);
                    add(at0);
                    if (wb + 32u < t1) add(at1);
                    if (__any_sync(0xffffffffu, z < q.zone)) {
                        zone_at(u0 < t1 ? u0 + o0 : 0xffffffffu);
                        zone_at(u1 < t1 ? u1 + o1 : 0xffffffffu);
                        z = 0xffffffffu;
                    }
                }
            }
            held += ((t1 - t0) >> 5) + 64u;
            if (held > 32000u) {
#pragma unroll
                for (int k = 0; k < H; ++k)
                    flush_columns(cols + k * colwords, q.ncol,
                                  p.counts + (uint64_t)__float_as_uint(c[k].w) * (uint64_t)p.nrads, lane);
                held = 0;
            }
        }
    }
    if (held) {
#pragma unroll
        for (int k = 0; k < H; ++k)
            flush_columns(cols + k * colwords, q.ncol, p.counts + (uint64_t)__float_as_uint(c[k].w) * (uint64_t)p.nrads,
                          lane);
    }
}

// Two neighbouring items of the list are counted together when they are two
// centres of one index no further apart than a radius: most candidates then
// serve both.
template <bool BY_WARPS>
__device__ __forceinline__ bool paired(const CountParams& p, const uint2* it, uint32_t n) {
    constexpr uint32_t kLater = ~((1u << kItemFrom) - 1u);  // an image's later part
    constexpr uint32_t kAlone = kItemZone | kItemFar | kItemShort | (BY_WARPS ? kLater : 0u);
    if (n < 2u || ((it[0].y | it[1].y) & kAlone) || (((it[0].y ^ it[1].y) >> 3) & 3u)) return false;
    const float4 a = item_centre(p, it[0]), b = item_centre(p, it[1]);
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    return dx * dx + dy * dy + dz * dz <= p.r2max;
}

// BY_WARPS: the list of a count that gives a warp to each halo, whose items may
// begin in a later part of their box (1 % of the time of heavy lists of lanes,
// hence two kernels).
template <int R, int BLOCKS, bool BY_WARPS>
__global__ void __launch_bounds__(HV_THREADS, BLOCKS)
k_listed_count(const __grid_constant__ CountParams p, const __grid_constant__ LaneParams q) {
    extern __shared__ uint32_t smem[];
    auto from = [](const uint2& it) { return BY_WARPS ? 32u * (it.y >> kItemFrom) : 0u; };
    if (q.gate && (*q.gate != 0u) != BY_WARPS) return;
    const uint32_t nhuge = min(q.ctl[1], BY_WARPS ? q.cap_huge : q.cap);
    const uint32_t nother = min(q.ctl[2], BY_WARPS ? q.cap_other : q.cap);
    if (nhuge + nother == 0u) return;
    // Warps claim (two items, part); only huge items have several parts.  With
    // fewer items than warps each is claimed alone, and blocks beyond the last
    // claim leave at once.
    const uint32_t warps = gridDim.x * HV_WARPS;
    const uint32_t uh = nhuge < warps / 16u ? 1u : 2u, uo = nother < warps ? 1u : 2u;
    const uint32_t mh = (nhuge + uh - 1u) / uh, mo = (nother + uo - 1u) / uo;
    const uint32_t ph = mh >= (1u << 28) ? 1u : max(8u, min(64u, 4u * warps / max(mh, 1u)));
    const uint32_t ch = mh * ph;
    if (blockIdx.x * HV_WARPS >= ch + mo) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int colwords = 2 * (q.ncol + 1) * 16;
    uint32_t* slots = smem + HV_WARPS * colwords;
    uint32_t* cols = smem + warp * colwords;
    for (int i = tid; i < q.nslots; i += HV_THREADS) slots[i] = q.slots[i];
    for (int i = lane; i < colwords; i += 32) cols[i] = 0u;
    __syncthreads();
    // Pairs first, then long rows alone, then the rest: warps of an SM run the
    // same loop at a time (the three together exceed the instruction cache).
#pragma unroll 1
    for (int phase = 0; phase < 3; ++phase) {
        for (;;) {
            uint32_t i = 0;
            if (lane == 0) i = atomicAdd(q.ctl + 3 + phase, 1u);
            i = __shfl_sync(0xffffffffu, i, 0);
            if (i >= ch + mo) break;
            const bool huge = i < ch;
            const uint32_t k = huge ? i / ph : i - ch, part = huge ? i % ph : 0u;
            const uint32_t nparts = huge ? ph : 1u, per = huge ? uh : uo;
            const uint32_t n = min(per, (huge ? nhuge : nother) - per * k);
            uint2 it[2];
#pragma unroll
            for (uint32_t j = 0; j < 2u; ++j)
                it[j] = j < n ? q.list[huge ? per * k + j : q.cap - 1u - (per * k + j)] : make_uint2(0u, 0u);
            if (paired<BY_WARPS>(p, it, n)) {
                if (phase == 0) count_items<R, 2, false>(p, q, it, part, nparts, cols, slots, lane);
            } else if (phase == 1) {
#pragma unroll 1
                for (uint32_t j = 0; j < n; ++j) {
                    const uint2 one = j ? it[1] : it[0];
                    if (!(one.y & (kItemZone | kItemFar | kItemShort)))
                        count_items<R, 1, false>(p, q, &one, part, nparts, cols, slots, lane, from(one));
                }
            } else if (phase == 2) {
#pragma unroll 1
                for (uint32_t j = 0; j < n; ++j) {
                    const uint2 one = j ? it[1] : it[0];
                    if (one.y & (kItemZone | kItemFar)) count_literal<R>(p, q, one, part, nparts, lane);
                    else if (one.y & kItemShort)
                        count_items<R, 1, true>(p, q, &one, part, nparts, cols, slots, lane, from(one));
                }
            }
        }
    }
}

// What the full list left: a warp claims the marks of 64 halos and counts the
// images one after the other.
template <int R>
__global__ void __launch_bounds__(HV_THREADS, HV_BLOCKS)
k_left_count(const __grid_constant__ CountParams p, const __grid_constant__ LaneParams q) {
    extern __shared__ uint32_t smem[];
    if (q.ctl[kCtlLeft] == 0u) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int colwords = (q.ncol + 1) * 16;
    uint32_t* slots = smem + HV_WARPS * colwords;
    uint32_t* cols = smem + warp * colwords;
    for (int i = tid; i < q.nslots; i += HV_THREADS) slots[i] = q.slots[i];
    for (int i = lane; i < colwords; i += 32) cols[i] = 0u;
    __syncthreads();
    const uint64_t words = (p.nhalos * (uint64_t)p.nidx + 1u) / 2u;
    for (;;) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(q.ctl + kCtlLeft + 1, 1u);
        i = __shfl_sync(0xffffffffu, i, 0);
        const uint64_t w0 = (uint64_t)i * 32u;
        if (w0 >= words) break;
        const uint32_t mine = w0 + lane < words ? q.left[w0 + lane] : 0u;
        uint32_t any = __ballot_sync(0xffffffffu, mine != 0u);
        for (; any; any &= any - 1u) {
            const int j = __ffs((int)any) - 1;
            for (uint32_t m = __shfl_sync(0xffffffffu, mine, j); m; m &= m - 1u) {
                const uint32_t b = (uint32_t)__ffs((int)m) - 1u;
                const uint64_t at16 = 2u * (w0 + (uint32_t)j) + (b >> 4), f = at16 / p.nhalos;
                const uint2 it = make_uint2((uint32_t)(at16 - f * p.nhalos),
                                            (b & 7u) | ((uint32_t)f << 3) | ((b & 8u) ? kItemZone : 0u));
                if ((b & 8u) || beyond(q, item_centre(p, it))) count_literal<R>(p, q, it, 0u, 1u, lane);
                else count_items<R, 1, true>(p, q, &it, 0u, 1u, cols, slots, lane);
            }
        }
    }
}

}  // namespace

bool lane_count_applies(const sjcs_query* q, const CountParams& p) {
    if (!q->lane.nslots || !p.prune || p.nhalos >= (1ull << 29)) return false;
    for (int i = 0; i < p.nidx; ++i)
        if (p.mn[i] >= kEndSlot) return false;
    return true;
}

bool ignores_schedule(const sjcs_query* q, const sjcs_index* idx) {
    CountParams p{};
    p.prune = q->monotone && std::isfinite(q->r2max) ? 1 : 0;
    p.nhalos = q->nhalos;
    p.nidx = 1;
    p.mn[0] = (uint32_t)idx->n;
    return lane_count_applies(q, p);
}

namespace {
// The list takes 1.5 items per halo and index.  An image is one item at most:
// lists of up to kExactItems (64 MB), and those of counts without images, have
// room for all of them and nothing is ever left (marks and an idle k_left_count
// cost about 5 us).
constexpr uint64_t kExactItems = 1u << 23;

// List, control words and marks of a count on stream s.  A pool that cannot
// give the whole list gives a shorter one, down to none.
int alloc_list(StreamScratch& scr, const CountParams& p, bool lean, LaneParams* q, cudaStream_t s) {
    const uint64_t n = p.nhalos * (uint64_t)p.nidx;
    // a lean query's list stays within what a server admits a request with
    const uint64_t part = n + (lean ? n / 4 : n / 2) + 1024;
    uint64_t cap = n * (p.periodic ? 8u : 1u), marks = 0;
    auto not_all = [&] {
        cap = std::min<uint64_t>(part, 0xf0000000ull);
        marks = (n + 1) / 2;
    };
    if (cap > std::max(lean ? 0 : kExactItems, part) || cap > 0xf0000000ull) not_all();
    uint32_t* ctl = nullptr;
    for (;;) {
        const cudaError_t e =
            scr.alloc(&ctl, (kLaneCtlWords + marks + (marks & 1u)) * sizeof(uint32_t) + cap * sizeof(uint2));
        if (e == cudaSuccess) break;
        if (e != cudaErrorMemoryAllocation || cap == 0) SJCS_CUDA_TRY(e);
        cudaGetLastError();
        if (!marks) not_all();
        cap = cap > 4096 ? cap / 4 : 0;
    }
    SJCS_CUDA_TRY(cudaMemsetAsync(ctl, 0, (kLaneCtlWords + marks) * sizeof(uint32_t), s));
    q->ctl = ctl;
    q->left = marks ? ctl + kLaneCtlWords : nullptr;
    q->list = reinterpret_cast<uint2*>(ctl + kLaneCtlWords + marks + (marks & 1u));
    q->cap = q->cap_huge = q->cap_other = (uint32_t)cap;
    return SJCS_OK;
}

// 1 to *gate if few of the halos sampled lie in clumps: if the 3 x 3 rows around
// a halo's, as far as its box in x (its own quad, in a Morton index), hold more
// than 2.5 times the particles of a uniform set there.
template <bool ROWS>
__global__ void __launch_bounds__(kSample) k_sample_density(const __grid_constant__ CountParams p,
                                                            uint32_t* __restrict__ gate) {
    const uint64_t h = (uint64_t)threadIdx.x * p.nhalos / kSample;
    const float4 c = p.halos[h];
    const Image im = make_image(p, c.x, c.y, c.z);
    const int y = cell_of(c.y, p.g.inv_h[1], p.g.G[1]), z = cell_of(c.z, p.g.inv_h[2], p.g.G[2]);
    const uint32_t* __restrict__ cs = p.mcs[0];
    uint32_t n = 0, cells = 0;
    if constexpr (ROWS) {
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int yy = y + k % 3 - 1, zz = z + k / 3 - 1;
            if (yy < 0 || yy >= p.g.G[1] || zz < 0 || zz >= p.g.G[2]) continue;
            const uint64_t rc = ((uint64_t)zz * (uint64_t)p.g.G[1] + (uint64_t)yy) * (uint64_t)p.g.G[0];
            n += __ldg(cs + rc + im.x1 + 1) - __ldg(cs + rc + im.x0);
            cells += (uint32_t)(im.x1 - im.x0 + 1);
        }
    } else {
        const uint32_t code = morton_cell((uint32_t)cell_of(c.x, p.g.inv_h[0], p.g.G[0]), (uint32_t)y, (uint32_t)z) & ~3u;
        n = __ldg(cs + code + 4u) - __ldg(cs + code);
        cells = 4u;
    }
    const bool dense = (float)n > 2.5f * (float)p.mn[0] * (float)cells / (float)p.g.ncells;
    const int all = __syncthreads_count(dense);
    if (threadIdx.x == 0) *gate = all <= kSampleDense ? 1u : 0u;
}

LaneParams lane_params(const sjcs_query* qq, const CountParams& p, const LaneModel* model) {
    const auto& L = qq->lane;
    LaneParams q{};
    q.slots = L.slots;
    q.nslots = L.nslots;
    q.kbase = L.kbase;
    q.shift = L.shift;
    q.khi = (L.nslots << L.shift) - 1;
    q.ncol = L.ncol;
    q.safe2 = L.safe2;
    uint32_t km;
    std::memcpy(&q.zone0, &L.safe2, 4);
    std::memcpy(&km, &p.r2max, 4);
    q.zone = km - q.zone0;
    q.cmax = L.cmax;
    if (model) {
        q.leaves = model->leaves;
        q.root = model->root;
        q.wpref = reinterpret_cast<const uint32_t*>(p.mpts[0]) + 3;
        q.key_shift = model->key_shift;
    }
    return q;
}

size_t listed_smem(const LaneParams& q) { return HV_WARPS * 2 * (size_t)(q.ncol + 1) * 64 + (size_t)q.nslots * 4; }

// The items of q's list (front and end), and what was marked beside it.
template <int R, bool BY_WARPS>
int launch_listed(sjcs_ctx* ctx, const CountParams& p, const LaneParams& q, bool noalloc, cudaStream_t s) {
    const size_t smem = listed_smem(q);
    int per_sm = 0;
    auto listed = k_listed_count<R, HV_BLOCKS, BY_WARPS>;
    if constexpr (R == RANGE_ROWS)
        if (noalloc) listed = k_listed_count<R, HV_BLOCKS_NOALLOC, BY_WARPS>;
    SJCS_CUDA_TRY(allow_block_smem(listed));
    SJCS_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, listed, HV_THREADS, smem));
    if (per_sm < 1) per_sm = 1;
    const unsigned blocks = (unsigned)(ctx->num_sms * per_sm);
    listed<<<blocks, HV_THREADS, smem, s>>>(p, q);
    SJCS_LAUNCH_CHECK();
    if (q.left) {
        SJCS_CUDA_TRY(allow_block_smem(k_left_count<R>));
        k_left_count<R><<<blocks, HV_THREADS, smem, s>>>(p, q);
        SJCS_LAUNCH_CHECK();
    }
    return SJCS_OK;
}

// Most candidates of a lane's walk: a batch lasts as long as its longest lane,
// so with few batches per SM long walks are left to the list (1e5 clustered
// halos on 2e7 particles at R = 10, 1.3 waves: 1.06 ms without this, 0.78 with
// it), but not below 160 (131072 x 20000, R = 40: 98 us a call with 96, 78 with
// 160).  Quads of Morton cells hold a quarter more candidates than rows (1e6 x
// 2e5 uniform at R = 20: 0.50 ms with 8, 0.35 with 10, 0.42 with 13).
uint32_t walk_limit(sjcs_ctx* ctx, const CountParams& p, bool rows) {
    const uint64_t nbatch = (p.nhalos + 31) / 32, per = rows ? 8 : 10;
    return (uint32_t)std::min<uint64_t>(kWalkMax, std::max<uint64_t>(160, nbatch * per / (uint64_t)ctx->num_sms));
}

// Fewer halos than a few for every warp.
bool few_halos(sjcs_ctx* ctx, const CountParams& p) {
    return p.nhalos < (uint64_t)ctx->num_sms * HV_WARPS * HV_BLOCKS * 4;
}

// The box of a halo far from the faces, were the particles uniform: about the
// candidates that the sphere leaves of it, and its ranges.
struct UniformBox {
    double candidates, ranges;
};
UniformBox uniform_box(const CountParams& p, bool rows) {
    const double e = std::min(p.half, p.reach);
    UniformBox b{0.0, 1.0};
    for (int f = 0; f < p.nidx; ++f) b.candidates += 0.625 * p.mn[f] / p.nidx;
    for (int a = 0; a < 3; ++a) {
        const double h = 1000.0 / p.g.G[a], unit = !rows && a < 2 ? 2.0 * h : h;  // quads begin and end at even cells
        const double w = std::min(1000.0, 2.0 * e + unit);
        b.candidates *= w / 1000.0;
        if (!rows || a > 0) b.ranges *= w / unit;
    }
    return b;
}

template <int R, bool PACK>
int launch_ranges(sjcs_ctx* ctx, const sjcs_query* qq, const CountParams& p, cudaStream_t s, const LaneScratch* given,
                  const LaneModel* model, const Warps& warps) {
    LaneParams q = lane_params(qq, p, model);
    StreamScratch scr(s);
    if (given) {
        q.ctl = given->ctl;
        q.list = given->list;
        q.cap = q.cap_huge = q.cap_other = given->cap;
    } else {
        const int rc = alloc_list(scr, p, qq->lean, &q, s);
        if (rc) return rc;
    }
    q.huge = few_halos(ctx, p) ? kHugeFew : kHuge;
    q.walk_max = walk_limit(ctx, p, R == RANGE_ROWS);
    if (warps) {
        CountParams w = p;
        w.gate = q.gate = q.ctl + kCtlGate;
        k_sample_density<R == RANGE_ROWS><<<1, kSample, 0, s>>>(p, q.gate);
        SJCS_LAUNCH_CHECK();
        w.heavy = (uint32_t)std::min(1e9, 1.5 * uniform_box(p, R == RANGE_ROWS).candidates);
        w.huge = q.huge;
        w.list_ctl = q.ctl;
        w.list = q.list;
        w.list_cap = q.cap;
        w.list_huge = q.cap_huge = q.cap / 8u;
        q.cap_other = q.cap - q.cap_huge;
        const int rc = warps(w);
        if (rc) return rc;
    }
    // one block per SM (neighbouring batches share its L1); blocks of fewer
    // warps when there are not enough batches for every SM
    const uint64_t nbatch = (p.nhalos + 31) / 32, sms = (uint64_t)ctx->num_sms;
    const size_t warp_a = sizeof(LaneRows<PACK>) + (size_t)(q.ncol + 1) * 64, table = (size_t)q.nslots * 4;
    const int fit = (int)std::min<size_t>(LN_WARPS, (kMaxBlockSmem - table) / warp_a);  // >= 15 for any table
    const int nw = (int)std::min<uint64_t>((uint64_t)fit, (nbatch + sms - 1) / sms);
    const uint64_t blocks = std::min<uint64_t>((nbatch + (uint64_t)nw - 1) / (uint64_t)nw, sms);
    SJCS_CUDA_TRY(allow_block_smem(k_lane_count<R, PACK>));
    k_lane_count<R, PACK><<<(unsigned)blocks, nw * 32, nw * warp_a + table, s>>>(p, q);
    SJCS_LAUNCH_CHECK();
    if (warps) {
        LaneParams w = q;
        w.left = nullptr;  // only lanes mark
        const int rc = launch_listed<R, true>(ctx, p, w, given != nullptr, s);
        if (rc) return rc;
    }
    return launch_listed<R, false>(ctx, p, q, given != nullptr, s);
}
}  // namespace

namespace {
bool few_batches(const sjcs_ctx* ctx, uint64_t nhalos) {
    return (nhalos + 31) / 32 <= (uint64_t)ctx->num_sms * kFewBatches;
}
}  // namespace

// An image or two of every halo on one to three indexes.
uint32_t count_by_warps_items(const sjcs_ctx* ctx, uint64_t nhalos) {
    return few_batches(ctx, nhalos) ? (uint32_t)(4 * nhalos) : 0u;
}

// Boxes that lanes would walk: by the number of batches.  Fuller ones are all
// listed by lanes: that is ahead in long rows, and behind in short ones unless
// the halos lie in clumps (1e5 on 3e7 particles, R = 15: uniform 805 us listed
// and 404 by warps, clustered 1388 and 1870), which a sample of 6 us tells; the
// extra launches take 15 us of a small count.  Below a batch per SM nothing
// pays for a sample, and rows are better off with warps (1000 on 2e7, R = 20:
// clustered 151 and 153, uniform 73 and 54), quads of the table with lanes (124
// and 212, 107 and 75), those of the model with warps (473 and 262, 350 and 91).
// Halos in no order (sorted false, the allocation-free call's): warps that take
// neighbours share no particle lines, so lanes from a batch per SM on (20000 on
// 131072 at R = 40 75 us a call, 81 by warps; 130 on them 69 and 61).
Counter who_counts(sjcs_ctx* ctx, const CountParams& p, RangesOf of, bool sorted) {
    if (!sorted) return (p.nhalos + 31) / 32 <= (uint64_t)ctx->num_sms ? Counter::Warps : Counter::Lanes;
    const bool rows = of == RangesOf::Rows, few = few_batches(ctx, p.nhalos);
    const UniformBox b = uniform_box(p, rows);
    if (b.candidates <= (double)walk_limit(ctx, p, rows)) return few ? Counter::Warps : Counter::Lanes;
    if (b.candidates >= (rows ? kLongRow : kLongQuad) * b.ranges) return Counter::Lanes;
    if (few && of == RangesOf::Model) return Counter::Warps;
    if ((p.nhalos + 31) / 32 <= (uint64_t)ctx->num_sms) return rows ? Counter::Warps : Counter::Lanes;
    return Counter::Sampled;
}

int list_for_warps(sjcs_ctx* ctx, const sjcs_query* q, CountParams* p, RangesOf ranges, StreamScratch& scr,
                   cudaStream_t s, const LaneScratch* given) {
    // What is ordinary at this density stays with its warp (listing from 1.1
    // times that on took 106 us for 10500 uniform halos on 1e7 particles at R =
    // 20, 1.3 to 2.5 times 97).  With less than a warp for every listed image
    // each is split; the more halos, the more of them are left to balance the
    // warps (clustered, 100 halos: 45 us from 512 on and 60 from 1024; 20000: 141
    // and 129).
    const bool split = (p->nhalos + 31) / 32 <= (uint64_t)ctx->num_sms;
    p->heavy = (uint32_t)std::min(
        1e9, std::max(split ? 512.0 : 1024.0, (split ? 1.2 : 1.5) * uniform_box(*p, ranges == RangesOf::Rows).candidates));
    p->huge = split ? 0u : kHugeFew;
    if (given) {
        p->list_ctl = given->ctl;
        p->list = given->list;
        p->list_cap = given->cap;
    } else {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        SJCS_CUDA_TRY(cudaStreamIsCapturing(s, &capture));
        uint32_t* base = q->list_ctl;
        if (capture != cudaStreamCaptureStatusNone) {
            // a graph may run beside other counts of its query
            SJCS_CUDA_TRY(scr.alloc(&base, count_by_warps_bytes(q->list_items)));
            SJCS_CUDA_TRY(cudaMemsetAsync(base, 0, kListWords * sizeof(uint32_t), s));
            p->list_ctl = base;
        } else {
            p->list_ctl = base + (q->list_turn & 1u) * kListWords;
            p->list_clear = base + (~q->list_turn & 1u) * kListWords;
            ++q->list_turn;
        }
        p->list = reinterpret_cast<uint2*>(base + 2 * kListWords);
        p->list_cap = q->list_items;
    }
    p->list_huge = split ? p->list_cap : p->list_cap / 2u;
    return SJCS_OK;
}

int launch_listed_images(sjcs_ctx* ctx, const sjcs_query* qq, const CountParams& p, RangesOf ranges, cudaStream_t s,
                         const LaneScratch* given, const LaneModel* model) {
    LaneParams q = lane_params(qq, p, model);
    q.ctl = p.list_ctl;
    q.list = p.list;
    q.cap = p.list_cap;
    q.cap_huge = p.list_huge;
    q.cap_other = p.list_cap - p.list_huge;
    if (ranges == RangesOf::Rows) return launch_listed<RANGE_ROWS, true>(ctx, p, q, given != nullptr, s);
    return model ? launch_listed<RANGE_MODEL, true>(ctx, p, q, false, s)
                 : launch_listed<RANGE_CELLS, true>(ctx, p, q, false, s);
}

int launch_lane_count(sjcs_ctx* ctx, const sjcs_query* q, const CountParams& p, cudaStream_t s,
                      const LaneScratch* given, const Warps& warps) {
    // Packed rows need the slots of a box's planes within 2^24 of each other;
    // with more than 2^29 particles ordinary boxes would not be.
    bool pack = true;
    for (int i = 0; i < p.nidx; ++i) pack &= p.mn[i] <= (1u << 29);
    return pack ? launch_ranges<RANGE_ROWS, true>(ctx, q, p, s, given, nullptr, warps)
                : launch_ranges<RANGE_ROWS, false>(ctx, q, p, s, given, nullptr, warps);
}

int launch_lane_count_cells(sjcs_ctx* ctx, const sjcs_query* q, const CountParams& p, cudaStream_t s,
                            const LaneModel* model, const Warps& warps) {
    return model ? launch_ranges<RANGE_MODEL, false>(ctx, q, p, s, nullptr, model, warps)
                 : launch_ranges<RANGE_CELLS, false>(ctx, q, p, s, nullptr, nullptr, warps);
}

}  // namespace sjcs
