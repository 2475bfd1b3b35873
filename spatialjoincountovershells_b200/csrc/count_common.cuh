// Device code shared by the shell-count kernels (grid rows and Morton cells):
// the kernel parameters, the exact acceptance test and shell binning, and the
// flattening of per-lane slot ranges into coalesced candidate windows.
// The arithmetic contract is documented in shell_count.cu.
#pragma once

#include <cmath>

#include "sjcs_internal.cuh"

namespace sjcs {
namespace count {

enum BinMode { BIN_LUT = 0, BIN_BSEARCH = 1, BIN_FIRST_MATCH = 2 };
constexpr int kMaxFused = kMaxFusedIndexes;  // indexes counted in one pass by k_shell_count_multi

struct CountParams {
    const float4* __restrict__ pts;  // particles grouped by cell (x, y, z; .w not read)
    const uint32_t* __restrict__ cs;
    GridGeom g;
    float h[3];                      // cell edge per axis, 1000 / G
    const float4* __restrict__ halos;
    uint64_t nhalos;
    const float* __restrict__ r2;    // [pad], +inf past nrads
    const uint32_t* __restrict__ lut;
    int nrads;
    int pad;
    int nlut;
    uint32_t lut_k0;                 // bit pattern of r2[0]
    int lut_shift;
    float half;
    float reach;                     // a counted particle lies within this of the centre on each axis (see make_image)
    float r2max;
    float r2p;                       // r2max * (1 + 1e-5)
    float r2slack;                   // r2max * 1e-5
    int periodic;
    int prune;
    uint32_t* __restrict__ counts;
    // several indexes of one grid counted in one pass (k_shell_count_multi)
    int nidx;
    const float4* mpts[kMaxFused];
    const uint32_t* mcs[kMaxFused];
    uint32_t mn[kMaxFused];  // particles of each index
    // Images of more than `heavy` candidates go to a list instead (LIST
    // variants of the kernels) for k_listed_count, which splits those of more
    // than `huge` over several warps.
    uint32_t heavy, huge;
    uint32_t list_cap, list_huge;  // room, and the part of it for huge ones
    uint32_t* list_ctl;            // [1] huge ones, from the front, [2] others, from the end
    uint32_t* list_clear;  // control words to clear for the next count, or null
    const uint32_t* gate;  // LIST variants count only if this holds a 1 (null: always)
    uint2* list;
};

// Item of a list of images: the halo's place, and bits 0-2 the shifted axes,
// bits 3-4 the index, from kItemFrom on the first 32 ranges still to count.
constexpr uint32_t kItemShort = 1u << 9;  // short rows: flattened before they are read
constexpr int kItemFrom = 10;
constexpr uint32_t kItemFromMax = 1u << 22;
constexpr int kListWords = 8;  // control words of a list

// The control words that the next count of the query will use (its counts take
// turns with two sets, so none needs a launch to clear its own).
__device__ __forceinline__ void clear_next_list(const CountParams& p) {
    if (p.list_clear && blockIdx.x == 0 && threadIdx.x < kListWords) p.list_clear[threadIdx.x] = 0u;
}

// Cycles of the data pipe that reading a listed item costs for one of its rows
// and for a candidate, in 1/32 cycles, when rows are read one by one and when
// they are flattened first (see lane_count.cu).
constexpr uint32_t kRowCost = 20, kRowCand = 9, kFlatCand = 22;
__device__ __forceinline__ bool short_rows(uint32_t T, uint32_t rows) {
    return ((kFlatCand - kRowCand) * T >> 5) < kRowCost * rows;
}

// Puts a warp's image of T candidates in `rows` ranges on the list; false: no
// room.
__device__ __forceinline__ bool list_image(const CountParams& p, uint2 it, uint32_t T, uint32_t rows, int lane) {
    bool fits = false;
    if (lane == 0) {
        const bool huge = T > p.huge;
        uint32_t* n = p.list_ctl + (huge ? 1 : 2);
        const uint32_t room = huge ? p.list_huge : p.list_cap - p.list_huge;
        // a full part is not counted on: no wrap, however many items come
        if (*const_cast<volatile uint32_t*>(n) < room) {
            const uint32_t i = atomicAdd(n, 1u);
            fits = i < room;
            if (short_rows(min(T, 1u << 24), rows)) it.y |= kItemShort;
            if (fits) p.list[huge ? i : p.list_cap - 1u - i] = it;
        }
    }
    return __shfl_sync(0xffffffffu, fits, 0);
}

// Lets kern use all the shared memory a block can have.  The limit belongs to
// the function on its device, not to a launch: every call sets the same value,
// so that host threads with contexts of their own cannot lower it between
// another's setting and launch.  Not for kernels with static shared memory.
constexpr size_t kMaxBlockSmem = 227 * 1024;
template <class Kernel>
inline cudaError_t allow_block_smem(Kernel kern) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxBlockSmem);
}

// CountParams::reach: with pruning, a bound above the square root of r2p plus
// the rounding of the differences; else no bound.
inline float reach_of(float r2max, bool prune) {
    return prune ? (float)(std::sqrt((double)r2max * (1.0 + 1e-5)) * (1.0 + 1e-6) + 4e-3) : INFINITY;
}

__device__ __forceinline__ float edge_margin(float v) { return 1e-3f + 2e-6f * fabsf(v); }

// Lower bound of |c - y| over every y whose cell index is k.
__device__ __forceinline__ float cell_gap(float c, int k, float h, int G) {
    const float lo_e = (float)k * h, hi_e = (float)(k + 1) * h;
    const float lo = (k == 0) ? -INFINITY : lo_e - edge_margin(lo_e);
    const float hi = (k == G - 1) ? INFINITY : hi_e + edge_margin(hi_e);
    return fmaxf(0.0f, fmaxf(lo - c, c - hi));
}

template <int BIN>
__device__ __forceinline__ int bin_of(const CountParams& p, const float* __restrict__ tab,
                                      const uint32_t* __restrict__ lut, float dist) {
    if (BIN == BIN_LUT) {
        const uint32_t key = __float_as_uint(dist);
        if (key < p.lut_k0) return 0;
        const int s = (int)lut[(key - p.lut_k0) >> p.lut_shift];
        return s + ((tab[s] <= dist) ? 1 : 0);
    } else {
        int s = 0;
        for (int step = p.pad >> 1; step > 0; step >>= 1) s += (tab[s + step - 1] <= dist) ? step : 0;
        return s;
    }
}

// Image set-up: the query box, its cell range and the clipping constants.
struct Image {
    float cx, cy, cz;
    float lox, hix, loy, hiy, loz, hiz;
    int x0, x1, y0, y1, z0, z1;
    int ny, nz;
    uint32_t nrows;  // saturated at 2^31
};

__device__ __forceinline__ Image make_image(const CountParams& p, float cx, float cy, float cz) {
    Image im;
    im.cx = cx;
    im.cy = cy;
    im.cz = cz;
    im.lox = __fsub_rn(cx, p.half);
    im.hix = __fadd_rn(cx, p.half);
    im.loy = __fsub_rn(cy, p.half);
    im.hiy = __fadd_rn(cy, p.half);
    im.loz = __fsub_rn(cz, p.half);
    im.hiz = __fadd_rn(cz, p.half);
    // Cells: those of the box, but no further from the centre than a counted
    // particle can be (non-periodic boxes are r2max wide, far wider than the
    // sphere when R > 1).  A NaN bound passes every particle on that side of
    // the box test, so it must open the cell range to the grid edge (cell_of
    // maps NaN to cell 0, which is right for a lower bound only).
    const float rx = p.reach + 1e-6f * fabsf(cx), ry = p.reach + 1e-6f * fabsf(cy), rz = p.reach + 1e-6f * fabsf(cz);
    const float hx = fminf(im.hix, cx + rx), hy = fminf(im.hiy, cy + ry), hz = fminf(im.hiz, cz + rz);
    im.x0 = cell_of(fmaxf(im.lox, cx - rx), p.g.inv_h[0], p.g.G[0]);
    im.x1 = (hx != hx) ? p.g.G[0] - 1 : cell_of(hx, p.g.inv_h[0], p.g.G[0]);
    im.y0 = cell_of(fmaxf(im.loy, cy - ry), p.g.inv_h[1], p.g.G[1]);
    im.y1 = (hy != hy) ? p.g.G[1] - 1 : cell_of(hy, p.g.inv_h[1], p.g.G[1]);
    im.z0 = cell_of(fmaxf(im.loz, cz - rz), p.g.inv_h[2], p.g.G[2]);
    im.z1 = (hz != hz) ? p.g.G[2] - 1 : cell_of(hz, p.g.inv_h[2], p.g.G[2]);
    im.ny = im.y1 - im.y0 + 1;
    im.nz = im.z1 - im.z0 + 1;
    const uint64_t nr = (uint64_t)im.ny * (uint64_t)im.nz;
    im.nrows = nr > 0x80000000ull ? 0x80000000u : (uint32_t)nr;
    return im;
}

// ZONE: only distances >= zone_lo are counted.
template <int BIN, bool BIG, bool ZONE = false>
__device__ __forceinline__ void test_candidate(const CountParams& p, const Image& im, const float4 pp, bool live,
                                               uint32_t* __restrict__ sink, const float* __restrict__ tab,
                                               const uint32_t* __restrict__ lut, float zone_lo = 0.0f) {
    const bool inb = !(pp.x < im.lox) & !(im.hix < pp.x) & !(pp.y < im.loy) & !(im.hiy < pp.y) &
                     !(pp.z < im.loz) & !(im.hiz < pp.z);
    const float dx = __fsub_rn(pp.x, im.cx), dy = __fsub_rn(pp.y, im.cy), dz = __fsub_rn(pp.z, im.cz);
    const float dist = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    if (BIN != BIN_FIRST_MATCH) {
        if (live && inb && dist < p.r2max && (!ZONE || dist >= zone_lo)) atomicAdd(sink + bin_of<BIN>(p, tab, lut, dist), 1u);
    } else if (live && inb) {
        for (int i = 0; i < p.nrads; ++i) {
            if (dist < tab[i]) {
                atomicAdd(sink + i, 1u);
                break;
            }
        }
    }
}

// Scan the lanes' row lengths and test every candidate of those rows,
// two windows of 32 candidates per iteration so two loads are in flight.
// LIST: rows of more than `most` candidates are left to the list as item it;
// returns the candidates counted, or kListed.
constexpr uint32_t kListed = 0xffffffffu;
template <int BIN, bool BIG, bool LIST = false>
__device__ __forceinline__ uint32_t run_rows(const CountParams& p, const Image& im, uint32_t start, uint32_t end,
                                             uint32_t* __restrict__ sink, const float* __restrict__ tab,
                                             const uint32_t* __restrict__ lut, int lane, uint32_t most = 0,
                                             uint2 it = make_uint2(0u, 0u)) {
    const uint32_t len = end - start;
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    if constexpr (LIST)
        if (total > most &&
            list_image(p, it, total, (uint32_t)__popc(__ballot_sync(0xffffffffu, len != 0u)), lane))
            return kListed;
    const uint32_t off = start - (incl - len);  // slot = t + off for t inside this row (mod 2^32)
    for (uint32_t wb = 0; wb < total; wb += 64) {
        const uint32_t t0 = wb + (uint32_t)lane, t1 = t0 + 32u;
        // row of t = #{rows j : incl_j <= t} (empty rows are skipped naturally)
        int r0 = 0, r1 = 0;
#pragma unroll
        for (int b = 16; b >= 1; b >>= 1) {
            const uint32_t v0 = __shfl_sync(0xffffffffu, incl, r0 + b - 1);
            const uint32_t v1 = __shfl_sync(0xffffffffu, incl, r1 + b - 1);
            r0 += (v0 <= t0) ? b : 0;
            r1 += (v1 <= t1) ? b : 0;
        }
        const uint32_t o0 = __shfl_sync(0xffffffffu, off, r0);
        const uint32_t o1 = __shfl_sync(0xffffffffu, off, r1);
        const bool l0 = t0 < total, l1 = t1 < total;
        const float4 p0 = l0 ? __ldg(p.pts + (t0 + o0)) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 p1 = l1 ? __ldg(p.pts + (t1 + o1)) : make_float4(0.f, 0.f, 0.f, 0.f);
        test_candidate<BIN, BIG>(p, im, p0, l0, sink, tab, lut);
        test_candidate<BIN, BIG>(p, im, p1, l1, sink, tab, lut);
    }
    return total;
}

// Piece `part` of `nparts` of the candidates of the lanes' rows: the
// contiguous share [total*part/nparts, total*(part+1)/nparts) of the
// flattened candidate sequence, so nparts warps sharing a halo split every
// row set evenly and together test each candidate once.
template <int BIN, bool BIG, bool ZONE = false>
__device__ __forceinline__ void run_rows_part(const CountParams& p, const Image& im, uint32_t start, uint32_t end,
                                              uint32_t* __restrict__ sink, const float* __restrict__ tab,
                                              const uint32_t* __restrict__ lut, int lane, uint32_t part,
                                              uint32_t nparts, float zone_lo = 0.0f) {
    const uint32_t len = end - start;
    uint32_t incl = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t off = start - (incl - len);
    const uint32_t tb = (uint32_t)(((uint64_t)total * part) / nparts);
    const uint32_t te = (uint32_t)(((uint64_t)total * (part + 1u)) / nparts);
    for (uint32_t wb = tb; wb < te; wb += 64) {
        const uint32_t t0 = wb + (uint32_t)lane, t1 = t0 + 32u;
        int r0 = 0, r1 = 0;
#pragma unroll
        for (int b = 16; b >= 1; b >>= 1) {
            const uint32_t v0 = __shfl_sync(0xffffffffu, incl, r0 + b - 1);
            const uint32_t v1 = __shfl_sync(0xffffffffu, incl, r1 + b - 1);
            r0 += (v0 <= t0) ? b : 0;
            r1 += (v1 <= t1) ? b : 0;
        }
        const uint32_t o0 = __shfl_sync(0xffffffffu, off, r0);
        const uint32_t o1 = __shfl_sync(0xffffffffu, off, r1);
        const bool l0 = t0 < te, l1 = t1 < te;
        const float4 p0 = l0 ? __ldg(p.pts + (t0 + o0)) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 p1 = l1 ? __ldg(p.pts + (t1 + o1)) : make_float4(0.f, 0.f, 0.f, 0.f);
        test_candidate<BIN, BIG, ZONE>(p, im, p0, l0, sink, tab, lut, zone_lo);
        test_candidate<BIN, BIG, ZONE>(p, im, p1, l1, sink, tab, lut, zone_lo);
    }
}

// Shell bucket of an estimated candidate count, for ordering work by size:
// 0 for none, else 1 + 8*floor(log2 e) + the next 3 bits of e (<= 256 values;
// neighbouring buckets differ by a factor <= 2^(1/8)).
__device__ __forceinline__ uint32_t est_bucket(uint32_t e) {
    if (e == 0) return 0u;
    const int lg = 31 - __clz(e);
    const uint32_t mant = lg >= 3 ? (e >> (lg - 3)) & 7u : (e << (3 - lg)) & 7u;
    const uint32_t b = 1u + 8u * (uint32_t)lg + mant;
    return b < 255u ? b : 255u;  // 8 bits
}

}  // namespace count
}  // namespace sjcs
