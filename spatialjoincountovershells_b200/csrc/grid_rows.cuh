// Rows of grid cells of a query box (device code shared by the grid count
// kernels): row numbering, clipping of a row to the sphere, and the row's
// slot range.  The margins are justified in shell_count.cu.
#pragma once

#include "count_common.cuh"

namespace sjcs {
namespace count {

// Row r of the image (r < nrows) -> (y cell, z cell); exact for all r < 2^31.
__device__ __forceinline__ void row_yz(const Image& im, uint32_t r, int* yy, int* zz) {
    uint32_t q;
    if (im.nrows <= (1u << 20)) {
        // float quotient estimate: relative error < 4e-7, so for r < 2^20 it is
        // off by at most one; corrected exactly below
        q = (uint32_t)__fmul_rz((float)r, __frcp_rn((float)im.ny));
        if (q * (uint32_t)im.ny > r) --q;
        else if ((q + 1u) * (uint32_t)im.ny <= r) ++q;
    } else {
        q = r / (uint32_t)im.ny;
    }
    *yy = im.y0 + (int)(r - q * (uint32_t)im.ny);
    *zz = im.z0 + (int)q;
}

// Lane `lane` takes row rb + lane of the image: clip its x cells to the
// sphere and fetch the row's first and one-past-last slots.  Returns the
// slot range through *start / *end (empty: start == end).  gy_l / gz_l are
// the lane-distributed gap tables of the image (valid when ny, nz <= 32).
__device__ __forceinline__ void row_issue(const CountParams& p, const Image& im, uint32_t rb, int lane,
                                          float gy_l, float gz_l, uint32_t* start, uint32_t* end) {
    const uint32_t r = rb + (uint32_t)lane;
    int yy = 0, zz = 0;
    const bool live = r < im.nrows;
    if (live) row_yz(im, r, &yy, &zz);
    int xa = im.x0, xb = im.x1;
    if (p.prune) {
        const bool small = im.ny <= 32 && im.nz <= 32;
        float gy = __shfl_sync(0xffffffffu, gy_l, (yy - im.y0) & 31);
        float gz = __shfl_sync(0xffffffffu, gz_l, (zz - im.z0) & 31);
        if (!small) {
            gy = cell_gap(im.cy, yy, p.h[1], p.g.G[1]);
            gz = cell_gap(im.cz, zz, p.h[2], p.g.G[2]);
        }
        const float rem =
            __fadd_rn(__fsub_rn(__fsub_rn(p.r2p, __fmul_rn(gy, gy)), __fmul_rn(gz, gz)), p.r2slack);
        if (rem < 0.0f) {
            xb = xa - 1;  // no particle of this row can be within R
        } else {
            // approximate square root: its error (< 1e-6 relative) is far inside the margin
            float xr = rem > 0.0f ? __fmul_rn(rem, rsqrtf(rem)) : 0.0f;
            xr = __fadd_rn(xr, 1e-3f + 1e-6f * (fabsf(im.cx) + xr));
            const float xl = __fsub_rn(im.cx, xr), xh = __fadd_rn(im.cx, xr);
            xa = max(xa, cell_of(xl, p.g.inv_h[0], p.g.G[0]));
            if (xh == xh) xb = min(xb, cell_of(xh, p.g.inv_h[0], p.g.G[0]));
        }
    }
    uint32_t s0 = 0, s1 = 0;
    if (live && xa <= xb) {
        const uint64_t rowcell = ((uint64_t)zz * (uint64_t)p.g.G[1] + (uint64_t)yy) * (uint64_t)p.g.G[0];
        s0 = __ldg(p.cs + rowcell + xa);
        s1 = __ldg(p.cs + rowcell + xb + 1);
    }
    *start = s0;
    *end = s1;
}

// Lane-distributed gap tables: lane j holds the gap of y cell y0 + j (and z).
__device__ __forceinline__ void gap_tables(const CountParams& p, const Image& im, int lane, float* gy, float* gz) {
    *gy = 0.0f;
    *gz = 0.0f;
    if (p.prune) {
        if (lane < im.ny) *gy = cell_gap(im.cy, im.y0 + lane, p.h[1], p.g.G[1]);
        if (lane < im.nz) *gz = cell_gap(im.cz, im.z0 + lane, p.h[2], p.g.G[2]);
    }
}

}  // namespace count
}  // namespace sjcs
