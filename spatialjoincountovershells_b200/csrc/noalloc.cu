// sjcs_count_noalloc: one particle file's shell counts for small inputs with
// no device allocation at all.
//
// Some callers cannot let a library call cudaMalloc: a host program whose
// framework has already reserved the GPU's memory for its own caching
// allocator (a library cudaMalloc then fails or fragments that pool), or a
// latency-critical loop that cannot absorb the device-wide synchronisation a
// cudaMalloc/cudaFree may imply.  For them this entry point builds the grid
// index and counts shells using only a fixed scratch area that lives in a
// file-scope __device__ array (SJCS_NOALLOC_SCRATCH_BYTES, about 9.3 MB),
// plus the caller's own input and output buffers.
//
// Every GPU that loads this library's module holds that array until the
// process exits.  With lazy module loading (the CUDA default since 12.2) the
// module, and with it the array, is loaded on a device by the first call made
// while that device is current -- its cudaGetSymbolAddress -- so that first
// call is when the driver sets the 9.3 MB aside: make it before a framework
// reserves the device's memory, or set CUDA_MODULE_LOADING=EAGER to load it
// with the library.  Make that first call before any stream capture too.
// All calls share the array and it keeps the last call's contents, so calls
// that overlap on the GPU (two streams, two host threads) race and must be
// serialised by the caller; what must start at zero (digit counts, list
// control words) is cleared by each call.
#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "count_common.cuh"
#include "lane_count.cuh"
#include "sjcs_internal.cuh"

namespace sjcs {
namespace {

constexpr uint64_t kNP = SJCS_NOALLOC_MAX_PARTICLES;
constexpr uint64_t kNH = SJCS_NOALLOC_MAX_HALOS;
constexpr uint64_t kNC = SJCS_NOALLOC_MAX_CELLS;
constexpr int kNR = SJCS_NOALLOC_MAX_SHELLS;
constexpr int kMaxTable = 640;  // lane slots that travel with the launch (parameters stay under 4 KB)

constexpr uint64_t align256(uint64_t x) { return (x + 255) & ~uint64_t(255); }
// byte offsets of the sub-buffers (each 256-byte aligned)
constexpr uint32_t kListItems = (uint32_t)(8 * kNH);  // every image of every halo
constexpr uint64_t kOffPts = 0;
constexpr uint64_t kOffCells = align256(kOffPts + kNP * 16);
constexpr uint64_t kOffTmp = align256(kOffCells + (kNC + 1) * 4);
constexpr uint64_t kOffTop = align256(kOffTmp + kNP * 16);
constexpr uint64_t kOffCursors = align256(kOffTop + 514 * 4);
constexpr uint64_t kOffHalos = align256(kOffCursors + 513 * 4);
constexpr uint64_t kOffR2 = align256(kOffHalos + kNH * 16);
constexpr uint64_t kOffSlots = align256(kOffR2 + (uint64_t)kNR * 4);
constexpr uint64_t kOffCtl = align256(kOffSlots + (uint64_t)kMaxTable * 4);
constexpr uint64_t kOffList = align256(kOffCtl + (uint64_t)kLaneCtlWords * 4);
constexpr uint64_t kOffDense = align256(kOffList + (uint64_t)kListItems * 8);
constexpr uint64_t kScratchBytes = align256(kOffDense + kGridDenseWords * 4);
static_assert(kScratchBytes <= SJCS_NOALLOC_SCRATCH_BYTES, "the scratch array holds every buffer");

static __device__ __align__(256) unsigned char g_noalloc_scratch[SJCS_NOALLOC_SCRATCH_BYTES];

// Pairs up to which every particle is tested against every halo: at 2^24 that
// took 35-39 us a call and the index 45-47, at 2^25 65 and about 47 (2^23: 21
// and 59; a call of 2003 x 97 24, of which the caller spends 20, was 73).
constexpr uint64_t kDirectPairs = 1ull << 24;

constexpr int kMaxDevices = 64;
std::mutex g_setup_mu;
void* g_scratch_addr[kMaxDevices];

// Device address of the scratch array on the current device (set up once).
int scratch_address(unsigned char** out) {
    int dev = 0;
    SJCS_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(SJCS_ERR_INVALID, "device %d beyond the supported %d", dev, kMaxDevices);
    std::lock_guard<std::mutex> lk(g_setup_mu);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return fail(SJCS_ERR_CUDA, "cudaGetSymbolAddress of the scratch array failed on device %d: %s", dev,
                        cudaGetErrorString(e));
        g_scratch_addr[dev] = p;
    }
    *out = static_cast<unsigned char*>(g_scratch_addr[dev]);
    return SJCS_OK;
}

// The padded radius table and the lane slots travel as kernel arguments
// (copied at launch), so no host buffer has to outlive the call.
struct R2Table {
    float v[kNR];
};
struct Tables {
    R2Table r2;
    uint32_t slots[kMaxTable];
};

// Everything the build and the count start from: the tables, the cleared
// digit counts and list control words, and the halos in the caller's order.
__global__ void __launch_bounds__(256) k_noalloc_prep(const __grid_constant__ Tables t, int pad, int nslots,
                                                      const char* __restrict__ base, size_t stride, uint64_t nh,
                                                      float* __restrict__ r2, uint32_t* __restrict__ slots,
                                                      uint32_t* __restrict__ top, uint32_t* __restrict__ ctl,
                                                      float4* __restrict__ halos) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0) {
        for (int k = threadIdx.x; k < pad; k += blockDim.x) r2[k] = t.r2.v[k];
        for (int k = threadIdx.x; k < nslots; k += blockDim.x) slots[k] = t.slots[k];
        for (int k = threadIdx.x; k < 514; k += blockDim.x) top[k] = 0u;
        if (threadIdx.x < kLaneCtlWords) ctl[threadIdx.x] = 0u;
    }
    if (i < nh) {
        const float* p = reinterpret_cast<const float*>(base + i * stride);
        halos[i] = make_float4(p[0], p[1], p[2], __uint_as_float((uint32_t)i));
    }
}

// Few enough pairs: every particle against every halo, no index.  A warp takes
// four halos and every nslice-th run of 32 particles, so a particle is loaded
// once for four tests.  Nearly all pairs fail the compare of the distance with
// r2max; one that does not, and every shifted image, takes the reference's
// predicate literally (test_candidate) into the warp's shared counters.
constexpr int kDirectWarps = 8, kDirectHalos = 4;
template <int BIN>
__global__ void __launch_bounds__(kDirectWarps * 32)
k_count_direct(const __grid_constant__ count::CountParams p, const __grid_constant__ R2Table t,
               const float* __restrict__ xyz, uint32_t n, const char* __restrict__ base, size_t stride, uint32_t nslice) {
    __shared__ float tab[kNR];
    extern __shared__ uint32_t cnt_all[];  // [warp][halo][shell]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t* cnt = cnt_all + warp * kDirectHalos * p.nrads;
    for (int i = threadIdx.x; i < p.pad; i += blockDim.x) tab[i] = t.v[i];
    for (int i = lane; i < kDirectHalos * p.nrads; i += 32) cnt[i] = 0u;
    __syncthreads();
    const uint32_t item = blockIdx.x * kDirectWarps + (uint32_t)warp;
    const uint32_t h0 = item / nslice * kDirectHalos, slice = item % nslice;
    if (h0 >= p.nhalos) return;
    float cx[kDirectHalos], cy[kDirectHalos], cz[kDirectHalos];
    uint32_t F[kDirectHalos], anyF = 0u;
#pragma unroll
    for (int k = 0; k < kDirectHalos; ++k) {
        cx[k] = cy[k] = cz[k] = NAN;  // no halo: no distance passes
        F[k] = 0u;
        if (h0 + k >= p.nhalos) continue;
        const float* hp = reinterpret_cast<const float*>(base + (uint64_t)(h0 + k) * stride);
        cx[k] = hp[0];
        cy[k] = hp[1];
        cz[k] = hp[2];
        if (p.periodic)
            F[k] = ((__fsub_rn(cx[k], p.half) < kBoxLow) | (__fadd_rn(cx[k], p.half) > kBoxUpp) ? 1u : 0u) |
                   ((__fsub_rn(cy[k], p.half) < kBoxLow) | (__fadd_rn(cy[k], p.half) > kBoxUpp) ? 2u : 0u) |
                   ((__fsub_rn(cz[k], p.half) < kBoxLow) | (__fadd_rn(cz[k], p.half) > kBoxUpp) ? 4u : 0u);
        anyF |= F[k];
    }
    auto literal = [&](float x, float y, float z, const float4& v, bool live, int k) {
        count::Image im;
        im.cx = x;
        im.cy = y;
        im.cz = z;
        im.lox = __fsub_rn(x, p.half);
        im.hix = __fadd_rn(x, p.half);
        im.loy = __fsub_rn(y, p.half);
        im.hiy = __fadd_rn(y, p.half);
        im.loz = __fsub_rn(z, p.half);
        im.hiz = __fadd_rn(z, p.half);
        count::test_candidate<BIN, false>(p, im, v, live, cnt + k * p.nrads, tab, nullptr);
    };
    auto image = [&](float c) {  // min_oob takes precedence over max_oob on an axis (MultiRangeCount.c:38-43)
        return __fsub_rn(c, p.half) < kBoxLow ? __fadd_rn(c, kBoxUpp) : __fsub_rn(c, kBoxUpp);
    };
#pragma unroll 2
    for (uint32_t j0 = slice * 32u; j0 < n; j0 += nslice * 32u) {
        const uint32_t j = j0 + (uint32_t)lane;
        const bool live = j < n;
        float4 v = make_float4(NAN, 0.f, 0.f, 0.f);
        if (live) v = make_float4(xyz[3 * (uint64_t)j], xyz[3 * (uint64_t)j + 1], xyz[3 * (uint64_t)j + 2], 0.f);
#pragma unroll
        for (int k = 0; k < kDirectHalos; ++k) {
            const float dx = __fsub_rn(v.x, cx[k]), dy = __fsub_rn(v.y, cy[k]), dz = __fsub_rn(v.z, cz[k]);
            const float dist = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
            if (BIN == count::BIN_FIRST_MATCH || dist < p.r2max) literal(cx[k], cy[k], cz[k], v, live, k);
        }
        if (anyF) {
#pragma unroll
            for (int k = 0; k < kDirectHalos; ++k)
                for (uint32_t S = F[k]; S; S = (S - 1u) & F[k])
                    literal((S & 1u) ? image(cx[k]) : cx[k], (S & 2u) ? image(cy[k]) : cy[k],
                            (S & 4u) ? image(cz[k]) : cz[k], v, live, k);
        }
    }
    __syncwarp();
    for (int i = lane; i < kDirectHalos * p.nrads; i += 32)
        if (cnt[i]) atomicAdd(p.counts + (uint64_t)h0 * (uint64_t)p.nrads + (uint64_t)i, cnt[i]);
}

}  // namespace
}  // namespace sjcs

using namespace sjcs;

extern "C" int sjcs_count_noalloc(const float* d_xyz, uint64_t n, const float* d_halo_xyz, size_t stride_bytes,
                                  uint64_t nhalos, const float* r2, int nrads, int flags, uint32_t* d_counts,
                                  void* stream) {
    if (n > kNP)
        return fail(SJCS_ERR_INVALID, "sjcs_count_noalloc: %llu particles exceed its limit of %llu",
                    (unsigned long long)n, (unsigned long long)kNP);
    if (nhalos > kNH)
        return fail(SJCS_ERR_INVALID, "sjcs_count_noalloc: %llu halos exceed its limit of %llu",
                    (unsigned long long)nhalos, (unsigned long long)kNH);
    if (nrads < 1 || nrads > kNR)
        return fail(SJCS_ERR_INVALID, "sjcs_count_noalloc: %d shells outside its limit of 1..%d", nrads, kNR);
    if (!r2) return fail(SJCS_ERR_INVALID, "sjcs_count_noalloc: r2 is NULL");
    if ((n && !d_xyz) || (nhalos && (!d_halo_xyz || !d_counts)))
        return fail(SJCS_ERR_INVALID, "sjcs_count_noalloc: NULL input or output pointer");
    if (stride_bytes < 3 * sizeof(float) || stride_bytes % sizeof(float))
        return fail(SJCS_ERR_INVALID, "sjcs_count_noalloc: stride_bytes must be a multiple of 4 and >= 12");
    if (flags & ~SJCS_QUERY_PERIODIC) return fail(SJCS_ERR_INVALID, "sjcs_count_noalloc: unknown flags 0x%x", flags);
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    unsigned char* base = nullptr;
    int rc = scratch_address(&base);
    if (rc) return rc;

    // radius table, as sjcs_query_create builds it (binary-search binning)
    Tables tab;
    int pad = 1;
    while (pad < nrads) pad <<= 1;
    bool mono = true;
    for (int i = 0; i < pad; ++i) tab.r2.v[i] = i < nrads ? r2[i] : INFINITY;
    for (int i = 0; i < nrads; ++i) {
        if (std::isnan(r2[i])) mono = false;
        if (i + 1 < nrads && !(r2[i] <= r2[i + 1])) mono = false;
    }
    const float R = (float)std::sqrt((double)r2[nrads - 1]);
    const float half = (flags & SJCS_QUERY_PERIODIC) ? R : r2[nrads - 1];
    if (n == 0 || nhalos == 0) return SJCS_OK;

    sjcs_ctx c;
    c.magic = kCtxMagic;
    SJCS_CUDA_TRY(cudaGetDevice(&c.device));
    SJCS_CUDA_TRY(cudaDeviceGetAttribute(&c.num_sms, cudaDevAttrMultiProcessorCount, c.device));

    if (n * nhalos <= kDirectPairs) {
        count::CountParams p{};
        p.nhalos = nhalos;
        p.nrads = nrads;
        p.pad = pad;
        p.half = half;
        p.r2max = r2[nrads - 1];
        p.periodic = (flags & SJCS_QUERY_PERIODIC) ? 1 : 0;
        p.counts = d_counts;
        // slices: enough warps for every SM, at least 4 runs of 32 particles each
        const uint64_t runs = (n + 31) / 32, warps = (uint64_t)c.num_sms * 32;
        const uint64_t groups = (nhalos + kDirectHalos - 1) / kDirectHalos;
        const uint32_t nslice = (uint32_t)std::max<uint64_t>(1, std::min((runs + 3) / 4, (warps + groups - 1) / groups));
        const unsigned blocks = (unsigned)((groups * nslice + kDirectWarps - 1) / kDirectWarps);
        auto kern = mono ? k_count_direct<count::BIN_BSEARCH> : k_count_direct<count::BIN_FIRST_MATCH>;
        kern<<<blocks, kDirectWarps * 32, (size_t)kDirectWarps * kDirectHalos * nrads * sizeof(uint32_t), s>>>(
            p, tab.r2, d_xyz, (uint32_t)n, reinterpret_cast<const char*>(d_halo_xyz), stride_bytes, nslice);
        SJCS_LAUNCH_CHECK();
        return SJCS_OK;
    }

    // objects that only point at the scratch
    sjcs_query q{};
    q.nhalos = nhalos;
    q.nrads = nrads;
    q.flags = flags;
    q.pad = pad;
    q.monotone = mono;
    q.r2max = r2[nrads - 1];
    q.R = R;
    q.half = half;
    q.halos = reinterpret_cast<float4*>(base + kOffHalos);
    q.counts = d_counts;
    q.d_r2 = reinterpret_cast<float*>(base + kOffR2);
    q.d_lut = nullptr;
    q.nlut = 0;
    std::vector<uint32_t> slots;
    if (mono) build_lane_table(r2, nrads, half, &slots, &q.lane);
    if (slots.size() > (size_t)kMaxTable) q.lane = {};
    std::copy(slots.begin(), slots.begin() + q.lane.nslots, tab.slots);
    q.lane.slots = reinterpret_cast<uint32_t*>(base + kOffSlots);
    LaneScratch list{};
    list.ctl = reinterpret_cast<uint32_t*>(base + kOffCtl);
    list.list = reinterpret_cast<uint2*>(base + kOffList);
    list.cap = kListItems;

    // the grid index, in the scratch array
    GridGeom g = auto_grid(n, std::isfinite(R) ? R : 0.0f, nullptr);
    while (g.ncells > kNC) {
        int G[3] = {std::max(1, g.G[0] * 7 / 8), std::max(1, g.G[1] * 7 / 8), std::max(1, g.G[2] * 7 / 8)};
        for (int a = 0; a < 3; ++a) {
            g.G[a] = G[a];
            g.inv_h[a] = (float)G[a] / 1000.0f;
        }
        g.ncells = (uint64_t)G[0] * G[1] * G[2];
    }
    GridBuildBuffers b{};
    b.pts = reinterpret_cast<float4*>(base + kOffPts);
    b.cell_start = reinterpret_cast<uint32_t*>(base + kOffCells);
    b.tmp = reinterpret_cast<float4*>(base + kOffTmp);
    b.top = reinterpret_cast<uint32_t*>(base + kOffTop);
    b.cursors = reinterpret_cast<uint32_t*>(base + kOffCursors);
    b.dense = reinterpret_cast<uint32_t*>(base + kOffDense);
    k_noalloc_prep<<<(unsigned)((nhalos + 255) / 256), 256, 0, s>>>(
        tab, pad, q.lane.nslots, reinterpret_cast<const char*>(d_halo_xyz), stride_bytes, nhalos, q.d_r2, q.lane.slots,
        b.top, list.ctl, q.halos);
    SJCS_LAUNCH_CHECK();
    rc = build_grid_into(c.num_sms, d_xyz, n, g, b, s);
    if (rc) return rc;

    sjcs_index idx{};
    idx.n = n;
    idx.geom = g;
    idx.pts = b.pts;
    idx.cell_start = b.cell_start;
    return launch_shell_count_noalloc(&c, &q, &idx, list, s);
}
