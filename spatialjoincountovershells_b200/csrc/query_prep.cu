// Halo preparation: order the halos along a coarse Morton curve so that the
// warps resident on an SM search neighbouring halos and share particle lines
// in L1/L2.  The order changes nothing in the counts (each halo's counts go
// back to its own row); the reference walks halos in file order in chunks of
// 100 (threadJoin, src/astr_rcount/main.c:802-823).
//
// The order only has to bring neighbours together, so it is a counting sort
// by Morton bucket with no order inside a bucket: one pass takes each halo's
// rank in its bucket from an atomic counter, a scan starts the buckets, one
// pass writes (x, y, z, index).  Bound by the scattered 16-byte writes.  A
// full 30-bit radix sort (four stable passes over 20-byte records, 20
// launches) bought the counts nothing.
#include "radix_sort.cuh"
#include "sjcs_internal.cuh"

namespace sjcs {
namespace {

__device__ __forceinline__ float3 load_halo(const char* base, size_t stride, uint64_t i) {
    const float* p = reinterpret_cast<const float*>(base + i * stride);
    return make_float3(p[0], p[1], p[2]);
}

// Morton bucket of 2^b cells per axis (b <= 10).
__device__ __forceinline__ uint32_t bucket_of(const float3 h, int b) { return morton30(h.x, h.y, h.z) >> (30 - 3 * b); }

__global__ void __launch_bounds__(256) k_halo_rank(const char* __restrict__ base, size_t stride, uint64_t n, int b,
                                                   uint32_t* __restrict__ count, uint32_t* __restrict__ rank) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < n;
    const uint32_t k = live ? bucket_of(load_halo(base, stride, i), b) : 0xffffffffu;
    // one atomic per bucket and warp, so that halos crowded into one bucket do
    // not queue up one by one
    const uint32_t peers = __match_any_sync(0xffffffffu, k);
    const int lane = threadIdx.x & 31, first = __ffs(peers) - 1;
    uint32_t at = 0;
    if (live && lane == first) at = atomicAdd(count + k, (uint32_t)__popc(peers));
    at = __shfl_sync(0xffffffffu, at, first);
    if (live) rank[i] = at + (uint32_t)__popc(peers & lanemask_lt());
}

__global__ void __launch_bounds__(256) k_halo_place(const char* __restrict__ base, size_t stride, uint64_t n, int b,
                                                    const uint32_t* __restrict__ start,
                                                    const uint32_t* __restrict__ rank, float4* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float3 h = load_halo(base, stride, i);
    const uint64_t o = (uint64_t)start[bucket_of(h, b)] + rank[i];
    if (o < n) out[o] = make_float4(h.x, h.y, h.z, __uint_as_float((uint32_t)i));  // in range unless the halos changed
}

__global__ void __launch_bounds__(256) k_halo_pack(const char* __restrict__ base, size_t stride, uint64_t n,
                                                   float4* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float3 h = load_halo(base, stride, i);
    out[i] = make_float4(h.x, h.y, h.z, __uint_as_float((uint32_t)i));
}

}  // namespace

int sort_halos(sjcs_ctx* ctx, const float* d_halo_xyz, size_t stride_bytes, uint64_t nhalos,
               float4* out, cudaStream_t s) {
    (void)ctx;
    if (nhalos == 0) return SJCS_OK;
    const char* base = reinterpret_cast<const char*>(d_halo_xyz);
    const unsigned blocks = (unsigned)((nhalos + 255) / 256);
    // Few halos lie too far apart to share particle lines: caller's order.
    if (nhalos <= 4096) {
        k_halo_pack<<<blocks, 256, 0, s>>>(base, stride_bytes, nhalos, out);
        SJCS_LAUNCH_CHECK();
        return SJCS_OK;
    }
    // 4096 to 2^21 buckets: 2 to 16 halos each, fewer below 8192 halos and more
    // above 3.4e7 (coarser buckets: the count of 1e7 halos on three files of 1e8,
    // 4.8 a bucket, took 14.0 instead of 13.0 ms; finer ones gained nothing)
    int b = 4;
    while (b < 7 && (1ull << (3 * b)) < nhalos / 16) ++b;
    const uint64_t nb = 1ull << (3 * b);
    StreamScratch scr(s);
    uint32_t *count = nullptr, *rank = nullptr;
    SJCS_CUDA_TRY(scr.alloc(&count, nb * sizeof(uint32_t)));
    SJCS_CUDA_TRY(scr.alloc(&rank, nhalos * sizeof(uint32_t)));
    SJCS_CUDA_TRY(cudaMemsetAsync(count, 0, nb * sizeof(uint32_t), s));
    k_halo_rank<<<blocks, 256, 0, s>>>(base, stride_bytes, nhalos, b, count, rank);
    SJCS_LAUNCH_CHECK();
    const int rc = exclusive_scan_u32(count, nb, s);
    if (rc) return rc;
    k_halo_place<<<blocks, 256, 0, s>>>(base, stride_bytes, nhalos, b, count, rank, out);
    SJCS_LAUNCH_CHECK();
    return SJCS_OK;
}

}  // namespace sjcs
