// Plain (grid) index build for one particle file.
//
// Replaces the STR bulk load of the reference (MakeTreeWithSameThreadPoolArraySTR,
// src/objects/ArraySTR/Build.c:845-963: per level, LSD radix sorts on the
// y, x, z centres, gather, pack 10 children per parent MBR).  The counts the
// reference produces do not depend on the tree shape -- a leaf is reached iff
// its point lies inside the query box, because every parent MBR is the exact
// hull of its children (adjustMbrArraySTRNode, src/objects/ArraySTR/Node.c:10-58)
// -- so any index that returns a superset of the in-box points gives the same
// counts.  Here the index is a uniform cell grid.  Cell keys of up to 30 bits
// (every automatic grid) are built by the partition build further down; wider
// keys by a stable LSD radix sort:
//   pass 0   key = cell of (x,y,z) and payload = (x,y,z), read from the AoS input
//            (staged in shared memory a tile at a time when 16-byte aligned)
//   passes   stable LSD radix sort of (key, payload), 8 bits per pass
//   last     writes the sorted particles as float4 and the sorted keys
//   offsets  cell_start[c] = first sorted slot of cell c (boundary fill)
#include <algorithm>
#include <cmath>

#include "morton.cuh"
#include "radix_sort.cuh"
#include "sjcs_internal.cuh"

namespace sjcs {
namespace {

struct KeysFromParticles {
    const float* __restrict__ xyz;
    GridGeom g;
    __device__ __forceinline__ uint32_t key_of(float x, float y, float z) const { return cell_key(g, x, y, z); }
    __device__ __forceinline__ uint32_t operator()(uint64_t i) const {
        return key_of(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]);
    }
};
struct PayFromParticles {
    const float* __restrict__ xyz;
    __device__ __forceinline__ uint4 operator()(uint64_t i) const {
        return make_uint4(__float_as_uint(xyz[3 * i]), __float_as_uint(xyz[3 * i + 1]),
                          __float_as_uint(xyz[3 * i + 2]), 0u);
    }
};
// Last pass: sorted key (for the offsets) and the particle as float4.
struct SinkParticles {
    uint32_t* __restrict__ keys;
    uint4* __restrict__ pts;
    __device__ __forceinline__ void operator()(uint32_t g, uint32_t k, const uint4& v) const {
        keys[g] = k;
        pts[g] = v;
    }
};

struct Gap {
    uint32_t lo, hi, val;  // cells [lo, hi] start at slot val
};
constexpr uint32_t kGapInline = 64;

// cell_start[c] = i for every cell c in [lo, hi] (lo > hi: nothing); runs
// longer than kGapInline go to the gap list.
__device__ __forceinline__ void fill_cells(uint64_t lo, uint64_t hi, uint32_t i, uint32_t* __restrict__ cs,
                                           Gap* __restrict__ gaps, uint32_t* __restrict__ ngaps,
                                           uint32_t max_gaps) {
    if (lo > hi) return;
    const uint64_t cnt = hi - lo + 1;
    const uint64_t inl = cnt < kGapInline ? cnt : kGapInline;
    for (uint64_t c = 0; c < inl; ++c) cs[lo + c] = i;
    if (cnt > kGapInline) {
        const uint32_t slot = atomicAdd(ngaps, 1u);
        if (slot < max_gaps) {
            gaps[slot] = Gap{(uint32_t)(lo + kGapInline), (uint32_t)hi, i};
        } else {
            for (uint64_t c = lo + kGapInline; c <= hi; ++c) cs[c] = i;
        }
    }
}

// cell_start[c] = i for every cell c in (key[i-1], key[i]] (key[-1] = -1,
// key[n] = ncells), so empty cells point at the next occupied slot and
// cell_start[ncells] = n.  Thread t takes boundaries i = 4t .. 4t+3, reading
// their keys with one 16-byte load when the key array is 16-byte aligned.
// Long runs of empty cells go to a gap list that a second kernel fills
// cooperatively.
__global__ void k_cell_start(const uint32_t* __restrict__ keys, uint64_t n, uint64_t ncells,
                             uint32_t* __restrict__ cs, Gap* __restrict__ gaps,
                             uint32_t* __restrict__ ngaps, uint32_t max_gaps, int vec) {
    const uint64_t i0 = 4 * ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x);
    if (i0 > n) return;
    uint64_t cur[4];
    if (vec && i0 + 4 <= n) {
        const uint4 v = *reinterpret_cast<const uint4*>(keys + i0);
        cur[0] = v.x;
        cur[1] = v.y;
        cur[2] = v.z;
        cur[3] = v.w;
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) cur[j] = (i0 + j < n) ? (uint64_t)keys[i0 + j] : ncells;
    }
    uint64_t lo = (i0 == 0) ? 0ull : (uint64_t)keys[i0 - 1] + 1ull;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint64_t i = i0 + (uint64_t)j;
        if (i > n) break;
        fill_cells(lo, cur[j], (uint32_t)i, cs, gaps, ngaps, max_gaps);
        lo = cur[j] + 1ull;
    }
}

__global__ void k_fill_gaps(const Gap* __restrict__ gaps, const uint32_t* __restrict__ ngaps,
                            uint32_t max_gaps, uint32_t* __restrict__ cs) {
    const uint32_t ng = min(*ngaps, max_gaps);
    for (uint32_t gi = blockIdx.x; gi < ng; gi += gridDim.x) {
        const Gap gp = gaps[gi];
        for (uint64_t c = (uint64_t)gp.lo + threadIdx.x; c <= gp.hi; c += blockDim.x) cs[c] = gp.val;
    }
}

// ---------------------------------------------------------------------------
// Partition build, for cell keys of at most 30 bits.
//
// The counts need each cell's particles together and the cells in key order;
// the order inside a cell is free (a count is a sum).  So the records are
// partitioned most significant digit first, without stable ranking: a block
// places each record of its tile with one shared-memory atomic and reserves
// room per digit with one global cursor atomic, and the last pass
// counting-sorts groups of 4096 cells in shared memory and writes their
// cell-table entries itself:
//   top     counts of the key's top digit (<= 9 bits) over x,y,z, in shared
//           memory; their prefix starts the top buckets
//   pass A  x,y,z -> (x, y, z, key) records by the top digit, and beside them
//           the next digit (16 bits per record)
//   mid     per tile of a top bucket: counts of the next digit in shared
//           memory, added to the segment counts (a segment is 2^sb cells,
//           sb = max(9, key bits - 18) <= 12); their prefix starts the segments
//   pass B  records by the next digit (<= 9 bits) inside each top bucket
//           (keys of more than sb + 9 bits; else the top digit is the segment)
//   cells   per group of 4096 cells (whole segments): cell counts, cell_start
//           of its cells, records written in cell order
// Records are 16 bytes with the cell key in .w, which the count kernel does
// not read.  (12-byte records, keys computed again in every pass, were
// measured slower: a record then leaves as three scattered 4-byte stores.)
constexpr int PB_THREADS = 512;
constexpr int PB_ITEMS = 8;
constexpr uint32_t PB_TILE = PB_THREADS * PB_ITEMS;  // records per block in a partition pass
constexpr int PB_MIN_SEG_BITS = 9;
constexpr int PB_GROUP_BITS = 12;
constexpr uint32_t PB_GROUP_CELLS = 1u << PB_GROUP_BITS;  // cells per block in the last pass
constexpr size_t PB_SMEM = (size_t)PB_TILE * sizeof(float4);  // exchange (pass A: staged x,y,z first)
constexpr size_t PB_STAGE_SMEM = (size_t)PB_TILE * 3 * sizeof(float);  // a tile's x,y,z
constexpr int PB_MAX_KEY_BITS = PB_GROUP_BITS + 18;  // segment + two digits of <= 9 bits

struct PbTile {
    uint32_t bucket, start, len;  // records [start, start + len) of top bucket `bucket`
};

// Exclusive scan over the block (PB_THREADS threads) of one value per thread;
// *total gets the sum.  ws holds PB_THREADS / 32 + 1 words; one call per kernel.
__device__ __forceinline__ uint32_t pb_block_scan(uint32_t v, uint32_t* ws, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) ws[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        constexpr int W = PB_THREADS / 32;
        const uint32_t w = lane < W ? ws[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += t;
        }
        if (lane < W) ws[lane] = wi - w;
        if (lane == W - 1) ws[W] = wi;
    }
    __syncthreads();
    *total = ws[PB_THREADS / 32];
    return incl - v + ws[warp];
}

__device__ __forceinline__ uint32_t pb_key(const float4& r) { return __float_as_uint(r.w); }

// One from counter lk of a group's cells for every lane (none, ~0: lk out of
// range); a warp whose lanes all want the same counter asks for it once.
__device__ __forceinline__ uint32_t pb_take(uint32_t* __restrict__ hist, uint32_t lk) {
    const uint32_t first = __shfl_sync(0xffffffffu, lk, 0);
    if (__all_sync(0xffffffffu, lk == first)) {
        if (first >= PB_GROUP_CELLS) return 0xffffffffu;
        const uint32_t lane = threadIdx.x & 31u;
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&hist[first], 32u);
        return __shfl_sync(0xffffffffu, at, 0) + lane;
    }
    return lk < PB_GROUP_CELLS ? atomicAdd(&hist[lk], 1u) : 0xffffffffu;
}

// Cell key of a particle: the grid's cell number, or the level-L Morton code.
struct GridKey {
    GridGeom g;
    __device__ __forceinline__ uint32_t operator()(float x, float y, float z) const { return cell_key(g, x, y, z); }
};
struct MortonKey {
    float scale;  // 2^L / 1000: the same cells as the top L bits of morton_q
    int G;
    __device__ __forceinline__ uint32_t operator()(float x, float y, float z) const {
        return morton_cell((uint32_t)cell_of(x, scale, G), (uint32_t)cell_of(y, scale, G),
                           (uint32_t)cell_of(z, scale, G));
    }
};

// top_hist[cell >> shift] += 1 for every particle (at most PB_THREADS bins,
// counted in shared memory first).  Block b takes tiles `tiles`*b ..
// (one reduction per bin for all of them); each tile's x,y,z are staged in
// shared memory with coalesced 16-byte copies (cp.async when the array is
// 16-byte aligned) and the keys taken from there.
constexpr uint32_t PB_TOP_TILES = 4;
template <class Key>
__global__ void __launch_bounds__(PB_THREADS)
k_pb_top_hist(const float* __restrict__ xyz, int aligned, uint64_t n, Key key, int shift,
              uint32_t* __restrict__ top_hist, uint32_t tiles) {
    __shared__ uint32_t sh[PB_THREADS];
    extern __shared__ float4 stage4[];
    float* sx = reinterpret_cast<float*>(stage4);
    const int tid = threadIdx.x;
    sh[tid] = 0u;
    for (uint32_t t = 0; t < tiles; ++t) {
        const uint64_t start = ((uint64_t)blockIdx.x * tiles + t) * PB_TILE;
        if (start >= n) break;  // uniform across the block
        const uint64_t rem = n - start;
        const uint32_t len = rem < PB_TILE ? (uint32_t)rem : PB_TILE;
        const float* src = xyz + 3 * start;
        const uint32_t words = 3u * len;
        uint32_t w0 = 0;
        __syncthreads();  // the previous tile's staged words have been read
        if (aligned) {
            const uint32_t chunks = words >> 2;
            for (uint32_t c = (uint32_t)tid; c < chunks; c += PB_THREADS) cp_async16(sx + 4 * c, src + 4 * c);
            w0 = chunks * 4u;
        }
        for (uint32_t w = w0 + (uint32_t)tid; w < words; w += PB_THREADS) sx[w] = src[w];
        cp_async_wait_all();
        __syncthreads();
#pragma unroll
        for (int i = 0; i < PB_ITEMS; ++i) {
            const uint32_t loc = (uint32_t)i * PB_THREADS + (uint32_t)tid;
            if (loc < len) atomicAdd(&sh[key(sx[3 * loc], sx[3 * loc + 1], sx[3 * loc + 2]) >> shift], 1u);
        }
    }
    __syncthreads();
    const uint32_t c = sh[tid];
    if (c) atomicAdd(&top_hist[tid], c);
}

// Tiles of the middle pass: each top bucket's records [top_start[t],
// top_start[t+1]) cut into tiles of at most PB_TILE, so a tile never mixes
// buckets.  Every block computes the buckets' tile offsets (ntop <=
// PB_THREADS) and writes tiles blockIdx.x * PB_THREADS + threadIdx.x.
__global__ void __launch_bounds__(PB_THREADS)
k_pb_tiles(const uint32_t* __restrict__ top_start, uint32_t ntop, PbTile* __restrict__ tiles,
           uint32_t* __restrict__ ntiles) {
    __shared__ uint32_t ws[PB_THREADS / 32 + 1];
    __shared__ uint32_t tend[PB_THREADS];  // inclusive tile prefix: tiles of buckets <= t
    const uint32_t t = threadIdx.x;
    const uint32_t lo = t < ntop ? top_start[t] : 0u, hi = t < ntop ? top_start[t + 1] : 0u;
    const uint32_t nt = (hi - lo + PB_TILE - 1) / PB_TILE;
    uint32_t total;
    const uint32_t base = pb_block_scan(nt, ws, &total);
    tend[t] = base + nt;
    __syncthreads();
    if (blockIdx.x == 0 && t == 0) *ntiles = total;
    const uint32_t i = blockIdx.x * PB_THREADS + t;
    if (i >= total) return;
    // bucket of tile i: the first b with tend[b] > i (it has tiles)
    uint32_t b = 0;
#pragma unroll
    for (uint32_t step = PB_THREADS / 2; step > 0; step >>= 1)
        if (tend[b + step - 1] <= i) b += step;
    const uint32_t b_lo = top_start[b], b_len = top_start[b + 1] - b_lo;
    const uint32_t off = (i - (tend[b] - (b_len + PB_TILE - 1) / PB_TILE)) * PB_TILE;
    tiles[i] = PbTile{b, b_lo + off, min(PB_TILE, b_len - off)};
}

// Segment counts for the middle pass: block i counts the middle digits of
// tiles 8i .. 8i+7 (mid[] as written by pass A) in shared memory and adds
// them to seg_hist[(bucket << bits_mid) + digit] whenever the bucket changes
// and at the end -- a reduction per (bucket run, digit) rather than per
// record.
constexpr uint32_t PB_MID_TILES = 8;
__global__ void __launch_bounds__(PB_THREADS)
k_pb_mid_hist(const uint16_t* __restrict__ mid, const PbTile* __restrict__ tiles,
              const uint32_t* __restrict__ ntiles, int bits_mid, uint64_t nseg, uint32_t* __restrict__ seg_hist) {
    __shared__ uint32_t sh[PB_THREADS];
    const uint32_t nt = *ntiles, t0 = blockIdx.x * PB_MID_TILES;
    if (t0 >= nt) return;
    const uint32_t t1 = min(t0 + PB_MID_TILES, nt);
    // masked: a slot that pass A left unwritten (only if the input changed
    // after the histogram) cannot index out of range
    const uint32_t mask = (1u << bits_mid) - 1u;
    sh[threadIdx.x] = 0u;
    uint32_t bucket = tiles[t0].bucket;
    __syncthreads();
    for (uint32_t t = t0; t < t1; ++t) {
        const PbTile tl = tiles[t];
        if (tl.bucket != bucket) {  // uniform across the block
            __syncthreads();
            const uint32_t c = sh[threadIdx.x];
            const uint64_t sg = ((uint64_t)bucket << bits_mid) + threadIdx.x;
            if (c && sg < nseg) atomicAdd(&seg_hist[sg], c);
            sh[threadIdx.x] = 0u;
            bucket = tl.bucket;
            __syncthreads();
        }
        for (uint32_t j = threadIdx.x; j < tl.len; j += PB_THREADS) atomicAdd(&sh[mid[tl.start + j] & mask], 1u);
    }
    __syncthreads();
    const uint32_t c = sh[threadIdx.x];
    const uint64_t sg = ((uint64_t)bucket << bits_mid) + threadIdx.x;
    if (c && sg < nseg) atomicAdd(&seg_hist[sg], c);
}

// Stage floats [w_src, w_src + words) of `base` (total_words long) in shared
// memory at sx[off ..], off = w_src mod 4: 16-byte cp.async chunks from the
// aligned word at or below w_src when `base` is 16-byte aligned (the chunks
// stay inside the array; words past the last whole chunk load plainly), else
// plain loads (off = 0).  sx holds at least words + 6 floats.  The copies are
// awaited by the caller (cp_async_wait_all, then a block barrier).
__device__ __forceinline__ uint32_t pb_stage(const float* __restrict__ base, int aligned, uint64_t w_src,
                                             uint32_t words, uint64_t total_words, float* sx) {
    const uint32_t tid = threadIdx.x;
    if (!aligned) {
        for (uint32_t w = tid; w < words; w += PB_THREADS) sx[w] = base[w_src + w];
        return 0u;
    }
    const uint64_t a0 = w_src & ~3ull, wend = w_src + words;
    const uint64_t cend = min((wend + 3ull) & ~3ull, total_words & ~3ull);
    const uint32_t chunks = cend > a0 ? (uint32_t)((cend - a0) >> 2) : 0u;
    for (uint32_t c = tid; c < chunks; c += PB_THREADS) cp_async16(sx + 4 * c, base + a0 + 4 * c);
    for (uint64_t w = a0 + 4ull * chunks + tid; w < wend; w += PB_THREADS) sx[w - a0] = base[w];
    return (uint32_t)(w_src - a0);
}

// One partition pass.  kTiles == false: tile blockIdx.x of the caller's
// x,y,z (the first pass; staged in shared memory, keys computed here);
// otherwise tile blockIdx.x of `tiles` over 16-byte (x, y, z, key) records.
// A record's digit is (key >> shift) & (2^bits - 1) and its room is reserved
// from cursors[(bucket << cur_shift) + digit].  With `mid` given, the pass
// also writes mid[slot] = (key >> sb) & mid_mask beside every record.
template <bool kTiles, class Key>
__global__ void __launch_bounds__(PB_THREADS, 2)
k_pb_partition(const float* __restrict__ xyz, int xyz_aligned, const float4* __restrict__ in,
               const PbTile* __restrict__ tiles, const uint32_t* __restrict__ ntiles, uint64_t n, Key key,
               int shift, int bits, int cur_shift, uint32_t* __restrict__ cursors, float4* __restrict__ out,
               uint16_t* __restrict__ mid, int sb, uint32_t mid_mask) {
    __shared__ uint32_t cnt[PB_THREADS];  // one bin per thread (digits of <= 9 bits)
    __shared__ uint32_t dstart[PB_THREADS];
    __shared__ uint32_t delta[PB_THREADS];
    __shared__ uint32_t ws[PB_THREADS / 32 + 1];
    extern __shared__ float4 xch[];
    const int tid = threadIdx.x;
    const uint32_t mask = (1u << bits) - 1u;
    uint64_t start;
    uint32_t len, bucket;
    if constexpr (!kTiles) {
        start = (uint64_t)blockIdx.x * PB_TILE;
        const uint64_t rem = n - start;
        len = rem < PB_TILE ? (uint32_t)rem : PB_TILE;
        bucket = 0;
    } else {
        if (blockIdx.x >= *ntiles) return;
        const PbTile tl = tiles[blockIdx.x];
        start = tl.start;
        len = tl.len;
        bucket = tl.bucket;
    }
    cnt[tid] = 0;
    float4 v[PB_ITEMS];
    if constexpr (!kTiles) {
        float* sx = reinterpret_cast<float*>(xch);
        const uint32_t off = pb_stage(xyz, xyz_aligned, 3 * start, 3u * len, 3 * n, sx);
        cp_async_wait_all();
        __syncthreads();
#pragma unroll
        for (int i = 0; i < PB_ITEMS; ++i) {
            const uint32_t loc = (uint32_t)i * PB_THREADS + (uint32_t)tid;
            if (loc < len) {
                const float x = sx[off + 3 * loc], y = sx[off + 3 * loc + 1], z = sx[off + 3 * loc + 2];
                v[i] = make_float4(x, y, z, __uint_as_float(key(x, y, z)));
            }
        }
    } else {
#pragma unroll
        for (int i = 0; i < PB_ITEMS; ++i) {
            const uint32_t loc = (uint32_t)i * PB_THREADS + (uint32_t)tid;
            if (loc < len) v[i] = in[start + loc];
        }
        __syncthreads();
    }
    uint32_t r[PB_ITEMS];
#pragma unroll
    for (int i = 0; i < PB_ITEMS; ++i) {
        const uint32_t loc = (uint32_t)i * PB_THREADS + (uint32_t)tid;
        if (loc < len) r[i] = atomicAdd(&cnt[(pb_key(v[i]) >> shift) & mask], 1u);
    }
    __syncthreads();  // ranks done; the staged x,y,z are no longer read
    const uint32_t c = cnt[tid];
    uint32_t gb = 0, total;
    if (c) gb = atomicAdd(&cursors[((uint64_t)bucket << cur_shift) + (uint64_t)tid], c);
    const uint32_t ds = pb_block_scan(c, ws, &total);
    dstart[tid] = ds;
    delta[tid] = gb - ds;  // slot of the record at tile position j of this digit: delta + j
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PB_ITEMS; ++i) {
        const uint32_t loc = (uint32_t)i * PB_THREADS + (uint32_t)tid;
        if (loc < len) xch[dstart[(pb_key(v[i]) >> shift) & mask] + r[i]] = v[i];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < PB_ITEMS; ++k) {
        const uint32_t j = (uint32_t)k * PB_THREADS + (uint32_t)tid;
        if (j < len) {
            const float4 w = xch[j];
            const uint32_t o = delta[(pb_key(w) >> shift) & mask] + j;
            if (o < n) {  // in range unless the input changed after the histogram
                out[o] = w;
                if (mid) mid[o] = (uint16_t)((pb_key(w) >> sb) & mid_mask);
            }
        }
    }
}

// Groups of the last pass with so many records that one block would be busy
// with them long after the others are listed and shared by all blocks.  A block
// moves about one record a nanosecond and all of them 130 (5e6 equal particles
// took 5.2 ms and take 0.19; 2e7, half of them in a clump of sigma 2, 9.6 and
// 0.71 ms by Morton cells), so a group counts as dense from about n / 100 on,
// and 32768 more for the two passes (20 to 50 us; 2e6 clustered by Morton cells:
// 101 us, 148 with groups from n / 128 on).
struct PbDense {
    uint32_t* n;      // groups listed (zeroed)
    uint32_t* group;  // [pb_dense_slots]
    uint32_t* done;   // [pb_dense_slots] pieces counted
    uint32_t* cur;    // [pb_dense_slots][PB_GROUP_CELLS] counts, then where the next record goes
};
// Records of a piece.  Small sets need the pieces (a clump of 131072 87 us by
// four tiles, 56 by one), a large one with many dense groups fewer counters to
// clear and add up (5e7 clustered, R = 20 by Morton cells: 1.32 ms, 2.0 by one).
__host__ __device__ constexpr uint32_t pb_piece_len(uint64_t n) { return n < (1u << 22) ? PB_TILE : 4 * PB_TILE; }

// Records from which on a group is dense, and how many groups can be.
__host__ __device__ constexpr uint32_t pb_dense(uint64_t n) {
    return 8 * PB_TILE + (uint32_t)(n / 100);
}
__host__ __device__ constexpr uint32_t pb_dense_slots(uint64_t n) { return (uint32_t)(n / pb_dense(n)); }
// Words of PbDense for n particles, without the count.
constexpr uint64_t pb_dense_words(uint64_t n) { return (uint64_t)pb_dense_slots(n) * (PB_GROUP_CELLS + 2); }
PbDense pb_dense_at(uint32_t* n, uint32_t* words, uint64_t particles) {
    const uint32_t k = pb_dense_slots(particles);
    return {n, words, words + k, words + 2 * (uint64_t)k};
}

// Last pass: block b counting-sorts the records of cells [4096 b, 4096 b +
// 4096) (whole segments of 2^sb cells, contiguous after the partition passes)
// and writes cell_start for those of its cells that are <= ncells.  A group
// of at most PB_TILE records goes through shared memory; a larger one is read
// twice (counts, then placement) and written in place, or left to the passes
// over dense groups.
__global__ void __launch_bounds__(PB_THREADS, 2)
k_pb_cells(const float4* __restrict__ in, const uint32_t* __restrict__ seg_start, uint64_t nseg, int sb,
           uint64_t ncells, uint32_t* __restrict__ cs, float4* __restrict__ out, PbDense dense, uint32_t slots,
           uint32_t limit) {
    __shared__ __align__(16) uint32_t hist[PB_GROUP_CELLS];
    __shared__ uint32_t ws[PB_THREADS / 32 + 1];
    extern __shared__ float4 xch[];
    static_assert(PB_GROUP_CELLS == 8 * PB_THREADS, "a thread scans 8 cells");
    const int tid = threadIdx.x;
    const uint64_t cell0 = (uint64_t)blockIdx.x * PB_GROUP_CELLS;
    const uint64_t seg0 = cell0 >> sb;
    const uint64_t seg1 = min(seg0 + (PB_GROUP_CELLS >> sb), nseg);
    const uint32_t lo = seg_start[seg0], cnt = seg_start[seg1] - lo;
    const uint32_t c0 = (uint32_t)cell0;
    if (cnt > limit && slots) {
        if (tid == 0) ws[0] = atomicAdd(dense.n, 1u);
        __syncthreads();
        const uint32_t slot = ws[0];
        if (slot < slots) {
            if (tid == 0) {
                dense.group[slot] = blockIdx.x;
                dense.done[slot] = 0u;
            }
            for (uint32_t c = (uint32_t)tid; c < PB_GROUP_CELLS; c += PB_THREADS)
                dense.cur[(uint64_t)slot * PB_GROUP_CELLS + c] = 0u;
            return;
        }
    }
    uint4* h4 = reinterpret_cast<uint4*>(hist);
    h4[2 * tid] = make_uint4(0u, 0u, 0u, 0u);
    h4[2 * tid + 1] = make_uint4(0u, 0u, 0u, 0u);
    const bool fits = cnt <= PB_TILE;
    float4 v[PB_ITEMS];
    uint32_t r[PB_ITEMS];
    if (fits) {
#pragma unroll
        for (int i = 0; i < PB_ITEMS; ++i) {
            const uint32_t j = (uint32_t)i * PB_THREADS + (uint32_t)tid;
            if (j < cnt) v[i] = in[lo + j];
        }
    }
    __syncthreads();
    if (fits) {
#pragma unroll
        for (int i = 0; i < PB_ITEMS; ++i) {
            const uint32_t j = (uint32_t)i * PB_THREADS + (uint32_t)tid;
            r[i] = 0xffffffffu;
            if (j < cnt) {
                // a key outside the group (only if the input changed after the
                // histogram) is dropped rather than counted out of range
                const uint32_t lk = pb_key(v[i]) - c0;
                if (lk < PB_GROUP_CELLS) r[i] = atomicAdd(&hist[lk], 1u);
            }
        }
    } else {
        for (uint32_t j = (uint32_t)tid; j < cnt; j += PB_THREADS) {
            const uint32_t lk = pb_key(in[lo + j]) - c0;
            if (lk < PB_GROUP_CELLS) atomicAdd(&hist[lk], 1u);
        }
    }
    __syncthreads();
    // exclusive scan of the 4096 cell counts; thread t owns cells 8t .. 8t+7
    const uint4 a = h4[2 * tid], b = h4[2 * tid + 1];
    uint32_t e[8];
    e[0] = 0u;
    e[1] = a.x;
    e[2] = e[1] + a.y;
    e[3] = e[2] + a.z;
    e[4] = e[3] + a.w;
    e[5] = e[4] + b.x;
    e[6] = e[5] + b.y;
    e[7] = e[6] + b.z;
    uint32_t total;
    const uint32_t base = pb_block_scan(e[7] + b.w, ws, &total);
#pragma unroll
    for (int k = 0; k < 8; ++k) e[k] += base;
    h4[2 * tid] = make_uint4(e[0], e[1], e[2], e[3]);
    h4[2 * tid + 1] = make_uint4(e[4], e[5], e[6], e[7]);
    const uint64_t c8 = cell0 + 8u * (uint64_t)tid;
    if (c8 + 7 <= ncells) {
        uint4* dst = reinterpret_cast<uint4*>(cs + c8);
        dst[0] = make_uint4(lo + e[0], lo + e[1], lo + e[2], lo + e[3]);
        dst[1] = make_uint4(lo + e[4], lo + e[5], lo + e[6], lo + e[7]);
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (c8 + k <= ncells) cs[c8 + k] = lo + e[k];
    }
    __syncthreads();
    if (fits) {
#pragma unroll
        for (int i = 0; i < PB_ITEMS; ++i) {
            if (r[i] != 0xffffffffu) xch[hist[pb_key(v[i]) - c0] + r[i]] = v[i];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < PB_ITEMS; ++k) {
            const uint32_t j = (uint32_t)k * PB_THREADS + (uint32_t)tid;
            if (j < cnt) out[lo + j] = xch[j];
        }
    } else {
        for (uint32_t j = (uint32_t)tid; j < cnt; j += PB_THREADS) {
            const float4 w = in[lo + j];
            const uint32_t lk = pb_key(w) - c0;
            if (lk < PB_GROUP_CELLS) out[lo + atomicAdd(&hist[lk], 1u)] = w;
        }
    }
}

// A piece of a dense group: its place in the list, records and first cell.
struct PbPiece {
    uint32_t slot, lo, cnt, c0, pieces, start, len;
};
// Piece `at` of all listed groups; false: there are fewer.
__device__ __forceinline__ bool pb_piece(const PbDense& dense, uint32_t nd, const uint32_t* __restrict__ seg_start,
                                         uint64_t nseg, int sb, uint32_t piece, uint32_t at,
                                         PbPiece* p) {
    for (uint32_t k = 0; k < nd; ++k) {
        const uint64_t cell0 = (uint64_t)dense.group[k] * PB_GROUP_CELLS, seg0 = cell0 >> sb;
        const uint32_t lo = seg_start[seg0];
        const uint32_t cnt = seg_start[min(seg0 + (PB_GROUP_CELLS >> sb), nseg)] - lo;
        const uint32_t pieces = (cnt + piece - 1u) / piece;
        if (at < pieces) {
            *p = {k, lo, cnt, (uint32_t)cell0, pieces, at * piece, min(piece, cnt - at * piece)};
            return true;
        }
        at -= pieces;
    }
    return false;
}

// Counts per cell of the dense groups, a piece to a block; the last block of a
// group turns them into cell_start and the cursors that begin there.
__global__ void __launch_bounds__(PB_THREADS, 2)
k_pb_dense_count(const float4* __restrict__ in, const uint32_t* __restrict__ seg_start, uint64_t nseg, int sb,
                 uint64_t ncells, uint32_t* __restrict__ cs, PbDense dense, uint32_t slots,
                 uint32_t piece) {
    __shared__ uint32_t hist[PB_GROUP_CELLS];
    __shared__ uint32_t ws[PB_THREADS / 32 + 1];
    __shared__ uint32_t last;
    const int tid = threadIdx.x;
    cudaGridDependencySynchronize();
    const uint32_t nd = min(*dense.n, slots);
    PbPiece p;
    for (uint32_t at = blockIdx.x; nd && pb_piece(dense, nd, seg_start, nseg, sb, piece, at, &p); at += gridDim.x) {
        uint32_t* cur = dense.cur + (uint64_t)p.slot * PB_GROUP_CELLS;
        for (uint32_t c = (uint32_t)tid; c < PB_GROUP_CELLS; c += PB_THREADS) hist[c] = 0u;
        __syncthreads();
        for (uint32_t j0 = 0; j0 < p.len; j0 += PB_TILE) {
            uint32_t lk[PB_ITEMS];
#pragma unroll
            for (int i = 0; i < PB_ITEMS; ++i) {
                const uint32_t j = j0 + (uint32_t)i * PB_THREADS + (uint32_t)tid;
                lk[i] = j < p.len ? pb_key(in[p.lo + p.start + j]) - p.c0 : 0xffffffffu;
            }
#pragma unroll
            for (int i = 0; i < PB_ITEMS; ++i) pb_take(hist, lk[i]);
        }
        __syncthreads();
        for (uint32_t c = (uint32_t)tid; c < PB_GROUP_CELLS; c += PB_THREADS)
            if (hist[c]) atomicAdd(cur + c, hist[c]);
        __threadfence();
        __syncthreads();
        if (tid == 0) last = atomicAdd(dense.done + p.slot, 1u) == p.pieces - 1u ? 1u : 0u;
        __syncthreads();
        if (!last) continue;  // the whole block
        __threadfence();
        uint32_t e[8], sum = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            e[k] = sum;
            sum += __ldcg(cur + 8u * (uint32_t)tid + k);
        }
        uint32_t total;
        const uint32_t base = pb_block_scan(sum, ws, &total) + p.lo;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t c = 8u * (uint32_t)tid + k;
            cur[c] = base + e[k];
            if ((uint64_t)p.c0 + c <= ncells) cs[p.c0 + c] = base + e[k];
        }
        __syncthreads();
    }
}

// The records of the dense groups to their cells: a tile's ranks from counters
// in shared memory, room for each of its cells from the group's cursors.
__global__ void __launch_bounds__(PB_THREADS, 2)
k_pb_dense_place(const float4* __restrict__ in, const uint32_t* __restrict__ seg_start, uint64_t nseg, int sb,
                 float4* __restrict__ out, PbDense dense, uint32_t slots, uint32_t piece) {
    __shared__ uint32_t hist[PB_GROUP_CELLS];
    const int tid = threadIdx.x;
    cudaGridDependencySynchronize();
    const uint32_t nd = min(*dense.n, slots);
    PbPiece p;
    for (uint32_t at = blockIdx.x; nd && pb_piece(dense, nd, seg_start, nseg, sb, piece, at, &p); at += gridDim.x) {
        uint32_t* cur = dense.cur + (uint64_t)p.slot * PB_GROUP_CELLS;
        for (uint32_t j0 = 0; j0 < p.len; j0 += PB_TILE) {
            for (uint32_t c = (uint32_t)tid; c < PB_GROUP_CELLS; c += PB_THREADS) hist[c] = 0u;
            __syncthreads();
            float4 v[PB_ITEMS];
            uint32_t lk[PB_ITEMS], r[PB_ITEMS];
#pragma unroll
            for (int i = 0; i < PB_ITEMS; ++i) {
                const uint32_t j = j0 + (uint32_t)i * PB_THREADS + (uint32_t)tid;
                if (j < p.len) v[i] = in[p.lo + p.start + j];
                lk[i] = j < p.len ? pb_key(v[i]) - p.c0 : 0xffffffffu;
            }
#pragma unroll
            for (int i = 0; i < PB_ITEMS; ++i) r[i] = pb_take(hist, lk[i]);
            __syncthreads();
            for (uint32_t c = (uint32_t)tid; c < PB_GROUP_CELLS; c += PB_THREADS) {
                const uint32_t k = hist[c];
                if (k) hist[c] = atomicAdd(cur + c, k);
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < PB_ITEMS; ++i) {
                if (r[i] == 0xffffffffu) continue;
                const uint32_t o = hist[lk[i]] + r[i];
                if (o - p.lo < p.cnt) out[o] = v[i];  // in range unless the input changed after the histogram
            }
            __syncthreads();
        }
    }
}

// The last pass and, where a group may be dense, the passes over those.
int launch_cells(const float4* tmp, const uint32_t* seg, uint64_t nseg, int sb, uint64_t n, uint64_t ncells, uint32_t* cs,
                 float4* pts, const PbDense& dense, int num_sms, cudaStream_t s) {
    const unsigned ngroups = (unsigned)(ncells / PB_GROUP_CELLS + 1);  // the last one holds cell_start[ncells]
    const uint32_t slots = pb_dense_slots(n);
    k_pb_cells<<<ngroups, PB_THREADS, PB_SMEM, s>>>(tmp, seg, nseg, sb, ncells, cs, pts, dense, slots,
                                                    pb_dense(n));
    SJCS_LAUNCH_CHECK();
    if (!slots) return SJCS_OK;
    const uint32_t piece = pb_piece_len(n);
    const unsigned blocks = (unsigned)std::min<uint64_t>(2 * (uint64_t)num_sms, (n + piece - 1) / piece);
    // launched while the kernel before drains: idle, they cost 3 us each without
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(PB_THREADS);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    SJCS_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_pb_dense_count, tmp, seg, nseg, sb, ncells, cs, dense, slots, piece));
    SJCS_LAUNCH_CHECK();
    SJCS_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_pb_dense_place, tmp, seg, nseg, sb, pts, dense, slots, piece));
    SJCS_LAUNCH_CHECK();
    return SJCS_OK;
}

// Segment bits of a key, <= PB_GROUP_BITS.  Keys of up to 21 bits take
// segments wide enough for one digit above them: one partition pass instead
// of two.
int segment_bits(int kb) {
    return kb <= PB_GROUP_BITS + 9 ? std::max(PB_MIN_SEG_BITS, kb - 9) : std::max(PB_MIN_SEG_BITS, kb - 18);
}

template <class Key>
int set_partition_smem() {
    SJCS_CUDA_TRY(cudaFuncSetAttribute(k_pb_top_hist<Key>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)PB_STAGE_SMEM));
    SJCS_CUDA_TRY(cudaFuncSetAttribute(k_pb_partition<true, Key>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)PB_SMEM));
    SJCS_CUDA_TRY(cudaFuncSetAttribute(k_pb_partition<false, Key>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)PB_SMEM));
    SJCS_CUDA_TRY(cudaFuncSetAttribute(k_pb_cells, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PB_SMEM));
    return SJCS_OK;
}

// The partition build into pts (n records) and cs (ncells + 1 entries) by a
// cell key of kb <= 30 bits.
template <class Key>
int build_partitioned(int num_sms, const float* d_xyz, uint64_t n, Key key, int kb, uint64_t ncells, float4* pts,
                      uint32_t* cs, cudaStream_t s) {
    if (n == 0) {
        SJCS_CUDA_TRY(cudaMemsetAsync(cs, 0, (ncells + 1) * sizeof(uint32_t), s));
        return SJCS_OK;
    }
    const int sb = segment_bits(kb);
    const int upper = kb > sb ? kb - sb : 0;  // bits above the segment
    const int bits_mid = upper > 9 ? upper - 9 : 0;
    const int bits_top = upper - bits_mid;
    const uint64_t nseg = (ncells + (1ull << sb) - 1) >> sb;
    const uint32_t ntop = (uint32_t)((nseg + (1ull << bits_mid) - 1) >> bits_mid);
    const uint64_t ntiles_in = (n + PB_TILE - 1) / PB_TILE;
    const uint64_t ntiles_mid = ntiles_in + ntop;  // bound on the middle pass's tiles
    const int aligned = (reinterpret_cast<uintptr_t>(d_xyz) & 15u) == 0;

    StreamScratch scr(s);
    uint32_t *top = nullptr, *cur_top = nullptr, *seg = nullptr, *cur_seg = nullptr, *ntiles = nullptr;
    float4* tmp = nullptr;
    PbTile* tiles = nullptr;
    uint16_t* mid = nullptr;
    // top digit counts and starts (ntop + 1 entries); without a middle pass
    // the top digit is the segment and these are the segment starts too.  The
    // word behind them counts the dense groups, whose room follows.
    SJCS_CUDA_TRY(scr.alloc(&top, ((uint64_t)ntop + 2 + pb_dense_words(n)) * sizeof(uint32_t)));
    SJCS_CUDA_TRY(scr.alloc(&cur_top, ((uint64_t)ntop + 1) * sizeof(uint32_t)));
    SJCS_CUDA_TRY(scr.alloc(&tmp, n * sizeof(float4)));
    if (bits_mid) {
        SJCS_CUDA_TRY(scr.alloc(&seg, (nseg + 1) * sizeof(uint32_t)));
        SJCS_CUDA_TRY(scr.alloc(&cur_seg, (nseg + 1) * sizeof(uint32_t)));
        SJCS_CUDA_TRY(scr.alloc(&tiles, ntiles_mid * sizeof(PbTile)));
        SJCS_CUDA_TRY(scr.alloc(&ntiles, sizeof(uint32_t)));
        SJCS_CUDA_TRY(scr.alloc(&mid, n * sizeof(uint16_t)));
        SJCS_CUDA_TRY(cudaMemsetAsync(seg, 0, (nseg + 1) * sizeof(uint32_t), s));
    } else {
        seg = top;
    }
    const int top_shift = sb + bits_mid;
    int rc = set_partition_smem<Key>();
    if (rc) return rc;
    SJCS_CUDA_TRY(cudaMemsetAsync(top, 0, ((uint64_t)ntop + 2) * sizeof(uint32_t), s));
    // four tiles a block once every SM has blocks enough
    const uint32_t per = ntiles_in >= (uint64_t)num_sms * 4 * PB_TOP_TILES ? PB_TOP_TILES : 1u;
    k_pb_top_hist<Key><<<(unsigned)((ntiles_in + per - 1) / per), PB_THREADS, PB_STAGE_SMEM, s>>>(d_xyz, aligned, n, key,
                                                                                          top_shift, top, per);
    SJCS_LAUNCH_CHECK();
    rc = exclusive_scan_u32(top, (uint64_t)ntop + 1, s, nullptr, cur_top);
    if (rc) return rc;
    // pass A writes pts when a middle pass follows (pts is free until the
    // last pass), else tmp; with a middle pass it also writes the middle digits
    float4* a_out = bits_mid ? pts : tmp;
    const uint32_t mid_mask = (1u << bits_mid) - 1u;
    k_pb_partition<false, Key><<<(unsigned)ntiles_in, PB_THREADS, PB_SMEM, s>>>(
        d_xyz, aligned, nullptr, nullptr, nullptr, n, key, top_shift, bits_top, 0, cur_top, a_out, mid, sb, mid_mask);
    SJCS_LAUNCH_CHECK();
    if (bits_mid) {
        const unsigned tile_blocks = (unsigned)((ntiles_mid + PB_THREADS - 1) / PB_THREADS);
        k_pb_tiles<<<tile_blocks, PB_THREADS, 0, s>>>(top, ntop, tiles, ntiles);
        SJCS_LAUNCH_CHECK();
        k_pb_mid_hist<<<(unsigned)((ntiles_mid + PB_MID_TILES - 1) / PB_MID_TILES), PB_THREADS, 0, s>>>(
            mid, tiles, ntiles, bits_mid, nseg, seg);
        SJCS_LAUNCH_CHECK();
        rc = exclusive_scan_u32(seg, nseg + 1, s, nullptr, cur_seg);
        if (rc) return rc;
        k_pb_partition<true, Key><<<(unsigned)ntiles_mid, PB_THREADS, PB_SMEM, s>>>(
            nullptr, 0, pts, tiles, ntiles, n, key, sb, bits_mid, bits_mid, cur_seg, tmp, nullptr, sb, 0u);
        SJCS_LAUNCH_CHECK();
    }
    return launch_cells(tmp, seg, nseg, sb, n, ncells, cs, pts, pb_dense_at(top + ntop + 1, top + ntop + 2, n), num_sms,
                        s);
}

}  // namespace

int build_grid_into(int num_sms, const float* d_xyz, uint64_t n, const GridGeom& g, const GridBuildBuffers& b,
                    cudaStream_t s) {
    static_assert(pb_dense_words(SJCS_NOALLOC_MAX_PARTICLES) <= kGridDenseWords, "room for the dense groups");
    if (pb_dense_words(n) > kGridDenseWords) return fail(SJCS_ERR_INVALID, "too many particles for the fixed buffers");
    if (n == 0) {
        SJCS_CUDA_TRY(cudaMemsetAsync(b.cell_start, 0, (g.ncells + 1) * sizeof(uint32_t), s));
        return SJCS_OK;
    }
    const int kb = grid_key_bits(g);
    if (kb > kGridMaxDirectBits) return fail(SJCS_ERR_INVALID, "grid of %d key bits needs two partition passes", kb);
    const int sb = segment_bits(kb), bits_top = std::max(0, kb - sb);
    const uint64_t nseg = (g.ncells + (1ull << sb) - 1) >> sb;  // <= 512
    const uint64_t ntiles = (n + PB_TILE - 1) / PB_TILE;
    const int aligned = (reinterpret_cast<uintptr_t>(d_xyz) & 15u) == 0;
    int rc = set_partition_smem<GridKey>();
    if (rc) return rc;
    k_pb_top_hist<GridKey><<<(unsigned)ntiles, PB_THREADS, PB_STAGE_SMEM, s>>>(
        d_xyz, aligned, n, GridKey{g}, sb, b.top, 1u);
    SJCS_LAUNCH_CHECK();
    rc = exclusive_scan_u32(b.top, nseg + 1, s, nullptr, b.cursors);
    if (rc) return rc;
    k_pb_partition<false, GridKey><<<(unsigned)ntiles, PB_THREADS, PB_SMEM, s>>>(d_xyz, aligned, nullptr, nullptr, nullptr, n,
                                                                        GridKey{g},
                                                                        sb, bits_top, 0, b.cursors, b.tmp, nullptr, sb,
                                                                        0u);
    SJCS_LAUNCH_CHECK();
    return launch_cells(b.tmp, b.top, nseg, sb, n, g.ncells, b.cell_start, b.pts, pb_dense_at(b.top + 513, b.dense, n),
                        num_sms, s);
}

GridGeom auto_grid(uint64_t n, float radius_hint, const uint32_t* grid_req) {
    GridGeom g{};
    int G[3];
    if (grid_req && grid_req[0] && grid_req[1] && grid_req[2]) {
        for (int a = 0; a < 3; ++a) G[a] = (int)grid_req[a];
    } else {
        // Rows of cells run along x and are looked up with two offsets, so x
        // can be finer than y/z for free: cells are 2.5x longer in y and z.
        // Target about 1.6 cells per particle, at most 2^28 cells (a 1 GB
        // cell table; keys of up to 30 bits take the partition build), and
        // keep y/z cells >= R/4: a query box then spans at most 9x9 rows.
        // A box spans at most 5x5 rows -- the per-batch row plan -- when
        // y/z cells are >= R/2, so cells go below R/2 only as far as the
        // 2^27-cell size would (the 5x5 plan counts far faster than 6x6
        // boxes without it, for the small gain of finer cells).
        constexpr double kMaxCells = 268435456.0;  // 2^28
        const double want = std::max(1.6 * (double)n, 4096.0);
        double hyz = std::cbrt(2.5e9 / std::min(want, kMaxCells));
        if (radius_hint > 0.0f) {
            const double h27 = std::cbrt(2.5e9 / std::min(want, 134217728.0));
            hyz = std::max(hyz, std::min(0.5 * (double)radius_hint, h27));
            hyz = std::max(hyz, 0.25 * (double)radius_hint);
        }
        for (;;) {
            const double hx = hyz / 2.5;
            G[0] = (int)std::min(std::max(std::ceil(1000.0 / hx), 1.0), 4096.0);
            G[1] = (int)std::min(std::max(std::ceil(1000.0 / hyz), 1.0), 4096.0);
            G[2] = G[1];
            if ((double)G[0] * G[1] * G[2] <= kMaxCells) break;
            hyz *= 1.002;  // rounding up per axis overshot the cap
        }
    }
    for (int a = 0; a < 3; ++a) {
        g.G[a] = G[a];
        g.inv_h[a] = (float)G[a] / 1000.0f;
    }
    g.ncells = (uint64_t)G[0] * G[1] * G[2];
    return g;
}

int grid_key_bits(const GridGeom& g) {
    int key_bits = 1;
    while (key_bits < 32 && (1ull << key_bits) < g.ncells) ++key_bits;
    return key_bits;
}

namespace {
// Buffers of the stable LSD sort (cell keys of more than 30 bits).
struct LsdBuffers {
    float4* pts;       // n sorted particles (output)
    uint32_t* kfinal;  // n sorted keys
    uint32_t *kx, *ky; // n
    uint4 *px, *py;    // n
    uint32_t* hist;    // RS_BINS * ceil(n / 4096)
};

template <class PayOp0>
int sort_particles(const float* d_xyz, uint64_t n, const GridGeom& g, const LsdBuffers& b, PayOp0 pop0, cudaStream_t s) {
    return radix_sort_records(n, grid_key_bits(g), KeysFromParticles{d_xyz, g}, pop0,
                              SinkParticles{b.kfinal, reinterpret_cast<uint4*>(b.pts)}, b.kx, b.px, b.ky, b.py,
                              b.hist, s);
}
}  // namespace

int fill_cell_table(const uint32_t* sorted_cells, uint64_t n, uint64_t ncells, uint32_t* cell_start, void* gaps,
                    uint32_t* ngaps, cudaStream_t s) {
    SJCS_CUDA_TRY(cudaMemsetAsync(ngaps, 0, sizeof(uint32_t), s));
    const uint64_t threads = n / 4 + 1;  // boundaries 0..n, four per thread
    const unsigned blocks = (unsigned)((threads + 255) / 256);
    const int vec = (reinterpret_cast<uintptr_t>(sorted_cells) & 15u) == 0;
    k_cell_start<<<blocks, 256, 0, s>>>(sorted_cells, n, ncells, cell_start, static_cast<Gap*>(gaps), ngaps,
                                        kGridGaps, vec);
    SJCS_LAUNCH_CHECK();
    k_fill_gaps<<<1024, 256, 0, s>>>(static_cast<Gap*>(gaps), ngaps, kGridGaps, cell_start);
    SJCS_LAUNCH_CHECK();
    return SJCS_OK;
}

int build_morton_table(int num_sms, const float* d_xyz, uint64_t n, int level, float4* pts, uint32_t* table,
                       cudaStream_t s) {
    const int G = 1 << level;
    return build_partitioned(num_sms, d_xyz, n, MortonKey{(float)G / 1000.0f, G}, std::max(1, 3 * level), 1ull << (3 * level),
                             pts, table, s);
}

int build_grid_index(sjcs_ctx* ctx, const float* d_xyz, uint64_t n, const GridGeom& g,
                     sjcs_index* idx, cudaStream_t s) {
    idx->geom = g;
    const uint64_t nalloc = n ? n : 1;
    SJCS_CUDA_TRY(cudaMallocAsync(&idx->pts, nalloc * sizeof(float4), s));
    SJCS_CUDA_TRY(cudaMallocAsync(&idx->cell_start, (g.ncells + 1) * sizeof(uint32_t), s));
    if (grid_key_bits(g) <= PB_MAX_KEY_BITS)
        return build_partitioned(ctx->num_sms, d_xyz, n, GridKey{g}, grid_key_bits(g), g.ncells, idx->pts, idx->cell_start, s);

    LsdBuffers b{};
    b.pts = idx->pts;
    const uint64_t ntiles = (n + RS_TILE - 1) / RS_TILE;
    StreamScratch scr(s);  // freed (stream-ordered) on every return path
    void* gaps = nullptr;
    uint32_t* ngaps = nullptr;
    SJCS_CUDA_TRY(scr.alloc(&b.kfinal, nalloc * sizeof(uint32_t)));
    SJCS_CUDA_TRY(scr.alloc(&b.kx, nalloc * sizeof(uint32_t)));  // keys of 31 bits: four passes
    SJCS_CUDA_TRY(scr.alloc(&b.px, nalloc * sizeof(uint4)));
    SJCS_CUDA_TRY(scr.alloc(&b.ky, nalloc * sizeof(uint32_t)));
    SJCS_CUDA_TRY(scr.alloc(&b.py, nalloc * sizeof(uint4)));
    SJCS_CUDA_TRY(scr.alloc(&b.hist, ((uint64_t)RS_BINS * (ntiles ? ntiles : 1)) * sizeof(uint32_t)));
    SJCS_CUDA_TRY(scr.alloc(&gaps, kGridGaps * sizeof(Gap)));
    SJCS_CUDA_TRY(scr.alloc(&ngaps, sizeof(uint32_t)));
    // A 16-byte-aligned particle array is staged tile by tile in the first
    // pass; any other alignment is read particle by particle.
    const bool staged = (reinterpret_cast<uintptr_t>(d_xyz) & 15u) == 0;
    const int rc = staged ? sort_particles(d_xyz, n, g, b, PayFromXyzStaged{d_xyz}, s)
                          : sort_particles(d_xyz, n, g, b, PayFromParticles{d_xyz}, s);
    if (rc) return rc;
    return fill_cell_table(b.kfinal, n, g.ncells, idx->cell_start, gaps, ngaps, s);
}

}  // namespace sjcs
