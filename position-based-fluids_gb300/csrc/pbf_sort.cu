// pbf_sort.cu — stable LSD radix sort of (cell key, particle index) pairs.
//
// The reference sorts with 6 passes of 5 bits over 2048 "virtual processors"
// (radixsort.cl:61-308, src/Simulation.cpp:456-536).  Its result is the
// stable sort of the keys (every key is below 2^30), and that order is the
// contract here: equal keys keep their input order.
//
// Here the keys are < gridBufSize, so only ceil(log2(gridBufSize) / 8)
// passes of 8-bit digits are run (3 at gridBufSize = 2^19).  Each pass is
//   upsweep   : per-tile 256-bin digit histogram -> hist[digit][tile]
//   scan      : per digit, an exclusive scan over the tiles (one block per
//               digit); the downsweep adds the exclusive scan of the digit
//               totals
//   downsweep : per-warp stable ranking with __match_any_sync and per-warp
//               digit counters in shared memory, then the scatter.
// A tile is 8 warps x kRounds rounds of 32 keys: 4096 keys (16 rounds) above
// 2^21 keys, 2048 (8 rounds) above 2^18 and 1024 (4 rounds) below, so that
// smaller sorts still spread over the SMs (at 2^20 keys, 512 tiles sort
// 12 % faster than 256).  Each warp owns consecutive keys taken round by
// round, so (warp, round, lane) order is input order.
//
// A substep whose key range is not much larger than its particle count sorts
// by counting instead (counting_scan_*, cell_scatter, cell_gather): predict
// counts each key's particles and keeps each particle's place of arrival among
// them, one scan over the key range turns the counts into first indices (which
// are the cell table as well), and the particles of a cell, few and in any
// order after the scatter, are put in input order by counting the smaller
// indices among them.

#include <cuda_runtime.h>
#include <cstdint>

#include "pbf_device.cuh"
#include "pbf_internal.h"

namespace pbf {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kSmallSortKeys = 1 << 18;     // at most this many keys: 4-round tiles
constexpr int kMidSortKeys = 1 << 21;       // at most this many keys: 8-round tiles

template <int kRounds>
__global__ void __launch_bounds__(kThreads)
radix_upsweep_kernel(const uint32_t* __restrict__ keys, int n, int shift, int tiles, uint32_t* __restrict__ hist) {
    constexpr int kTile = kThreads * kRounds;
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * kTile;
#pragma unroll 4
    for (int r = 0; r < kRounds; ++r) {
        const size_t idx = base + (size_t)r * kThreads + threadIdx.x;
        if (idx < (size_t)n) atomicAdd(&h[(keys[idx] >> shift) & 0xFFu], 1u);
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

// Per-digit exclusive scan over the tiles: block d scans row d of
// hist[digit][tile] in place and writes the row's total to totals[d].
__global__ void __launch_bounds__(kThreads)
radix_scan_kernel(uint32_t* __restrict__ hist, int tiles, uint32_t* __restrict__ totals) {
    __shared__ uint32_t warpSums[kWarps];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t* row = hist + (size_t)blockIdx.x * tiles;
    uint32_t carry = 0;
    for (int base = 0; base < tiles; base += kThreads) {
        const int k = base + t;
        const uint32_t v = k < tiles ? row[k] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += u;
        }
        if (lane == 31) warpSums[warp] = incl;
        __syncthreads();
        uint32_t before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t ws = warpSums[w];
            before += w < warp ? ws : 0u;
            all += ws;
        }
        if (k < tiles) row[k] = carry + before + incl - v;
        carry += all;
        __syncthreads();
    }
    if (t == 0) totals[blockIdx.x] = carry;
}

template <int kRounds>
__global__ void __launch_bounds__(kThreads)
radix_downsweep_kernel(const uint32_t* __restrict__ keysIn, const uint32_t* __restrict__ permIn,
                       uint32_t* __restrict__ keysOut, uint32_t* __restrict__ permOut, int n, int shift,
                       int tiles, const uint32_t* __restrict__ hist, const uint32_t* __restrict__ totals) {
    constexpr int kTile = kThreads * kRounds;
    constexpr int kWarpKeys = 32 * kRounds;
    __shared__ uint32_t warpCount[kWarps][256];
    __shared__ uint32_t digitBase[256];
    __shared__ uint32_t warpSums[kWarps];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) warpCount[w][t] = 0;
    {   // digitBase[d] = keys of all tiles with a smaller digit (exclusive scan of the totals)
        const uint32_t v = totals[t];
        uint32_t incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += u;
        }
        if (lane == 31) warpSums[warp] = incl;
        __syncthreads();
        uint32_t before = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) before += w < warp ? warpSums[w] : 0u;
        digitBase[t] = before + incl - v;
    }
    __syncthreads();

    const size_t base = (size_t)blockIdx.x * kTile + (size_t)warp * kWarpKeys;
    const unsigned ltMask = (1u << lane) - 1u;
    uint32_t key[kRounds], rank[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const size_t idx = base + (size_t)r * 32 + lane;
        const bool valid = idx < (size_t)n;
        const unsigned active = __ballot_sync(0xFFFFFFFFu, valid);
        uint32_t k = 0, rk = 0, peers = 0, prior = 0;
        if (valid) {
            k = keysIn[idx];
            const uint32_t d = (k >> shift) & 0xFFu;
            peers = __match_any_sync(active, d);
            prior = warpCount[warp][d];
            rk = prior + __popc(peers & ltMask);
        }
        __syncwarp();
        if (valid && (__ffs(peers) - 1) == lane) warpCount[warp][(k >> shift) & 0xFFu] = prior + __popc(peers);
        __syncwarp();
        key[r] = k;
        rank[r] = rk;
    }
    __syncthreads();
    {   // exclusive scan over warps for digit t
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t c = warpCount[w][t];
            warpCount[w][t] = run;
            run += c;
        }
        digitBase[t] += hist[(size_t)t * tiles + blockIdx.x];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const size_t idx = base + (size_t)r * 32 + lane;
        if (idx < (size_t)n) {
            const uint32_t d = (key[r] >> shift) & 0xFFu;
            const uint32_t dst = digitBase[d] + warpCount[warp][d] + rank[r];
            keysOut[dst] = key[r];
            permOut[dst] = permIn[idx];
        }
    }
}

// ---- counting sort ----
constexpr int kScanChunk = 4 * kThreads;  // counters a block takes at a time

// Sum of each block's tile of counters.
__global__ void __launch_bounds__(kThreads)
counting_sums_kernel(const uint4* counts, uint32_t chunks, uint32_t chunksPerBlock,
                     uint32_t* sums) {
    chain_wait();
    __shared__ uint32_t warpSums[kWarps];
    const uint32_t first = blockIdx.x * chunksPerBlock, last = min(first + chunksPerBlock, chunks);
    uint32_t sum = 0;
    for (uint32_t k = first; k < last; ++k) {
        const uint4 v = counts[(size_t)k * kThreads + threadIdx.x];
        sum += (v.x + v.y) + (v.z + v.w);
    }
    sum = __reduce_add_sync(0xFFFFFFFFu, sum);
    if ((threadIdx.x & 31) == 0) warpSums[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t all = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) all += warpSums[w];
        sums[blockIdx.x] = all;
    }
}

// starts[k] = number of particles with a smaller key than k, for every key and
// one beyond the last; the counters are left at zero for the next substep.
// Every block adds up the sums of the blocks before it (at most kMaxScanBlocks
// of them), so no block waits for another.
constexpr uint32_t kMaxScanBlocks = 1024, kOneBlockChunks = 16;
__global__ void __launch_bounds__(kThreads)
counting_scan_kernel(uint4* counts, uint32_t chunks, uint32_t chunksPerBlock,
                     const uint32_t* sums, uint4* starts) {
    chain_wait();
    __shared__ uint32_t warpSums[kWarps];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t before = 0;
    for (uint32_t b = t; b < blockIdx.x; b += kThreads) before += sums[b];
    before = __reduce_add_sync(0xFFFFFFFFu, before);
    if (lane == 0) warpSums[warp] = before;
    __syncthreads();
    uint32_t carry = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) carry += warpSums[w];
    const uint32_t first = blockIdx.x * chunksPerBlock, last = min(first + chunksPerBlock, chunks);
    for (uint32_t k = first; k < last; ++k) {
        const size_t at = (size_t)k * kThreads + t;
        const uint4 v = counts[at];
        const uint32_t sum = (v.x + v.y) + (v.z + v.w);
        if (sum) counts[at] = make_uint4(0u, 0u, 0u, 0u);
        uint32_t incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += u;
        }
        __syncthreads();  // warpSums is read by all before it is written again
        if (lane == 31) warpSums[warp] = incl;
        __syncthreads();
        uint32_t base = carry, all = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t ws = warpSums[w];
            base += w < warp ? ws : 0u;
            all += ws;
        }
        base += incl - sum;
        starts[at] = make_uint4(base, base + v.x, base + v.x + v.y, base + v.x + v.y + v.z);
        carry += all;
    }
}

// order[first index of the key + place of arrival] = particle
__global__ void __launch_bounds__(kThreads)
cell_scatter_kernel(int n, const uint32_t* keys, const uint32_t* place,
                    const uint32_t* starts, uint32_t* order, uint32_t keyLimit, int* err) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t first = starts[checked_index(keys[i], keyLimit, err, kErrCellKey)];
    order[checked_index(first + place[i], (uint32_t)n, err, kErrSortIndex)] = (uint32_t)i;
}

// The particle in slot s of the scattered order goes to its cell's first index
// plus the number of smaller indices in the cell: the stable order.  With it go
// its key, index, position, prediction and id (radixsort.cl:22-37; velocities
// are not permuted, they are recomputed before any read, update_velocities.cl:13).
__global__ void __launch_bounds__(kThreads)
cell_gather_kernel(int n, const uint32_t* keys, const uint32_t* starts,
                   const uint32_t* order, uint32_t* keysOut, uint32_t* permOut,
                   uint32_t* permCopy,
                   const float4* pos, const float4* pred, const uint32_t* ids,
                   float4* posOut, float4* predOut, uint32_t* idsOut,
                   uint32_t keyLimit, int* err) {
    chain_wait();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t i = checked_index(order[s], (uint32_t)n, err, kErrSortIndex);
    const float4 x = pos[i], p = pred[i];
    const uint32_t id = ids[i], key = checked_index(keys[i], keyLimit, err, kErrCellKey);
    const uint32_t first = starts[key], end = checked_index(starts[key + 1], (uint32_t)n + 1u, err, kErrSortIndex);
    uint32_t to = first;
    for (uint32_t q = first; q < end; ++q) to += order[q] < i;
    to = checked_index(to, (uint32_t)n, err, kErrSortIndex);
    keysOut[to] = key;
    permOut[to] = i;
    if (permCopy) permCopy[to] = i;
    posOut[to] = x;
    predOut[to] = p;
    idsOut[to] = id;
}

// The stable order without the records: permOut from the scattered order.  The
// comparisons are as many as the cell holds, for each particle; cells of more
// than kCrowdedCell go to the list `crowded` (its length first, zero before the
// launch).
constexpr uint32_t kCrowdedCell = 1024;
__global__ void __launch_bounds__(kThreads)
cell_rank_kernel(int n, uint32_t keyLimit, const uint32_t* keys, const uint32_t* starts,
                 const uint32_t* order, uint32_t* permOut, uint32_t* crowded) {
    chain_wait();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= (uint32_t)n) return;
    const uint32_t i = checked_index(order[s], (uint32_t)n, nullptr, kErrSortIndex);
    const uint32_t key = checked_index(keys[i], keyLimit, nullptr, kErrCellKey);
    const uint32_t first = starts[key], end = checked_index(starts[key + 1], (uint32_t)n + 1u, nullptr, kErrSortIndex);
    if (end - first > kCrowdedCell) {
        if (s == first) crowded[1u + atomicAdd(crowded, 1u)] = key;
        return;
    }
    uint32_t to = first;
    for (uint32_t q = first; q < end; ++q) to += order[q] < i;
    permOut[to] = i;
}

// The sorted keys and the cell table (first and last particle of a key, both
// all ones for none) from the first indices; the table may be NULL.  The last
// particle of the only one of n = 1 is not written (update_cells.cl:11-25).
// A warp writes the keys of the cells of more than 16 particles, one thread 512
// of them one after another took 100 us; those of crowded cells are left to
// crowded_cells_kernel.
__global__ void __launch_bounds__(kThreads)
cell_table_kernel(int n, uint32_t keys, const uint32_t* starts, uint32_t* keysOut,
                  uint32_t* cells) {
    chain_wait();
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    uint32_t first = 0, end = 0;
    if (k < keys) {
        first = starts[k];
        end = starts[k + 1];
        if (cells) {
            cells[2 * (size_t)k] = first < end ? first : kEmpty;
            cells[2 * (size_t)k + 1] = first < end && n > 1 ? end - 1u : kEmpty;
        }
    }
    const bool many = end - first > 16u;
    if (!many)
        for (uint32_t q = first; q < end; ++q) keysOut[q] = k;
    for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, many && end - first <= kCrowdedCell); todo; todo &= todo - 1u) {
        const int src = __ffs(todo) - 1;
        const uint32_t f = __shfl_sync(0xFFFFFFFFu, first, src), e = __shfl_sync(0xFFFFFFFFu, end, src);
        for (uint32_t q = f + lane; q < e; q += 32) keysOut[q] = k - lane + src;
    }
}

// The crowded cells, each by one block, or by up to kMostParts that take an
// equal part of the span of the cell's indices: the indices in the part are
// marked in a bitmap and read out in order, behind those below the part.  So a
// cell costs its particles and its span, however many it holds (2^20 particles,
// 16,384 to a cell: 0.12 ms, all in one: 0.24; a comparison with each would take
// 0.13 us for every particle that a cell holds).  Word w of the map is at
// [w % each][w / each], a thread's words in a column.
constexpr int kCrowdedThreads = 1024, kCrowdedBlocks = 152;
constexpr uint32_t kMostParts = 16, kPartCell = 16384;
constexpr int kMostShift = 5;  // 2^5 words to a thread
static_assert(PBF_NOALLOC_MAX_KEYS == (kCrowdedThreads * 32) << kMostShift, "the bitmap holds every index");
__global__ void __launch_bounds__(kCrowdedThreads)
crowded_cells_kernel(const uint32_t* crowded, const uint32_t* starts,
                     const uint32_t* order, uint32_t* keysOut, uint32_t* permOut) {
    chain_wait();
    extern __shared__ uint32_t marks[];  // kCrowdedThreads words for every word to a thread
    __shared__ uint32_t warpSums[kCrowdedThreads / 32], below, least, largest;
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t count = crowded[0];
    for (uint32_t c = 0; c < count; ++c) {
        const uint32_t part = (blockIdx.x + kCrowdedBlocks - c * 17u % kCrowdedBlocks) % kCrowdedBlocks;
        if (part >= kMostParts) continue;
        const uint32_t key = crowded[1u + c], first = starts[key], end = starts[key + 1];
        int parts = 0;  // 2^parts of them
        while ((1u << parts) < kMostParts && (end - first) >> parts > kPartCell) ++parts;
        if (part >= 1u << parts) continue;
        if (t == 0) {
            below = largest = 0u;
            least = 0xFFFFFFFFu;
        }
        __syncthreads();
        uint32_t low = 0xFFFFFFFFu, high = 0u;
#pragma unroll 4
        for (uint32_t s = first + t; s < end; s += kCrowdedThreads) {
            low = min(low, order[s]);
            high = max(high, order[s]);
            if (part == 0) keysOut[s] = key;
        }
        low = __reduce_min_sync(0xFFFFFFFFu, low);
        high = __reduce_max_sync(0xFFFFFFFFu, high);
        if (lane == 0) {
            atomicMin(&least, low);
            atomicMax(&largest, high);
        }
        __syncthreads();
        const uint32_t begin = least & ~31u, span = largest - begin;  // the bitmap's first index, its last one's place
        int shift = 0;  // 2^shift words to a thread of all parts
        while (shift < kMostShift && span >> shift >= kCrowdedThreads * 32u) ++shift;
        const int down = max(shift - parts, 0);  // 2^down words to a thread of this part
        const uint32_t each = 1u << down, lo = begin + part * ((uint32_t)kCrowdedThreads << down) * 32u;
        if (lo <= largest) {
            for (uint32_t r = 0; r < each; ++r) marks[r * kCrowdedThreads + t] = 0u;
            __syncthreads();
            uint32_t less = 0;
#pragma unroll 4
            for (uint32_t s = first + t; s < end; s += kCrowdedThreads) {
                const uint32_t i = order[s], w = (i - lo) >> 5;
                less += i < lo;
                if (i >= lo && w >> down < kCrowdedThreads)
                    atomicOr(&marks[(w & (each - 1u)) * kCrowdedThreads + (w >> down)], 1u << (i & 31u));
            }
            less = __reduce_add_sync(0xFFFFFFFFu, less);
            if (lane == 0 && less) atomicAdd(&below, less);
            __syncthreads();
            uint32_t mine = 0;
            for (uint32_t r = 0; r < each; ++r) mine += __popc(marks[r * kCrowdedThreads + t]);
            uint32_t incl = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if (lane >= (uint32_t)d) incl += u;
            }
            if (lane == 31) warpSums[warp] = incl;
            __syncthreads();
            uint32_t to = first + below + incl - mine;
            for (uint32_t w = 0; w < warp; ++w) to += warpSums[w];
            for (uint32_t r = 0; r < each; ++r)
                for (uint32_t m = marks[r * kCrowdedThreads + t]; m; m &= m - 1u)
                    permOut[to++] = lo + 32u * ((t << down) + r) + (uint32_t)__ffs(m) - 1u;
        }
        __syncthreads();  // all is read before the next cell writes it
    }
}

}  // namespace

cudaError_t launch_cell_finish(int n, uint32_t keyCount, const uint32_t* starts, const uint32_t* order, uint32_t* keys,
                               uint32_t* permOut, uint32_t* cells, uint32_t* crowded, cudaStream_t s) {
    launch_chained(cell_rank_kernel, (n + kThreads - 1) / kThreads, kThreads, s, n, keyCount, keys, starts, order, permOut, crowded);
    launch_chained(cell_table_kernel, (keyCount + kThreads - 1) / kThreads, kThreads, s, n, keyCount, starts, keys, cells);
    if ((uint32_t)n <= kCrowdedCell) return cudaGetLastError();
    int shift = 0;
    while (shift < kMostShift && ((uint64_t)kCrowdedThreads * 32 << shift) < (uint64_t)n) ++shift;
    constexpr size_t kRow = kCrowdedThreads * sizeof(uint32_t);
    // always the same limit: callers on other threads launch the kernel too
    const cudaError_t e = cudaFuncSetAttribute(crowded_cells_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(kRow << kMostShift));
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kCrowdedBlocks);
    cfg.blockDim = dim3(kCrowdedThreads);
    cfg.dynamicSmemBytes = kRow << shift;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, crowded_cells_kernel, static_cast<const uint32_t*>(crowded), starts, order, keys, permOut);
}

CountingPlan make_counting_plan(int n, uint64_t keys) {
    if ((keys > kCountingSmall && keys > kCountingRatio * (uint64_t)n) || (uint64_t)n > kCountingLoad * keys)
        return CountingPlan{};
    return make_scan_plan(keys);
}

CountingPlan make_scan_plan(uint64_t keys) {
    CountingPlan p;
    p.chunks = (uint32_t)((keys + 1 + kScanChunk - 1) / kScanChunk);  // one start beyond the last key
    // a key range of a few chunks is scanned by one block, which needs no sums of others before it
    p.chunksPerBlock = p.chunks <= kOneBlockChunks ? p.chunks : (p.chunks + kMaxScanBlocks - 1) / kMaxScanBlocks;
    p.blocks = (p.chunks + p.chunksPerBlock - 1) / p.chunksPerBlock;
    p.words = (size_t)p.chunks * kScanChunk;
    return p;
}

void launch_counting_scan(const CountingPlan& plan, uint32_t* counts, uint32_t* sums, uint32_t* starts, cudaStream_t s) {
    uint4* c4 = reinterpret_cast<uint4*>(counts);
    if (plan.blocks > 1)
        launch_chained(counting_sums_kernel, plan.blocks, kThreads, s, c4, plan.chunks, plan.chunksPerBlock,
                                                                      sums);
    launch_chained(counting_scan_kernel, plan.blocks, kThreads, s, c4, plan.chunks, plan.chunksPerBlock, sums,
                                                          reinterpret_cast<uint4*>(starts));
}

void launch_counting_sort(const CountingPlan& plan, int n, uint32_t* counts, uint32_t* sums, uint32_t* starts,
                          const uint32_t* keys, const uint32_t* place, uint32_t* order, uint32_t keyLimit, int* err,
                          cudaStream_t s) {
    launch_counting_scan(plan, counts, sums, starts, s);
    launch_chained(cell_scatter_kernel, (n + kThreads - 1) / kThreads, kThreads, s, n, keys, place, starts, order, keyLimit, err);
}

void launch_cell_gather(int n, const uint32_t* keys, const uint32_t* starts, const uint32_t* order, uint32_t* keysOut,
                        uint32_t* permOut, uint32_t* permCopy, const float4* pos, const float4* pred,
                        const uint32_t* ids, float4* posOut, float4* predOut, uint32_t* idsOut, uint32_t keyLimit, int* err,
                        cudaStream_t s) {
    launch_chained(cell_gather_kernel, (n + kThreads - 1) / kThreads, kThreads, s, n, keys, starts, order, keysOut, permOut, permCopy, pos,
                                                                          pred, ids, posOut, predOut, idsOut, keyLimit, err);
}

SortPlan make_sort_plan(int n, uint32_t gridBufSize) {
    SortPlan p;
    p.n = n;
    int bits = 0;
    while (bits < 32 && ((uint64_t)1 << bits) < (uint64_t)gridBufSize) ++bits;  // keys <= gridBufSize-1
    p.passes = (bits + 7) / 8;
    p.rounds = n <= kSmallSortKeys ? 4 : (n <= kMidSortKeys ? 8 : 16);
    const int tile = kThreads * p.rounds;
    p.tiles = (n + tile - 1) / tile;
    p.histWords = (size_t)256 * p.tiles + 256;  // per-tile histograms, then the 256 digit totals
    return p;
}

int radix_sort_launches(const SortPlan& plan) { return 3 * plan.passes; }

int launch_radix_sort(const SortPlan& plan, uint32_t* keys[2], uint32_t* perm[2], uint32_t* hist,
                      const float4*, const float4*, float4*, float4*, cudaStream_t s) {
    int cur = 0;
    uint32_t* totals = hist + (size_t)256 * plan.tiles;
    for (int pass = 0; pass < plan.passes; ++pass) {
        const int shift = 8 * pass;
        if (plan.rounds == 4)
            radix_upsweep_kernel<4><<<plan.tiles, kThreads, 0, s>>>(keys[cur], plan.n, shift, plan.tiles, hist);
        else if (plan.rounds == 8)
            radix_upsweep_kernel<8><<<plan.tiles, kThreads, 0, s>>>(keys[cur], plan.n, shift, plan.tiles, hist);
        else
            radix_upsweep_kernel<16><<<plan.tiles, kThreads, 0, s>>>(keys[cur], plan.n, shift, plan.tiles, hist);
        radix_scan_kernel<<<256, kThreads, 0, s>>>(hist, plan.tiles, totals);
        if (plan.rounds == 4)
            radix_downsweep_kernel<4><<<plan.tiles, kThreads, 0, s>>>(keys[cur], perm[cur], keys[cur ^ 1],
                                                                      perm[cur ^ 1], plan.n, shift, plan.tiles, hist,
                                                                      totals);
        else if (plan.rounds == 8)
            radix_downsweep_kernel<8><<<plan.tiles, kThreads, 0, s>>>(keys[cur], perm[cur], keys[cur ^ 1],
                                                                      perm[cur ^ 1], plan.n, shift, plan.tiles, hist,
                                                                      totals);
        else
            radix_downsweep_kernel<16><<<plan.tiles, kThreads, 0, s>>>(keys[cur], perm[cur], keys[cur ^ 1],
                                                                       perm[cur ^ 1], plan.n, shift, plan.tiles, hist,
                                                                       totals);
        cur ^= 1;
    }
    return cur;
}

}  // namespace pbf
