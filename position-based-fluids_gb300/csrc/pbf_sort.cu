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

// order[first index of the key + place of arrival] = particle.  crowded (may be
// NULL; words of it, the first two zero): the keys of the cells that
// launch_cell_finish does not order by comparing, by the first particle to arrive
// in each: [0] and [1] count those of up to kBlockCell particles, listed from [2]
// on, and the larger ones, listed from the end on downwards.
constexpr uint32_t kComparedCell = 128, kWarpCell = 512, kBlockCell = 4096;
__global__ void __launch_bounds__(kThreads)
cell_scatter_kernel(int n, const uint32_t* keys, const uint32_t* place,
                    const uint32_t* starts, uint32_t* order, uint32_t* crowded, uint32_t words, uint32_t keyLimit, int* err) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t key = checked_index(keys[i], keyLimit, err, kErrCellKey), first = starts[key], at = place[i];
    order[checked_index(first + at, (uint32_t)n, err, kErrSortIndex)] = (uint32_t)i;
    if (!crowded || at != 0u) return;
    const uint32_t holds = starts[key + 1] - first;
    if (holds > kBlockCell) crowded[words - 1u - atomicAdd(crowded + 1, 1u)] = key;
    else if (holds > kComparedCell) crowded[2u + atomicAdd(crowded, 1u)] = key;
}

// Particles of the cell [first, end) of the scattered order whose index is below i.
// The particles that one warp brings to a cell lie together in it, by index
// (place_of_arrival), so most of a crowded cell whose particles were sorted before
// are the 32 of a whole warp, or its last ones, and are counted at once: 65,536
// particles in one cell take 1.6 ms to compare, 0.36 like this.
// Out of line: inlined it costs the substep of 2,048 particles 0.7 us.
constexpr uint32_t kLongCell = 256;
__device__ __noinline__ uint32_t smaller_in_long_cell(const uint32_t* order, uint32_t first, uint32_t end, uint32_t i) {
    uint32_t less = 0, q = first;
    // of the `count` consecutive indices from a on
    auto run = [&](uint32_t a, uint32_t count) { return i > a ? min(i - a, count) : 0u; };
    while (q + 32u <= end) {
        const uint32_t a = order[q], rest = 32u - (a & 31u);
        if (rest == 32u && q + 128u <= end) {
            uint32_t from[3], last[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) last[k] = order[q + 32 * k + 31];
#pragma unroll
            for (int k = 0; k < 3; ++k) from[k] = order[q + 32 * k + 32];
            bool whole = last[0] == a + 31u;
#pragma unroll
            for (int k = 0; k < 3; ++k) whole = whole && (from[k] & 31u) == 0u && last[k + 1] == from[k] + 31u;
            if (whole) {
                less += run(a, 32u) + run(from[0], 32u) + run(from[1], 32u) + run(from[2], 32u);
                q += 128u;
                continue;
            }
        }
        if (order[q + rest - 1u] == a + rest - 1u) {
            less += run(a, rest);
            q += rest;
        } else {
#pragma unroll 8
            for (uint32_t k = 0; k < 32u; ++k) less += order[q + k] < i;
            q += 32u;
        }
    }
    for (; q < end; ++q) less += order[q] < i;
    return less;
}

// The runs of same-cell particles, for sparse_scene: each thread draws a slot from its
// part of the scattered order, where a warp's particles of a key lie together, and
// counts it if the slot before holds a particle of another cell.  The gather's first
// blocks do that and nothing else: they end long before its last.
__device__ __forceinline__ void sample_runs(int n, float perH, const uint32_t* order, const float4* pred, uint32_t* sampled) {
    const uint32_t k = blockIdx.x * kThreads + threadIdx.x, part = (uint32_t)n / (kSampleBlocks * kThreads);
    const uint32_t s = max(k * part + ((k * 2654435761u) >> 8) % part, 1u);
    const float4 p = pred[order[s]], o = pred[order[s - 1u]];
    const bool head = __float2int_rz(p.x * perH) != __float2int_rz(o.x * perH) ||
                      __float2int_rz(p.y * perH) != __float2int_rz(o.y * perH) ||
                      __float2int_rz(p.z * perH) != __float2int_rz(o.z * perH);
    const int heads = __popc(__ballot_sync(0xFFFFFFFFu, head));
    if ((threadIdx.x & 31) == 0) atomicAdd(sampled, (uint32_t)heads);
}

// The particle in slot s of the scattered order goes to its cell's first index
// plus the number of smaller indices in the cell: the stable order.  With it go
// its key, index, position, prediction and id (radixsort.cl:22-37; velocities
// are not permuted, they are recomputed before any read, update_velocities.cl:13).
template <bool Sample>
__global__ void __launch_bounds__(kThreads, 8)
cell_gather_kernel(int n, float h, uint32_t* sampled, const uint32_t* keys, const uint32_t* starts,
                   const uint32_t* order, uint32_t* keysOut, uint32_t* permOut,
                   uint32_t* permCopy,
                   const float4* pos, const float4* pred, const uint32_t* ids,
                   float4* posOut, float4* predOut, uint32_t* idsOut,
                   uint32_t keyLimit, int* err) {
    chain_wait();
    if (Sample && blockIdx.x < kSampleBlocks) {
        sample_runs(n, 1.0f / h, order, pred, sampled);
        return;
    }
    const int s = (blockIdx.x - (Sample ? kSampleBlocks : 0u)) * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t i = checked_index(order[s], (uint32_t)n, err, kErrSortIndex);
    const float4 x = pos[i], p = pred[i];
    const uint32_t id = ids[i], key = checked_index(keys[i], keyLimit, err, kErrCellKey);
    const uint32_t first = starts[key], end = checked_index(starts[key + 1], (uint32_t)n + 1u, err, kErrSortIndex);
    uint32_t to = first;
    if (end - first > kLongCell) to += smaller_in_long_cell(order, first, end, i);
    else
        for (uint32_t q = first; q < end; ++q) to += order[q] < i;
    to = checked_index(to, (uint32_t)n, err, kErrSortIndex);
    keysOut[to] = key;
    permOut[to] = i;
    if (permCopy) permCopy[to] = i;
    posOut[to] = x;
    predOut[to] = p;
    idsOut[to] = id;
}

// ---- the stable order without the records ----
//
// cell_scatter leaves a cell's particles in any order.  Up to kComparedCell of them
// are ranked by comparing, up to kWarpCell are sorted by a warp, up to kBlockCell by
// a block, and the particles of larger cells, at most kMostBig of them, are counted
// and placed tile by tile of the particles' own order, as a radix pass does with
// its digits.  A call with 2^20 particles in 2^17 keys, sorted before / in random
// order, us: 128 to a cell 53 / 80, 512 45 / 73, 2,100 42 / 67, 4,096 45 / 90,
// 16,384 37 / 71, all in one 34; by radix passes 81-85 / 85-106 whatever they hold;
// comparing with every other one takes 104 / 145 at 512 and 181 / 284 at 1,024.

constexpr uint32_t kMostBig = PBF_NOALLOC_MAX_KEYS / (kBlockCell + 1);
constexpr int kTileRounds = 16, kTileKeys = kThreads * kTileRounds;
constexpr uint32_t kMostTiles = PBF_NOALLOC_MAX_KEYS / kTileKeys;
constexpr uint32_t kBigSlots = 512;  // of the table, a power of two above kMostBig
static_assert(kMostBig < kBigSlots / 2 + 1 && kMostTiles <= kBlockCell, "bins and tiles of the large cells");

// The large cells' numbers by key, and their first indices by number, for a block.  The
// counts and the probes are limited to what a call can need: calls must not overlap on
// the array, and where they do all the same no loop here runs on what the other left.
struct BigCells {
    uint32_t key[kBigSlots], bin[kBigSlots], first[kMostBig];
    __device__ __forceinline__ static uint32_t slot(uint32_t k) { return (k * 2654435761u) >> 23; }
    // All threads; they are in step afterwards.
    __device__ __forceinline__ void fill(const uint32_t* crowded, uint32_t words, uint32_t big, const uint32_t* starts) {
        for (uint32_t q = threadIdx.x; q < kBigSlots; q += kThreads) key[q] = kEmpty;
        __syncthreads();
        for (uint32_t b = threadIdx.x; b < big; b += kThreads) {
            const uint32_t k = crowded[words - 1u - b];
            uint32_t q = slot(k);
            for (uint32_t tries = 0; tries < kBigSlots && atomicCAS(&key[q], kEmpty, k) != kEmpty; ++tries) q = (q + 1u) % kBigSlots;
            bin[q] = b;
            first[b] = starts[k];
        }
        __syncthreads();
    }
    // kEmpty: not a large cell's key.
    __device__ __forceinline__ uint32_t find(uint32_t k) const {
        for (uint32_t q = slot(k), tries = 0; tries < kBigSlots; q = (q + 1u) % kBigSlots, ++tries) {
            const uint32_t at = key[q];
            if (at == k) return bin[q];
            if (at == kEmpty) break;
        }
        return kEmpty;
    }
};

// permOut of the cells that are ranked by comparing.  The first `tiles` blocks also
// count the particles that each tile has of each large cell, into the cell's slots
// of permOut, one per tile.
__global__ void __launch_bounds__(kThreads)
cell_rank_kernel(int n, uint32_t keyLimit, const uint32_t* keys, const uint32_t* starts, const uint32_t* order,
                 uint32_t* permOut, const uint32_t* crowded, uint32_t words, uint32_t tiles) {
    chain_wait();
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < (uint32_t)n) {
        const uint32_t i = checked_index(order[s], (uint32_t)n, nullptr, kErrSortIndex);
        const uint32_t key = checked_index(keys[i], keyLimit, nullptr, kErrCellKey);
        const uint32_t first = starts[key], end = checked_index(starts[key + 1], (uint32_t)n + 1u, nullptr, kErrSortIndex);
        if (end - first <= kComparedCell) {
            uint32_t to = first;
            for (uint32_t q = first; q < end; ++q) to += order[q] < i;
            permOut[to] = i;
        }
    }
    if (blockIdx.x >= tiles) return;
    const uint32_t big = min(crowded[1], kMostBig);
    if (big == 0u) return;
    __shared__ BigCells cells;
    __shared__ uint32_t counts[kMostBig];
    for (uint32_t b = threadIdx.x; b < big; b += kThreads) counts[b] = 0u;
    cells.fill(crowded, words, big, starts);
    uint32_t key[kTileRounds];
#pragma unroll
    for (int r = 0; r < kTileRounds; ++r) {
        const uint32_t i = blockIdx.x * kTileKeys + r * kThreads + threadIdx.x;
        key[r] = i < (uint32_t)n ? keys[i] : kEmpty;
    }
#pragma unroll
    for (int r = 0; r < kTileRounds; ++r) {
        const uint32_t bin = key[r] != kEmpty ? cells.find(key[r]) : kEmpty;
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, bin);
        if (bin != kEmpty && (threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&counts[bin], (uint32_t)__popc(peers));
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < big; b += kThreads) permOut[cells.first[b] + blockIdx.x] = counts[b];
}

// Sorts the particles of one cell of more than kComparedCell and at most 16 G, G
// threads (a warp or the block): a counting sort by the upper bits of their indices,
// about as many buckets as particles, and the few of a bucket are put in order by
// comparing them.
template <uint32_t G>
struct SharedCell {
    static constexpr uint32_t kMost = 16 * G;
    uint32_t index[kMost], buckets[kMost];
    uint32_t warpSums[G / 32], least, largest;
};
static_assert(kWarpCell == SharedCell<32>::kMost && kBlockCell == SharedCell<kThreads>::kMost, "what a warp and a block sort");
template <uint32_t G>
__device__ __forceinline__ void sort_cell(SharedCell<G>& sh, uint32_t first, uint32_t count, const uint32_t* order, uint32_t* permOut) {
    const uint32_t t = threadIdx.x % G, lane = t & 31, warp = t >> 5;
    auto sync = [] {
        if constexpr (G == 32) __syncwarp();
        else __syncthreads();
    };
    int log = 0;  // 2^log buckets to a thread, bucket b at [b % 2^log][b / 2^log]
    while (G << log < count) ++log;
    const uint32_t each = 1u << log;
    if (t == 0) {
        sh.least = 0xFFFFFFFFu;
        sh.largest = 0u;
    }
    for (uint32_t r = 0; r < each; ++r) sh.buckets[r * G + t] = 0u;
    sync();
    uint32_t low = 0xFFFFFFFFu, high = 0u;
#pragma unroll 4
    for (uint32_t q = t; q < count; q += G) {
        const uint32_t i = order[first + q];
        low = min(low, i);
        high = max(high, i);
    }
    low = __reduce_min_sync(0xFFFFFFFFu, low);
    high = __reduce_max_sync(0xFFFFFFFFu, high);
    if (lane == 0) {
        atomicMin(&sh.least, low);
        atomicMax(&sh.largest, high);
    }
    sync();
    const uint32_t begin = sh.least, span = sh.largest - begin;
    int shift = 0;  // 2^shift indices to a bucket
    while (span >> shift >> log >= G) ++shift;
    auto place = [&](uint32_t b) -> uint32_t& { return sh.buckets[(b & (each - 1u)) * G + (b >> log)]; };
#pragma unroll 4
    for (uint32_t q = t; q < count; q += G) atomicAdd(&place((order[first + q] - begin) >> shift), 1u);
    sync();
    uint32_t mine = 0;
    for (uint32_t r = 0; r < each; ++r) mine += sh.buckets[r * G + t];
    uint32_t incl = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= (uint32_t)d) incl += u;
    }
    uint32_t run = incl - mine;
    if constexpr (G > 32) {
        if (lane == 31) sh.warpSums[warp] = incl;
        sync();
        for (uint32_t w = 0; w < warp; ++w) run += sh.warpSums[w];
    }
    for (uint32_t r = 0; r < each; ++r) {
        const uint32_t c = sh.buckets[r * G + t];
        sh.buckets[r * G + t] = run;
        run += c;
    }
    sync();
#pragma unroll 4
    for (uint32_t q = t; q < count; q += G) {
        const uint32_t i = order[first + q];
        sh.index[atomicAdd(&place((i - begin) >> shift), 1u)] = i;
    }
    sync();
    for (uint32_t q = t; q < count; q += G) {  // a bucket's place is its end now
        const uint32_t i = sh.index[q], b = (i - begin) >> shift, from = b ? place(b - 1u) : 0u, end = place(b);
        uint32_t to = from;
        for (uint32_t k = from; k < end; ++k) to += sh.index[k] < i;
        permOut[first + to] = i;
    }
    sync();  // all is read before the next cell writes it
}

// The cells that a block sorts go to permOut, a block taking one after another; of
// the larger ones, block b places the particles of tile b into the cells' slots of
// `order`, behind those of the tiles before it.
struct BigTile {
    BigCells cells;
    uint32_t warpCount[kWarps][kMostBig], base[kMostBig];
};
__global__ void __launch_bounds__(kThreads)
crowded_cells_kernel(int n, const uint32_t* keys, const uint32_t* starts, uint32_t* order, uint32_t* permOut,
                     const uint32_t* crowded, uint32_t words, uint32_t tiles) {
    chain_wait();
    __shared__ union {
        SharedCell<32> warpCell[kWarps];
        SharedCell<kThreads> cell;
        BigTile tile;
    } sh;
    const uint32_t count = min(crowded[0], words - 2u), big = min(crowded[1], kMostBig), t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (uint32_t c = blockIdx.x * kWarps + warp; c < count; c += gridDim.x * kWarps) {
        const uint32_t key = crowded[2u + c], first = starts[key], holds = starts[key + 1] - first;
        if (holds <= kWarpCell) sort_cell<32>(sh.warpCell[warp], first, holds, order, permOut);
    }
    __syncthreads();
    for (uint32_t c = blockIdx.x; c < count; c += gridDim.x) {
        const uint32_t key = crowded[2u + c], first = starts[key], holds = starts[key + 1] - first;
        if (holds > kWarpCell && holds <= kBlockCell) sort_cell<kThreads>(sh.cell, first, holds, order, permOut);
    }
    if (big == 0u || blockIdx.x >= tiles) return;
    BigTile& tile = sh.tile;
    tile.cells.fill(crowded, words, big, starts);
    for (uint32_t b = warp; b < big; b += kWarps) {
        const uint32_t first = tile.cells.first[b];
        uint32_t before = 0;
#pragma unroll
        for (uint32_t q = lane; q < kMostTiles; q += 32) before += q < blockIdx.x ? permOut[first + q] : 0u;
        before = __reduce_add_sync(0xFFFFFFFFu, before);
        if (lane == 0) tile.base[b] = first + before;
        for (uint32_t w = lane; w < kWarps; w += 32) tile.warpCount[w][b] = 0u;
    }
    __syncthreads();
    const uint32_t from = blockIdx.x * kTileKeys + warp * (32 * kTileRounds) + lane;  // a warp's particles are consecutive
    uint32_t bins[kTileRounds], rank[kTileRounds];
#pragma unroll
    for (int r = 0; r < kTileRounds; ++r) bins[r] = from + 32 * r < (uint32_t)n ? keys[from + 32 * r] : kEmpty;
#pragma unroll
    for (int r = 0; r < kTileRounds; ++r) {
        const uint32_t bin = bins[r] != kEmpty ? tile.cells.find(bins[r]) : kEmpty;
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, bin);
        const uint32_t prior = bin != kEmpty ? tile.warpCount[warp][bin] : 0u;
        __syncwarp();
        if (bin != kEmpty && lane == (uint32_t)__ffs(peers) - 1u) tile.warpCount[warp][bin] = prior + (uint32_t)__popc(peers);
        __syncwarp();
        bins[r] = bin;
        rank[r] = prior + (uint32_t)__popc(peers & ((1u << lane) - 1u));
    }
    __syncthreads();
    for (uint32_t b = t; b < big; b += kThreads) {
        uint32_t run = tile.base[b];
        for (int w = 0; w < kWarps; ++w) {
            const uint32_t c = tile.warpCount[w][b];
            tile.warpCount[w][b] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kTileRounds; ++r)
        if (bins[r] != kEmpty)
            order[checked_index(tile.warpCount[warp][bins[r]] + rank[r], (uint32_t)n, nullptr, kErrSortIndex)] = from + 32 * r;
}

// The sorted keys and the cell table (first and last particle of a key, both
// all ones for none) from the first indices; the table may be NULL.  The last
// particle of the only one of n = 1 is not written (update_cells.cl:11-25).
// A warp writes the keys of the cells of more than 16 particles (one thread 512 of
// them one after another took 100 us), a block those of the cells of more than
// kComparedCell, and all blocks those of the large ones, with their order.
__global__ void __launch_bounds__(kThreads)
cell_table_kernel(int n, uint32_t keys, const uint32_t* starts, const uint32_t* order, uint32_t* keysOut, uint32_t* permOut,
                  uint32_t* cells, const uint32_t* crowded, uint32_t words) {
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
    for (uint32_t todo = __ballot_sync(0xFFFFFFFFu, many && end - first <= kComparedCell); todo; todo &= todo - 1u) {
        const int src = __ffs(todo) - 1;
        const uint32_t f = __shfl_sync(0xFFFFFFFFu, first, src), e = __shfl_sync(0xFFFFFFFFu, end, src);
        for (uint32_t q = f + lane; q < e; q += 32) keysOut[q] = k - lane + src;
    }
    if ((uint32_t)n <= kComparedCell) return;
    const uint32_t count = min(crowded[0], words - 2u), big = min(crowded[1], kMostBig);
    for (uint32_t b = blockIdx.x; b < count; b += gridDim.x) {
        const uint32_t key = crowded[2u + b], e = min(starts[key + 1], (uint32_t)n);
        for (uint32_t q = starts[key] + threadIdx.x; q < e; q += kThreads) keysOut[q] = key;
    }
    if (big == 0u) return;
    const uint32_t parts = max(gridDim.x / big, 1u), part = blockIdx.x % parts;  // blocks to a cell
    for (uint32_t b = blockIdx.x / parts; b < big; b += gridDim.x) {
        const uint32_t key = crowded[words - 1u - b], e = min(starts[key + 1], (uint32_t)n);
        for (uint32_t q = starts[key] + part * kThreads + threadIdx.x; q < e; q += parts * kThreads) {
            keysOut[q] = key;
            permOut[q] = order[q];
        }
    }
}

}  // namespace

void launch_cell_finish(const CountingPlan& plan, int n, uint32_t keyCount, const uint32_t* starts, uint32_t* order,
                        uint32_t* keys, uint32_t* permOut, uint32_t* cells, const uint32_t* crowded, cudaStream_t s) {
    const uint32_t words = (uint32_t)plan.words, tiles = (uint32_t)n > kBlockCell ? ((uint32_t)n + kTileKeys - 1) / kTileKeys : 0u;
    launch_chained(cell_rank_kernel, (n + kThreads - 1) / kThreads, kThreads, s, n, keyCount, keys, starts, order, permOut,
                   crowded, words, tiles);
    if ((uint32_t)n > kComparedCell) {
        const uint32_t most = min((uint32_t)n / kComparedCell, 912u);  // 6 blocks to an SM
        launch_chained(crowded_cells_kernel, max(most, tiles), kThreads, s, n, keys, starts, order, permOut, crowded, words, tiles);
    }
    launch_chained(cell_table_kernel, (keyCount + kThreads - 1) / kThreads, kThreads, s, n, keyCount, starts, order, keys,
                   permOut, cells, crowded, words);
}

CountingPlan make_counting_plan(int n, uint64_t keys) {
    if ((keys > kCountingSmall && keys > kCountingRatio * (uint64_t)n) || (uint64_t)n > kCountingLoad * keys)
        return CountingPlan{};
    return make_scan_plan(keys);
}

CountingPlan make_scan_plan(uint64_t keys) {
    CountingPlan p;
    p.chunks = (uint32_t)((keys + 2 + kScanChunk - 1) / kScanChunk);  // one start beyond the last key; two counts (cell_scatter)
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
                          const uint32_t* keys, const uint32_t* place, uint32_t* order, uint32_t* crowded,
                          uint32_t keyLimit, int* err, cudaStream_t s) {
    launch_counting_scan(plan, counts, sums, starts, s);
    launch_chained(cell_scatter_kernel, (n + kThreads - 1) / kThreads, kThreads, s, n, keys, place, starts, order, crowded,
                   (uint32_t)plan.words, keyLimit, err);
}

void launch_cell_gather(const DevConsts& c, const uint32_t* keys, const uint32_t* starts, const uint32_t* order, uint32_t* keysOut,
                        uint32_t* permOut, uint32_t* permCopy, const float4* pos, const float4* pred,
                        const uint32_t* ids, float4* posOut, float4* predOut, uint32_t* idsOut, uint32_t keyLimit, int* err,
                        cudaStream_t s) {
    const int n = c.n;
    const bool sample = n >= kSparseLeast;
    auto k = sample ? cell_gather_kernel<true> : cell_gather_kernel<false>;
    launch_chained(k, (n + kThreads - 1) / kThreads + (sample ? kSampleBlocks : 0u), kThreads, s, n, c.h, c.epoch + 1, keys, starts, order, keysOut, permOut, permCopy, pos,
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

int launch_radix_sort(const SortPlan& plan, uint32_t* keys[2], uint32_t* perm[2], uint32_t* hist, cudaStream_t s) {
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
