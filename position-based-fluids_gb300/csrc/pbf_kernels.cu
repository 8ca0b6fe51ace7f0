// pbf_kernels.cu — the per-substep PBF stages on sm_103a.
//
// Arithmetic contract (shared with the CPU oracle): this file is compiled
// with --fmad=false, IEEE division and IEEE sqrt, so every float operation
// below is one correctly rounded IEEE operation, evaluated in the order of
// the reference kernel it stands for.  With the same inputs the results are
// bit-identical to a strict IEEE evaluation of the reference's kernels.
//   dot(a,b)       = (a.x*b.x + a.y*b.y) + a.z*b.z
//   cross(a,b)     = (a.y*b.z - a.z*b.y, a.z*b.x - a.x*b.z, a.x*b.y - a.y*b.x)
//   fast_length(a) = sqrtf(dot(a,a))
//   convert_int    = __float2int_rz (truncating, saturating, NaN -> 0)
//
// Data layout in device memory (N particles, all arrays dense):
//   pos, pred, vel, omega : float4[N]  (16-byte records, coalesced 128-bit I/O)
//   keys, perm            : uint32[N]
//   cells                 : uint2[gridBufSize]  (start, inclusive end)
//   rows                  : uint4[ceil(circles * perCircle / 4)][N]: particle
//                           i's friends that the density pass keeps, in
//                           summation order, four per entry; written by the
//                           friends build and walked by the passes after it.
//   meta                  : uint2[N] per particle: 7-bit friend count of each
//                           of up to 8 circles (bits 0-55), the circles the
//                           density pass keeps (bits 56-59) and the circles
//                           the other passes keep (bits 60-63).

#include <cuda_runtime.h>
#include <cstdint>

#include "pbf_device.cuh"
#include "pbf_internal.h"

namespace pbf {
namespace {

constexpr int kBlock = 256;

inline unsigned blocks_for(int n, int block = kBlock) { return (unsigned)((n + block - 1) / block); }

// Scene values of particle i: from the batch table, or DevConsts for a
// single scene.
__device__ __forceinline__ uint32_t key_base(const Batch& b, int i) {
    return b.scenes ? b.scenes[b.sceneOf[i]].keyBase : 0u;
}

// Adds the lanes of `valid` to their keys' counts; returns the lane's place
// among its key's particles.  The particles come nearly sorted, a few keys to a
// warp: one atomic per key and warp.
__device__ __forceinline__ uint32_t place_of_arrival(unsigned valid, uint32_t key, uint32_t* counts) {
    const unsigned peers = __match_any_sync(valid, key);
    const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
    uint32_t place = 0;
    if (lane == leader) place = atomicAdd(&counts[key], (uint32_t)__popc(peers));
    return __shfl_sync(valid, place, leader) + (uint32_t)__popc(peers & ((1u << lane) - 1u));
}

// ------------------------------------------------------------- predict --
// predict_positions.cl:8-17 fused with computeKeys (radixsort.cl:7-19).
__global__ void predict_keys_kernel(DevConsts c, Batch b, const float4* pos, float4* vel,
                                    float4* pred, uint32_t* keys,
                                    uint32_t* perm, uint32_t* counts, int paused) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned valid = __ballot_sync(0xFFFFFFFFu, i < c.n);
    if (i >= c.n) return;
    float4 v = vel[i];
    float gx = c.gx, gy = c.gy, gz = c.gz;
    uint32_t base = 0;
    if (b.scenes) {
        const SceneParams& sp = b.scenes[b.sceneOf[i]];
        gx = sp.gx; gy = sp.gy; gz = sp.gz;
        base = sp.keyBase;
    }
    if (!paused) {
        v.x = v.x + c.dt * gx;
        v.y = v.y + c.dt * gy;
        v.z = v.z + c.dt * gz;
        vel[i] = v;
    }
    const float4 p = pos[i];
    const float4 q = make_float4(p.x + c.dt * v.x, p.y + c.dt * v.y, p.z + c.dt * v.z, p.w + c.dt * v.w);
    pred[i] = q;
    if (i == 0) {
        c.epoch[0] += 1u;  // a new substep: earlier taint marks lapse
        c.epoch[1] = c.epoch[2] = 0u;
    }
    if (!paused) {
        const uint32_t key = base + grid_hash(__float2int_rz(q.x / c.h), __float2int_rz(q.y / c.h), __float2int_rz(q.z / c.h), c.grid);
        keys[i] = key;
        if (!counts) {
            perm[i] = (uint32_t)i;
            return;
        }
        perm[i] = place_of_arrival(valid, key, counts);
    }
}

// radixsort.cl:1-20 alone (keys of given predicted positions, no padding).
// With `hot` given and set (clear_counts): the keys of many particles in few cells,
// unsorted, where an atomic for every key of every warp on the same few counters
// took 80 us for 2^20 particles in 1,024 cells and 180 in 256 (34 and 28 now).  The
// first blocks take a tile of kHotTile each, count in shared memory, and add up a
// tile's count of a key with one atomic.
constexpr int kKeyThreads = 1024, kHotLeast = 65536;  // fewer particles do not contend
constexpr uint32_t kHotTile = 4096;                   // as many slots as particles: the table does not overflow
template <int Threads>
__global__ void __launch_bounds__(Threads)
compute_keys_kernel(DevConsts c, Batch b, const float4* pred, uint32_t* keys, uint32_t* perm, uint32_t* counts,
                    const uint32_t* hot) {
    chain_wait();
    auto key_of = [&](int i) {
        const float4 q = pred[i];
        return key_base(b, i) + grid_hash(__float2int_rz(q.x / c.h), __float2int_rz(q.y / c.h), __float2int_rz(q.z / c.h), c.grid);
    };
    if (Threads < kKeyThreads || *hot == 0u) {
        const int i = blockIdx.x * Threads + threadIdx.x;
        const unsigned valid = __ballot_sync(0xFFFFFFFFu, i < c.n);
        if (i >= c.n) return;
        const uint32_t key = key_of(i);
        keys[i] = key;
        perm[i] = counts ? place_of_arrival(valid, key, counts) : (uint32_t)i;
        return;
    }
    if (blockIdx.x * kHotTile >= (uint32_t)c.n) return;
    constexpr int kRounds = kHotTile / kKeyThreads;
    constexpr uint32_t kSlots = Threads < kKeyThreads ? 1 : kHotTile;
    __shared__ uint32_t slotKey[kSlots], slotCount[kSlots];  // a slot's count, then its first place
    for (uint32_t q = threadIdx.x; q < kHotTile; q += kKeyThreads) {
        slotKey[q] = kEmpty;
        slotCount[q] = 0u;
    }
    __syncthreads();
    uint32_t key[kRounds], slot[kRounds], place[kRounds];
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const int i = (int)(blockIdx.x * kHotTile) + r * kKeyThreads + (int)threadIdx.x;
        key[r] = i < c.n ? key_of(i) : kEmpty;
    }
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, key[r]);
        const int leader = __ffs(peers) - 1;
        uint32_t q = (key[r] * 2654435761u) >> 20, at = 0;
        if (lane == leader && key[r] != kEmpty) {
            for (;; q = (q + 1u) % kHotTile) {
                const uint32_t found = atomicCAS(&slotKey[q], kEmpty, key[r]);
                if (found == kEmpty || found == key[r]) break;
            }
            at = atomicAdd(&slotCount[q], (uint32_t)__popc(peers));
        }
        slot[r] = __shfl_sync(0xFFFFFFFFu, q, leader);
        place[r] = __shfl_sync(0xFFFFFFFFu, at, leader) + (uint32_t)__popc(peers & ((1u << lane) - 1u));
    }
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < kHotTile; q += kKeyThreads)
        if (slotKey[q] != kEmpty) slotCount[q] = atomicAdd(&counts[slotKey[q]], slotCount[q]);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const int i = (int)(blockIdx.x * kHotTile) + r * kKeyThreads + (int)threadIdx.x;
        if (i >= c.n) break;
        keys[i] = key[r];
        perm[i] = slotCount[slot[r]] + place[r];
    }
}

// Clears the counts and, by its first block, looks whether few cells hold the
// particles: as many as it has threads, drawn from all parts, of which more than an
// eighth lie in the cell of another (270 to a cell; sorted particles of one cell lie too
// close together for that unless they are as many, and need no help).
__global__ void __launch_bounds__(kKeyThreads)
clear_counts_kernel(DevConsts c, const float4* pred, uint4* counts, uint32_t quads, uint32_t* hot) {
    chain_wait();
    if (blockIdx.x > 0) {
        for (uint32_t q = (blockIdx.x - 1u) * kKeyThreads + threadIdx.x; q < quads; q += (gridDim.x - 1u) * kKeyThreads)
            counts[q] = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    constexpr uint32_t kSlots = 4 * kKeyThreads;
    __shared__ uint32_t table[kSlots];
    int again = 0;
    if (c.n > kHotLeast) {
        // somewhere in its part of them: evenly spaced ones of a lattice fall into the same few rows
        const uint32_t part = (uint32_t)c.n / kKeyThreads;
        const float4 p = pred[threadIdx.x * part + ((threadIdx.x * 2654435761u) >> 8) % part];
        for (uint32_t q = threadIdx.x; q < kSlots; q += kKeyThreads) table[q] = kEmpty;
        __syncthreads();
        const uint32_t key = grid_hash(__float2int_rz(p.x / c.h), __float2int_rz(p.y / c.h), __float2int_rz(p.z / c.h), c.grid);
        for (uint32_t q = (key * 2654435761u) >> 20;; q = (q + 1u) % kSlots) {
            const uint32_t found = atomicCAS(&table[q], kEmpty, key);
            again = found == key;
            if (found == kEmpty || found == key) break;
        }
    }
    const int shared = __syncthreads_count(again);
    if (threadIdx.x == 0) *hot = shared > kKeyThreads / 8;
}

// radixsort.cl:22-37 (velocities are not permuted; they are recomputed
// before any read, update_velocities.cl:13).
// Particle ids (the original index of each record) follow the same
// permutation into idsOut.
__global__ void gather_sorted_kernel(int n, const uint32_t* perm, const float4* pos,
                                     const float4* pred, const uint32_t* ids,
                                     float4* posOut, float4* predOut,
                                     uint32_t* idsOut, int* err) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t j = checked_index(perm[i], (uint32_t)n, err, kErrSortIndex);
    posOut[i] = pos[j];
    predOut[i] = pred[j];
    idsOut[i] = ids[j];
}

// --------------------------------------------------------------- cells --
// update_cells.cl:6-25 on a table that holds END_OF_CELL_LIST everywhere.
// cellStart (may be NULL) also receives each occupied cell's first particle;
// it is never reset (taint_around checks an entry against the keys).
__global__ void update_cells_kernel(int n, const uint32_t* keys, uint32_t* cells,
                                    uint32_t keyLimit, int* err, uint32_t* cellStart) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t k = checked_index(keys[i], keyLimit, err, kErrCellKey);
    if (i > 0) {
        const uint32_t kp = checked_index(keys[i - 1], keyLimit, err, kErrCellKey);
        if (kp != k) {
            cells[2 * (size_t)k] = (uint32_t)i;
            cells[2 * (size_t)kp + 1] = (uint32_t)(i - 1);
            if (cellStart) cellStart[k] = (uint32_t)i;
        }
        if (i == n - 1) cells[2 * (size_t)k + 1] = (uint32_t)i;
    } else {
        cells[2 * (size_t)k] = 0u;
        if (cellStart) cellStart[k] = 0u;
    }
}

// reset_grid.cl:6-14
__global__ void reset_cells_kernel(int n, const uint32_t* keys, uint2* cells,
                                   uint32_t keyLimit, int* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    cells[checked_index(keys[i], keyLimit, err, kErrCellKey)] = make_uint2(kEmpty, kEmpty);
}

// Number of leading circles a pass keeps: circles are visited in order and
// skipped once processed/total exceeds the threshold (compute_scaling.cl:47-54
// with 0.6f; compute_delta.cl:97-104, apply_viscosity.cl:25-32 and
// apply_vorticity.cl:23-30 with 0.5f).  The rounded quotient of two counts of
// at most 512 exceeds 0.6f exactly when 5 processed > 3 total, and 0.5f when
// 2 processed > total: 0.6f is the float nearest 3/5, and a quotient that is
// not 3/5 differs from it by at least 1/2560.
__device__ __forceinline__ bool density_keeps(const DevConsts& c, int processed, int total) {
    return c.complete || 5 * processed <= 3 * total;
}
__device__ __forceinline__ bool others_keep(const DevConsts& c, int processed, int total) {
    return c.complete || 2 * processed <= total;
}

// The meta words (see the head of this file) of a particle whose circles'
// counts are the bytes of cnt; *dense receives the friends the density pass
// keeps.
__device__ __forceinline__ uint2 make_meta(const DevConsts& c, uint64_t cnt, int* dense) {
    const int C = c.circles;
    int total = 0;
    for (int k = 0; k < C; ++k) total += (int)byte_of(cnt, k);
    uint64_t mt = 0;
    int before = 0, keptL = 0, keptO = 0;
    *dense = 0;
    for (int k = 0; k < C; ++k) {
        const int nk = (int)byte_of(cnt, k);
        mt |= (uint64_t)nk << (7 * k);
        const bool d = density_keeps(c, before, total), o = others_keep(c, before, total);
        before += nk;
        if (d) { keptL = k + 1; *dense = before; }
        if (o) keptO = k + 1;
    }
    mt |= (uint64_t)keptL << 56 | (uint64_t)keptO << 60;
    return make_uint2((uint32_t)mt, (uint32_t)(mt >> 32));
}

// The particles of a cell, from either form of the cell table (CellTable).
struct CellTable {
    const uint2* ranges;     // first and last particle, kEmpty for none (update_cells.cl)
    const uint32_t* starts;  // or the first particle of every key, and one beyond the last
};
__device__ __forceinline__ void cell_range(const CellTable& cells, uint32_t key, int n, int* err,
                                           uint32_t& first, uint32_t& count) {
    uint32_t last;
    count = 0;
    if (cells.starts) {
        first = cells.starts[key];
        last = cells.starts[key + 1];  // one beyond
        if (first == last) return;
        --last;
    } else {
        const uint2 range = cells.ranges[key];
        first = range.x;
        last = range.y;
        if (first == kEmpty) return;
    }
    last = min(last, (uint32_t)(n - 1));
    if (first > last) atomicOr(err, kErrCellTable);
    else count = last - first + 1u;
}

// Friend `pos` of particle i in the rows.
__device__ __forceinline__ void put_friend(uint4* rows, int n, int i, int pos, uint32_t j) {
    char* entry = reinterpret_cast<char*>(rows + i) + (uint64_t)((uint32_t)pos >> 2) * (16u * (uint32_t)n);
    *reinterpret_cast<uint32_t*>(entry + 4u * ((uint32_t)pos & 3u)) = j;
}

__device__ __forceinline__ uint32_t friend_at(const uint4* rows, int n, int i, int pos) {
    const char* entry = reinterpret_cast<const char*>(rows + i) + (uint64_t)((uint32_t)pos >> 2) * (16u * (uint32_t)n);
    return *reinterpret_cast<const volatile uint32_t*>(entry + 4u * ((uint32_t)pos & 3u));  // another lane may have written it
}

// The friend circle of r^2 < h^2: min(int(adj^3 * C), C-1) with
// adj = max(0, (r - 0.3h) / 0.7h) (build_friends_list.cl:58-95), read off
// precomputed r^2 thresholds (DevConsts::circT): the same integer the sqrt /
// divide / cube / truncate sequence gives, without computing it.  Thresholds
// past C-1 are +inf.
__device__ __forceinline__ int circle_of(const DevConsts& c, float r2) {
    int circ = 0;  // the thresholds do not decrease: the last one reached counts
    if (r2 >= c.circT[0]) circ = 1;
    if (r2 >= c.circT[1]) circ = 2;
    if (r2 >= c.circT[2]) circ = 3;
    if (r2 >= c.circT[3]) circ = 4;
    if (c.circles > 5) {
        if (r2 >= c.circT[4]) circ = 5;
        if (r2 >= c.circT[5]) circ = 6;
        if (r2 >= c.circT[6]) circ = 7;
    }
    return circ;
}

// build_friends_list.cl:29-102 for particle i: one scan of the 27 neighbour
// cells in the reference's order (x, then y, then z offsets; particles of a
// cell in sorted order), self excluded, candidates read through L1 with two
// loads in flight: consider(j, r^2) for every candidate that is not out of
// reach (a NaN distance is taken, as in the reference's test).  The 27 hashes
// are formed from the three spread coordinates of each axis.
template <typename F>
__device__ __forceinline__ void scan_neighbours(const DevConsts& c, uint32_t base, const float4* pred,
                                                const CellTable& cells, int* err, int i,
                                                const float4 pi, int cx, int cy, int cz, F consider) {
    const int n = c.n;
    const bool pow2 = (c.grid & (c.grid - 1)) == 0;
    const uint32_t mask = c.grid - 1;
    const uint32_t exm = expand_bits(cx - 1), ex0 = expand_bits(cx), exp_ = expand_bits(cx + 1);
    const uint32_t eym = expand_bits(cy - 1) << 1, ey0 = expand_bits(cy) << 1, eyp = expand_bits(cy + 1) << 1;
    const uint32_t ezm = expand_bits(cz - 1) << 2, ez0 = expand_bits(cz) << 2, ezp = expand_bits(cz + 1) << 2;
    const uint32_t selfHash = pow2 ? ((ex0 | ey0 | ez0) & mask) : ((ex0 | ey0 | ez0) % c.grid);
    auto test = [&](uint32_t j, const float4 pj) {
        const float rx = pi.x - pj.x, ry = pi.y - pj.y, rz = pi.z - pj.z;
        const float r2 = dot3(rx, ry, rz, rx, ry, rz);
        if (!(r2 >= c.h2)) consider(j, r2);
    };
    auto scan = [&](uint32_t lo, uint32_t hi) {
        uint32_t j = lo;
        for (; j + 1 <= hi; j += 2) {
            const float4 p0 = pred[j], p1 = pred[j + 1];
            test(j, p0);
            test(j + 1, p1);
        }
        if (j <= hi) test(j, pred[j]);
    };
    for (int x = -1; x <= 1; ++x) {
        const uint32_t ex = x < 0 ? exm : (x > 0 ? exp_ : ex0);
        for (int y = -1; y <= 1; ++y) {
            const uint32_t exy = ex | (y < 0 ? eym : (y > 0 ? eyp : ey0));
            for (int z = -1; z <= 1; ++z) {
                const uint32_t m = exy | (z < 0 ? ezm : (z > 0 ? ezp : ez0));
                const uint32_t hm = pow2 ? (m & mask) : (m % c.grid);
                uint32_t first, count;
                cell_range(cells, base + hm, n, err, first, count);
                if (count == 0u) continue;
                const uint32_t last = first + count - 1u;
                if (hm == selfHash && first <= (uint32_t)i && (uint32_t)i <= last) {
                    // the particle's own table entry: skip itself (build_friends_list.cl:62)
                    if ((uint32_t)i > first) scan(first, (uint32_t)i - 1);
                    if ((uint32_t)i < last) scan((uint32_t)i + 1, last);
                } else {
                    scan(first, last);
                }
            }
        }
    }
}

// Moves the kept friends of particle i up from the places of their circles
// (friend q of circle k at perCircle * k + q), none past one that has yet to move.
__device__ __forceinline__ void close_up(const DevConsts& c, uint4* rows, int i, uint64_t cnt, int dense) {
    int to = (int)byte_of(cnt, 0);
    for (int k = 1; to < dense; ++k) {
        const int nk = (int)byte_of(cnt, k);
        if (to < c.perCircle * k)
            for (int q = 0; q < nk; ++q) put_friend(rows, c.n, i, to + q, friend_at(rows, c.n, i, c.perCircle * k + q));
        to += nk;
    }
}

// Particle i's friends by one thread, in one scan: they go to the places of their
// circles and are closed up when the circles' counts are known.  Circle counts
// saturate at perCircle (later candidates are dropped,
// build_friends_list.cl:79-83).
__device__ __noinline__ void friends_of_one(const DevConsts& c, uint32_t base, const float4* pred,
                                            const CellTable& cells, uint4* rows,
                                            uint2* meta, int* err, int i, const float4 pi,
                                            int cx, int cy, int cz) {
    uint64_t cnt = 0;  // 8 circles x 8-bit counters
    scan_neighbours(c, base, pred, cells, err, i, pi, cx, cy, cz, [&](uint32_t j, float r2) {
        const int k = circle_of(c, r2), have = (int)byte_of(cnt, k);
        if (have >= c.perCircle) return;
        cnt += 1ull << (8 * k);
        put_friend(rows, c.n, i, c.perCircle * k + have, j);
    });
    int dense;
    meta[i] = make_meta(c, cnt, &dense);
    close_up(c, rows, i, cnt, dense);
    for (int t = dense; t & 3; ++t) put_friend(rows, c.n, i, t, (uint32_t)i);
}

__global__ void __launch_bounds__(kMaxBlock)
build_friends_scan_kernel(const __grid_constant__ DevConsts c, Batch b, const float4* pred, CellTable cells,
                          uint4* rows, uint2* meta, int* err) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const float4 pi = pred[i];
    const int cx = __float2int_rz(pi.x / c.h), cy = __float2int_rz(pi.y / c.h), cz = __float2int_rz(pi.z / c.h);
    const uint32_t base = key_base(b, i);
    record_cell(c, i, pi, cx, cy, cz, base);
    friends_of_one(c, base, pred, cells, rows, meta, err, i, pi, cx, cy, cz);
}

// Least and largest value of a warp's lanes, NaN if any lane holds one.
__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.NaN.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
// The larger one, NaN if either is.
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

// The same rows, built by warps.  A warp takes its 32 particles run by run (a
// run: consecutive particles in one cell of one scene, which share the 27-cell
// candidate sequence).  The sequence goes to shared memory once per run, in
// order, without the candidates farther than h from the box around the run's
// members (their r^2 to every member is at least their r^2 to the box, which
// the same rounded operations form).  Then all lanes test the candidates
// against one member after another, 64 at a time, and append the accepted ones
// to a list, in order; then they sort the list by circle, which ballots over
// the thresholds of r^2 do stably, and write the member's rows.
//
// What bounds it is instruction issue.  A scan by one thread per particle
// tests 424 candidates in lockstep for each, at about 49 instructions, and
// stores friends 4 bytes at a time into rows N apart; here a member costs about
// 4 steps of 64 candidates and the sorting of its list, and its friends are
// stored 16 bytes together.  1M particles, mid-collapse: 641M -> 453M warp
// instructions, 649 -> 462 us at 81 % issue active, DRAM writes 489 -> 160 MB,
// and the density pass that used to copy the friends into rows (149 us) is one
// of the others (100 us).  Per particle the candidate sequence takes about 100
// instructions, the tests 160 and the sorting 170.  Against the scan by threads:
// 0.105 / 0.095 / 0.174 / 0.156 / 0.180 ms at 0.5 / 1 / 2 / 4 / 8 particles to a
// cell and 0.062 / 0.063 / 0.162 / 0.217 / 0.310 there (200,000 particles for the
// first two, then 500,000; sparse_scene).
// Runs with
// coordinates that are not finite take the scan.  A run with up to half as many
// candidates again as fit is split across the longest side of its box, and the
// candidates of others pass through in chunks (friends_in_chunks): at once where the
// cells hold twice as many as fit, of which a run keeps about three of four.  262,144
// particles in two colliding columns, where 560 candidates are common: a frame
// takes 0.76 ms with that line, 0.84 with chunks alone.  A substep of 400,000
// particles with 30 / 50 / 80 to a cell takes 1.61 / 2.15 / 2.74 ms (1.74 / 2.19 /
// 2.76 when the chunks wait for the first walk's count; without chunks 1.9 / 3.6 /
// 7.1; two scans by one thread each, with the passes of then, 1.69 / 2.51 / 3.33).
// A run that is a small part of what its key holds takes the walk all the same:
// 150,000 particles in 1,024 keys 1.28 ms (1.96 in chunks at once, 1.32 the scans).
// In chunks of more than 8 times as many candidates, circles at their limit take no
// part: 65,536 particles in 16 clusters of 4,096 take 1.1 ms (1.8), 32,768 in one
// cell 2.9 (5.2; the scans 4.7).
// 384 candidates leave room for 7 blocks per SM: 320 is 2 % faster on the scene
// above and 10 % slower where 560 are common, 448 is 5 % slower on the former.
constexpr int kFriendWarps = 4, kCandidates = 384, kMostFriends = 128;
struct FriendShared {
    float x[kCandidates], y[kCandidates], z[kCandidates];
    uint32_t j[kCandidates];
    uint2 list[kMostFriends + 64];  // candidate, bits of r^2
};

// Sorts the cnt <= 32 NR entries of the list by circle, at most perCircle to a
// circle (later candidates are dropped, build_friends_list.cl:79-83), and
// writes the rows of particle ip.  Returns the circles' counts, one byte each.
// The counts stay below 256, so that four bytes of a word are added, and
// summed up to each circle by one multiplication, at once.
template <int NR>
__device__ __forceinline__ uint64_t sort_friends(const DevConsts& c, const FriendShared& sh, int lane, uint32_t ltMask,
                                                 int cnt, int ip, uint4* rows) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    constexpr uint32_t kOnes = 0x01010101u;
    uint32_t j[NR], circ[NR], rank[NR];
    uint32_t lo = 0, hi = 0;  // counts of circles 0-3 and 4-7
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int e = 32 * r + lane;
        const uint2 entry = sh.list[e];
        j[r] = sh.j[e < cnt ? entry.x : 0u];
        const bool valid = e < cnt && (int)j[r] != ip;  // not itself (build_friends_list.cl:62)
        circ[r] = valid ? (uint32_t)circle_of(c, __uint_as_float(entry.y)) : 8u;
        const uint32_t peers = __match_any_sync(kFull, circ[r]);
        const uint32_t one = valid ? 1u << (8u * (circ[r] & 3u)) : 0u, one0 = circ[r] < 4u ? one : 0u;
        rank[r] = (uint32_t)__popc(peers & ltMask) + (r ? __byte_perm(lo, hi, circ[r] & 7u) & 0xFFu : 0u);
        lo += __reduce_add_sync(kFull, one0);
        hi += __reduce_add_sync(kFull, one - one0);
    }
    const uint32_t over = (127u - (uint32_t)c.perCircle) * kOnes;
    if (((lo + over) | (hi + over)) & 0x80808080u) {  // a circle is over its limit
        auto clip = [&](uint32_t w) {
            uint32_t v = 0;
            for (int k = 0; k < 4; ++k) v |= min((w >> (8 * k)) & 0xFFu, (uint32_t)c.perCircle) << (8 * k);
            return v;
        };
        lo = clip(lo);
        hi = clip(hi);
    }
    const uint32_t ends = lo * kOnes, upTo3 = ends >> 24, endsHi = (hi + upTo3) * kOnes;
    const uint32_t begins = ends << 8, beginsHi = (endsHi << 8) | upTo3;
    const int total = (int)(endsHi >> 24);
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int first = (int)__byte_perm(begins, beginsHi, circ[r] & 7u);  // the zero byte 0 fills the other bytes
        if (circ[r] < 8u && (int)rank[r] < c.perCircle && density_keeps(c, first, total))
            put_friend(rows, c.n, ip, first + (int)rank[r], j[r]);
    }
    return (uint64_t)lo | ((uint64_t)hi << 32);
}

// The same for a particle with more than kMostFriends accepted candidates: the
// shared candidates are walked twice, to count the circles and to put each
// friend in its place.
__device__ __noinline__ uint64_t sort_many_friends(const DevConsts& c, const FriendShared& sh, int lane, uint32_t ltMask,
                                                   uint32_t kept, float px, float py, float pz, int ip,
                                                   uint4* rows) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const uint32_t limit = (uint32_t)c.perCircle * 0x01010101u;
    uint32_t lo = 0, hi = 0;  // counts of circles 0-3 and 4-7, a byte each, at most perCircle
    int total = 0;
    for (int pass = 0; pass < 2; ++pass) {
        const uint64_t all = (uint64_t)lo | ((uint64_t)hi << 32);
        for (int k = 0; k < 8; ++k) total += (int)byte_of(all, k);
        lo = hi = 0;
        for (uint32_t k = 0; k < kept; k += 32) {
            const uint32_t e = k + (uint32_t)lane;
            const float rx = px - sh.x[e], ry = py - sh.y[e], rz = pz - sh.z[e];
            const float r2 = dot3(rx, ry, rz, rx, ry, rz);
            const uint32_t j = sh.j[e];
            const bool valid = e < kept && !(r2 >= c.h2) && (int)j != ip;
            const uint32_t circ = valid ? (uint32_t)circle_of(c, r2) : 8u;
            const uint32_t peers = __match_any_sync(kFull, circ);
            const int rank = __popc(peers & ltMask) + (int)(__byte_perm(lo, hi, circ & 7u) & 0xFFu);
            if (pass == 1 && valid && rank < c.perCircle) {
                int first = 0;
                for (int q = 0; q < (int)circ; ++q) first += (int)byte_of(all, q);
                if (density_keeps(c, first, total)) put_friend(rows, c.n, ip, first + rank, j);
            }
            const uint32_t one = valid ? 1u << (8u * (circ & 3u)) : 0u, one0 = circ < 4u ? one : 0u;
            lo = __vminu4(lo + __reduce_add_sync(kFull, one0), limit);
            hi = __vminu4(hi + __reduce_add_sync(kFull, one - one0), limit);
        }
    }
    return (uint64_t)lo | ((uint64_t)hi << 32);
}

// The members of a run with far more candidates than fit, which pass through shared
// memory in chunks; friends go to the places of their circles and
// are closed up at the end.  end, shift: the cells (see below).  Returns the lane's
// circle counts.
__device__ __noinline__ uint64_t friends_in_chunks(const DevConsts& c, FriendShared& sh, const float4* pred,
                                                   uint4* rows, uint32_t total, uint32_t end, uint32_t shift,
                                                   float lx, float ly, float lz, float hx, float hy, float hz,
                                                   uint32_t runMask, const float4 pi, int warpBase, uint64_t counts) {
    constexpr unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const uint32_t ltMask = (1u << lane) - 1u, limit = (uint32_t)c.perCircle * 0x01010101u;
    uint32_t kept = 0;
    int firstCell = 0;
    for (uint32_t t0 = 0; t0 < total; t0 += 32) {
        const uint32_t t = t0 + (uint32_t)lane;
        const uint32_t ending = __reduce_or_sync(kFull, end - t0 < 32u ? 1u << (end - t0) : 0u);
        const int q = firstCell + __popc(ending & (ltMask | (1u << lane)));
        firstCell += __popc(ending);
        const uint32_t j = t + __shfl_sync(kFull, shift, q);
        const float4 pj = t < total ? pred[j] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float dx = max_nan(max_nan(lx - pj.x, pj.x - hx), 0.0f), dy = max_nan(max_nan(ly - pj.y, pj.y - hy), 0.0f),
                    dz = max_nan(max_nan(lz - pj.z, pj.z - hz), 0.0f);
        const bool keep = t < total && !(dot3(dx, dy, dz, dx, dy, dz) >= c.h2);
        const uint32_t km = __ballot_sync(kFull, keep);
        if (keep) {
            const uint32_t pos = kept + (uint32_t)__popc(km & ltMask);
            sh.x[pos] = pj.x;
            sh.y[pos] = pj.y;
            sh.z[pos] = pj.z;
            sh.j[pos] = j;
        }
        kept += (uint32_t)__popc(km);
        if (t0 + 32u < total && kept + 32u <= (uint32_t)kCandidates) continue;
        for (uint32_t e = kept + (uint32_t)lane; e < ((kept + 63u) & ~63u); e += 32) {
            sh.x[e] = __int_as_float(0x7F800000);
            sh.y[e] = sh.z[e] = 0.0f;
        }
        __syncwarp();
        for (uint32_t rm = runMask; rm; rm &= rm - 1u) {
            const int pl = __ffs(rm) - 1, ip = warpBase + pl;
            const F2 px = both(__shfl_sync(kFull, pi.x, pl)), py = both(__shfl_sync(kFull, pi.y, pl)),
                     pz = both(__shfl_sync(kFull, pi.z, pl));
            uint32_t lo = __shfl_sync(kFull, (uint32_t)counts, pl), hi = __shfl_sync(kFull, (uint32_t)(counts >> 32), pl);
            int cnt = 0;
            uint32_t full = 0;  // of many chunks most candidates belong to circles that take no more
            if (total > 8u * (uint32_t)kCandidates)
                for (int k = 0; k < 8; ++k) full |= (__byte_perm(lo, hi, k) & 0xFFu) == (uint32_t)c.perCircle ? 1u << k : 0u;
            for (uint32_t k = 0; k < kept; k += 64) {
                const uint32_t e = k + 2u * (uint32_t)lane;
                const F2 rx = sub2(px, load2(sh.x + e)), ry = sub2(py, load2(sh.y + e)), rz = sub2(pz, load2(sh.z + e));
                const float2 r2 = unpack2(dot2(c, rx, ry, rz, rx, ry, rz));
                bool a0 = !(r2.x >= c.h2), a1 = !(r2.y >= c.h2);
                if (full) {
                    a0 = a0 && !((full >> circle_of(c, r2.x)) & 1u);
                    a1 = a1 && !((full >> circle_of(c, r2.y)) & 1u);
                }
                const uint32_t m0 = __ballot_sync(kFull, a0), m1 = __ballot_sync(kFull, a1);
                const int pos = cnt + __popc(m0 & ltMask) + __popc(m1 & ltMask);
                if (a0) sh.list[pos] = make_uint2(e, __float_as_uint(r2.x));
                if (a1) sh.list[pos + (a0 ? 1 : 0)] = make_uint2(e + 1u, __float_as_uint(r2.y));
                cnt += __popc(m0) + __popc(m1);
                if (cnt <= kMostFriends && k + 64u < kept) continue;
                __syncwarp();
                for (int r = 0; r < cnt; r += 32) {
                    const uint2 entry = sh.list[r + lane];
                    const uint32_t friendOf = sh.j[r + lane < cnt ? entry.x : 0u];
                    const bool valid = r + lane < cnt && (int)friendOf != ip;
                    const uint32_t circ = valid ? (uint32_t)circle_of(c, __uint_as_float(entry.y)) : 8u;
                    const uint32_t peers = __match_any_sync(kFull, circ);
                    const int rank = __popc(peers & ltMask) + (int)(__byte_perm(lo, hi, circ & 7u) & 0xFFu);
                    if (valid && rank < c.perCircle) put_friend(rows, c.n, ip, c.perCircle * (int)circ + rank, friendOf);
                    const uint32_t one = valid ? 1u << (8u * (circ & 3u)) : 0u, one0 = circ < 4u ? one : 0u;
                    lo = __vminu4(lo + __reduce_add_sync(kFull, one0), limit);
                    hi = __vminu4(hi + __reduce_add_sync(kFull, one - one0), limit);
                }
                cnt = 0;
                __syncwarp();  // the list is read before it is written again
            }
            if (lane == pl) counts = (uint64_t)lo | ((uint64_t)hi << 32);
        }
        __syncwarp();
        kept = 0;
    }
    return counts;
}

// Whether the scene's runs have fewer than two members on average (sample_runs),
// because cells hold few or many cells share a key: a warp then takes a run for every
// particle or two, and the scan by threads is the faster one.  A substep of 1M random
// particles at 0.5 / 1 / 1.5 / 2 / 3 to a cell of space takes 736 / 784 / 787 / 797 /
// 809 us by warps and 563 / 661 / 728 by threads up to 1.5 (4M at 0.5 / 1 / 2: 3,983 /
// 4,092 / 3,834 and 2,606 / 2,988 / 3,408); two scans by one thread each, with the
// passes of then, took 704 / 776 / - / 894 / 985 (3,516 / 3,703 / 3,845).  The friends
// of 3M dense particles in 2^16 keys: 8.0 ms and 6.9.  Decided for single warps it is
// slower: the few of a dense scene take 30 to 70 us after all others have ended.
// Dense scenes pay 3 us a substep for the question.
__device__ __forceinline__ bool sparse_scene(const DevConsts& c) {
    return 2u * c.epoch[1] > kSampleBlocks * 256u;
}

// The friends of a sparse scene by one thread each, where build_friends_kernel<32>
// leaves them; an idle launch (about 1.5 us) in others.
__global__ void __launch_bounds__(kBlock, 6)
build_friends_sparse_kernel(const __grid_constant__ DevConsts c, Batch b, const float4* pred, CellTable cells, uint4* rows,
                            uint2* meta, int* err) {
    chain_wait();
    if (!sparse_scene(c)) return;
    __shared__ uint32_t tile;
    while (true) {  // tiles of particles, from a counter: they differ in cost
        __syncthreads();
        if (threadIdx.x == 0) tile = atomicAdd(c.epoch + 2, 1u);
        __syncthreads();
        if (tile * kBlock >= (uint32_t)c.n) return;
        const int i = (int)(tile * kBlock + threadIdx.x);
        if (i >= c.n) continue;
        const float4 pi = pred[i];
        const int cx = __float2int_rz(pi.x / c.h), cy = __float2int_rz(pi.y / c.h), cz = __float2int_rz(pi.z / c.h);
        friends_of_one(c, key_base(b, i), pred, cells, rows, meta, err, i, pi, cx, cy, cz);
    }
}

// W particles to a warp: 32, or fewer where that leaves the chip without warps
// (a warp takes its members one after another).
template <int W>
__global__ void __launch_bounds__(32 * kFriendWarps)
build_friends_kernel(const __grid_constant__ DevConsts c, Batch b, const float4* pred, CellTable cells,
                     uint4* rows, uint2* meta, int* err) {
    chain_wait();
    constexpr unsigned kFull = 0xFFFFFFFFu;
    __shared__ FriendShared shared[kFriendWarps];
    FriendShared& sh = shared[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int warpBase = (int)(blockIdx.x * kFriendWarps + (threadIdx.x >> 5)) * W;
    const int i = warpBase + lane;
    const int n = c.n;
    if (warpBase >= n) return;  // whole warp idle
    const bool valid = lane < W && i < n;
    const bool sparse = W == 32 && c.n >= kSparseLeast && sparse_scene(c);  // read beside the position
    const float4 pi = valid ? pred[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int cx = __float2int_rz(pi.x / c.h), cy = __float2int_rz(pi.y / c.h), cz = __float2int_rz(pi.z / c.h);
    const uint32_t base = valid ? key_base(b, i) : 0u;
    if (valid) record_cell(c, i, pi, cx, cy, cz, base);
    if (W == 32 && sparse) return;
    const bool pow2 = (c.grid & (c.grid - 1)) == 0;
    const uint32_t gmask = c.grid - 1;
    const int ux = __shfl_up_sync(kFull, cx, 1), uy = __shfl_up_sync(kFull, cy, 1), uz = __shfl_up_sync(kFull, cz, 1);
    const uint32_t ub = __shfl_up_sync(kFull, base, 1);
    const bool head = valid && (lane == 0 || cx != ux || cy != uy || cz != uz || base != ub);
    uint32_t heads = __ballot_sync(kFull, head);
    const uint32_t validMask = __ballot_sync(kFull, valid);
    const uint32_t ltMask = (1u << lane) - 1u;
    const float inf = __int_as_float(0x7F800000);
    uint32_t scan = 0;   // lanes whose particles take the scan
    uint64_t counts = 0; // this lane's particle: its circles' counts
    uint32_t spread = 0; // lanes whose particles' friends are at the places of their circles
    uint32_t now = 0, later = 0;  // the parts of a split run: the one to do next, and the rest
    while (heads | now | later) {
        uint32_t runMask = now;
        if (now == 0 && later == 0) {
            const uint32_t first = heads & (0u - heads);
            heads ^= first;
            runMask = validMask & (heads ? (heads & (0u - heads)) - 1u : kFull) & ~(first - 1u);
        } else if (now == 0) {
            runMask = later;
            later = 0;
        }
        now = 0;
        const int h0 = __ffs(runMask) - 1;
        const bool member = (runMask >> lane) & 1u;
        const float lx = warp_min(member ? pi.x : inf), ly = warp_min(member ? pi.y : inf), lz = warp_min(member ? pi.z : inf);
        const float hx = warp_max(member ? pi.x : -inf), hy = warp_max(member ? pi.y : -inf), hz = warp_max(member ? pi.z : -inf);
        const float sum = (lx + hx) + (ly + hy) + (lz + hz);
        if (!(fabsf(sum) < inf)) {
            scan |= runMask;
            continue;
        }
        const int rx0 = __shfl_sync(kFull, cx, h0), ry0 = __shfl_sync(kFull, cy, h0), rz0 = __shfl_sync(kFull, cz, h0);
        const uint32_t rbase = __shfl_sync(kFull, base, h0);
        // lane q < 27: neighbour cell q in the scan order (x, then y, then z offsets)
        uint32_t start = 0, count = 0;
        if (lane < 27) {
            const int x = lane / 9 - 1, y = (lane / 3) % 3 - 1, z = lane % 3 - 1;
            const uint32_t m = expand_bits(rx0 + x) | (expand_bits(ry0 + y) << 1) | (expand_bits(rz0 + z) << 2);
            cell_range(cells, rbase + (pow2 ? (m & gmask) : (m % c.grid)), n, err, start, count);
        }
        uint32_t end = count;  // inclusive scan: candidates up to and including cell q
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(kFull, end, d);
            if (lane >= d) end += v;
        }
        const uint32_t total = __shfl_sync(kFull, end, 31);
        // the cells that hold any, in order: candidate t of the q-th is particle t + shift
        const uint32_t occupied = __ballot_sync(kFull, count > 0u);
        if (count > 0u) sh.list[__popc(occupied & ltMask)] = make_uint2(end, start - (end - count));
        __syncwarp();
        const uint2 cell = sh.list[lane];
        end = lane < __popc(occupied) ? cell.x : 0xFFFFFFFFu;
        const uint32_t shift = cell.y;
        __syncwarp();
        // cells this full keep about three of four, too many to split, unless it is other cells' particles that fill their keys
        if (total > 2u * (uint32_t)kCandidates && 2 * __popc(runMask) >= (int)min(__shfl_sync(kFull, count, 13), (uint32_t)W)) {
            counts = friends_in_chunks(c, sh, pred, rows, total, end, shift, lx, ly, lz, hx, hy, hz, runMask, pi, warpBase, counts);
            spread |= runMask;
            continue;
        }
        uint32_t kept = 0;
        int firstCell = 0;  // of candidate t0
        for (uint32_t t0 = 0; t0 < total; t0 += 32) {
            const uint32_t t = t0 + (uint32_t)lane;
            // bit l: a cell ends at candidate t0 + l
            const uint32_t ending = __reduce_or_sync(kFull, end - t0 < 32u ? 1u << (end - t0) : 0u);
            const int q = firstCell + __popc(ending & (ltMask | (1u << lane)));
            firstCell += __popc(ending);
            const uint32_t j = t + __shfl_sync(kFull, shift, q);
            const float4 pj = t < total ? pred[j] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float dx = max_nan(max_nan(lx - pj.x, pj.x - hx), 0.0f), dy = max_nan(max_nan(ly - pj.y, pj.y - hy), 0.0f),
                        dz = max_nan(max_nan(lz - pj.z, pj.z - hz), 0.0f);
            const bool keep = t < total && !(dot3(dx, dy, dz, dx, dy, dz) >= c.h2);
            const uint32_t km = __ballot_sync(kFull, keep);
            const uint32_t pos = kept + (uint32_t)__popc(km & ltMask);
            if (keep && pos < (uint32_t)kCandidates) {
                sh.x[pos] = pj.x;
                sh.y[pos] = pj.y;
                sh.z[pos] = pj.z;
                sh.j[pos] = j;
            }
            kept += (uint32_t)__popc(km);
        }
        if (kept > (uint32_t)kCandidates) {
            // the members on one side of the box's middle first, across its longest side
            const float ex = hx - lx, ey = hy - ly, ez = hz - lz;
            const bool low = ex >= ey && ex >= ez ? pi.x < lx + 0.5f * ex : ey >= ez ? pi.y < ly + 0.5f * ey : pi.z < lz + 0.5f * ez;
            uint32_t part = __ballot_sync(kFull, member && low);
            if (part == 0u || part == runMask) part = runMask & (0u - runMask);
            if (2u * kept > 3u * (uint32_t)kCandidates || part == runMask) {  // too many for that, or a single member
                counts = friends_in_chunks(c, sh, pred, rows, total, end, shift, lx, ly, lz, hx, hy, hz, runMask, pi, warpBase, counts);
                spread |= runMask;
            } else {
                now = part;
                later |= runMask & ~part;
            }
            continue;
        }
        for (uint32_t e = kept + (uint32_t)lane; e < ((kept + 63u) & ~63u); e += 32) {  // up to a step of 64: out of reach
            sh.x[e] = inf;
            sh.y[e] = sh.z[e] = 0.0f;
        }
        __syncwarp();
        for (uint32_t rm = runMask; rm; rm &= rm - 1u) {
            const int pl = __ffs(rm) - 1;
            const F2 px = both(__shfl_sync(kFull, pi.x, pl)), py = both(__shfl_sync(kFull, pi.y, pl)),
                     pz = both(__shfl_sync(kFull, pi.z, pl));
            int cnt = 0;
            for (uint32_t k = 0; k < kept && cnt <= kMostFriends; k += 64) {
                const uint32_t e = k + 2u * (uint32_t)lane;
                const F2 rx = sub2(px, load2(sh.x + e)), ry = sub2(py, load2(sh.y + e)), rz = sub2(pz, load2(sh.z + e));
                const float2 r2 = unpack2(dot2(c, rx, ry, rz, rx, ry, rz));
                const bool a0 = !(r2.x >= c.h2), a1 = !(r2.y >= c.h2);  // a NaN distance is taken, as in the scan
                const uint32_t m0 = __ballot_sync(kFull, a0), m1 = __ballot_sync(kFull, a1);
                const int pos = cnt + __popc(m0 & ltMask) + __popc(m1 & ltMask);
                if (a0) sh.list[pos] = make_uint2(e, __float_as_uint(r2.x));
                if (a1) sh.list[pos + (a0 ? 1 : 0)] = make_uint2(e + 1u, __float_as_uint(r2.y));
                cnt += __popc(m0) + __popc(m1);
            }
            __syncwarp();
            const int ip = warpBase + pl;
            uint64_t mine = 0;
            if (cnt <= 32) mine = sort_friends<1>(c, sh, lane, ltMask, cnt, ip, rows);
            else if (cnt <= 64) mine = sort_friends<2>(c, sh, lane, ltMask, cnt, ip, rows);
            else if (cnt <= 96) mine = sort_friends<3>(c, sh, lane, ltMask, cnt, ip, rows);
            else if (cnt <= kMostFriends) mine = sort_friends<4>(c, sh, lane, ltMask, cnt, ip, rows);
            else mine = sort_many_friends(c, sh, lane, ltMask, kept, unpack2(px).x, unpack2(py).x, unpack2(pz).x, ip, rows);
            if (lane == pl) counts = mine;
            __syncwarp();  // the list is read before the next member's is written
        }
    }
    __syncwarp();  // spread friends are read by the lane that closes them up
    if (!valid) return;
    if ((scan >> lane) & 1u) {
        friends_of_one(c, base, pred, cells, rows, meta, err, i, pi, cx, cy, cz);
        return;
    }
    int dense;
    meta[i] = make_meta(c, counts, &dense);
    if ((spread >> lane) & 1u) close_up(c, rows, i, counts, dense);
    for (int t = dense; t & 3; ++t) put_friend(rows, n, i, t, (uint32_t)i);
}

// ------------------------------------------------- balanced thread map --
// The block's particles handed to its threads in decreasing order of their
// friend count, so that the lanes of a warp walk lists of similar length;
// a particle's result does not depend on which thread computes it.  Counting
// sort in shared memory over the kept-circle count (saturated at 255), ties
// in any order.  Every thread of the block must call it (it synchronises);
// returns the particle index, or -1 for threads beyond the block's particles.
__device__ __forceinline__ int balanced_particle(const uint2* meta, int n, bool densityPass, int tile) {
    __shared__ uint32_t bins[256];
    __shared__ int order[kMaxBlock];
    const int t = threadIdx.x;
    const int i = tile * blockDim.x + t;
    for (int k = t; k < 256; k += blockDim.x) bins[k] = 0u;
    __syncthreads();
    int key = -1;
    if (i < n) {
        const uint64_t mt = load_meta(meta, i);
        const int kept = densityPass ? kept_density(mt) : kept_other(mt);
        int tot = 0;
        for (int c = 0; c < kept; ++c) tot += (int)circle_count(mt, c);
        key = 255 - min(tot, 255);
        atomicAdd(&bins[key], 1u);
    }
    __syncthreads();
    if (t < 32) {  // exclusive scan of the 256 bins: 8 per lane
        uint32_t v[8], s = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) { v[k] = bins[8 * t + k]; s += v[k]; }
        uint32_t incl = s;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (t >= d) incl += u;
        }
        uint32_t run = incl - s;
#pragma unroll
        for (int k = 0; k < 8; ++k) { bins[8 * t + k] = run; run += v[k]; }
    }
    __syncthreads();
    if (key >= 0) order[atomicAdd(&bins[key], 1u)] = i;
    __syncthreads();
    const int valid = min(n - tile * (int)blockDim.x, (int)blockDim.x);
    return t < valid ? order[t] : -1;
}

// Registers of the solver passes.  __launch_bounds__(512) makes the compiler
// aim at the occupancy of 512-thread blocks and schedule the loads of a step
// late; a register limit without it does not.  1M particles, two substeps:
// density pass 0.835 ms with the bounds, 0.787 / 0.771 / 0.772 with limits of
// 56 / 64 / 96; XSPH 0.259, 0.252 with 72; vorticity 0.190, 0.175 with 56; the
// position pass 0.792, 0.797 / 0.794 with 56 / 64, so it keeps the bounds.
// Limits below 52 spill and are slower.  512 threads of 72 registers fit an SM.

// ---------------------------------------------------- tiles of a launch --
// A launch covers `tiles` tiles of blockDim particles.  With tiles == 0, one
// block per tile (tile = blockIdx.x).  Otherwise a persistent grid of at
// most the resident blocks takes the tiles in order from counter[0], one
// atomic per tile, so busy SMs take fewer tiles; no block waits on another.
// The last block to find the tiles exhausted resets counter[0] and
// counter[1] to 0 for the next launch on the stream.  Every thread of a
// block runs every tile the block takes (the balanced thread map
// synchronises).
template <typename F>
__device__ __forceinline__ void for_tiles(int tiles, int* counter, F body) {
    if (tiles == 0) {
        body((int)blockIdx.x);
        return;
    }
    __shared__ int nextTile;
    while (true) {
        if (threadIdx.x == 0) nextTile = atomicAdd(&counter[0], 1);
        __syncthreads();
        const int t = nextTile;
        __syncthreads();
        if (t >= tiles) break;
        body(t);
    }
    if (threadIdx.x == 0 && atomicAdd(&counter[1], 1) == (int)gridDim.x - 1) {
        counter[0] = 0;
        counter[1] = 0;
    }
}

// -------------------------------------------------------------- scaling --
// Relaxed variants (R = true, relaxedMath): per pair one reciprocal square
// root w = 1/|r| replaces sqrt(r^2) and the divisions by |r|, and sums are
// fused multiply-adds: the reference's kernels as its own
// -cl-fast-relaxed-math -cl-mad-enable build may evaluate them.
// Spiky gradient magnitude over |r|: (h - |r|)^2 / |r| with |r| = r^2 w.  The
// scalar operations of each friend are those named here, packed for two.
__device__ __forceinline__ F2 spiky_over_r2(const DevConsts& c, F2 r2, F2& w) {
    const float2 r = unpack2(r2);
    w = pack2(rsqrtf(r.x), rsqrtf(r.y));
    const F2 hr = fma2(neg2(r2), w, both(c.h));
    return mul2(mul2(hr, hr), w);
}

// compute_scaling.cl:27-112 followed by pack_data.cl (w = lambda).  Q: the
// exact quotients by |r| through one reciprocal (quotient_rn).
template <bool R, bool Q, int L>
__device__ __forceinline__ void compute_scaling_body(const DevConsts& c, const float4* pred,
                                                     float4* predPacked, float* density,
                                                     float4* tapeSums, float* tapeRho,
                                                     const uint4* rows, int i, uint4 head, const float4 pi, uint64_t mt) {
    const int n = c.n;
    // complete neighbour sets count the particle itself first: d = h^2 - 0
    float ds = c.complete ? c.h2 * c.h2 * c.h2 : 0.0f, gsk = 0.0f, gx = 0.0f, gy = 0.0f, gz = 0.0f;
    auto load = [&](uint32_t j) { return pred[checked_index(j, (uint32_t)n, c.err, kErrFriendIndex)]; };
    auto one = [&](float rx, float ry, float rz, float r2) {  // a friend in support, divided the IEEE way
        const float rl = sqrtf(r2);
        const float hr = c.h - rl;
        const float sc = c.gradSpiky * hr * hr;
        const float g0 = (sc * rx) / rl, g1 = (sc * ry) / rl, g2 = (sc * rz) / rl;
        const float d = c.h2 - r2;
        ds = ds + d * d * d;
        gsk = gsk + dot3(g0, g1, g2, g0, g1, g2);
        gx = gx + g0;
        gy = gy + g1;
        gz = gz + g2;
    };
    constexpr bool kLaneSums = L > 1 && Q && !R;  // the other forms go in_turn
    __shared__ __align__(16) float terms[kLaneSums ? kMaxBlock / L * LaneSums<L, 5>::kStride : 1];
    LaneSums<L, 5> sums(terms, {ds, gsk, gx, gy, gz});
    auto pass = [&](auto from) { ds = from(ds); gsk = from(gsk); gx = from(gx); gy = from(gy); gz = from(gz); };
    walk_pairs<L>(rows, n, i, head, FlatFriends(mt, kept_density(mt)).total, load, [&](const float4& pa, const float4& pb, bool va, bool vb) {
        const F2 rx = pack2(pi.x - pa.x, pi.x - pb.x), ry = pack2(pi.y - pa.y, pi.y - pb.y),
                 rz = pack2(pi.z - pa.z, pi.z - pb.z);
        const F2 r2 = R ? fma2(rz, rz, fma2(ry, ry, mul2(rx, rx))) : dot2(c, rx, ry, rz, rx, ry, rz);
        const float2 s2 = unpack2(r2);
        va = va && in_support(c, s2.x);
        vb = vb && in_support(c, s2.y);
        if (!R && !Q) {
            const float2 x = unpack2(rx), y = unpack2(ry), z = unpack2(rz);
            in_turn<L>([&] {
                if (va) one(x.x, y.x, z.x, s2.x);
                if (vb) one(x.y, y.y, z.y, s2.y);
            }, pass);
            return;
        }
        F2 g0, g1, g2;
        if (R) {
            F2 w;
            const F2 s = mul2(both(c.gradSpiky), spiky_over_r2(c, r2, w));
            g0 = mul2(s, rx);
            g1 = mul2(s, ry);
            g2 = mul2(s, rz);
        } else {
            F2 nrl, y;
            sqrt_recip_rn2(r2, nrl, y);
            const F2 hr = add2(both(c.h), nrl);
            const F2 sc = mul2(mul2(both(c.gradSpiky), hr), hr);
            g0 = quotient_rn2(mul2(sc, rx), nrl, y);
            g1 = quotient_rn2(mul2(sc, ry), nrl, y);
            g2 = quotient_rn2(mul2(sc, rz), nrl, y);
        }
        const F2 d = sub2(both(c.h2), r2);
        const float2 x = unpack2(g0), y = unpack2(g1), z = unpack2(g2);
        if (R) {
            const float2 dd = unpack2(mul2(d, d)), d1 = unpack2(d);
            in_turn<L>([&] {
                if (va) {
                    ds = fmaf(dd.x, d1.x, ds);
                    gsk = fmaf(z.x, z.x, fmaf(y.x, y.x, fmaf(x.x, x.x, gsk)));
                    gx += x.x; gy += y.x; gz += z.x;
                }
                if (vb) {
                    ds = fmaf(dd.y, d1.y, ds);
                    gsk = fmaf(z.y, z.y, fmaf(y.y, y.y, fmaf(x.y, x.y, gsk)));
                    gx += x.y; gy += y.y; gz += z.y;
                }
            }, pass);
        } else {
            const float2 d3 = unpack2(mul2(mul2(d, d), d)), gg = unpack2(dot2(c, g0, g1, g2, g0, g1, g2));
            if constexpr (kLaneSums) {
                sums.add(va, vb, {d3, gg, x, y, z});
                return;
            }
            in_turn<L>([&] {
                if (va) {
                    ds = ds + d3.x;
                    gsk = gsk + gg.x;
                    gx = gx + x.x; gy = gy + y.x; gz = gz + z.x;
                }
                if (vb) {
                    ds = ds + d3.y;
                    gsk = gsk + gg.y;
                    gx = gx + x.y; gy = gy + y.y; gz = gz + z.y;
                }
            }, pass);
        }
    });
    if constexpr (kLaneSums) {
        ds = sums.template get<0>();
        gsk = sums.template get<1>();
        gx = sums.template get<2>();
        gy = sums.template get<3>();
        gz = sums.template get<4>();
    }
    if (threadIdx.x % L) return;  // the sums are the first lane's
    ds = ds * c.poly6;
    density[i] = ds;
    gsk = gsk + dot3(gx, gy, gz, gx, gy, gz);
    if (tapeSums) {
        tapeSums[i] = make_float4(gx, gy, gz, gsk);
        tapeRho[i] = ds;
    }
    const float constraint = (ds / c.rho0) - 1.0f;
    const float lambda = -1.0f * constraint / (gsk / c.rho0sq + c.eps);
    predPacked[i] = make_float4(pi.x, pi.y, pi.z, lambda);
}

template <bool R, bool B, int L>
__global__ void __maxnreg__(64)
compute_scaling_kernel(const __grid_constant__ DevConsts c, const float4* pred, float4* predPacked,
                       float* density, float4* tapeSums, float* tapeRho,
                       const uint2* meta, const uint4* rows, int tiles, int* tileCounter) {
    chain_wait();
    for_tiles(tiles, tileCounter, [&](int tile) {
        const int i = B ? balanced_particle(meta, c.n, true, tile) : (tile * (int)blockDim.x + (int)threadIdx.x) / L;
        if (i < 0 || i >= c.n) return;
        const float4 pi = pred[i];
        const uint4 head = first_entry<L>(rows, c.n, i);
        const uint64_t mt = load_meta(meta, i);
        // a particle that may hold a friend at an irregular position divides the IEEE way
        if (!R && c.quotients && !quotients_tainted<L>(c, i)) compute_scaling_body<R, true, L>(c, pred, predPacked, density, tapeSums, tapeRho, rows, i, head, pi, mt);
        else compute_scaling_body<R, false, L>(c, pred, predPacked, density, tapeSums, tapeRho, rows, i, head, pi, mt);
    });
}

// update_velocities.cl:11-14 (the GL texture write is dropped) for particle i
// at its final prediction p, from its position q.  Also moves the sorted
// particle ids back to their fixed buffer.
__device__ __forceinline__ void end_of_step(const DevConsts& c, const StepEnd& end, int i, const float4& p, const float4& q) {
    if (end.idsIn) end.idsOut[i] = end.idsIn[i];
    float4 v = end.vel[i];
    v.x = (p.x - q.x) / c.dt;
    v.y = (p.y - q.y) / c.dt;
    v.z = (p.z - q.z) / c.dt;
    end.vel[i] = v;
    if (end.tapeP) {
        end.tapeP[i] = p;
        end.tapeV[i] = v;
    }
    end.posOut[i] = make_float4(p.x, p.y, p.z, sqrtf(dot3(v.x, v.y, v.z, v.x, v.y, v.z)));
}

// ---------------------------------------------------------------- delta --
// compute_delta.cl:54-185 (force planes: identity for an all-zero mask) with
// the optional box clamp on `future`, then update_predicted.cl.  After the
// last iteration w carries the density (pack_data.cl with the density source,
// src/Simulation.cpp:591), and the velocities are updated there as well
// (end.posOut), which saves a launch and the prediction's way through memory.
template <bool R, bool Q, int L>
__device__ __forceinline__ void compute_delta_body(const DevConsts& c, const Batch& b, const float4* pp,
                                                   const float4* posPrev, const StepEnd& end,
                                                   float4* predOut,
                                                   const float* density, int lastIteration,
                                                   uint8_t* clampMask, const uint4* rows,
                                                   int i, uint4 head, const float4 pi, uint64_t mt) {
    const int n = c.n;
    float sx = 0.0f, sy = 0.0f, sz = 0.0f;
    auto load = [&](uint32_t j) { return pp[checked_index(j, (uint32_t)n, c.err, kErrFriendIndex)]; };
    auto one = [&](float rx, float ry, float rz, float r2, float wj) {  // a friend in support, divided the IEEE way
        const float rl = sqrtf(r2);
        const float hr = c.h - rl;
        const float g0 = (rx / rl) * hr * hr, g1 = (ry / rl) * hr * hr, g2 = (rz / rl) * hr * hr;
        const float d = c.h2 - r2;
        const float p6 = d * d * d;
        const float rq = p6 / c.poly6q;
        const float scorr = c.K * rq * rq * rq * rq;
        const float a = pi.w + wj + scorr;
        sx = sx + a * g0;
        sy = sy + a * g1;
        sz = sz + a * g2;
    };
    constexpr bool kLaneSums = L > 1 && Q && !R;  // the other forms go in_turn
    __shared__ __align__(16) float terms[kLaneSums ? kMaxBlock / L * LaneSums<L, 3>::kStride : 1];
    LaneSums<L, 3> sums(terms, {0.0f, 0.0f, 0.0f});
    auto pass = [&](auto from) { sx = from(sx); sy = from(sy); sz = from(sz); };
    walk_pairs<L>(rows, n, i, head, FlatFriends(mt, kept_other(mt)).total, load, [&](const float4& pa, const float4& pb, bool va, bool vb) {
        const F2 rx = pack2(pi.x - pa.x, pi.x - pb.x), ry = pack2(pi.y - pa.y, pi.y - pb.y),
                 rz = pack2(pi.z - pa.z, pi.z - pb.z);
        const F2 r2 = R ? fma2(rz, rz, fma2(ry, ry, mul2(rx, rx))) : dot2(c, rx, ry, rz, rx, ry, rz);
        const float2 s2 = unpack2(r2);
        va = va && in_support(c, s2.x);
        vb = vb && in_support(c, s2.y);
        if (!R && !Q) {
            const float2 x = unpack2(rx), y = unpack2(ry), z = unpack2(rz);
            in_turn<L>([&] {
                if (va) one(x.x, y.x, z.x, s2.x, pa.w);
                if (vb) one(x.y, y.y, z.y, s2.y, pb.w);
            }, pass);
            return;
        }
        const F2 d = sub2(both(c.h2), r2);
        const F2 p6 = mul2(mul2(d, d), d);
        const F2 wij = pack2(pi.w + pa.w, pi.w + pb.w);
        if (R) {
            F2 w;
            const F2 k = spiky_over_r2(c, r2, w);
            const F2 rq = mul2(p6, both(c.invPoly6q));
            const F2 rq2 = mul2(rq, rq);
            const float2 a = unpack2(mul2(fma2(mul2(both(c.K), rq2), rq2, wij), k));
            const float2 x = unpack2(rx), y = unpack2(ry), z = unpack2(rz);
            in_turn<L>([&] {
                if (va) { sx = fmaf(a.x, x.x, sx); sy = fmaf(a.x, y.x, sy); sz = fmaf(a.x, z.x, sz); }
                if (vb) { sx = fmaf(a.y, x.y, sx); sy = fmaf(a.y, y.y, sy); sz = fmaf(a.y, z.y, sz); }
            }, pass);
        } else {
            F2 nrl, y;
            sqrt_recip_rn2(r2, nrl, y);
            const F2 hr = add2(both(c.h), nrl);
            const F2 g0 = mul2(mul2(quotient_rn2(rx, nrl, y), hr), hr), g1 = mul2(mul2(quotient_rn2(ry, nrl, y), hr), hr),
                     g2 = mul2(mul2(quotient_rn2(rz, nrl, y), hr), hr);
            F2 rq;
            if (c.quotientPoly6q) {
                rq = quotient_rn2(p6, both(-c.poly6q), both(c.recipPoly6q));
            } else {
                const float2 p = unpack2(p6);
                rq = pack2(p.x / c.poly6q, p.y / c.poly6q);
            }
            const F2 a = add2(wij, product2(c, mul2(mul2(mul2(both(c.K), rq), rq), rq), rq));
            const float2 x = unpack2(mul2(a, g0)), v = unpack2(mul2(a, g1)), z = unpack2(mul2(a, g2));
            if constexpr (kLaneSums) {
                sums.add(va, vb, {x, v, z});
                return;
            }
            in_turn<L>([&] {
                if (va) { sx = sx + x.x; sy = sy + v.x; sz = sz + z.x; }
                if (vb) { sx = sx + x.y; sy = sy + v.y; sz = sz + z.y; }
            }, pass);
        }
    });
    if constexpr (kLaneSums) {
        sx = sums.template get<0>();
        sy = sums.template get<1>();
        sz = sums.template get<2>();
    }
    if (threadIdx.x % L) return;  // the sums are the first lane's
    float fx, fy, fz;
    if (R) {
        fx = fmaf(c.dpScale, sx, pi.x);
        fy = fmaf(c.dpScale, sy, pi.y);
        fz = fmaf(c.dpScale, sz, pi.z);
    } else {
        fx = pi.x + (c.negGradSpiky * sx) / c.rho0;
        fy = pi.y + (c.negGradSpiky * sy) / c.rho0;
        fz = pi.z + (c.negGradSpiky * sz) / c.rho0;
    }
    if (c.nquads > 0) {  // force planes, in order (compute_delta.cl:157-182)
        const float4 prev = posPrev[i];
        const float edge = plane_edge_offset(c, fx, fy, fz);
        for (int q = 0; q < c.nquads; ++q) bounce_point_quad(c, c.quads[q], prev.x, prev.y, prev.z, fx, fy, fz, edge);
    }
    if (c.clamp) {
        const float* lo = c.lo;
        const float* hi = c.hi;
        if (b.scenes) {
            const SceneParams& sp = b.scenes[b.sceneOf[i]];
            lo = sp.lo;
            hi = sp.hi;
        }
        // the wave generator's moving wall: xMin + wavePos (pbf_set_wave_position)
        const float lx = c.wave ? lo[0] + *c.wave : lo[0];
        if (clampMask)  // which coordinates the clamp moves: 2 bits per axis, 1 low, 2 high
            clampMask[i] = (uint8_t)((fx < lx ? 1 : (fx > hi[0] ? 2 : 0)) | (fy < lo[1] ? 4 : (fy > hi[1] ? 8 : 0)) |
                                     (fz < lo[2] ? 16 : (fz > hi[2] ? 32 : 0)));
        fx = fx < lx ? lx : (fx > hi[0] ? hi[0] : fx);
        fy = fy < lo[1] ? lo[1] : (fy > hi[1] ? hi[1] : fy);
        fz = fz < lo[2] ? lo[2] : (fz > hi[2] ? hi[2] : fz);
    } else if (clampMask) {
        clampMask[i] = 0;
    }
    const float dx = fx - pi.x, dy = fy - pi.y, dz = fz - pi.z;
    const float4 out = make_float4(pi.x + dx, pi.y + dy, pi.z + dz, lastIteration ? density[i] : pi.w + 0.0f);
    predOut[i] = out;
    if (!R) note_position(c, i, out.x, out.y, out.z);
    if (end.posOut) end_of_step(c, end, i, out, posPrev[i]);
}

template <bool R, bool B, int L>
__global__ void __launch_bounds__(kMaxBlock)
compute_delta_kernel(const __grid_constant__ DevConsts c, Batch b, const float4* pp, const float4* posPrev,
                     StepEnd end, float4* predOut, const float* density,
                     const uint2* meta, int lastIteration, uint8_t* clampMask,
                     const uint4* rows, int tiles, int* tileCounter) {
    chain_wait();
    for_tiles(tiles, tileCounter, [&](int tile) {
        const int i = B ? balanced_particle(meta, c.n, false, tile) : (tile * (int)blockDim.x + (int)threadIdx.x) / L;
        if (i < 0 || i >= c.n) return;
        const float4 pi = pp[i];
        const uint4 head = first_entry<L>(rows, c.n, i);
        const uint64_t mt = load_meta(meta, i);
        // a particle that may hold a friend at an irregular position divides the IEEE way
        if (!R && c.quotients && !quotients_tainted<L>(c, i)) compute_delta_body<R, true, L>(c, b, pp, posPrev, end, predOut, density, lastIteration, clampMask, rows, i, head, pi, mt);
        else compute_delta_body<R, false, L>(c, b, pp, posPrev, end, predOut, density, lastIteration, clampMask, rows, i, head, pi, mt);
    });
}

// ----------------------------------------------------------- velocities --
// The end of a step without solver iterations.
__global__ void update_velocities_kernel(DevConsts c, StepEnd end, const float4* pred,
                                         const float4* posIn) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < c.n) end_of_step(c, end, i, pred[i], posIn[i]);
}

// apply_viscosity.cl:12-86, every neighbour read from the pre-pass
// velocities (Jacobi).  near receives the one record that the vorticity pass
// reads of a neighbour: its position and |omega| (as apply_vorticity.cl:55
// forms it for each neighbour), with x = infinity, which is out of every
// support, where the neighbour's density is too small to count
// (apply_vorticity.cl:44).  The vorticity pass was bound by the L1 wavefronts
// of its two gathers per friend (79 %); with one it takes 0.191 ms instead of
// 0.214 (1M particles, mid-collapse, two substeps).
template <bool R, bool Q, int L>
__device__ __forceinline__ void apply_viscosity_body(const DevConsts& c, const Batch& b, const float4* pred,
                                                     const float4* velIn, float4* velOut,
                                                     float4* omega, float4* near,
                                                     const uint4* rows, int i, uint4 head, const float4 pi,
                                                     const float4 vi, uint64_t mt) {
    const int n = c.n;
    float vsx = 0.0f, vsy = 0.0f, vsz = 0.0f, ox = 0.0f, oy = 0.0f, oz = 0.0f;
    auto load = [&](uint32_t j) { j = checked_index(j, (uint32_t)n, c.err, kErrFriendIndex); return PairRec{pred[j], velIn[j]}; };
    constexpr bool kLaneSums = L > 1 && Q && !R;  // the other forms go in_turn
    __shared__ __align__(16) float terms[kLaneSums ? kMaxBlock / L * LaneSums<L, 6>::kStride : 1];
    LaneSums<L, 6> sums(terms, {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f});
    auto pass = [&](auto from) { ox = from(ox); oy = from(oy); oz = from(oz); vsx = from(vsx); vsy = from(vsy); vsz = from(vsz); };
    walk_pairs<L, true>(rows, n, i, head, FlatFriends(mt, kept_other(mt)).total, load, [&](const PairRec& qa, const PairRec& qb, bool va, bool vb) {
        const float4 pa = qa.a, pb = qb.a;
        const F2 rx = pack2(pi.x - pa.x, pi.x - pb.x), ry = pack2(pi.y - pa.y, pi.y - pb.y),
                 rz = pack2(pi.z - pa.z, pi.z - pb.z);
        const F2 r2 = dot2(c, rx, ry, rz, rx, ry, rz);
        const float2 s2 = unpack2(r2);
        va = va && in_support(c, s2.x) && fabsf(pa.w) > 1e-8f;
        vb = vb && in_support(c, s2.y) && fabsf(pb.w) > 1e-8f;
        const F2 ux = pack2(qa.b.x - vi.x, qb.b.x - vi.x), uy = pack2(qa.b.y - vi.y, qb.b.y - vi.y),
                 uz = pack2(qa.b.z - vi.z, qb.b.z - vi.z);
        F2 g0, g1, g2;
        if (R) {
            F2 w;
            const F2 k = spiky_over_r2(c, r2, w);
            g0 = mul2(k, rx);
            g1 = mul2(k, ry);
            g2 = mul2(k, rz);
        } else if (Q) {
            F2 nrl, y;
            sqrt_recip_rn2(r2, nrl, y);
            const F2 hr = add2(both(c.h), nrl);
            g0 = mul2(mul2(quotient_rn2(rx, nrl, y), hr), hr);
            g1 = mul2(mul2(quotient_rn2(ry, nrl, y), hr), hr);
            g2 = mul2(mul2(quotient_rn2(rz, nrl, y), hr), hr);
        } else {
            const float la = sqrtf(s2.x), lb = sqrtf(s2.y);
            const F2 hr = pack2(c.h - la, c.h - lb);
            const float2 x = unpack2(rx), y = unpack2(ry), z = unpack2(rz);
            g0 = mul2(mul2(pack2(x.x / la, x.y / lb), hr), hr);
            g1 = mul2(mul2(pack2(y.x / la, y.y / lb), hr), hr);
            g2 = mul2(mul2(pack2(z.x / la, z.y / lb), hr), hr);
        }
        const F2 d = sub2(both(c.h2), r2);
        const F2 d3 = mul2(mul2(d, d), d);
        if (R) {
            const float2 x = unpack2(fma2(uy, g2, neg2(mul2(uz, g1)))), y = unpack2(fma2(uz, g0, neg2(mul2(ux, g2)))),
                         z = unpack2(fma2(ux, g1, neg2(mul2(uy, g0)))), t = unpack2(d3), a0 = unpack2(ux),
                         a1 = unpack2(uy), a2 = unpack2(uz);
            in_turn<L>([&] {
                if (va) {
                    ox += x.x; oy += y.x; oz += z.x;
                    vsx = fmaf(a0.x, t.x, vsx); vsy = fmaf(a1.x, t.x, vsy); vsz = fmaf(a2.x, t.x, vsz);
                }
                if (vb) {
                    ox += x.y; oy += y.y; oz += z.y;
                    vsx = fmaf(a0.y, t.y, vsx); vsy = fmaf(a1.y, t.y, vsy); vsz = fmaf(a2.y, t.y, vsz);
                }
            }, pass);
        } else {
            const float2 p0 = unpack2(mul2(uy, g2)), p1 = unpack2(mul2(uz, g0)), p2 = unpack2(mul2(ux, g1)),
                         q0 = unpack2(mul2(uz, g1)), q1 = unpack2(mul2(ux, g2)), q2 = unpack2(mul2(uy, g0)),
                         a0 = unpack2(mul2(ux, d3)), a1 = unpack2(mul2(uy, d3)), a2 = unpack2(mul2(uz, d3));
            if constexpr (kLaneSums) {
                sums.add(va, vb, {make_float2(p0.x - q0.x, p0.y - q0.y), make_float2(p1.x - q1.x, p1.y - q1.y),
                                  make_float2(p2.x - q2.x, p2.y - q2.y), a0, a1, a2});
                return;
            }
            in_turn<L>([&] {
                if (va) {
                    ox = ox + (p0.x - q0.x); oy = oy + (p1.x - q1.x); oz = oz + (p2.x - q2.x);
                    vsx = vsx + a0.x; vsy = vsy + a1.x; vsz = vsz + a2.x;
                }
                if (vb) {
                    ox = ox + (p0.y - q0.y); oy = oy + (p1.y - q1.y); oz = oz + (p2.y - q2.y);
                    vsx = vsx + a0.y; vsy = vsy + a1.y; vsz = vsz + a2.y;
                }
            }, pass);
        }
    });
    if constexpr (kLaneSums) {
        ox = sums.template get<0>();
        oy = sums.template get<1>();
        oz = sums.template get<2>();
        vsx = sums.template get<3>();
        vsy = sums.template get<4>();
        vsz = sums.template get<5>();
    }
    if (threadIdx.x % L) return;  // the sums are the first lane's
    vsx = vsx * c.poly6;
    vsy = vsy * c.poly6;
    vsz = vsz * c.poly6;
    const float visc = b.scenes ? b.scenes[b.sceneOf[i]].visc : c.visc;
    velOut[i] = make_float4(vi.x + visc * vsx, vi.y + visc * vsy, vi.z + visc * vsz, vi.w + visc * 0.0f);
    const float wx = ox * c.negGradSpiky, wy = oy * c.negGradSpiky, wz = oz * c.negGradSpiky;
    float size;
    if (R) {
        const float o2 = fmaf(wz, wz, fmaf(wy, wy, wx * wx));
        size = o2 > 0.0f ? o2 * rsqrtf(o2) : 0.0f;
    } else {
        size = sqrtf(dot3(wx, wy, wz, wx, wy, wz));
    }
    omega[i] = make_float4(wx, wy, wz, size);
    near[i] = make_float4(fabsf(pi.w) > 1e-8f ? pi.x : __int_as_float(0x7F800000), pi.y, pi.z, size);
}

template <bool R, bool B, int L>
__global__ void __maxnreg__(72)
apply_viscosity_kernel(const __grid_constant__ DevConsts c, Batch b, const float4* pred, const float4* velIn,
                       float4* velOut, float4* omega, float4* near,
                       const uint2* meta, const uint4* rows, int tiles, int* tileCounter) {
    chain_wait();
    for_tiles(tiles, tileCounter, [&](int tile) {
        const int i = B ? balanced_particle(meta, c.n, false, tile) : (tile * (int)blockDim.x + (int)threadIdx.x) / L;
        if (i < 0 || i >= c.n) return;
        const float4 pi = pred[i], vi = velIn[i];
        const uint4 head = first_entry<L>(rows, c.n, i);
        const uint64_t mt = load_meta(meta, i);
        // a particle that may hold a friend at an irregular position divides the IEEE way
        if (!R && c.quotients && !quotients_tainted<L>(c, i)) apply_viscosity_body<R, true, L>(c, b, pred, velIn, velOut, omega, near, rows, i, head, pi, vi, mt);
        else apply_viscosity_body<R, false, L>(c, b, pred, velIn, velOut, omega, near, rows, i, head, pi, vi, mt);
    });
}

// apply_vorticity.cl:12-86; neighbours are read from near (apply_viscosity).
template <bool R, bool Q, int L>
__device__ __forceinline__ void apply_vorticity_body(const DevConsts& c, const float4* near,
                                                     const float4* omega,
                                                     const float4* velIn, float4* velOut,
                                                     const uint4* rows, int i,
                                                     uint4 head, const float4 pi, uint64_t mt) {
    const int n = c.n;
    float ex = 0.0f, ey = 0.0f, ez = 0.0f;
    auto load = [&](uint32_t j) { return near[checked_index(j, (uint32_t)n, c.err, kErrFriendIndex)]; };
    constexpr bool kLaneSums = L > 1 && Q && !R;  // the other forms go in_turn
    __shared__ __align__(16) float terms[kLaneSums ? kMaxBlock / L * LaneSums<L, 3>::kStride : 1];
    LaneSums<L, 3> sums(terms, {0.0f, 0.0f, 0.0f});
    auto pass = [&](auto from) { ex = from(ex); ey = from(ey); ez = from(ez); };
    walk_pairs<L>(rows, n, i, head, FlatFriends(mt, kept_other(mt)).total, load, [&](const float4& pa, const float4& pb, bool va, bool vb) {
        const F2 rx = pack2(pi.x - pa.x, pi.x - pb.x), ry = pack2(pi.y - pa.y, pi.y - pb.y),
                 rz = pack2(pi.z - pa.z, pi.z - pb.z);
        const F2 r2 = dot2(c, rx, ry, rz, rx, ry, rz);
        const float2 s2 = unpack2(r2);
        va = va && in_support(c, s2.x);
        vb = vb && in_support(c, s2.y);
        if (R) {
            F2 w;
            const float2 k = unpack2(spiky_over_r2(c, r2, w)), x = unpack2(rx), y = unpack2(ry), z = unpack2(rz);
            auto add = [&](float ol, float kj, float x1, float y1, float z1) {
                const float s = ol > 0.0f ? ol * kj : 0.0f;
                ex = fmaf(s, x1, ex);
                ey = fmaf(s, y1, ey);
                ez = fmaf(s, z1, ez);
            };
            in_turn<L>([&] {
                if (va) add(pa.w, k.x, x.x, y.x, z.x);
                if (vb) add(pb.w, k.y, x.y, y.y, z.y);
            }, pass);
        } else {
            F2 g0, g1, g2;
            if (Q) {
                F2 nrl, y;
                sqrt_recip_rn2(r2, nrl, y);
                const F2 hr = add2(both(c.h), nrl);
                g0 = mul2(mul2(quotient_rn2(rx, nrl, y), hr), hr);
                g1 = mul2(mul2(quotient_rn2(ry, nrl, y), hr), hr);
                g2 = mul2(mul2(quotient_rn2(rz, nrl, y), hr), hr);
            } else {
                const float la = sqrtf(s2.x), lb = sqrtf(s2.y);
                const F2 hr = pack2(c.h - la, c.h - lb);
                const float2 x = unpack2(rx), y = unpack2(ry), z = unpack2(rz);
                g0 = mul2(mul2(pack2(x.x / la, x.y / lb), hr), hr);
                g1 = mul2(mul2(pack2(y.x / la, y.y / lb), hr), hr);
                g2 = mul2(mul2(pack2(z.x / la, z.y / lb), hr), hr);
            }
            const F2 ol = pack2(pa.w, pb.w);
            const float2 x = unpack2(mul2(ol, g0)), y = unpack2(mul2(ol, g1)), z = unpack2(mul2(ol, g2));
            if constexpr (kLaneSums) {
                sums.add(va, vb, {x, y, z});
                return;
            }
            in_turn<L>([&] {
                if (va) { ex = ex + x.x; ey = ey + y.x; ez = ez + z.x; }
                if (vb) { ex = ex + x.y; ey = ey + y.y; ez = ez + z.y; }
            }, pass);
        }
    });
    if constexpr (kLaneSums) {
        ex = sums.template get<0>();
        ey = sums.template get<1>();
        ez = sums.template get<2>();
    }
    if (threadIdx.x % L) return;  // the sums are the first lane's
    ex = ex * c.negGradSpiky;
    ey = ey * c.negGradSpiky;
    ez = ez * c.negGradSpiky;
    if (R) {
        const float l2 = fmaf(ez, ez, fmaf(ey, ey, ex * ex));
        if (l2 > 0.0f) {
            const float w = rsqrtf(l2);
            ex *= w;
            ey *= w;
            ez *= w;
        }
    } else {
        const float l = sqrtf(dot3(ex, ey, ez, ex, ey, ez));
        if (l > 0.0f) {
            ex = ex / l;
            ey = ey / l;
            ez = ez / l;
        }
    }
    const float4 oi = omega[i];
    const float fx = c.vort * (ey * oi.z - ez * oi.y);
    const float fy = c.vort * (ez * oi.x - ex * oi.z);
    const float fz = c.vort * (ex * oi.y - ey * oi.x);
    const float4 v = velIn[i];
    velOut[i] = make_float4(v.x + fx * c.dt, v.y + fy * c.dt, v.z + fz * c.dt, v.w + 0.0f);
}

template <bool R, bool B, int L>
__global__ void __maxnreg__(56)
apply_vorticity_kernel(const __grid_constant__ DevConsts c, const float4* pred, const float4* near,
                       const float4* omega, const float4* velIn, float4* velOut,
                       const uint2* meta,
                       const uint4* rows, int tiles, int* tileCounter, int tileOffset) {
    chain_wait();
    for_tiles(tiles, tileCounter, [&](int tile) {
        tile += tileOffset * L;  // a launch over part of the tiles (L blocks per tile)
        const int i = B ? balanced_particle(meta, c.n, false, tile) : (tile * (int)blockDim.x + (int)threadIdx.x) / L;
        if (i < 0 || i >= c.n) return;
        const float4 pi = pred[i];
        const uint4 head = first_entry<L>(rows, c.n, i);
        const uint64_t mt = load_meta(meta, i);
        // a particle that may hold a friend at an irregular position divides the IEEE way
        if (!R && c.quotients && !quotients_tainted<L>(c, i)) apply_vorticity_body<R, true, L>(c, near, omega, velIn, velOut, rows, i, head, pi, mt);
        else apply_vorticity_body<R, false, L>(c, near, omega, velIn, velOut, rows, i, head, pi, mt);
    });
}

}  // namespace

// ------------------------------------------------------------- launchers --
void launch_predict_keys(const DevConsts& c, Batch b, const float4* pos, float4* vel, float4* pred, uint32_t* keys,
                         uint32_t* perm, uint32_t* counts, int paused, cudaStream_t s) {
    launch_chained(predict_keys_kernel, blocks_for(c.n), kBlock, s, c, b, pos, vel, pred, keys, perm, counts, paused);
}

void launch_compute_keys(const DevConsts& c, Batch b, const float4* pred, uint32_t* keys, uint32_t* perm, uint32_t* counts,
                         const uint32_t* hot, cudaStream_t s) {
    if (hot) launch_chained(compute_keys_kernel<kKeyThreads>, blocks_for(c.n, kKeyThreads), kKeyThreads, s, c, b, pred, keys, perm, counts, hot);
    else launch_chained(compute_keys_kernel<kBlock>, blocks_for(c.n), kBlock, s, c, b, pred, keys, perm, counts, hot);
}

void launch_clear_counts(const DevConsts& c, const float4* pred, uint32_t* counts, size_t words, uint32_t* hot, cudaStream_t s) {
    const uint32_t quads = (uint32_t)(words / 4);
    launch_chained(clear_counts_kernel, 1u + min((quads + kKeyThreads - 1) / kKeyThreads, 303u), kKeyThreads, s, c, pred,
                   reinterpret_cast<uint4*>(counts), quads, hot);
}

void launch_gather_sorted(int n, const uint32_t* perm, const float4* pos, const float4* pred, const uint32_t* ids,
                          float4* posOut, float4* predOut, uint32_t* idsOut, int* err, cudaStream_t s) {
    launch_chained(gather_sorted_kernel, blocks_for(n), kBlock, s, n, perm, pos, pred, ids, posOut, predOut, idsOut, err);
}

void launch_update_cells(int n, const uint32_t* keys, uint32_t* cells, uint32_t keyLimit, int* err, cudaStream_t s,
                         uint32_t* cellStart) {
    update_cells_kernel<<<blocks_for(n), kBlock, 0, s>>>(n, keys, cells, keyLimit, err, cellStart);
}

void launch_reset_cells(int n, const uint32_t* keys, uint32_t* cells, uint32_t keyLimit, int* err, cudaStream_t s) {
    reset_cells_kernel<<<blocks_for(n), kBlock, 0, s>>>(n, keys, reinterpret_cast<uint2*>(cells), keyLimit, err);
}

// Lanes that share a particle in a solver pass (walk_pairs).  A substep of 2,048
// / 4,096 / 8,192 / 16,384 / 24,576 / 32,768 particles takes 68 / 77 / 86 / 99 /
// 102 / 109 us with one lane, 54 / 60 / 66 / 84 / 96 / 112 with four and 52 / 57 /
// 68 / 96 / 118 / 136 with eight: beyond, the chip is full, and what the lanes
// exchange costs more than the shorter chains save.  Relaxed sums go in turns: 60 /
// 68 / 75 / 85 / 86 / 89 us with one lane, 56 / 63 / 68 / 82 / 95 / 118 with four.
int lanes_per_particle(const DevConsts& c, int balance, const int* tileCounter) {
    if (balance || tileCounter) return 1;
    if (c.relaxed) return c.n <= 16384 ? 4 : 1;
    return c.n <= 4096 ? 8 : c.n <= 24576 ? 4 : 1;
}

// Grid of a neighbour pass: one block per tile of `block` particles, or
// (persistent) at most as many blocks as the device keeps resident, which
// then take the tiles from a counter (*tiles receives their count; 0 for one
// block per tile).  A launcher's tileCounter (two words, zero between
// launches) selects the persistent grid; NULL, one block per tile.
template <typename K>
unsigned grid_for_tiles(K kernel, int n, int block, bool persistent, int* tiles) {
    const unsigned all = blocks_for(n, block);
    *tiles = 0;
    if (!persistent) return all;  // no tile counter: one block per tile
    static int sms[64] = {};  // per device, filled on first use
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return all;
    if (!sms[dev]) cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
    int resident = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, block, 0) != cudaSuccess || resident < 1 ||
        sms[dev] < 1) {
        cudaGetLastError();
        return all;
    }
    const unsigned cap = (unsigned)resident * (unsigned)sms[dev];
    if (all <= cap) return all;
    *tiles = (int)all;
    return cap;
}

int launch_build_friends(const DevConsts& c, Batch b, const float4* pred, const uint32_t* cells,
                          const uint32_t* starts, uint4* rows, uint2* meta, int* errorWord, int block, int algorithm,
                          cudaStream_t s) {
    const CellTable table{reinterpret_cast<const uint2*>(cells), starts};
    if (algorithm == 1) {
        launch_chained(build_friends_scan_kernel, blocks_for(c.n, block), block, s, c, b, pred, table, rows, meta, errorWord);
        return 1;
    }
    // a substep of 1,024 / 2,048 / 4,096 / 8,192 particles takes 43 / 48 / 54 / 68 us with one particle to a warp,
    // 46 / 52 / 56 / 66 with 4 (nothing else fills the chip, and a warp takes its members one after another);
    // friends of 2,048 / 16,384 / 65,536 / 131,072 / 262,144 particles, us: 13 / 20 / 45 / 81 / 152 with 4 to a
    // warp, 17 / 23 / 38 / 65 / 120 with 8, 22 / 32 / 38 / 58 / 105 with 16, 34 / 41 / 47 / 63 / 104 with 32
    const int w = c.n <= 4096 ? 1 : c.n <= 16384 ? 4 : c.n <= 49152 ? 8 : c.n <= 196608 ? 16 : 32;
    auto k = w == 1 ? build_friends_kernel<1> : w == 4 ? build_friends_kernel<4> : w == 8 ? build_friends_kernel<8> : w == 16 ? build_friends_kernel<16> : build_friends_kernel<32>;
    launch_chained(k, blocks_for(c.n, w * kFriendWarps), 32 * kFriendWarps, s, c, b, pred, table, rows, meta, errorWord);
    if (c.n < kSparseLeast) return 1;
    launch_chained(build_friends_sparse_kernel, 912u, kBlock, s, c, b, pred, table, rows, meta, errorWord);
    return 2;
}

void launch_compute_scaling(const DevConsts& c, const float4* pred, float4* predPacked, float* density,
                            float4* tapeSums, float* tapeRho, const uint2* meta, const uint4* rows, int block, int balance, int* tileCounter,
                            cudaStream_t s) {
    const int lanes = lanes_per_particle(c, balance, tileCounter);
    auto k = c.relaxed ? (lanes > 1 ? compute_scaling_kernel<true, false, 4> : balance ? compute_scaling_kernel<true, true, 1> : compute_scaling_kernel<true, false, 1>)
                       : (lanes == 8 ? compute_scaling_kernel<false, false, 8> : lanes == 4 ? compute_scaling_kernel<false, false, 4> : balance ? compute_scaling_kernel<false, true, 1> : compute_scaling_kernel<false, false, 1>);
    int tiles = 0;
    const unsigned grid = grid_for_tiles(k, c.n * lanes, block, tileCounter != nullptr, &tiles);
    launch_chained(k, grid, block, s, c, pred, predPacked, density, tapeSums, tapeRho, meta, rows, tiles, tileCounter);
}

void launch_compute_delta(const DevConsts& c, Batch b, const float4* predPacked, const float4* posPrev,
                          const StepEnd& end, float4* predOut, const float* density, const uint2* meta, int lastIteration,
                          uint8_t* clampMask, const uint4* rows, int block, int balance, int* tileCounter,
                          cudaStream_t s) {
    const int lanes = lanes_per_particle(c, balance, tileCounter);
    auto k = c.relaxed ? (lanes > 1 ? compute_delta_kernel<true, false, 4> : balance ? compute_delta_kernel<true, true, 1> : compute_delta_kernel<true, false, 1>)
                       : (lanes == 8 ? compute_delta_kernel<false, false, 8> : lanes == 4 ? compute_delta_kernel<false, false, 4> : balance ? compute_delta_kernel<false, true, 1> : compute_delta_kernel<false, false, 1>);
    int tiles = 0;
    const unsigned grid = grid_for_tiles(k, c.n * lanes, block, tileCounter != nullptr, &tiles);
    launch_chained(k, grid, block, s, c, b, predPacked, posPrev, end, predOut, density, meta, lastIteration, clampMask, rows, tiles,
                             tileCounter);
}

void launch_update_velocities(const DevConsts& c, const StepEnd& end, const float4* pred, const float4* posIn,
                              cudaStream_t s) {
    update_velocities_kernel<<<blocks_for(c.n), kBlock, 0, s>>>(c, end, pred, posIn);
}

void launch_apply_viscosity(const DevConsts& c, Batch b, const float4* pred, const float4* velIn, float4* velOut,
                            float4* omega, float4* near, const uint2* meta, const uint4* rows, int block, int balance,
                            int* tileCounter, cudaStream_t s) {
    const int lanes = lanes_per_particle(c, balance, tileCounter);
    auto k = c.relaxed ? (lanes > 1 ? apply_viscosity_kernel<true, false, 4> : balance ? apply_viscosity_kernel<true, true, 1> : apply_viscosity_kernel<true, false, 1>)
                       : (lanes == 8 ? apply_viscosity_kernel<false, false, 8> : lanes == 4 ? apply_viscosity_kernel<false, false, 4> : balance ? apply_viscosity_kernel<false, true, 1> : apply_viscosity_kernel<false, false, 1>);
    int tiles = 0;
    const unsigned grid = grid_for_tiles(k, c.n * lanes, block, tileCounter != nullptr, &tiles);
    launch_chained(k, grid, block, s, c, b, pred, velIn, velOut, omega, near, meta, rows, tiles, tileCounter);
}

void launch_apply_vorticity(const DevConsts& c, const float4* pred, const float4* near, const float4* omega,
                            const float4* velIn, float4* velOut, const uint2* meta, const uint4* rows, int block, int balance,
                            int* tileCounter, cudaStream_t s, int firstTile, int tileCount) {
    const int lanes = lanes_per_particle(c, balance, tileCounter);
    auto k = c.relaxed ? (lanes > 1 ? apply_vorticity_kernel<true, false, 4> : balance ? apply_vorticity_kernel<true, true, 1> : apply_vorticity_kernel<true, false, 1>)
                       : (lanes == 8 ? apply_vorticity_kernel<false, false, 8> : lanes == 4 ? apply_vorticity_kernel<false, false, 4> : balance ? apply_vorticity_kernel<false, true, 1> : apply_vorticity_kernel<false, false, 1>);
    if (tileCount > 0) {  // tiles [firstTile, firstTile + tileCount), one block each
        launch_chained(k, (unsigned)(tileCount * lanes), block, s, c, pred, near, omega, velIn, velOut, meta, rows, 0, nullptr, firstTile);
        return;
    }
    int tiles = 0;
    const unsigned grid = grid_for_tiles(k, c.n * lanes, block, tileCounter != nullptr, &tiles);
    launch_chained(k, grid, block, s, c, pred, near, omega, velIn, velOut, meta, rows, tiles, tileCounter, 0);
}

}  // namespace pbf
