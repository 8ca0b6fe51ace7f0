// pbf_internal.h — declarations shared by the library's translation units.
#pragma once

#include <cstdint>
#include <string>

#include "pbf_capi.h"

#include <cuda_runtime.h>

namespace pbf {

// Constants every solver kernel reads, formed once on the host from the
// parameters (src/Simulation.cpp:169-183 bakes the same values into the
// OpenCL build as -D literals).
// One force plane with its per-plane constants formed on the host
// (compute_delta.cl:3-9): a, b, c, invdet = 1.0 / (a c - b b) taken in
// double and rounded once (the literal 1.0 is a double), and
// planeNorm = normalize(cross(E0, E1)) as cross / sqrt(dot).
struct QuadDev {
    float B[3], E0[3], E1[3], n[3];
    float a, b, c, invdet;
    int maskYOffset, maskHeight;
};

// Bits of the device error word (pbf_synchronize reports it).
constexpr int kErrCellTable = 1;    // a cell range that runs backwards
constexpr int kErrFriendIndex = 2;  // a friend-list entry >= N (bounds-checked builds)
constexpr int kErrSortIndex = 4;    // a permutation entry >= N (bounds-checked builds)
constexpr int kErrCellKey = 8;      // a key beyond the cell table (bounds-checked builds)

struct DevConsts {
    float dt, h, h2, minR, hMinusMinR;
    float poly6, gradSpiky, negGradSpiky, poly6q;
    float rho0, rho0sq, eps, K, visc, vort;
    float gx, gy, gz;
    float lo[3], hi[3];
    int clamp, guard;
    int relaxed;                 // relaxedMath: the neighbour passes' relaxed variants
    int complete;                // completeNeighbours: all circles in every pass, self in the density
    int nquads, maskW, maskH;    // force planes (pbf_set_force_quads) and their mask
    const QuadDev* quads;
    const uint32_t* mask;        // NULL: the empty mask
    const float* wave;           // device scalar: the moving wall's offset from xMin (NULL: none)
    int* err;                    // the context's error word (bounds-checked builds record bad indices there)
    float dpScale, invPoly6q;    // -gradSpiky / rho0 and 1 / poly6q (relaxed variants only)
    // Exact passes: quotients by |r| and by poly6q through a reciprocal and
    // one remainder correction (quotient_rn, sqrt_recip_rn), where the
    // parameters keep every numerator and quotient in the range that makes it
    // equal to IEEE division (make_consts decides), for the particles whose
    // friends all sit at regular positions (quotients_tainted).
    int quotients;               // divisions by |r| in the four neighbour passes
    int quotientPoly6q;          // the s_corr division by poly6q in the position pass
    float recipPoly6q;           // RN(1 / poly6q)
    uint32_t* epoch;             // device words: the substep's number, counted by the predict kernel, the runs of
                                 // same-cell particles among those that the counting sort samples (kSparseLeast), and
                                 // the tiles that the scan of a sparse scene has taken
    uint32_t* taint;             // per particle: the last substep that tainted it (quotients_tainted)
    int4* cellXYZ;               // per particle: the cell its friends were taken around, and the scene's first key
                                 // (NULL in relaxed mode: nothing is tainted)
    const uint32_t* cellStart;   // per cell key: its first particle, when the substep's keys confirm it
    const uint32_t* keys;        // the substep's sorted cell keys (set per substep)
    unsigned long long negZero2; // two floats -0 (product2 in pbf_device.cuh)
    int circles, perCircle;
    uint32_t grid;
    int n;
    // circT[k-1]: the smallest r^2 whose friend circle is >= k (k = 1..C-1),
    // +inf where no r^2 < h^2 reaches circle k.  The circle of r^2 is the
    // number of thresholds it reaches.
    float circT[PBF_MAX_CIRCLES];
};

// Records `msg` as the last error of `ctx` (or of the calling thread when ctx
// is NULL) and returns `code`.
int fail(pbf_ctx* ctx, int code, const std::string& msg);

DevConsts make_consts(const PbfParameters& p, int n);

// The values that may differ between the scenes of a batch.  A batch keeps
// all scenes in one particle array; scene s owns a fixed index range (its
// keys are offset by s * gridBufSize, so the stable sort never moves a
// particle out of it) and sceneOf[i] names the scene of particle i.
struct SceneParams {
    float gx, gy, gz;
    float lo[3], hi[3];
    float visc;
    uint32_t keyBase;  // s * gridBufSize
    uint32_t pad;
};
// scenes == nullptr: a single scene whose values are those of DevConsts.
struct Batch {
    const SceneParams* scenes;
    const uint16_t* sceneOf;
    int nscenes = 0;
};
SceneParams make_scene_params(const PbfParameters& p, uint32_t keyBase);

// Threads per block of the kernels whose block size the autotuner chooses.
struct LaunchShape {
    int friends = 256, scaling = 256, delta = 256, viscosity = 256, vorticity = 256;
    int friendsAlgorithm = 0;  // 1: one thread scans per particle; else: built by warps, run by run
    int balance = 0;           // solver passes: threads take the block's particles by friend count
    int persistent = 0;        // the four solver passes: a grid of the resident blocks takes
                               // the particle tiles from a counter (no waits between blocks)
};
constexpr int kMaxBlock = 512;
// Particles from which on a substep that sorts by counting looks whether the scene is
// sparse (sparse_scene): an idle launch more, and below the build by warps is no slower
// than the two scans that it replaced (200,000 at 0.5 to a cell 207 us a substep and
// 224; 500,000 404 and 393).  kSampleBlocks x 256 particles are asked.
constexpr int kSparseLeast = 600000;
constexpr uint32_t kSampleBlocks = 32;

// Launches a kernel of the substep's chain: it may start before the kernel
// before it on the stream has ended, and waits for that one's end itself
// (chain_wait in pbf_device.cuh) before it touches memory.
template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t s, A&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// ---- kernels (pbf_kernels.cu) ----
// counts (may be NULL): the number of particles of each key is added up there,
// and perm receives each particle's place of arrival among them instead of its
// own index (launch_compute_keys too).
void launch_predict_keys(const DevConsts& c, Batch b, const float4* pos, float4* vel, float4* pred,
                         uint32_t* keys, uint32_t* perm, uint32_t* counts, int paused, cudaStream_t s);
// hot: NULL, or the word that launch_clear_counts set.
void launch_compute_keys(const DevConsts& c, Batch b, const float4* pred, uint32_t* keys, uint32_t* perm, uint32_t* counts,
                         const uint32_t* hot, cudaStream_t s);
// Clears the counts (words: a multiple of 4) before launch_compute_keys, and tells
// in *hot whether few cells hold most of the particles of this single scene.
void launch_clear_counts(const DevConsts& c, const float4* pred, uint32_t* counts, size_t words, uint32_t* hot, cudaStream_t s);
// err (may be NULL): the error word that bounds-checked builds report bad
// permutation entries or keys to; keyLimit: the number of cell-table entries.
void launch_gather_sorted(int n, const uint32_t* perm, const float4* pos, const float4* pred, const uint32_t* ids,
                          float4* posOut, float4* predOut, uint32_t* idsOut, int* err, cudaStream_t s);
// cellStart (may be NULL): also each occupied cell's first particle.
void launch_update_cells(int n, const uint32_t* keys, uint32_t* cells, uint32_t keyLimit, int* err, cudaStream_t s,
                         uint32_t* cellStart = nullptr);
void launch_reset_cells(int n, const uint32_t* keys, uint32_t* cells, uint32_t keyLimit, int* err, cudaStream_t s);
// tileCounter (two device words, zero between launches; NULL for one block
// per tile of particles): the solver passes' persistent grid, whose
// blocks take the tiles from it (LaunchShape::persistent).
// Writes the rows (walk_pairs in pbf_device.cuh) and meta.  algorithm:
// LaunchShape::friendsAlgorithm; block is the scan's.
// The cells come as ranges (launch_update_cells) or, where starts is given, as
// the first index of every key and one beyond the last.  Returns the launches.
int launch_build_friends(const DevConsts& c, Batch b, const float4* pred, const uint32_t* cells,
                          const uint32_t* starts, uint4* rows, uint2* meta, int* errorWord, int block, int algorithm,
                          cudaStream_t s);
// uint4 entries per particle of the rows for `slots` friends, at least the four
// that eight lanes read ahead (first_entry in pbf_device.cuh).
inline size_t row_entries(int slots) { return slots > 16 ? ((size_t)slots + 3) / 4 : 4; }
// tapeSums, tapeRho below: a rollout's tape (AdjointTape; NULL without).
void launch_compute_scaling(const DevConsts& c, const float4* pred, float4* predPacked, float* density,
                            float4* tapeSums, float* tapeRho, const uint2* meta, const uint4* rows, int block, int balance, int* tileCounter,
                            cudaStream_t s);
// What the last position pass of a substep also writes: the new positions and
// velocities, and the particle ids (idsIn NULL: they stay); for a rollout's tape
// (NULL without one) the final predictions and the velocities again.  posOut
// NULL: not the last pass.
struct StepEnd {
    float4* posOut = nullptr;
    float4* vel = nullptr;
    const uint32_t* idsIn = nullptr;
    uint32_t* idsOut = nullptr;
    float4* tapeP = nullptr;
    float4* tapeV = nullptr;
};
// posPrev: the sorted positions, read by the force planes and the step's end.
void launch_compute_delta(const DevConsts& c, Batch b, const float4* predPacked, const float4* posPrev,
                          const StepEnd& end, float4* predOut, const float* density, const uint2* meta, int lastIteration,
                          uint8_t* clampMask, const uint4* rows, int block, int balance, int* tileCounter,
                          cudaStream_t s);
void launch_update_velocities(const DevConsts& c, const StepEnd& end, const float4* pred, const float4* posIn,
                              cudaStream_t s);
// near: the neighbour records that launch_apply_vorticity reads.
void launch_apply_viscosity(const DevConsts& c, Batch b, const float4* pred, const float4* velIn, float4* velOut,
                            float4* omega, float4* near, const uint2* meta, const uint4* rows, int block, int balance,
                            int* tileCounter, cudaStream_t s);
// tileCount > 0: only the particle tiles [firstTile, firstTile + tileCount)
// of `block` particles, one block per tile (a frame's read-back splits the
// last vorticity pass so that the first part's velocities copy out while the
// rest runs).
void launch_apply_vorticity(const DevConsts& c, const float4* pred, const float4* near, const float4* omega,
                            const float4* velIn, float4* velOut, const uint2* meta, const uint4* rows, int block, int balance,
                            int* tileCounter, cudaStream_t s, int firstTile = 0, int tileCount = 0);

// ---- radix sort (pbf_sort.cu) ----
struct SortPlan {
    int n = 0;
    int passes = 0;       // 8-bit digits needed for keys < gridBufSize
    int rounds = 16;      // keys per thread and tile: 256 x rounds per tile (4 at <= 2^18 keys)
    int tiles = 0;        // ceil(n / (256 * rounds))
    size_t histWords = 0; // 256 * tiles
};
SortPlan make_sort_plan(int n, uint32_t gridBufSize);
// Sorts (keys[0], perm[0]) by key, stably, ping-ponging through keys[1] /
// perm[1]; returns the index (0 or 1) of the buffers holding the result.
int launch_radix_sort(const SortPlan& plan, uint32_t* keys[2], uint32_t* perm[2], uint32_t* hist, cudaStream_t s);
// Kernels launched by one launch_radix_sort call.
int radix_sort_launches(const SortPlan& plan);

// ---- counting sort (pbf_sort.cu) ----
// Taken by a substep whose keys are at most kCountingRatio times its particles
// (or at most kCountingSmall), so that the scan over the key range (12 bytes a
// key: 35 us for 2^24 keys at the measured copy rate) stays below the radix
// passes that it replaces (65 us at 1M particles and three passes), and at least
// a kCountingLoad-th of them: a particle reads its key's other particles.  The
// radix sort above takes the others.
constexpr uint64_t kCountingSmall = 1u << 20, kCountingRatio = 16, kCountingLoad = 64;
struct CountingPlan {
    uint32_t blocks = 0;          // of the scan; 0: the radix sort
    uint32_t chunks = 0, chunksPerBlock = 0;
    size_t words = 0;             // counters, and first indices, as allocated
};
CountingPlan make_counting_plan(int n, uint64_t keys);
CountingPlan make_scan_plan(uint64_t keys);  // whatever the number of particles
// The first index of every key, and one beyond the last, from the counts, which
// it leaves at zero.
void launch_counting_scan(const CountingPlan& plan, uint32_t* counts, uint32_t* sums, uint32_t* starts, cudaStream_t s);
// From the counts and the particles' places of arrival (launch_predict_keys):
// the first index of every key into `starts`, and the particles grouped by key,
// in any order within a key, into `order`.  Zeroes the counts.  crowded: `counts`
// where launch_cell_finish follows, else NULL.  keyLimit, err: as for
// launch_update_cells.
void launch_counting_sort(const CountingPlan& plan, int n, uint32_t* counts, uint32_t* sums, uint32_t* starts,
                          const uint32_t* keys, const uint32_t* place, uint32_t* order, uint32_t* crowded,
                          uint32_t keyLimit, int* err, cudaStream_t s);
// The stable order from it, with the records gathered (launch_gather_sorted);
// permCopy (may be NULL) receives the permutation too; c: its n, h and epoch.
void launch_cell_gather(const DevConsts& c, const uint32_t* keys, const uint32_t* starts, const uint32_t* order, uint32_t* keysOut,
                        uint32_t* permOut, uint32_t* permCopy, const float4* pos, const float4* pred,
                        const uint32_t* ids, float4* posOut, float4* predOut, uint32_t* idsOut, uint32_t keyLimit, int* err,
                        cudaStream_t s);
// For the entry point that sorts without records (at most PBF_NOALLOC_MAX_KEYS
// particles): the stable permutation, the sorted keys (in place of the
// particles' own) and the cell table (may be NULL) from `order`, which it uses up,
// `starts` and the list of crowded cells.
void launch_cell_finish(const CountingPlan& plan, int n, uint32_t keyCount, const uint32_t* starts, uint32_t* order,
                        uint32_t* keys, uint32_t* permOut, uint32_t* cells, const uint32_t* crowded, cudaStream_t s);

// ---- adjoint (pbf_adjoint.cu) ----
// What one substep of a rollout leaves for its reverse pass.
struct AdjointTape {
    int iterations = 0;
    uint32_t* perm = nullptr;      // sorted index k came from perm[k]
    uint4* rows = nullptr;         // the substep's kept friends in order, four per entry (walk_pairs)
    uint2* meta = nullptr;
    float4* q[64] = {};            // (p^t, lambda^t), t < iterations
    float4* sums[64] = {};         // per iteration sum g and sum |g|^2 + |sum g|^2, g the density pass' gradients
    float* rho[64] = {};           // per iteration the density
    uint8_t* mask = nullptr;       // iterations x N box-clamp decisions (NULL: no clamp)
    float4* pI = nullptr;          // final predictions, w = density
    float4* v2 = nullptr;          // velocities before XSPH
    float4* omega = nullptr;
};
// Adjoint state; xb / vb hold the adjoints of the substep's output on entry
// and of its input on return (the pointers are swapped with xo / vo).
struct AdjointScalars {
    double visc;       // dL/d viscosityFactor
    float gravity[3];  // dL/d gravity
};
struct AdjointBuffers {
    float4 *xb, *vb, *xo, *vo, *pb, *pbt, *omb, *v2b, *xsb;
    AdjointScalars* scalars;  // on the device
};
// Between substeps pb, pbt, omb and v2b are zero.
void adjoint_substep(const DevConsts& c, const AdjointTape& tp, AdjointBuffers& ab, cudaStream_t s);
int adjoint_launches(int iterations);
void scatter_by_id(int n, const uint32_t* ids, const float4* byId, float4* out, cudaStream_t s);
void gather_to_id(int n, const uint32_t* ids, const float4* in, float4* byId, cudaStream_t s);

// ---- headless render (pbf_render.cu) ----
struct RenderBuffers {
    int width = 0, height = 0, n = 0;
    unsigned long long* dkey = nullptr;  // per pixel: (depth bits, ~particle index) of the nearest fragment
    float4* splat = nullptr;             // particles_color.fs output
    float4* smooth = nullptr;            // fluid_depth_smoothing.fs output
    float4* out = nullptr;               // the frame
    uint8_t* vis = nullptr;              // per particle: seen in the splat
    uint32_t* keys = nullptr;            // per particle: its bucket
    uint32_t* place = nullptr;           // per particle: its place of arrival in the bucket
    uint32_t* order = nullptr;           // the visible particles grouped by bucket
    float4* sorted = nullptr;            // their positions, by index within a bucket
    uint32_t* counts = nullptr;          // per bucket (2048^2): its particles; zero between frames
    uint32_t* starts = nullptr;          // per bucket: its first particle, and one beyond the last bucket
    uint32_t* sums = nullptr;
    CountingPlan plan{};
    int* err = nullptr;                  // the context's error word (bounds-checked builds)
};
// Returns the launches.
int render_frame(const PbfCamera& cam, int mode, int n, float h, const float4* pos, RenderBuffers& rb, cudaStream_t s);
uint64_t render_grid_buckets();

}  // namespace pbf
