// pbf_render.cu — the reference's particle renderer as CUDA kernels into
// device images (no graphics API).
//
// The passes follow src/visual/visual.cpp:340-440 (CVisual::renderParticles,
// smooth mode) and its shaders:
//   splat     particles.vs + particles_color.fs: each particle is a sphere
//             impostor of gl_PointSize = widthOfNearPlane * pointSize / w
//             pixels; a fragment's depth is that of the sphere surface; the
//             LEQUAL depth test (visual.cpp:101) keeps the nearest fragment,
//             the last drawn of equal ones.  Here: one 64-bit atomicMin per
//             fragment on (depth bits, ~index), then a resolve pass.
//   visible   vis_scan.cms: every pixel marks the particle its colour names.
//   grid      grid_chain_reset.cms + grid_build.cms: visible particles hashed
//             into 2048 x 2048 buckets.  The shader chains them with atomic
//             exchanges (order left to the hardware); here the chain of a
//             bucket is its particles in decreasing index order, from a
//             counting sort of the visible ones by bucket.
//   smooth    fluid_depth_smoothing.fs: two Newton steps of the pixel's point
//             along the camera ray towards the density shell sum (h^2 - r^2)^3
//             = 1; colour = (window depth, normalized gradient).
//   final     fluid_final_render.fs: diffuse + specular lighting with the
//             smoothed gradient as normal.
// Every step is one IEEE FP32 operation in the shaders' order (this file is
// compiled with --fmad=false); the oracle restates the same arithmetic.
// Pixel (i, j) has its centre at (i + 0.5, j + 0.5), row 0 at the bottom.

#include <cuda_runtime.h>
#include <cstdint>

#include "pbf_device.cuh"
#include "pbf_internal.h"

namespace pbf {
namespace {

constexpr uint32_t kGridBuckets = 2048u * 2048u;  // grid_build.cms: GRID_BUF_SIZE
constexpr uint64_t kEmptyKey = ~0ull;

struct V4 {
    float x, y, z, w;
};

// column-major 4x4 times (x, y, z, w), summed left to right
__device__ __forceinline__ V4 mat_mul(const float* m, float x, float y, float z, float w) {
    V4 r;
    r.x = ((m[0] * x + m[4] * y) + m[8] * z) + m[12] * w;
    r.y = ((m[1] * x + m[5] * y) + m[9] * z) + m[13] * w;
    r.z = ((m[2] * x + m[6] * y) + m[10] * z) + m[14] * w;
    r.w = ((m[3] * x + m[7] * y) + m[11] * z) + m[15] * w;
    return r;
}

__device__ __forceinline__ float dot3f(float ax, float ay, float az, float bx, float by, float bz) {
    return (ax * bx + ay * by) + az * bz;
}

// GLSL max / min / clamp: max(x, y) = x < y ? y : x
__device__ __forceinline__ float gmax(float x, float y) { return x < y ? y : x; }
__device__ __forceinline__ float gmin(float x, float y) { return y < x ? y : x; }
__device__ __forceinline__ float gclamp(float x, float a, float b) { return gmin(gmax(x, a), b); }

// GLSL int(float): truncation; NaN gives 0 and out-of-range values saturate
__device__ __forceinline__ int to_int(float v) { return __float2int_rz(v); }

__device__ __forceinline__ uint32_t expand_bits_i(int xi) {
    uint32_t x = (uint32_t)xi;
    x = (x | (x << 16)) & 0x030000FFu;
    x = (x | (x << 8)) & 0x0300F00Fu;
    x = (x | (x << 4)) & 0x030C30C3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

// grid_build.cms calcGridHash: mortonNumber(gridPos) % (2048 * 2048)
__device__ __forceinline__ uint32_t render_hash(int x, int y, int z) {
    const int m = (int)(expand_bits_i(x) | (expand_bits_i(y) << 1) | (expand_bits_i(z) << 2));
    return (uint32_t)(m % (int)kGridBuckets);
}

// One fragment of particle `p` (eye-space centre e, clip w, window centre
// xw, yw, sprite size s) at pixel (i, j): the sphere normal and the window
// depth, or false where particles_color.fs discards it.
struct Frag {
    float nx, ny, nz, depth;
};
__device__ __forceinline__ bool fragment(const PbfCamera& cam, float ex, float ey, float ez, float xw, float yw, float s,
                                         int i, int j, Frag& f) {
    const float pcx = 0.5f + (((float)i + 0.5f) - xw) / s;        // gl_PointCoord.s
    const float pcy = 0.5f - (((float)j + 0.5f) - yw) / s;        // gl_PointCoord.t (upper-left origin)
    f.nx = pcx * 2.0f + -1.0f;
    f.ny = pcy * 2.0f + -1.0f;
    const float mag = f.nx * f.nx + f.ny * f.ny;
    if (mag > 1.0f) return false;
    f.nz = sqrtf(1.0f - mag);
    const V4 c = mat_mul(cam.projection, ex + f.nx * cam.pointSize, ey + f.ny * cam.pointSize,
                         ez + f.nz * cam.pointSize, 1.0f);
    const float ndc = c.z / c.w;
    if (ndc < -1.0f) return false;
    f.depth = ((1.0f * ndc + 0.0f) + 1.0f) / 2.0f;
    return f.depth <= 1.0f;  // LEQUAL against the cleared depth 1.0
}

// particles.vs for particle p: eye position, clip w, window centre and
// sprite size; false when the point is clipped.
__device__ __forceinline__ bool sprite(const PbfCamera& cam, float4 p, float& ex, float& ey, float& ez, float& xw,
                                       float& yw, float& s) {
    const V4 e = mat_mul(cam.modelView, p.x, p.y, p.z, 1.0f);
    const V4 c = mat_mul(cam.projection, e.x, e.y, e.z, e.w);
    if (!(c.w > 0.0f)) return false;
    const float nx = c.x / c.w, ny = c.y / c.w, nz = c.z / c.w;
    if (!(fabsf(nx) <= 1.0f && fabsf(ny) <= 1.0f && fabsf(nz) <= 1.0f)) return false;
    s = cam.widthOfNearPlane * cam.pointSize / c.w;
    s = fminf(fmaxf(s, 1.0f), 1024.0f);
    const float hw = 0.5f * (float)cam.width, hh = 0.5f * (float)cam.height;
    xw = nx * hw + hw;
    yw = ny * hh + hh;
    ex = e.x;
    ey = e.y;
    ez = e.z;
    return true;
}

// The pixels of a sprite's square.
struct Rect {
    int i0, i1, j0, j1;
};
__device__ __forceinline__ Rect sprite_rect(const PbfCamera& cam, float xw, float yw, float s) {
    return {max(0, (int)ceilf(xw - s * 0.5f - 0.5f)), min(cam.width - 1, (int)ceilf(xw + s * 0.5f - 0.5f) - 1),
            max(0, (int)ceilf(yw - s * 0.5f - 0.5f)), min(cam.height - 1, (int)ceilf(yw + s * 0.5f - 0.5f) - 1)};
}

// ---- occlusion ----
//
// A volume of particles is tens of sprites deep, and all but the nearest
// fragments lose the depth test.  Under a perspective projection (checked on the
// host: depth depends on the eye-space z alone, and grows with the distance) a
// sprite that covers a tile of 8 x 8 pixels bounds the tile's final depth: its
// farthest fragment there.  occlude_kernel takes the least such bound of every
// tile; splat_kernel drops the tiles of a sprite whose nearest possible fragment
// lies behind the bound, and most sprites altogether (262,144 particles at 1280 x
// 720: 572 us for all fragments, one thread and one atomic after another for each
// sprite; 45 us for the bounds, the list and the listed sprites).  The bounds leave kSlack,
// above the few 2^-24 that the rounded depths can be off, so no fragment that
// could win is dropped and the image is the same.
constexpr int kTilePixels = 8;
constexpr float kSlack = 1.0e-6f;
__device__ __forceinline__ float depth_at(const PbfCamera& cam, float z) {
    return ((cam.projection[10] * z + cam.projection[14]) / -z + 1.0f) / 2.0f;
}

// A fragment's depth test.  Most fragments lie behind what is drawn already: one
// whose sprite's nearest depth does is dropped before its own is formed (1M
// sprites of 5 pixels, 48M -> 33M warp instructions in splat_kernel, and 61 -> 43
// us with four pixels' loads in flight; one by one they took the gain away).  An old
// value of the pixel is larger, so a stale read only costs the work.
__device__ __forceinline__ void draw(const PbfCamera& cam, float ex, float ey, float ez, float xw, float yw, float s,
                                     uint32_t nearest, int p, int i, int j, unsigned long long* at,
                                     unsigned long long drawn) {
    if (nearest > (uint32_t)(drawn >> 32)) return;
    Frag f;
    if (!fragment(cam, ex, ey, ez, xw, yw, s, i, j, f)) return;
    const unsigned long long key = ((unsigned long long)__float_as_uint(f.depth) << 32) | (0xFFFFFFFFu - (uint32_t)p);
    if (key < drawn) atomicMin(at, key);
}

__device__ __forceinline__ uint32_t nearest_depth(const PbfCamera& cam, float ez) {
    const float nearest = ez + cam.pointSize < 0.0f ? depth_at(cam, ez + cam.pointSize) - kSlack : 0.0f;
    return nearest > 0.0f ? __float_as_uint(nearest) : 0u;
}

// Also clears what a frame starts from: no fragment, and no particle seen (visWords
// words).  tileDepth NULL: that alone.  Each had a clear of its own; with those, and
// the launches up to the resolve not chained, 262,144 sprites of 2 pixels at 640 x 480
// took 48 us in a colour mode, 27 like this.
constexpr uint32_t kNoSprites = 0x7F7F7F7Fu;  // what the sprites' counter and the bounds start from
__global__ void __launch_bounds__(128)
occlude_kernel(PbfCamera cam, int n, const float4* pos, uint32_t* tileDepth, unsigned long long* dkey, uint32_t* vis,
               uint32_t visWords) {
    chain_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const size_t pixels = (size_t)cam.width * cam.height, stride = gridDim.x * (size_t)blockDim.x;
    for (size_t k = p; k < pixels; k += stride) dkey[k] = kEmptyKey;
    for (size_t k = p; k < visWords; k += stride) vis[k] = 0u;
    if (p >= n || !tileDepth) return;
    const float4 at = pos[p];
    // only sprites that lie inside the depth range as a whole, and wide enough to cover a tile: the size is known from
    // the eye-space z alone (w = -z)
    const float* m = cam.modelView;
    const float z = ((m[2] * at.x + m[6] * at.y) + m[10] * at.z) + m[14] * 1.0f;
    if (!(z + cam.pointSize < 0.0f) || cam.widthOfNearPlane * cam.pointSize / -z < 1.5f * kTilePixels) return;
    float ex, ey, ez, xw, yw, s;
    if (!sprite(cam, at, ex, ey, ez, xw, yw, s)) return;
    if (!(depth_at(cam, ez + cam.pointSize) > kSlack) || !(depth_at(cam, ez) < 1.0f - kSlack)) return;
    const Rect r = sprite_rect(cam, xw, yw, s);
    const int tilesX = (cam.width + kTilePixels - 1) / kTilePixels;
    const float scale = 2.0f / s;
    for (int tj = r.j0 / kTilePixels; tj <= r.j1 / kTilePixels; ++tj) {
        const float y0 = ((float)(tj * kTilePixels) + 0.5f - yw) * scale, y1 = y0 + (float)(kTilePixels - 1) * scale;
        const float y = fmaxf(fabsf(y0), fabsf(y1));
        for (int ti = r.i0 / kTilePixels; ti <= r.i1 / kTilePixels; ++ti) {
            const float x0 = ((float)(ti * kTilePixels) + 0.5f - xw) * scale, x1 = x0 + (float)(kTilePixels - 1) * scale;
            const float x = fmaxf(fabsf(x0), fabsf(x1));
            const float mag = x * x + y * y;  // of the tile's farthest pixel centre
            if (!(mag < 0.99f)) continue;
            const float far = depth_at(cam, ez + 0.999f * sqrtf(1.0f - mag) * cam.pointSize) + kSlack;
            uint32_t* bound = tileDepth + (size_t)tj * tilesX + ti;
            if (__float_as_uint(far) < *bound) atomicMin(bound, __float_as_uint(far));
        }
    }
}

// Draws the small sprites, a thread each, and lists the others (*counter of them)
// that are not hidden in every tile.  tileDepth NULL: no bounds.
// Pixels that one thread draws: sprites too small to cover a tile (494,820
// particles at 750 x 981, 10 pixels wide: 355 us a frame; a warp to each of more than
// 36 pixels: 642; every fragment formed: 522).
// Below kEarlyLeast particles the chip has too few threads to hide the loads of the
// early depth test (30,000 of 6 pixels at 640 x 480 93 us a frame with it, 57 without
// it and without the look at the tiles).  Tiny sprites skip both too: they cost as
// much as the few fragments do (1M of 2 to 3 pixels: 46 us in this kernel with them,
// 38 to 40 without; at 3 to 4 pixels a frame of 262,144, many over one another, takes
// 39 and 51).
constexpr int kSmallSprite = 144, kEarlyLeast = 100000;
template <bool Early>
__global__ void __launch_bounds__(128)
splat_kernel(PbfCamera cam, int n, const float4* pos, const uint32_t* tileDepth, unsigned long long* dkey, uint32_t* shown,
             uint32_t* counter) {
    chain_wait();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    float ex, ey, ez, xw, yw, s;
    if (!sprite(cam, pos[p], ex, ey, ez, xw, yw, s)) return;
    const Rect r = sprite_rect(cam, xw, yw, s);
    const int tilesX = (cam.width + kTilePixels - 1) / kTilePixels;
    const bool tiny = s <= (Early ? 3.0f : 8.0f);
    const uint32_t nearest = tileDepth ? nearest_depth(cam, ez) : 0u;
    bool visible = tiny || tileDepth == nullptr;
    for (int tj = r.j0 / kTilePixels; !visible && tj <= r.j1 / kTilePixels; ++tj)
        for (int ti = r.i0 / kTilePixels; !visible && ti <= r.i1 / kTilePixels; ++ti)
            visible = nearest <= tileDepth[(size_t)tj * tilesX + ti];
    if (!visible) return;
    if ((r.i1 - r.i0 + 1) * (r.j1 - r.j0 + 1) > kSmallSprite) {
        shown[atomicAdd(counter, 1u) - kNoSprites] = (uint32_t)p;
        return;
    }
    for (int j = r.j0; j <= r.j1; ++j) {
        unsigned long long* row = dkey + (size_t)j * cam.width;
        for (int i = r.i0; i <= r.i1; i += 4) {  // four pixels' loads in flight
            unsigned long long drawn[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) drawn[k] = !Early || tiny ? kEmptyKey : i + k <= r.i1 ? row[i + k] : 0ull;  // 0: nothing is in front of it
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (i + k <= r.i1) draw(cam, ex, ey, ez, xw, yw, s, nearest, p, i + k, j, row + i + k, drawn[k]);
        }
    }
}

// The sprites that remain, a warp each, tile by tile: they lie together in memory, so
// they are dealt out over the whole chip.  tileDepth NULL: no occlusion bounds.
constexpr int kDrawBlocks = 152 * 16, kDrawWarps = 4;
__global__ void __launch_bounds__(32 * kDrawWarps)
draw_kernel(PbfCamera cam, int n, const float4* pos, const uint32_t* tileDepth, unsigned long long* dkey,
            const uint32_t* shown, const uint32_t* shownCount, int* err) {
    chain_wait();
    const int lane = threadIdx.x & 31;
    const uint32_t count = checked_index(*shownCount - kNoSprites, (uint32_t)n + 1u, err, kErrSortIndex);
    const int tilesX = (cam.width + kTilePixels - 1) / kTilePixels;
    for (uint32_t k = blockIdx.x * kDrawWarps + (threadIdx.x >> 5); k < count; k += kDrawBlocks * kDrawWarps) {
        const int p = (int)checked_index(shown[k], (uint32_t)n, err, kErrSortIndex);
        float ex, ey, ez, xw, yw, s;
        sprite(cam, pos[p], ex, ey, ez, xw, yw, s);
        const Rect r = sprite_rect(cam, xw, yw, s);
        const uint32_t nearest = tileDepth ? nearest_depth(cam, ez) : 0u;
        for (int tj = r.j0 / kTilePixels; tj <= r.j1 / kTilePixels; ++tj)
            for (int ti = r.i0 / kTilePixels; ti <= r.i1 / kTilePixels; ++ti) {
                if (tileDepth && nearest > tileDepth[(size_t)tj * tilesX + ti]) continue;
                const int i = ti * kTilePixels + lane % kTilePixels;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int j = tj * kTilePixels + 4 * half + lane / kTilePixels;
                    if (i < r.i0 || i > r.i1 || j < r.j0 || j > r.j1) continue;
                    unsigned long long* at = dkey + (size_t)j * cam.width + i;
                    draw(cam, ex, ey, ez, xw, yw, s, nearest, p, i, j, at, *at);
                }
            }
    }
}

// hsv2rgb of particles_color.fs, mix(a, b, t) = a (1 - t) + b t
__device__ __forceinline__ float hsv_channel(float h, float k, float s, float v) {
    const float x = h + k;
    const float fr = x - floorf(x);
    const float p = fabsf(fr * 6.0f - 3.0f);
    const float q = gclamp(p - 1.0f, 0.0f, 1.0f);
    return v * (1.0f * (1.0f - s) + q * s);
}

__global__ void __launch_bounds__(256)
resolve_kernel(PbfCamera cam, int n, int mode, const float4* pos, const unsigned long long* dkey, float4* splat,
               uint8_t* vis, float4* out) {
    chain_wait();
    const int pix = blockIdx.x * blockDim.x + threadIdx.x;
    const bool inside = pix < cam.width * cam.height;
    const unsigned long long key = inside ? dkey[pix] : 0ull;
    // vis_scan.cms, in mode 0: the particle that the pixel's colour names, also an empty pixel's (particle 0; one
    // store by a block, not by every warp: about 3 us of a frame)
    auto mark = [&](float colour) {
        const uint32_t x = (uint32_t)(colour + 0.5f);
        if (x < (uint32_t)n && vis[x] == 0) vis[x] = 1;
    };
    if (mode == 0 && __syncthreads_or(inside && key == kEmptyKey) && threadIdx.x == 0) mark(0.0f);
    if (!inside) return;
    if (key == kEmptyKey) {
        splat[pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (mode != 0) out[pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);  // the colour modes' frame is the splat
        return;
    }
    const uint32_t p = 0xFFFFFFFFu - (uint32_t)(key & 0xFFFFFFFFu);
    const float depth = __uint_as_float((uint32_t)(key >> 32));
    if (mode == 0) {
        splat[pix] = make_float4(depth, (float)(int)p, 0.0f, 1.0f);
        mark((float)(int)p);
        return;
    }
    const int i = pix % cam.width, j = pix / cam.width;
    const float4 q = pos[p];
    float ex, ey, ez, xw, yw, s;
    Frag f{};
    sprite(cam, q, ex, ey, ez, xw, yw, s);
    fragment(cam, ex, ey, ez, xw, yw, s, i, j, f);
    const float cosA = gclamp(dot3f(f.nx, f.ny, f.nz, 1.0f, 1.0f, 1.0f), 0.0f, 1.0f);
    float r, g, b;
    if (mode == 1) {
        const float v = q.w / 20.0f;
        r = v;
        g = v;
        b = 1.0f;
    } else {
        const float hue = (float)(int)p / (float)n * 0.7f;
        r = hsv_channel(hue, 1.0f, 0.9f, 0.9f);
        g = hsv_channel(hue, 2.0f / 3.0f, 0.9f, 0.9f);
        b = hsv_channel(hue, 1.0f / 3.0f, 0.9f, 0.9f);
    }
    splat[pix] = out[pix] = make_float4(r * cosA, g * cosA, b * cosA, 1.0f * cosA);
}

// Bucket and place of arrival of the visible particles (kGridBuckets: not visible).
__global__ void grid_count_kernel(int n, float h, const float4* __restrict__ pos, const uint8_t* __restrict__ vis,
                                  uint32_t* __restrict__ keys, uint32_t* __restrict__ place, uint32_t* __restrict__ counts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t key = kGridBuckets;
    if (vis[i]) {
        const float4 p = pos[i];
        key = render_hash(to_int(p.x / h), to_int(p.y / h), to_int(p.z / h));
        place[i] = atomicAdd(&counts[key], 1u);
    }
    keys[i] = key;
}

__global__ void grid_scatter_kernel(int n, const uint32_t* __restrict__ keys, const uint32_t* __restrict__ place,
                                    const uint32_t* __restrict__ starts, uint32_t* __restrict__ order, int* err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || keys[i] >= kGridBuckets) return;
    order[checked_index(starts[keys[i]] + place[i], (uint32_t)n, err, kErrSortIndex)] = (uint32_t)i;
}

// The positions of each bucket's particles by decreasing index, the order of its chain.
__global__ void grid_rank_kernel(int n, const uint32_t* __restrict__ keys, const uint32_t* __restrict__ starts,
                                 const uint32_t* __restrict__ order, const float4* __restrict__ pos,
                                 float4* __restrict__ sorted, int* err) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x, limit = (uint32_t)n;
    if (s >= checked_index(starts[kGridBuckets], limit + 1u, err, kErrSortIndex)) return;
    const uint32_t i = checked_index(order[s], limit, err, kErrSortIndex), key = checked_index(keys[i], kGridBuckets, err, kErrCellKey);
    const uint32_t first = starts[key], end = checked_index(starts[key + 1], limit + 1u, err, kErrSortIndex);
    uint32_t to = first;
    for (uint32_t q = first; q < end; ++q) to += order[q] > i;
    sorted[checked_index(to, limit, err, kErrSortIndex)] = pos[i];
}

// fluid_depth_smoothing.fs SampleDensityAndGradient
__device__ void sample_density(float h, int n, const float4* __restrict__ sorted, const uint32_t* __restrict__ starts,
                               int* err, float wx, float wy, float wz, float& density, float& gx, float& gy, float& gz) {
    const float h2 = h * h;
    density = 0.0f;
    gx = gy = gz = 0.0f;
    const int cx = to_int(wx / h), cy = to_int(wy / h), cz = to_int(wz / h);
    // render_hash of the 27 buckets from the spread coordinates of each axis; the Morton number is below 2^30.  x is
    // its lowest bit: of three buckets in a row the first two (cx odd) or the last two lie together, and are one range
    const uint32_t sx0 = expand_bits_i(cx - 1), sx1 = expand_bits_i(cx), sx2 = expand_bits_i(cx + 1);
    const bool odd = cx & 1;
    const uint32_t from[2] = {sx0, odd ? sx2 : sx1}, length[2] = {odd ? 2u : 1u, odd ? 1u : 2u};
#pragma unroll 1
    for (int iz = -1; iz <= 1; ++iz)
#pragma unroll 1
        for (int iy = -1; iy <= 1; ++iy) {
            const uint32_t yz = (expand_bits_i(cy + iy) << 1) | (expand_bits_i(cz + iz) << 2);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                const uint32_t b = (from[part] | yz) & (kGridBuckets - 1u);
                const int end = (int)checked_index(starts[b + length[part]], (uint32_t)n + 1u, err, kErrSortIndex);
#pragma unroll 4
                for (int k = (int)starts[b]; k < end; ++k) {
                    const float4 pp = __ldg(sorted + k);
                    const float dx = pp.x - wx, dy = pp.y - wy, dz = pp.z - wz;
                    const float r2 = dot3f(dx, dy, dz, dx, dy, dz);
                    if (r2 < h2) {
                        const float d = h2 - r2;
                        gx = gx + dx * d * d;
                        gy = gy + dy * d * d;
                        gz = gz + dz * d * d;
                        density = density + d * d * d;
                    }
                }
            }
        }
    density = density * 1.0f;
    gx = gx * -6.0f;
    gy = gy * -6.0f;
    gz = gz * -6.0f;
}

// uvToWorld / uvToViewSpace: the point of pixel (i, j) at buffer depth z
__device__ __forceinline__ V4 pixel_world(const PbfCamera& cam, int i, int j, float z) {
    const float nearv = cam.depthRange[0], farv = cam.depthRange[1];
    const float lz = nearv / (farv - z * (farv - nearv)) * farv;
    const float u = (((float)i + 0.5f) / (float)cam.width * 2.0f - 1.0f) * cam.invFocalLen[0];
    const float v = (((float)j + 0.5f) / (float)cam.height * 2.0f - 1.0f) * cam.invFocalLen[1];
    return mat_mul(cam.invModelView, u * lz, v * lz, -lz, 1.0f);
}

__device__ __forceinline__ void normalize3(float& x, float& y, float& z) {
    const float l = sqrtf(dot3f(x, y, z, x, y, z));
    x = x / l;
    y = y / l;
    z = z / l;
}

// A warp takes 8 x 4 pixels, whose points lie in the same few buckets; bound by
// instruction issue (85 %): 141 us with a row of pixels and the positions behind
// the permutation, 118 like this, and 110 with two buckets to a range (the scene
// above; pairs of candidates in packed arithmetic: 105, and slower at 1M sprites).
__global__ void __launch_bounds__(128)
smooth_kernel(PbfCamera cam, float h, int n, const float4* __restrict__ sorted, const uint32_t* __restrict__ starts,
              const float4* __restrict__ splat, float4* __restrict__ out, int* err) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * 16 + 8 * (warp & 1) + (lane & 7), j = blockIdx.y * 8 + 4 * (warp >> 1) + (lane >> 3);
    if (i >= cam.width || j >= cam.height) return;
    const int pix = j * cam.width + i;
    const float z = splat[pix].x;
    out[pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (z == 1.0f) return;  // the far plane: discard
    const V4 m = pixel_world(cam, i, j, z);
    const float camx = cam.invModelView[12], camy = cam.invModelView[13], camz = cam.invModelView[14];
    float nx = camx - m.x, ny = camy - m.y, nz = camz - m.z;
    normalize3(nx, ny, nz);
    float tp = 0.0f, sx = m.x, sy = m.y, sz = m.z;
    float density, gx = 0.0f, gy = 0.0f, gz = 0.0f;
    for (int it = 0; it < 2; ++it) {
        sample_density(h, n, sorted, starts, err, sx, sy, sz, density, gx, gy, gz);
        const float dd = density - 1.0f;
        const float ga = dot3f(nx, ny, nz, gx, gy, gz);
        tp += dd / ga;
        sx = m.x + tp * nx;
        sy = m.y + tp * ny;
        sz = m.z + tp * nz;
    }
    const V4 vs = mat_mul(cam.modelView, sx, sy, sz, 1.0f);
    const V4 c = mat_mul(cam.projection, vs.x, vs.y, vs.z, 1.0f);
    const float ndc = c.z / c.w;
    if (ndc < -1.0f) return;
    const float zb = ((1.0f * ndc + 0.0f) + 1.0f) / 2.0f;
    normalize3(gx, gy, gz);
    out[pix] = make_float4(zb, gx, gy, gz);
}

// pow(x, 50) by binary powers (x^32 x^16 x^2); negative and NaN give NaN
__device__ __forceinline__ float pow50(float x) {
    if (!(x >= 0.0f)) return __int_as_float(0x7FC00000);
    const float x2 = x * x, x4 = x2 * x2, x8 = x4 * x4, x16 = x8 * x8, x32 = x16 * x16;
    return (x32 * x16) * x2;
}

__global__ void final_kernel(PbfCamera cam, const float4* __restrict__ smooth, float4* __restrict__ out) {
    const int pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= cam.width * cam.height) return;
    const int i = pix % cam.width, j = pix / cam.width;
    out[pix] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    // uvToEye of the pixel and its four neighbours: any at the far plane discards
    const int di[5] = {0, 1, -1, 0, 0}, dj[5] = {0, 0, 0, 1, -1};
    for (int k = 0; k < 5; ++k) {
        const int a = i + di[k], b = j + dj[k];
        const float z = (a >= 0 && a < cam.width && b >= 0 && b < cam.height) ? smooth[(size_t)b * cam.width + a].x : 0.0f;
        if (z == 1.0f) return;
    }
    const float4 s = smooth[pix];
    const float nx = s.y, ny = s.z, nz = s.w;
    const V4 w = pixel_world(cam, i, j, s.x);
    float ex = cam.invModelView[12] - w.x, ey = cam.invModelView[13] - w.y, ez = cam.invModelView[14] - w.z;
    normalize3(ex, ey, ez);
    const float lx = 0.0f, ly = 1.0f, lz = 0.0f;  // normalize(vec3(0, 1, 0))
    float hx = lx + ex, hy = ly + ey, hz = lz + ez;
    normalize3(hx, hy, hz);
    const float diff = gclamp(dot3f(lx, ly, lz, nx, ny, nz), 0.0f, 1.0f);
    const float spec = gmax(0.0f, pow50(dot3f(nx, ny, nz, hx, hy, hz)));
    out[pix] = make_float4(0.0f * diff + 1.0f * spec, 0.0f * diff + 1.0f * spec, 0.5f * diff + 1.0f * spec, 1.0f);
}

inline unsigned blocks(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

// A perspective projection as depth_at takes it: the clip z and w depend on the
// eye-space z alone, w is the distance, and depth grows with it.
bool plain_perspective(const PbfCamera& cam) {
    const float* m = cam.projection;
    return m[2] == 0.0f && m[6] == 0.0f && m[3] == 0.0f && m[7] == 0.0f && m[11] == -1.0f && m[15] == 0.0f &&
           m[10] < 0.0f && m[10] >= -2.0f && m[14] < 0.0f && m[14] > -1.0e6f && cam.pointSize > 0.0f &&
           cam.pointSize < 1.0e6f;
}

}  // namespace

int render_frame(const PbfCamera& cam, int mode, int n, float h, const float4* pos, RenderBuffers& rb, cudaStream_t s) {
    const size_t pixels = (size_t)cam.width * cam.height;
    // the counter of the listed sprites and the bounds of the tiles live in the smoothed image, and the list in the
    // grid's order: both are written later
    uint32_t* counter = reinterpret_cast<uint32_t*>(rb.smooth);
    uint32_t* tileDepth = plain_perspective(cam) ? counter + 1 : nullptr;
    const size_t tiles = (size_t)((cam.width + kTilePixels - 1) / kTilePixels) * ((cam.height + kTilePixels - 1) / kTilePixels);
    cudaMemsetAsync(counter, 0x7F, 4 * (1 + tiles), s);  // no sprite, and a depth above every other
    launch_chained(occlude_kernel, max(blocks(n, 128), min(blocks(pixels, 128), 1216u)), 128, s, cam, n, pos, tileDepth, rb.dkey,
                   reinterpret_cast<uint32_t*>(rb.vis), mode == 0 ? (uint32_t)((n + 3) / 4) : 0u);
    launch_chained(n >= kEarlyLeast ? splat_kernel<true> : splat_kernel<false>, blocks(n, 128), 128, s, cam, n, pos, tileDepth,
                   rb.dkey, rb.order, counter);
    launch_chained(draw_kernel, kDrawBlocks, 32 * kDrawWarps, s, cam, n, pos, tileDepth, rb.dkey, rb.order, counter, rb.err);
    launch_chained(resolve_kernel, blocks(pixels, 256), 256, s, cam, n, mode, pos, rb.dkey, rb.splat, rb.vis, rb.out);
    if (mode != 0) return 4;
    grid_count_kernel<<<blocks(n, 256), 256, 0, s>>>(n, h, pos, rb.vis, rb.keys, rb.place, rb.counts);
    launch_counting_scan(rb.plan, rb.counts, rb.sums, rb.starts, s);
    grid_scatter_kernel<<<blocks(n, 256), 256, 0, s>>>(n, rb.keys, rb.place, rb.starts, rb.order, rb.err);
    grid_rank_kernel<<<blocks(n, 256), 256, 0, s>>>(n, rb.keys, rb.starts, rb.order, pos, rb.sorted, rb.err);
    smooth_kernel<<<dim3(blocks(cam.width, 16), blocks(cam.height, 8)), 128, 0, s>>>(cam, h, n, rb.sorted, rb.starts, rb.splat,
                                                                                    rb.smooth, rb.err);
    final_kernel<<<blocks(pixels, 256), 256, 0, s>>>(cam, rb.smooth, rb.out);
    return 9 + (rb.plan.blocks > 1 ? 2 : 1);
}

uint64_t render_grid_buckets() { return kGridBuckets; }

}  // namespace pbf
