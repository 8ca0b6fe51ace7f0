// pbf_adjoint.cu — reverse accumulation through one substep, over a fixed
// neighbour structure (the substep's sort permutation, friend lists and box
// clamp decisions are constants of the derivative).
//
// With r = p_i - p_j, k(r) = (h - |r|)^2 r/|r| and W(r) = (h^2 - |r|^2)^3, the
// forward of a substep is (compute_scaling.cl, compute_delta.cl,
// update_velocities.cl, apply_viscosity.cl, apply_vorticity.cl):
//   lambda_i = -(rho_i/rho0 - 1) / (D_i/rho0^2 + eps),
//     rho_i = POLY6 sum W,  D_i = sum |G k|^2 + |sum G k|^2
//   p'_i = clamp(p_i - (G/rho0) sum (lambda_i + lambda_j + K (W/Wq)^4) k)
//   v2 = (p^I - x)/dt,  v3 = v2 + c POLY6 sum (v2_j - v2_i) W,
//   omega_i = -G sum (v2_j - v2_i) x k,  eta_i = -G sum |omega_j| k,
//   v4 = v3 + dt eps_v (eta/|eta|) x omega_i.
// Each kernel below walks the same friends as its forward kernel (the rows
// the substep recorded) and scatters neighbour terms with atomics, so the sums
// are not ordered: these are FP32 gradients, not bit-reproducible ones.  The derivation is the same
// as the FP64 adjoint the tests compare against.

#include <cuda_runtime.h>
#include <cstdint>

#include "pbf_device.cuh"
#include "pbf_internal.h"

namespace pbf {
namespace {

constexpr int kAdjBlock = 128;

struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 f3(const float4& a) { return {a.x, a.y, a.z}; }
__device__ __forceinline__ F3 operator+(F3 a, F3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ F3 operator-(F3 a, F3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F3 operator*(float s, F3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ float dot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ F3 cross(F3 a, F3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
__device__ __forceinline__ float len(F3 a) { return sqrtf(dot(a, a)); }
// a . a with its roundings written out, whatever the compiler contracts.
__device__ __forceinline__ float dot_fused(F3 a) { return fmaf(a.z, a.z, fmaf(a.x, a.x, __fmul_rn(a.y, a.y))); }

__device__ __forceinline__ void add3(float4* a, F3 v, float w = 0.0f) { atomicAdd(a, make_float4(v.x, v.y, v.z, w)); }

// A friend's records as the walks below load them: its index and one or two
// float4 records.
struct Friend1 {
    uint32_t j;
    float4 a;
};
struct Friend2 {
    uint32_t j;
    float4 a, b;
};

// Four lanes share a particle: lane `sub` takes the friends sub, sub + 4, ...,
// one word of each row entry, two in flight.  The sums are not ordered here, and
// at 65,536 particles one thread per particle leaves 13 warps on an SM, each
// waiting for its own loads (reverse pass of 20 substeps: 6.3 ms with one lane,
// 5.8 with four).
constexpr int kSplit = 4;
template <typename LoadF, typename BodyF>
__device__ __forceinline__ void walk_split(const uint4* rows, int n, int i, int total, int sub, LoadF load,
                                           BodyF body) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(rows + i) + sub;
    const size_t stride = 4 * (size_t)n;
    int t = sub;
    for (; t + kSplit < total; t += 2 * kSplit, p += 2 * stride) {
        const uint32_t j0 = *p, j1 = p[stride];
        const auto f0 = load(j0), f1 = load(j1);
        body(f0);
        body(f1);
    }
    if (t < total) body(load(*p));
}
// The sum of w v, (v, w) = term(record), over a particle's friends in list order,
// one fused multiply-add each, as one thread would take it, in all of its lanes:
// each computes its own friends' terms, and every lane adds the four of an entry
// in turn.  A friend without a term has zeros, which change no sum that starts at
// +0.  All lanes of the warp come here; those without a particle with a total of 0.
template <typename LoadF, typename TermF>
__device__ __forceinline__ F3 ordered_sum(const uint4* rows, int n, int i, int total, int sub, LoadF load,
                                          TermF term) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(rows + i) + sub;
    const size_t stride = 4 * (size_t)n;
    const int most = __reduce_max_sync(0xFFFFFFFFu, total);
    F3 sum = {0.0f, 0.0f, 0.0f};
    auto add_in_turn = [&](const float4& t) {
#pragma unroll
        for (int k = 0; k < kSplit; ++k) {
            const float w = __shfl_sync(0xFFFFFFFFu, t.w, k, kSplit);
            sum.x = fmaf(w, __shfl_sync(0xFFFFFFFFu, t.x, k, kSplit), sum.x);
            sum.y = fmaf(w, __shfl_sync(0xFFFFFFFFu, t.y, k, kSplit), sum.y);
            sum.z = fmaf(w, __shfl_sync(0xFFFFFFFFu, t.z, k, kSplit), sum.z);
        }
    };
    for (int t = sub; t - sub < most; t += 2 * kSplit, p += 2 * stride) {
        float4 t0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), t1 = t0;
        if (t + kSplit < total) {
            const uint32_t j0 = *p, j1 = p[stride];
            const auto f0 = load(j0), f1 = load(j1);
            t0 = term(f0);
            t1 = term(f1);
        } else if (t < total) {
            t0 = term(load(*p));
        }
        add_in_turn(t0);
        add_in_turn(t1);
    }
    return sum;
}
// The sum over a particle's lanes, in all of them.
__device__ __forceinline__ float lanes_sum(float v) {
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
    return v;
}
__device__ __forceinline__ F3 lanes_sum(F3 v) { return {lanes_sum(v.x), lanes_sum(v.y), lanes_sum(v.z)}; }

// k(r) and the adjoint of its argument: d/dr [k . kb] = f kb + f'(|r|)(kb.r) r/|r|
// with f = (h-|r|)^2/|r|, f' = -(h-|r|)(h+|r|)/|r|^2.  y is 1/|r| within an
// ulp (sqrt_recip_rn): the adjoint is an FP32 gradient, not a bit-exact one.
__device__ __forceinline__ F3 kvec(F3 r, float rl, float y, float h) {
    const float hr = h - rl;
    return (hr * hr * y) * r;
}
__device__ __forceinline__ F3 kvec_adj(F3 r, float rl, float y, float h, F3 kb) {
    const float hr = h - rl;
    const float f = hr * hr * y;
    const float fp = -hr * (h + rl) * y * y;
    return f * kb + (fp * dot(kb, r) * y) * r;
}
// |r| and 1/|r| of a pair.
__device__ __forceinline__ float pair_length(float r2, float& y) {
    float rl;
    sqrt_recip_rn(r2, rl, y);
    return rl;
}

__device__ __forceinline__ bool xsph_pair(const DevConsts& c, float r2, float rhoj) {
    return in_support(c, r2) && fabsf(rhoj) > 1e-8f;
}

template <typename T> __device__ __forceinline__ T block_sum(T v) {
    __shared__ T part[kAdjBlock / 32];
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, d);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    T s = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kAdjBlock / 32; ++w) s += part[w];
    return s;
}

// The kernels leave the accumulators they are done with at zero for the next
// use (each particle's own element, where only that particle reads it), so that
// a substep starts with omb, v2b, pb and pbt zero and clears nothing.

// v4 = v3 + dt*vort*(N x omega_i): adjoints of omega (omb) and of p^I (pb).
// eta is summed here, in list order and with fused multiply-adds, although the
// forward pass has summed it too, with each operation rounded: where eta nearly
// cancels, 1/|eta| magnifies its rounding errors.  Against this reverse pass in 64
// bits, dv0 of 20 substeps of 65,536 particles is 1.6e-5 off in one scene and 4.5e-5
// in another, and with the forward pass' eta 3.6e-5 and 5.7e-5.  The sum takes
// 0.03 ms of the 5.27 of those 20 substeps' reverse pass.
__global__ void __launch_bounds__(kAdjBlock)
adj_vorticity_kernel(DevConsts c, const float4* pI, const float4* omega,
                     const uint4* rows, const uint2* meta,
                     const float4* vb, float4* omb, float4* pb) {
    chain_wait();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / kSplit, sub = threadIdx.x % kSplit;
    const int n = c.n;
    const bool valid = i < n;
    const F3 pi = valid ? f3(pI[i]) : F3{0.0f, 0.0f, 0.0f};
    const uint64_t mt = valid ? load_meta(meta, i) : 0u;
    const int total = FlatFriends(mt, kept_other(mt)).total;
    const float G = c.gradSpiky;
    auto loadPO = [&](uint32_t j) {
        j = checked_index(j, (uint32_t)n, c.err, kErrFriendIndex);
        return Friend2{j, pI[j], omega[j]};
    };
    const F3 eta = -G * ordered_sum(rows, n, i, total, sub, loadPO, [&](const Friend2& f) {
        const F3 r = pi - f3(f.a), o = f3(f.b);
        const float r2 = dot_fused(r);
        if (!xsph_pair(c, r2, f.a.w)) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float y;
        const float rl = pair_length(r2, y);
        const F3 k = kvec(r, rl, y, c.h);
        return make_float4(k.x, k.y, k.z, sqrtf(dot_fused(o)));
    });
    const float l = len(eta);
    const bool turns = valid && l > 0.0f;
    F3 etab = {0.0f, 0.0f, 0.0f};
    if (turns) {
        const F3 N = (1.0f / l) * eta;
        const F3 ub = (c.vort * c.dt) * f3(vb[i]);
        const F3 oi = f3(omega[i]);
        const F3 Nb = cross(oi, ub);
        if (sub == 0) add3(&omb[i], cross(ub, N));
        etab = (1.0f / l) * (Nb - dot(N, Nb) * N);
    }
    F3 pbi = {0.0f, 0.0f, 0.0f};  // particle i's own terms, added once
    walk_split(rows, n, i, turns ? total : 0, sub, loadPO, [&](const Friend2& f) {
        const F3 r = pi - f3(f.a);
        const float r2 = dot(r, r);
        if (!xsph_pair(c, r2, f.a.w)) return;
        float y;
        const float rl = pair_length(r2, y);
        const F3 k = kvec(r, rl, y, c.h);
        const F3 oj = f3(f.b);
        const float ol = len(oj);
        if (ol > 0.0f) add3(&omb[f.j], (-G * dot(etab, k) / ol) * oj);
        const F3 rb = kvec_adj(r, rl, y, c.h, (-G * ol) * etab);
        pbi = pbi + rb;
        add3(&pb[f.j], -1.0f * rb);
    });
    pbi = lanes_sum(pbi);
    if (turns && sub == 0) add3(&pb[i], pbi);
}

// v3 = v2 + c POLY6 sum (v2_j - v2_i) W and omega = -G sum (v2_j - v2_i) x k:
// adjoints of v2 (v2b), p^I (pb) and of the XSPH factor (cbar).  The blocks of all
// substeps add to cbar, so it is a double: as a float it rounds at each of them,
// and four lanes a particle make four times the blocks (65,536 particles, 20
// substeps, ten scenes: r.m.s. 1.3e-6 off the reverse pass in 64 bits with one
// lane a particle, 3.1e-6 with four, 3.0e-7 as a double, the last two both in 5.24 ms).
__global__ void __launch_bounds__(kAdjBlock)
adj_viscosity_kernel(DevConsts c, const float4* pI, const float4* v2,
                     float4* omb, const float4* vb, const uint4* rows,
                     const uint2* meta, float4* v2b, float4* pb,
                     double* cbar) {
    chain_wait();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / kSplit, sub = threadIdx.x % kSplit;
    const int n = c.n;
    const bool valid = i < n;
    float cacc = 0.0f;
    F3 v2bi = {0.0f, 0.0f, 0.0f}, pbi = {0.0f, 0.0f, 0.0f};  // particle i's own terms, added once
    if (valid) {
        const uint64_t mt = load_meta(meta, i);
        const F3 pi = f3(pI[i]), v3b = f3(vb[i]), ob = f3(omb[i]), vi = f3(v2[i]);
        const float G = c.gradSpiky;
        if (sub == 0) v2bi = v3b;
        auto loadPV = [&](uint32_t j) {
            j = checked_index(j, (uint32_t)n, c.err, kErrFriendIndex);
            return Friend2{j, pI[j], v2[j]};
        };
        walk_split(rows, n, i, FlatFriends(mt, kept_other(mt)).total, sub, loadPV, [&](const Friend2& f) {
            const uint32_t j = f.j;
            const F3 r = pi - f3(f.a);
            const float r2 = dot(r, r);
            if (!xsph_pair(c, r2, f.a.w)) return;
            float y;
            const float rl = pair_length(r2, y);
            const F3 u = f3(f.b) - vi;
            const float d = c.h2 - r2;
            const float w = c.poly6 * d * d * d;
            const F3 k = kvec(r, rl, y, c.h);
            cacc += w * dot(v3b, u);
            const F3 ub = (c.visc * w) * v3b + (-G) * cross(k, ob);
            add3(&v2b[j], ub);
            v2bi = v2bi - ub;
            const float Wb = c.visc * c.poly6 * dot(v3b, u);
            const F3 rb = (Wb * -6.0f * d * d) * r + kvec_adj(r, rl, y, c.h, (-G) * cross(ob, u));
            pbi = pbi + rb;
            add3(&pb[j], -1.0f * rb);
        });
    }
    v2bi = lanes_sum(v2bi);
    pbi = lanes_sum(pbi);  // every lane has read omb[i] before this
    if (valid && sub == 0) {
        add3(&v2b[i], v2bi);
        add3(&pb[i], pbi);
        omb[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    const float s = block_sum(cacc);
    if (threadIdx.x == 0 && s != 0.0f) atomicAdd(cbar, (double)s);
}

// v2 = (p^I - x)/dt and x' = p^I.
__global__ void adj_velocity_kernel(DevConsts c, const float4* xb, float4* v2b,
                                    float4* pb, float4* xsb) {
    chain_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= c.n) return;
    const F3 v = f3(v2b[i]);
    v2b[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const F3 p = f3(pb[i]) + f3(xb[i]) + (1.0f / c.dt) * v;
    pb[i] = make_float4(p.x, p.y, p.z, 0.0f);
    xsb[i] = make_float4(-v.x / c.dt, -v.y / c.dt, -v.z / c.dt, 0.0f);
}

// p^{t+1} = clamp(p^t + delta(p^t, lambda^t)): adjoints of p^t (pbt) and
// lambda^t (in pbt's w: one atomic for both) from that of p^{t+1} (pbn).
// q = (p^t, lambda^t).
__global__ void __launch_bounds__(kAdjBlock)
adj_delta_kernel(DevConsts c, const float4* q, const uint8_t* mask,
                 const float4* pbn, const uint4* rows, const uint2* meta,
                 float4* pbt) {
    chain_wait();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / kSplit, sub = threadIdx.x % kSplit;
    const int n = c.n;
    const bool valid = i < n;
    F3 pbi = {0.0f, 0.0f, 0.0f};  // particle i's own terms, added once
    float lbi = 0.0f;
    if (valid) {
        F3 fb = f3(pbn[i]);
        if (mask) {
            const uint8_t m = mask[i];
            if (m & 3) fb.x = 0.0f;
            if (m & 12) fb.y = 0.0f;
            if (m & 48) fb.z = 0.0f;
        }
        if (sub == 0) pbi = fb;
        const float4 qi = q[i];
        const F3 pi = f3(qi);
        const float a0 = -c.gradSpiky / c.rho0;
        const uint64_t mt = load_meta(meta, i);
        auto loadQ = [&](uint32_t j) {
            j = checked_index(j, (uint32_t)n, c.err, kErrFriendIndex);
            return Friend1{j, q[j]};
        };
        walk_split(rows, n, i, FlatFriends(mt, kept_other(mt)).total, sub, loadQ, [&](const Friend1& f) {
            const uint32_t j = f.j;
            const float4 qj = f.a;
            const F3 r = pi - f3(qj);
            const float r2 = dot(r, r);
            if (!in_support(c, r2)) return;
            float y;
            const float rl = pair_length(r2, y);
            const float d = c.h2 - r2;
            const float rq = d * d * d / c.poly6q;
            const float a = qi.w + qj.w + c.K * rq * rq * rq * rq;
            const F3 k = kvec(r, rl, y, c.h);
            const float ab = a0 * dot(fb, k);
            lbi += ab;
            const float sW = ab * 4.0f * c.K * rq * rq * rq / c.poly6q;
            const F3 rb = (sW * -6.0f * d * d) * r + kvec_adj(r, rl, y, c.h, (a0 * a) * fb);
            pbi = pbi + rb;
            add3(&pbt[j], -1.0f * rb, ab);
        });
    }
    lbi = lanes_sum(lbi);
    pbi = lanes_sum(pbi);
    if (valid && sub == 0) add3(&pbt[i], pbi, lbi);
}

// lambda^t from p^t: adjoint of p^t (pbt) from that of lambda^t (pbt's w, which
// nothing changes here).  Clears pbn, which becomes the next iteration's pbt.
// The sums over the friends are the forward pass' (sums, density).
__global__ void __launch_bounds__(kAdjBlock)
adj_scaling_kernel(DevConsts c, const float4* q, const float4* sums,
                   const float* density, const uint4* rows,
                   const uint2* meta, float4* pbt, float4* pbn) {
    chain_wait();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / kSplit, sub = threadIdx.x % kSplit;
    const int n = c.n;
    const bool valid = i < n;
    const float lbar = valid ? __ldcg(&pbt[i].w) : 0.0f;
    const uint64_t mt = lbar != 0.0f ? load_meta(meta, i) : 0u;
    const int total = FlatFriends(mt, kept_density(mt)).total;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const F3 pi = valid ? f3(q[i]) : f3(zero);
    const float4 sum = valid ? sums[i] : zero;
    const float rho = valid ? density[i] : 0.0f, G = c.gradSpiky, D = sum.w;
    const F3 S = f3(sum);
    auto loadQ = [&](uint32_t j) {
        j = checked_index(j, (uint32_t)n, c.err, kErrFriendIndex);
        return Friend1{j, q[j]};
    };
    const float den = D / c.rho0sq + c.eps, Cc = rho / c.rho0 - 1.0f;
    const float rhob = (-lbar / den) / c.rho0;
    const float Db = lbar * Cc / (den * den) / c.rho0sq;
    F3 pbi = {0.0f, 0.0f, 0.0f};  // particle i's own terms, added once
    walk_split(rows, n, i, total, sub, loadQ, [&](const Friend1& f) {
        const uint32_t j = f.j;
        const F3 r = pi - f3(f.a);
        const float r2 = dot(r, r);
        if (!in_support(c, r2)) return;
        float y;
        const float rl = pair_length(r2, y);
        const float d = c.h2 - r2;
        const F3 g = G * kvec(r, rl, y, c.h);
        const F3 rb = (rhob * c.poly6 * -6.0f * d * d) * r + kvec_adj(r, rl, y, c.h, (G * 2.0f * Db) * (g + S));
        pbi = pbi + rb;
        add3(&pbt[j], -1.0f * rb);
    });
    pbi = lanes_sum(pbi);
    if (valid && sub == 0) {
        if (total > 0) add3(&pbt[i], pbi);
        pbn[i] = zero;
    }
}

// Undo the sort and the prediction p0 = x + dt (v + dt g): adjoints of the
// substep's inputs x, v (previous order) and of g.
__global__ void __launch_bounds__(kAdjBlock)
adj_unsort_predict_kernel(DevConsts c, const uint32_t* perm, const float4* xsb,
                          float4* pb0, float4* xo, float4* vo,
                          float* gbar) {
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    F3 g = {0.0f, 0.0f, 0.0f};
    if (k < c.n) {
        const uint32_t i = checked_index(perm[k], (uint32_t)c.n, c.err, kErrSortIndex);
        const F3 p = f3(pb0[k]);
        pb0[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const F3 x = f3(xsb[k]) + p;
        xo[i] = make_float4(x.x, x.y, x.z, 0.0f);
        vo[i] = make_float4(c.dt * p.x, c.dt * p.y, c.dt * p.z, 0.0f);
        g = (c.dt * c.dt) * p;
    }
    const float gx = block_sum(g.x);
    __syncthreads();
    const float gy = block_sum(g.y);
    __syncthreads();
    const float gz = block_sum(g.z);
    if (threadIdx.x == 0) {
        atomicAdd(&gbar[0], gx);
        atomicAdd(&gbar[1], gy);
        atomicAdd(&gbar[2], gz);
    }
}

// xb[k] = src[ids[k]] (to the current order) or dst[ids[k]] = xb[k] (back).
__global__ void scatter_by_id_kernel(int n, const uint32_t* ids, const float4* byId,
                                     float4* out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) out[k] = byId[ids[k]];
}
__global__ void gather_to_id_kernel(int n, const uint32_t* ids, const float4* in,
                                    float4* byId) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) byId[ids[k]] = in[k];
}

inline unsigned grid_for(int n) { return (unsigned)((n + kAdjBlock - 1) / kAdjBlock); }

}  // namespace

void adjoint_substep(const DevConsts& c, const AdjointTape& tp, AdjointBuffers& ab, cudaStream_t s) {
    const int n = c.n;
    const unsigned wide = (unsigned)(((int64_t)n * kSplit + kAdjBlock - 1) / kAdjBlock);
    launch_chained(adj_vorticity_kernel, wide, kAdjBlock, s, c, tp.pI, tp.omega, tp.rows, tp.meta, ab.vb, ab.omb,
                   ab.pb);
    launch_chained(adj_viscosity_kernel, wide, kAdjBlock, s, c, tp.pI, tp.v2, ab.omb, ab.vb, tp.rows, tp.meta, ab.v2b,
                   ab.pb, &ab.scalars->visc);
    launch_chained(adj_velocity_kernel, grid_for(n), kAdjBlock, s, c, ab.xb, ab.v2b, ab.pb, ab.xsb);
    for (int t = tp.iterations - 1; t >= 0; --t) {
        launch_chained(adj_delta_kernel, wide, kAdjBlock, s, c, tp.q[t], tp.mask ? tp.mask + (size_t)t * n : nullptr,
                       ab.pb, tp.rows, tp.meta, ab.pbt);
        launch_chained(adj_scaling_kernel, wide, kAdjBlock, s, c, tp.q[t], tp.sums[t], tp.rho[t], tp.rows, tp.meta, ab.pbt, ab.pb);
        float4* tmp = ab.pb;
        ab.pb = ab.pbt;
        ab.pbt = tmp;
    }
    launch_chained(adj_unsort_predict_kernel, grid_for(n), kAdjBlock, s, c, tp.perm, ab.xsb, ab.pb, ab.xo, ab.vo,
                   ab.scalars->gravity);
    float4* t1 = ab.xb;
    ab.xb = ab.xo;
    ab.xo = t1;
    float4* t2 = ab.vb;
    ab.vb = ab.vo;
    ab.vo = t2;
}

int adjoint_launches(int iterations) { return 4 + 2 * iterations; }

void scatter_by_id(int n, const uint32_t* ids, const float4* byId, float4* out, cudaStream_t s) {
    scatter_by_id_kernel<<<grid_for(n), kAdjBlock, 0, s>>>(n, ids, byId, out);
}

void gather_to_id(int n, const uint32_t* ids, const float4* in, float4* byId, cudaStream_t s) {
    gather_to_id_kernel<<<grid_for(n), kAdjBlock, 0, s>>>(n, ids, in, byId);
}

}  // namespace pbf
