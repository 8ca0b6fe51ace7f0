// Test kernels: the packed forms of the passes' arithmetic (two friends per
// instruction) against the scalar forms, bit for bit.  Built by
// tests/test_gpu_packed.py with nvcc and loaded through ctypes; not part of the
// library.
#include <cstdint>

#include "pbf_device.cuh"

namespace {

using namespace pbf;

__device__ __forceinline__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// Every r2 in [first, last), with r2's bit-reversed partner as the second friend.
__global__ void sqrt_kernel(uint32_t first, uint32_t last, unsigned long long* bad) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t b = first + blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; b < last; b += stride) {
        const float r0 = __uint_as_float((uint32_t)b);
        const float r1 = __uint_as_float(last - 1u - ((uint32_t)b - first));
        float l0, y0, l1, y1;
        sqrt_recip_rn(r0, l0, y0);
        sqrt_recip_rn(r1, l1, y1);
        F2 nrl, y;
        sqrt_recip_rn2(pack2(r0, r1), nrl, y);
        const float2 l = unpack2(nrl), q = unpack2(y);
        if (!same(-l.x, l0) || !same(-l.y, l1) || !same(q.x, y0) || !same(q.y, y1)) atomicAdd(bad, 1ull);
    }
}

// Seeded differences r: r^2, the quotients r / |r| and the square of their sum
// term, as the density pass chains them.
__global__ void chain_kernel(DevConsts c, uint32_t seed, int rounds, unsigned long long* bad) {
    uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) * 2654435761u + seed;
    auto draw = [&] {
        s = s * 1664525u + 1013904223u;
        return ((int)(s >> 8) - (1 << 23)) * 0x1p-27f;
    };
    for (int k = 0; k < rounds; ++k) {
        float v[6];
        for (float& x : v) x = draw();
        const F2 rx = pack2(v[0], v[3]), ry = pack2(v[1], v[4]), rz = pack2(v[2], v[5]);
        const F2 r2 = dot2(c, rx, ry, rz, rx, ry, rz);
        F2 nrl, y;
        sqrt_recip_rn2(r2, nrl, y);
        const F2 gx = quotient_rn2(rx, nrl, y), gy = quotient_rn2(ry, nrl, y), gz = quotient_rn2(rz, nrl, y);
        const float2 gg = unpack2(dot2(c, gx, gy, gz, gx, gy, gz)), d = unpack2(sub2(both(c.h2), r2));
        for (int f = 0; f < 2; ++f) {
            const float* a = v + 3 * f;
            const float s2 = dot3(a[0], a[1], a[2], a[0], a[1], a[2]);
            float l, w;
            sqrt_recip_rn(s2, l, w);
            const float x = quotient_rn(a[0], l, w), z0 = quotient_rn(a[1], l, w), z1 = quotient_rn(a[2], l, w);
            const float want = dot3(x, z0, z1, x, z0, z1);
            if (!same(f ? gg.y : gg.x, want) || !same(f ? d.y : d.x, c.h2 - s2)) atomicAdd(bad, 1ull);
        }
    }
}

int finish(unsigned long long* d, unsigned long long* out) {
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(out, d, 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}

}  // namespace

extern "C" int packed_sqrt_check(uint32_t first, uint32_t last, unsigned long long* out) {
    unsigned long long* d = nullptr;
    if (cudaMalloc((void**)&d, 8) != cudaSuccess) return -1;
    cudaMemset(d, 0, 8);
    sqrt_kernel<<<1216, 256>>>(first, last, d);
    return finish(d, out);
}

extern "C" int packed_chain_check(float h2, uint32_t seed, int rounds, unsigned long long* out) {
    unsigned long long* d = nullptr;
    if (cudaMalloc((void**)&d, 8) != cudaSuccess) return -1;
    cudaMemset(d, 0, 8);
    DevConsts c{};
    c.h2 = h2;
    c.negZero2 = 0x8000000080000000ull;
    chain_kernel<<<1216, 256>>>(c, seed, rounds, d);
    return finish(d, out);
}
