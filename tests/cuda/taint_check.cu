// Test kernel: quotients_tainted of lanes that find different marks (each lane
// looks at a particle of its own here).  Built by tests/test_gpu_taint_lanes.py
// with nvcc and loaded through ctypes; not part of the library.
#include <cstdint>

#include "pbf_device.cuh"

namespace {

template <int L>
__global__ void taint_kernel(pbf::DevConsts c, uint32_t* answers) {
    answers[threadIdx.x] = pbf::quotients_tainted<L>(c, (int)threadIdx.x);
}

}  // namespace

// marks, answers: 64 words of the host; a mark of 1 is this substep's.
extern "C" int taint_check(int lanes, const uint32_t* marks, uint32_t* answers) {
    uint32_t* d = nullptr;  // marks, answers, the substep's number
    if (cudaMalloc((void**)&d, 4 * 129) != cudaSuccess) return -1;
    const uint32_t epoch = 1;
    cudaMemcpy(d, marks, 4 * 64, cudaMemcpyHostToDevice);
    cudaMemcpy(d + 128, &epoch, 4, cudaMemcpyHostToDevice);
    pbf::DevConsts c{};
    c.taint = d;
    c.epoch = d + 128;
    if (lanes == 1) taint_kernel<1><<<1, 64>>>(c, d + 64);
    else if (lanes == 4) taint_kernel<4><<<1, 64>>>(c, d + 64);
    else taint_kernel<8><<<1, 64>>>(c, d + 64);
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(answers, d + 64, 4 * 64, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
