// The counting sort's kernels of a bounds-checked build on keys of which some lie
// beyond the table's limit.  The buffers hold more than the limit says, so that
// such a key stays inside them.  Built by tests/test_gpu_checked_keys.py with nvcc
// (-DPBF_CHECK_BOUNDS, together with csrc/pbf_sort.cu) and loaded through ctypes;
// not part of the library.
#include <vector>

#include "pbf_internal.h"

// Sorts n particles by keys of which the table holds `limit`; the error words after
// the scatter and after the gather.
extern "C" int checked_sort(int n, uint32_t limit, const uint32_t* keys, const uint32_t* place, int* errors) {
    const pbf::CountingPlan plan = pbf::make_scan_plan(limit);
    if (plan.blocks != 1 || plan.words <= limit + 64) return -1;
    uint32_t* d[8] = {};  // keys, place, counts, sums, starts, order, keysOut, permOut
    float4* v = nullptr;
    uint32_t* ids = nullptr;
    int* err = nullptr;
    for (auto& p : d)
        if (cudaMalloc((void**)&p, 4 * (plan.words + n)) != cudaSuccess) return -2;
    if (cudaMalloc((void**)&v, 64 * (size_t)n) != cudaSuccess || cudaMalloc((void**)&ids, 8 * (size_t)n) != cudaSuccess ||
        cudaMalloc((void**)&err, 4) != cudaSuccess)
        return -2;
    std::vector<uint32_t> counts(plan.words, 0u);
    for (int i = 0; i < n; ++i) ++counts[keys[i]];
    cudaMemcpy(d[0], keys, 4 * (size_t)n, cudaMemcpyHostToDevice);
    cudaMemcpy(d[1], place, 4 * (size_t)n, cudaMemcpyHostToDevice);
    cudaMemcpy(d[2], counts.data(), 4 * plan.words, cudaMemcpyHostToDevice);
    cudaMemset(v, 0, 64 * (size_t)n);
    cudaMemset(ids, 0, 8 * (size_t)n);
    cudaMemset(err, 0, 4);
    pbf::launch_counting_sort(plan, n, d[2], d[3], d[4], d[0], d[1], d[5], nullptr, limit, err, nullptr);
    cudaMemcpy(errors, err, 4, cudaMemcpyDeviceToHost);
    cudaMemset(err, 0, 4);
    pbf::DevConsts c{};
    c.n = n;
    c.h = 0.1f;
    pbf::launch_cell_gather(c, d[0], d[4], d[5], d[6], d[7], nullptr, v, v + n, ids, v + 2 * n, v + 3 * n, ids + n, limit,
                            err, nullptr);
    cudaError_t e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(errors + 1, err, 4, cudaMemcpyDeviceToHost);
    for (auto& p : d) cudaFree(p);
    cudaFree(v);
    cudaFree(ids);
    cudaFree(err);
    return (int)e;
}
