// Entry points for the tests: device steps and launchers of the frame path, one at a time, as the
// library's kernels use them.  Built into a library of its own (libgps_check.so) on top of
// libgps_b200.so, with the same flags; no part of the renderer calls anything here.
#include <cstdint>
#include <vector>
#include <cuda_runtime.h>
#include "frame_kernels.h"

namespace {

template <class T>
struct DeviceArray {
    T* p = nullptr;
    explicit DeviceArray(size_t n, int fill = 0) {
        if (cudaMalloc(&p, n * sizeof(T)) == cudaSuccess) cudaMemset(p, fill, n * sizeof(T));
        else p = nullptr;
    }
    ~DeviceArray() { cudaFree(p); }
};

}  // namespace

// The block cull of n Gaussians of which no block is culled, its chunk count starting at `stale`:
// list[0 .. 2 * chunks) (0xFFFFFFFF where nothing was written) and the count after it.
extern "C" int gps_check_cull_list(uint32_t n, uint32_t stale, uint32_t* list, uint32_t* count) {
    using namespace gps;
    const uint32_t nodes = (n + 3u) / 4u, words = (nodes + 31u) / 32u, chunks = (n + 31u) / 32u;
    DeviceArray<float4> boxes(2 * (size_t)words * 32), supers(2 * (size_t)words);
    DeviceArray<uint32_t> culled(words + 1), outside(words + 1), mask(chunks + 1), iter(1), number(1), out(2 * (size_t)chunks, 0xFF);
    if (!boxes.p || !supers.p || !culled.p || !outside.p || !mask.p || !iter.p || !number.p || !out.p) return 1;
    cudaMemcpy(number.p, &stale, sizeof(stale), cudaMemcpyHostToDevice);
    CullArgs a{};
    a.b.nodes = boxes.p;
    a.b.culled = culled.p;
    a.b.node_count = nodes;
    a.b.words = words;
    a.b.per_block = 4;
    a.b.chunk_count = number.p;
    a.b.supers = supers.p;
    a.b.outside = outside.p;
    a.n = n;
    a.list = out.p;
    a.mask_pair[0] = a.mask_pair[1] = mask.p;
    a.mask_iter = iter.p;
    launch_cull(a, 0);
    cudaMemcpy(list, out.p, 2 * (size_t)chunks * sizeof(uint32_t), cudaMemcpyDeviceToHost);
    cudaMemcpy(count, number.p, sizeof(uint32_t), cudaMemcpyDeviceToHost);
    return (int)cudaGetLastError();
}

namespace {
__global__ void no_kernel() {}
}  // namespace

// allow_dynamic_smem asked for more than a device has, after an earlier error (or none): whether it
// refused, and whether an error is pending after it.
extern "C" void gps_check_smem_refusal(int earlier_error, int* refused, int* pending) {
    cudaGetLastError();
    if (earlier_error) cudaSetDevice(-1);
    *refused = gps::allow_dynamic_smem(reinterpret_cast<const void*>(no_kernel), 1 << 20) ? 0 : 1;
    *pending = cudaGetLastError() != cudaSuccess ? 1 : 0;
}

namespace {
__global__ void depths_kernel(const uint32_t* __restrict__ keys, uint32_t n, float near_plane, float far_plane, float* __restrict__ out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        out[i] = gps::depth_of_key(keys[i] << 4, near_plane, far_plane);
}
}  // namespace

// The NDC depths of n 28-bit keys (host arrays).
extern "C" int gps_check_depths(const uint32_t* keys, uint32_t n, float near_plane, float far_plane, float* out) {
    DeviceArray<uint32_t> k(n);
    DeviceArray<float> d(n);
    if (!k.p || !d.p) return 1;
    cudaMemcpy(k.p, keys, (size_t)n * 4, cudaMemcpyHostToDevice);
    depths_kernel<<<148 * 8, 256>>>(k.p, n, near_plane, far_plane, d.p);
    cudaMemcpy(out, d.p, (size_t)n * 4, cudaMemcpyDeviceToHost);
    return (int)cudaGetLastError();
}

// Whether the library's sweep over all keys finds a depth that falls as the key grows (-1: an error).
extern "C" int gps_check_depth_falls(float near_plane, float far_plane) {
    DeviceArray<uint32_t> falls(1);
    if (!falls.p) return -1;
    gps::launch_depth_monotone(near_plane, far_plane, falls.p, 0);
    uint32_t n = 0;
    cudaMemcpy(&n, falls.p, sizeof(n), cudaMemcpyDeviceToHost);
    return cudaGetLastError() == cudaSuccess ? (n ? 1 : 0) : -1;
}
