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

namespace {

void upload(void* d, const void* h, size_t bytes) { cudaMemcpy(d, h, bytes, cudaMemcpyHostToDevice); }
void download(void* h, const void* d, size_t bytes) { cudaMemcpy(h, d, bytes, cudaMemcpyDeviceToHost); }

__global__ void divide_kernel(const float* __restrict__ a, const float* __restrict__ b, uint32_t n, float* __restrict__ out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = a[i] / b[i];
}

__global__ void hiz_level_kernel(uint32_t n, int* __restrict__ out) {
    for (uint32_t d = blockIdx.x * blockDim.x + threadIdx.x; d < n; d += gridDim.x * blockDim.x)
        out[d] = (int)ceilf(log2f((float)(int)d / 2.0f));
}

}  // namespace

// a / b as the library's flags compile it, and the Hi-Z level of extents 0..n - 1 pixels.
extern "C" int gps_check_divide(const float* a, const float* b, uint32_t n, float* out) {
    DeviceArray<float> x(n), y(n), z(n);
    if (!x.p || !y.p || !z.p) return 1;
    upload(x.p, a, (size_t)n * 4);
    upload(y.p, b, (size_t)n * 4);
    divide_kernel<<<148 * 8, 256>>>(x.p, y.p, n, z.p);
    download(out, z.p, (size_t)n * 4);
    return (int)cudaGetLastError();
}

extern "C" int gps_check_hiz_levels(uint32_t n, int* out) {
    DeviceArray<int> d(n);
    if (!d.p) return 1;
    hiz_level_kernel<<<32, 256>>>(n, d.p);
    download(out, d.p, (size_t)n * 4);
    return (int)cudaGetLastError();
}

// Both passes of a frame's block cull on `count` node boxes (8 floats each) of n Gaussians: the culled
// bits, the chunk list with its length and the mask words (all ones before) of each pass.  mips: a Hi-Z
// chain of width x height per pass, coarsest level first.
extern "C" int gps_check_cull(const float* nodes, uint32_t count, uint32_t per_block, uint32_t n, const float* planes24,
                              const float* vp16, const float* const* mips, int width, int height, uint32_t* const* culled,
                              uint32_t* const* list, uint32_t* const* mask, uint32_t* lengths) {
    using namespace gps;
    const uint32_t words = (count + 31u) / 32u, chunks = (n + 31u) / 32u;
    CullArgs a{};
    a.hiz.width = width;
    a.hiz.height = height;
    int top = 0;
    while ((1 << top) < (width > height ? width : height)) ++top;
    a.hiz.levels = top + 1;
    for (int l = 0; l <= top; ++l) {
        a.hiz.level_w[l] = (width + (1 << (top - l)) - 1) >> (top - l);
        a.hiz.level_h[l] = (height + (1 << (top - l)) - 1) >> (top - l);
        a.hiz.level_off[l] = a.hiz.mip_size;
        a.hiz.mip_size += (uint64_t)a.hiz.level_w[l] * (uint64_t)a.hiz.level_h[l];
    }
    DeviceArray<float> mip(a.hiz.mip_size);
    DeviceArray<float4> boxes(2 * (size_t)count), supers(2 * (size_t)words);
    DeviceArray<uint32_t> bits(words + 1), outside(words + 1), masks(chunks + 1), iter(1), number(1), out(chunks + 1);
    if (!mip.p || !boxes.p || !supers.p || !bits.p || !outside.p || !masks.p || !iter.p || !number.p || !out.p) return 1;
    upload(boxes.p, nodes, (size_t)count * 32);
    launch_super_bounds(boxes.p, count, supers.p, 0);
    a.hiz.mip = mip.p;
    a.b = {boxes.p, bits.p, count, words, per_block, number.p, supers.p, outside.p};
    for (int i = 0; i < 6; ++i) a.fc.planes[i] = make_v4(planes24[4 * i], planes24[4 * i + 1], planes24[4 * i + 2], planes24[4 * i + 3]);
    for (int c = 0; c < 4; ++c) a.fc.vp.c[c] = make_v4(vp16[4 * c], vp16[4 * c + 1], vp16[4 * c + 2], vp16[4 * c + 3]);
    a.fc.enable_occlusion = a.fc.enable_hier = 1;
    a.n = n;
    a.list = out.p;
    a.mask_pair[0] = a.mask_pair[1] = masks.p;
    a.mask_iter = iter.p;
    for (int pass = 0; pass < 2; ++pass) {
        upload(mip.p, mips[pass], a.hiz.mip_size * 4);
        cudaMemset(number.p, 0, 4);
        cudaMemset(masks.p, 0xFF, (size_t)chunks * 4);
        a.second_pass = pass;
        launch_cull(a, 0);
        download(culled[pass], bits.p, (size_t)words * 4);
        download(&lengths[pass], number.p, 4);
        download(list[pass], out.p, (size_t)chunks * 4);
        download(mask[pass], masks.p, (size_t)chunks * 4);
    }
    return (int)cudaGetLastError();
}
