// Entry points for the tests: device steps and launchers of the frame path, one at a time, as the
// library's kernels use them.  Built into a library of its own (libgps_check.so) on top of
// libgps_b200.so, with the same flags; no part of the renderer calls anything here.
#include <cstdint>
#include <vector>
#include <cuda_runtime.h>
#include "frame_kernels.h"
#include "gps_draw.cuh"

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

namespace {

using Tally = unsigned long long;

// Over all floats: where the draw's steps differ from CUDA's functions.
__global__ void draw_steps_kernel(Tally* differ) {
    using namespace gps;
    const uint64_t threads = (uint64_t)gridDim.x * blockDim.x;
    uint32_t d[6] = {0, 0, 0, 0, 0, 0};
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < (1ull << 32); i += threads) {
        const float v = __uint_as_float((uint32_t)i);
        if (v >= 1.e-37f && v <= 1.0f) {
            const float l = __logf(v);
            d[0] += l > 0.0f;
            d[1] += -neg_root(2.0f * l) != __fsqrt_rn(fmaxf(-2.0f * l, 0.0f));
        }
        if (v >= 1.e-7f && v <= 171.0f) {
            const float2 r = neg_root2(make_float2(-v, -v));
            d[2] += -r.x != __fsqrt_rn(v) || -r.y != __fsqrt_rn(v) || -neg_root(-v) != __fsqrt_rn(v);
        }
        const float2 f = floor_bits2(make_float2(v, v));
        const uint32_t b = __float_as_uint(floor_bits(v)) - kFloorBits;
        if (fabsf(v) < 4194304.0f) d[3] += (int)b != (int)floorf(v) || __float_as_uint(f.x) - kFloorBits != b || __float_as_uint(f.y) - kFloorBits != b;
        else d[4] += b < 200000u || __float_as_uint(f.x) - kFloorBits < 200000u || __float_as_uint(f.y) - kFloorBits < 200000u;
        if (v >= 0.0f && v <= 2.0f) {
            const float2 p = by_li2_max2(make_float2(v, v));
            d[5] += p.x != v / kLi2Max || p.y != v / kLi2Max;
        }
    }
    for (int k = 0; k < 6; ++k)
        if (d[k]) atomicAdd(differ + k, (Tally)d[k]);
}

// Samples of random Gaussians: those that draw_pair and draw_one draw otherwise than draw_sample; live ones.
__global__ void draws_kernel(uint32_t gaussians, uint32_t draws, uint32_t salt, Tally* out) {
    using namespace gps;
    uint32_t differ = 0, live = 0;
    FrameConst fc{};
    fc.num_passes = 4;
    fc.up_width = 3840;
    fc.up_height = 2160;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < gaussians; g += gridDim.x * blockDim.x) {
        u32x2 r = make_seed(g, salt);
        const vec2 a = pcg2d(r), b = pcg2d(r), c = pcg2d(r);
        const float mx = a.x * 3900.0f - 30.0f, my = a.y * 2220.0f - 30.0f;
        const float sx = exp2f(b.x * 12.0f - 2.0f), sy = exp2f(b.y * 12.0f - 2.0f), rho = (c.x - 0.5f) * 1.99f;
        const float xx = sx * sx + 0.3f, yy = sy * sy + 0.3f, xy = rho * sx * sy, inv = 1.0f / (xx * yy - xy * xy);
        SplatRecord rec;
        rec.a = make_float4(mx, my, sqrtf(xx), xy / sqrtf(xx));
        rec.b = make_float4(sqrtf(yy - rec.a.w * rec.a.w), yy * inv, -xy * inv, xx * inv);
        rec.c = make_float4(g & 7u ? c.y * 0.996f + 0.004f : 1.0f, 0.0f, 0.0f, 0.0f);
        ivec2 lo, hi;
        if (!gaussian_tile_bounds(lo, hi, {fc.up_width, fc.up_height}, make_v3(xx, xy, yy), make_v2(mx, my))) continue;
        rec.d = make_uint4((uint32_t)lo.x | ((uint32_t)lo.y << 16), (uint32_t)hi.x | ((uint32_t)hi.y << 16), 0u, 0u);
        const SampleConst k = sample_const(rec, fc, nullptr);
        u32x2 one = make_seed(g, salt + 1u), two = one, single = one;
        for (uint32_t s = 0; s < draws; s += 2u) {
            uint32_t tile[2], code[2];
            bool on[2];
            draw_pair(two, k, tile, code, on);
            for (int j = 0; j < 2; ++j) {
                uint32_t t0, c0, t1, c1;
                const bool l0 = draw_sample(one, k, t0, c0), l1 = draw_one(single, k, t1, c1);
                live += l0;
                differ += l0 != on[j] || l0 != l1 || (l0 && (t0 != tile[j] || c0 != code[j] || t1 != tile[j] || c1 != code[j]));
            }
        }
        differ += one.x != two.x || one.y != two.y || one.x != single.x;
    }
    if (differ) atomicAdd(out, (Tally)differ);
    atomicAdd(out + 1, (Tally)live);
}

}  // namespace

// differ[6]: logarithms above zero, neg_root of one, neg_root of any radicand, floor_bits, floor_bits out
// of range, by_li2_max2.
extern "C" int gps_check_draw_steps(unsigned long long* differ) {
    DeviceArray<Tally> d(6);
    if (!d.p) return 1;
    draw_steps_kernel<<<148 * 8, 256>>>(d.p);
    download(differ, d.p, 6 * sizeof(Tally));
    return (int)cudaGetLastError();
}

// out[2]: samples drawn otherwise, live samples.
extern "C" int gps_check_draws(uint32_t gaussians, uint32_t draws, uint32_t salt, unsigned long long* out) {
    DeviceArray<Tally> d(2);
    if (!d.p) return 1;
    draws_kernel<<<148 * 8, 128>>>(gaussians, draws, salt, d.p);
    download(out, d.p, 2 * sizeof(Tally));
    return (int)cudaGetLastError();
}

namespace {

struct SplatCase {
    const gps::SplatRecord* records;
    const uint32_t *gid, *start;
    uint32_t survivors, points;
    int frame_seed, width, height, passes, k, unbiased;
};

// One thread per point, one sample after the other in the reference's form, no pre-test.
__global__ void plain_splat_kernel(SplatCase a, unsigned long long* buffer) {
    using namespace gps;
    FrameConst fc{};
    fc.num_passes = a.passes;
    fc.up_width = a.width;
    fc.up_height = a.height;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < a.points; p += gridDim.x * blockDim.x) {
        uint32_t r = 0;  // the last survivor that starts at or before p
        for (uint32_t n = a.survivors; n > 1u;) {
            const uint32_t half = n / 2u;
            if (a.start[r + half] <= p) {
                r += half;
                n -= half;
            } else {
                n = half;
            }
        }
        const SplatRecord rec = a.records[a.gid[r]];
        const SampleConst c = sample_const(rec, fc, nullptr);
        const uint64_t key = (uint64_t)rec.d.z | ((uint64_t)rec.d.w << 32);
        u32x2 seed = make_seed(p, (uint32_t)a.frame_seed);
        for (int i = 0; i < a.passes * a.k; ++i) {
            if (a.unbiased) {
                uint32_t tile, code;
                if (draw_sample(seed, c, tile, code)) atomicMin(buffer + sample_slot(c, tile, code, i / a.k), (unsigned long long)key);
                continue;
            }
            const vec2 u = pcg2d(seed), xy = box_muller(u.x, u.y);
            const float px = floorf(c.pixel_mean.x + c.c0 * xy.x), py = floorf(c.pixel_mean.y + c.c1 * xy.x + c.c2 * xy.y);
            const int x = (int)px, y = (int)py;
            if (x < c.minx || x >= c.maxx || y < c.miny || y >= c.maxy) continue;
            if (c.opacity * gaussian_value(c.conic, make_v2(c.pixel_mean.x - px, c.pixel_mean.y - py)) < 1.0f / 255.0f) continue;
            unsigned long long* at = buffer + splat_index(x, y, i / a.k, a.passes, a.width, a.height);
            for (unsigned long long old = *at;;) {
                if ((key & kDepthMask) > (old & kDepthMask)) break;
                const unsigned long long now = (key & kDepthMask) < (old & kDepthMask)
                                                   ? key : (old & kDepthMask) | (((old & kColorMask) + (key & kColorMask)) & kColorMask);
                const unsigned long long was = atomicCAS(at, old, now);
                if (was == old) break;
                old = was;
            }
        }
    }
}

}  // namespace

// The splat of a pass from its records and survivors (device arrays) into a buffer of `entries` that starts at `initial`.
extern "C" int gps_check_splat(const float* d_records, const uint32_t* d_gid, const uint32_t* d_start, uint32_t survivors,
                               uint32_t points, int frame_seed, int width, int height, int passes, int k, int unbiased,
                               uint64_t initial, uint64_t entries, uint64_t* out) {
    DeviceArray<unsigned long long> buffer(entries);
    if (!buffer.p) return 1;
    gps::launch_clear(reinterpret_cast<uint64_t*>(buffer.p), entries, initial, 0);
    const SplatCase a{reinterpret_cast<const gps::SplatRecord*>(d_records), d_gid, d_start, survivors, points, frame_seed, width, height, passes, k, unbiased};
    plain_splat_kernel<<<148 * 4, 128>>>(a, buffer.p);
    download(out, buffer.p, entries * 8);
    return (int)cudaGetLastError();
}
