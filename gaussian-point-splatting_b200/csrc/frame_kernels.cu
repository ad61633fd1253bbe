// sm_100a kernels of the Gaussian point-splatting frame path.
//
//   block cull    gaussian_bvh.cu:215-329          one thread per block node, warp ballot, boxes of 32 first
//   preprocess    gaussian_point_splatting.cu:17-65,147-307
//   scan          workload_distributor.cu:52-145   tile reduce -> tile scan -> downsweep that
//                                                  compacts survivors and keeps P on the device
//   splat         gaussian_point_splatting.cu:67-141,383-432  persistent, tile-of-points blocks
//   clear/resolve gaussian_point_splatting.cu:484-548,580-585
//   Hi-Z          depth_mip_chain.cu:7-145, depth_mip_chain.cuh:172-215
//   TAA/progress  post_processing_kernels.cuh:108-285
//
// Every floating-point expression that decides a sample position, a count or a packed
// value follows the reference's expression shape (see gps_math.cuh) so that the 64-bit
// splat buffer is bit-identical to the reference kernels' for the same inputs.
#include <algorithm>
#include <type_traits>
#include <cstdio>
#include <mutex>
#include <string>
#include "../../include/gps_b200.h"
#include "frame_kernels.h"
#include "gps_draw.cuh"
#include "gps_rng.cuh"
#include "host_io.hpp"

namespace gps {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;   // per thread and round
constexpr int kScanRoundsMax = 4;  // a thread covers kScanItems * rounds consecutive Gaussians:
                                   // 1 round (4096-Gaussian tiles) below kScanBigScene, else 4
constexpr uint32_t kScanTile = kScanThreads * kScanItems * kScanRoundsMax;  // largest tile, 16384
constexpr uint32_t kScanTileSmall = kScanThreads * kScanItems;             // 4096
constexpr uint32_t kScanBigScene = 32u << 20;

// First statement of every kernel that launch_k starts: such a kernel may be scheduled while the
// previous kernel of its stream drains, so it reads and writes nothing before that kernel's
// memory is complete.
__device__ __forceinline__ void previous_kernel_done() { cudaGridDependencySynchronize(); }

// ---------------------------------------------------------------------------------
// Hi-Z query (depth_mip_chain.cuh:172-215, the non-tree variant the reference compiles)
// ---------------------------------------------------------------------------------
__device__ __forceinline__ bool hiz_occluded(const HizView& c, float depth, ivec2 mn, ivec2 mx) {
    mn.x = max(0, mn.x);
    mn.y = max(0, mn.y);
    mx.x = min(c.width - 1, mx.x);
    mx.y = min(c.height - 1, mx.y);
    int w = mx.x - mn.x + 1;
    int h = mx.y - mn.y + 1;
    int d = max(w, h);
    int lod = (int)ceilf(log2f((float)d / 2.0f));
    lod = min(max(lod, 0), c.levels - 1);
    int l = (c.levels - 1) - lod;
    const int wl = c.level_w[l];
    const int hl = c.level_h[l];
    int tile_w = max(1, min(c.width, 1 << (c.levels - l - 1)));
    int tile_h = max(1, min(c.height, 1 << (c.levels - l - 1)));
    int tx0 = max(0, min(wl - 1, mn.x / tile_w));
    int ty0 = max(0, min(hl - 1, mn.y / tile_h)) * wl;
    int tx1 = max(0, min(wl - 1, mx.x / tile_w));
    int ty1 = max(0, min(hl - 1, mx.y / tile_h)) * wl;
    const float* base = c.mip + c.level_off[l];
    float zmax = fmaxf(base[tx0 + ty0], fmaxf(base[tx1 + ty0], fmaxf(base[tx0 + ty1], base[tx1 + ty1])));
    return zmax < depth;
}

__device__ __forceinline__ bool block_culled(const BlockView& b, uint32_t g) {
    uint32_t node = g / b.per_block;
    return ((__ldg(&b.culled[node >> 5]) >> (node & 31)) & 1u) != 0u;
}

__device__ __forceinline__ bool mask_bit(const uint32_t* m, uint32_t g) {
    return ((__ldg(&m[g >> 5]) >> (g & 31)) & 1u) != 0u;
}

// ---------------------------------------------------------------------------------
// Block cull (gaussian_bvh.cu:215-329)
// ---------------------------------------------------------------------------------
// The sums of both tests are spelled out in the rounding that the reference's kernel is compiled to.
// Left to the compiler, which products are fused depends on the kernel they are inlined into, and one
// to seven of 8.4M boxes a frame were then culled otherwise, with other point indices and hence other
// samples for all that follow (the forms were told apart by the culled bits of 40 such frames).
__device__ __forceinline__ bool aabb_outside_frustum(vec3 bmin, vec3 bmax, const vec4* planes) {
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const vec3 n = make_v3(planes[i].x, planes[i].y, planes[i].z);
        const float d = planes[i].w;
        vec3 v = make_v3(n.x >= 0.0f ? bmax.x : bmin.x, n.y >= 0.0f ? bmax.y : bmin.y, n.z >= 0.0f ? bmax.z : bmin.z);
        if (__fadd_rn(__fmaf_rn(n.z, v.z, __fmaf_rn(n.x, v.x, __fmul_rn(n.y, v.y))), d) < 0.0f) return true;
    }
    return false;
}

// One row of view-projection * (v, 1).
__device__ __forceinline__ float project_row(float a, float b, float c, float d, vec3 v) {
    return __fadd_rn(__fmaf_rn(a, v.x, __fmul_rn(b, v.y)), __fmaf_rn(c, v.z, d));
}
__device__ __forceinline__ vec4 project_corner(const mat4& m, vec3 v) {
    return make_v4(project_row(m.c[0].x, m.c[1].x, m.c[2].x, m.c[3].x, v), project_row(m.c[0].y, m.c[1].y, m.c[2].y, m.c[3].y, v),
                   project_row(m.c[0].z, m.c[1].z, m.c[2].z, m.c[3].z, v), project_row(m.c[0].w, m.c[1].w, m.c[2].w, m.c[3].w, v));
}

__device__ __forceinline__ bool aabb_project_bounds(vec3 bmin, vec3 bmax, const mat4& vp, int width, int height,
                                                    ivec2& out_min, ivec2& out_max, float& out_depth) {
    vec3 corners[8] = {{bmin.x, bmin.y, bmin.z}, {bmax.x, bmin.y, bmin.z}, {bmin.x, bmax.y, bmin.z},
                       {bmax.x, bmax.y, bmin.z}, {bmin.x, bmin.y, bmax.z}, {bmax.x, bmin.y, bmax.z},
                       {bmin.x, bmax.y, bmax.z}, {bmax.x, bmax.y, bmax.z}};
    int minx = width - 1, miny = height - 1, maxx = 0, maxy = 0;
    float min_depth = 1e30f;
    bool any_front = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const vec4 clip = project_corner(vp, corners[i]);
        if (clip.w <= 0.0f) continue;
        any_front = true;
        vec3 ndc = make_v3(clip.x / clip.w, clip.y / clip.w, clip.z / clip.w);
        int px = int((ndc.x * 0.5f + 0.5f) * width);
        int py = int((ndc.y * 0.5f + 0.5f) * height);
        minx = min(minx, px);
        miny = min(miny, py);
        maxx = max(maxx, px);
        maxy = max(maxy, py);
        min_depth = fminf(min_depth, ndc.z);
    }
    if (!any_front) return false;
    minx = max(minx, 0);
    miny = max(miny, 0);
    maxx = min(maxx, width - 1);
    maxy = min(maxy, height - 1);
    if (minx > maxx || miny > maxy) return false;
    out_min = {minx, miny};
    out_max = {maxx, maxy};
    out_depth = min_depth;
    return true;
}

// A box that holds 32 nodes' boxes is outside only by more than the rounding of a node's own test:
// in exact arithmetic a node's support vertex lies no further in than the large box's, and both
// sums are off by at most 4 roundings of the terms' magnitudes (2.4e-7 of them).
__device__ __forceinline__ bool aabb_surely_outside_frustum(vec3 bmin, vec3 bmax, const vec4* planes) {
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const vec4 n = planes[i];
        const float x = n.x * (n.x >= 0.0f ? bmax.x : bmin.x), y = n.y * (n.y >= 0.0f ? bmax.y : bmin.y),
                    z = n.z * (n.z >= 0.0f ? bmax.z : bmin.z);
        if (x + y + z + n.w < -1.0e-6f * (fabsf(x) + fabsf(y) + fabsf(z) + fabsf(n.w))) return true;
    }
    return false;
}

// The splat buffer's clear beside a frame's first kernel: block `part` of `parts`.
__device__ __forceinline__ void clear_beside(const ClearArgs& c, uint32_t part, uint32_t parts) {
    const ulonglong2 v = make_ulonglong2(c.value, c.value);
    for (uint64_t i = (uint64_t)part * blockDim.x + threadIdx.x; i < c.pairs; i += (uint64_t)parts * blockDim.x) c.buffer[i] = v;
}

// Whether a node is culled: outside the frustum or behind the Hi-Z depth.
__device__ __forceinline__ bool node_culled(const BlockView& b, const FrameConst& fc, const HizView& hiz, uint32_t idx,
                                            bool test_frustum, bool& outside) {
    const float4 lo = __ldg(&b.nodes[2 * (size_t)idx]), hi = __ldg(&b.nodes[2 * (size_t)idx + 1]);
    const vec3 bmin = make_v3(lo.x, lo.y, lo.z), bmax = make_v3(hi.x, hi.y, hi.z);
    outside = test_frustum && aabb_outside_frustum(bmin, bmax, fc.planes);
    if (outside) return true;
    if (!fc.enable_occlusion) return false;
    ivec2 mn, mx;
    float front;
    return aabb_project_bounds(bmin, bmax, fc.vp, hiz.width, hiz.height, mn, mx, front) && hiz_occluded(hiz, front, mn, mx);
}

// The culled bits of the 32 nodes of a word, by one warp; `outside` are the nodes known to lie
// outside the frustum, which the frame's first pass finds out here.
__device__ __forceinline__ uint32_t cull_word(const CullArgs& a, uint32_t word, uint32_t& outside) {
    const uint32_t lane = threadIdx.x & 31u, idx = (word << 5) + lane;
    const bool node = idx < a.b.node_count && !((outside >> lane) & 1u);
    bool out = false, culled = false;
    if (node) culled = node_culled(a.b, a.fc, a.hiz, idx, !a.second_pass, out);
    outside |= __ballot_sync(0xffffffffu, out);
    return outside | __ballot_sync(0xffffffffu, culled);
}

// Block cull and the list of visible chunks: a chunk is 32 Gaussians (one survivor-mask word),
// visible if it holds an unculled block; the others' mask words are zeroed here, since the
// preprocess skips them.  The frame's first launch clears the splat buffer beside it, on the blocks
// after the first `cull_blocks`.
//
// Most of a scene is outside the frustum, and a node's test is a chain of dependent loads (its box,
// then the Hi-Z texels) that costs 2-3 us however few of a warp's nodes need it.  So a thread first
// tests the box around a word's 32 nodes (first pass) or looks whether all 32 were outside in the
// first pass (second pass, same camera), the words that are left go to a list in shared memory,
// and the warps take those.  A block has a.words_per_block words (8 to 64: enough blocks to fill the
// GPU where the scene is small) and lists their chunks: a word's 32 nodes of per_block Gaussians are exactly
// per_block chunks, so a chunk's nodes are all in one word.
// One launch instead of three; cull and clear 225 -> 133 us a frame with 8.4M nodes (33.6M town, of
// which the boxes are 42 us at the copy rate), the frame 1530 -> 1434; 1M nodes 1009 -> 999; taking 256
// nodes a block one group after the other instead, 253.
constexpr uint32_t kCullWords = 64;

__global__ void __launch_bounds__(256) cull_kernel(CullArgs a) {
    previous_kernel_done();
    if (blockIdx.x >= a.cull_blocks) {
        clear_beside(a.clear, blockIdx.x - a.cull_blocks, gridDim.x - a.cull_blocks);
        return;
    }
    __shared__ uint32_t culled[kCullWords], outside[kCullWords], todo[kCullWords], todo_count;
    const BlockView& b = a.b;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const uint32_t w0 = blockIdx.x * a.words_per_block, n0 = w0 << 5, pb = b.per_block;
    const uint32_t words = min(a.words_per_block, b.words - w0);
    if (t == 0u) todo_count = 0u;
    __syncthreads();
    if (t < words) {
        const uint32_t word = w0 + t, left = b.node_count - (word << 5);
        const uint32_t all = left >= 32u ? 0xffffffffu : (1u << left) - 1u;
        uint32_t out = 0u;
        if (a.second_pass) {
            out = b.outside[word];
        } else {
            const float4 lo = __ldg(&b.supers[2 * (size_t)word]), hi = __ldg(&b.supers[2 * (size_t)word + 1]);
            if (aabb_surely_outside_frustum(make_v3(lo.x, lo.y, lo.z), make_v3(hi.x, hi.y, hi.z), a.fc.planes)) out = all;
        }
        outside[t] = culled[t] = out;
        if (out != all) todo[atomicAdd(&todo_count, 1u)] = t;
    }
    __syncthreads();
    for (uint32_t i = warp; i < todo_count; i += 8u) {
        const uint32_t w = todo[i];
        uint32_t out = outside[w];
        const uint32_t m = cull_word(a, w0 + w, out);
        if (lane == 0u) {
            culled[w] = m;
            outside[w] = out;
        }
    }
    __syncthreads();
    if (t < words) {
        b.culled[w0 + t] = culled[t];
        if (!a.second_pass) b.outside[w0 + t] = outside[t];
    }
    uint32_t* mask = (*a.mask_iter & 1u) ? a.mask_pair[1] : a.mask_pair[0];
    const uint32_t chunks = (a.n + 31u) >> 5;
    const uint32_t c0 = w0 * pb, c1 = min((w0 + words) * pb, chunks);
    for (uint32_t base = c0 + (warp << 5); base < c1; base += 256u) {
        const uint32_t c = base + lane;
        bool vis = false;
        if (c < c1) {
            const uint32_t first = (c << 5) / pb - n0, last = min((c << 5) + 31u, a.n - 1u) / pb - n0;
            const uint32_t nodes = 0xffffffffu << (first & 31u) & 0xffffffffu >> (31u - (last & 31u));
            vis = (~culled[first >> 5] & nodes) != 0u;
            if (!vis) mask[c] = 0u;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, vis);
        if (m == 0u) continue;
        uint32_t slot = 0;
        if (lane == 0u) slot = atomicAdd(b.chunk_count, (uint32_t)__popc(m));
        slot = __shfl_sync(0xffffffffu, slot, 0);
        slot += (uint32_t)__popc(m & ((1u << lane) - 1u));
        if (vis && slot < chunks) a.list[slot] = c;  // (always, if the count started at zero)
    }
}

// The boxes around every 32 nodes (load time); one with a coordinate that is not finite in it gets
// NaN, which no test calls outside.
__global__ void super_bounds_kernel(const float4* __restrict__ nodes, uint32_t node_count, float4* __restrict__ supers,
                                    uint32_t words) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= words) return;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    bool finite = true;
    for (uint32_t i = w << 5; i < min((w + 1u) << 5, node_count); ++i) {
        const float4 a = nodes[2 * (size_t)i], b = nodes[2 * (size_t)i + 1];
        const float x[3] = {a.x, a.y, a.z}, y[3] = {b.x, b.y, b.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            // (by the bits: fast math may take a test against infinity for always true)
            finite &= (__float_as_uint(x[k]) & 0x7F800000u) != 0x7F800000u && (__float_as_uint(y[k]) & 0x7F800000u) != 0x7F800000u;
            lo[k] = fminf(lo[k], x[k]);
            hi[k] = fmaxf(hi[k], y[k]);
        }
    }
    const float nan = __uint_as_float(0x7FFFFFFFu);
    supers[2 * (size_t)w] = finite ? make_float4(lo[0], lo[1], lo[2], 0.0f) : make_float4(nan, nan, nan, 0.0f);
    supers[2 * (size_t)w + 1] = finite ? make_float4(hi[0], hi[1], hi[2], 0.0f) : make_float4(nan, nan, nan, 0.0f);
}

// ---------------------------------------------------------------------------------
// Preprocess (gaussian_point_splatting.cu:17-65 + 147-307)
// ---------------------------------------------------------------------------------
__device__ __forceinline__ void splat_samples_biased(u32x2& seed, const SplatRecord& rec, const FrameConst& fc,
                                                     uint64_t* __restrict__ buffer, int first, int last);
__device__ __forceinline__ void splat_samples_unbiased(u32x2& seed, const SplatRecord& rec, const FrameConst& fc,
                                                       uint64_t* __restrict__ buffer, const uint32_t* spread, int first,
                                                       int last);

// One Gaussian: true if it splats this pass (record and count written).  kImmediate: a
// Gaussian of at most a.immediate_threshold points is splatted here instead, its samples
// drawn from the seed state the point count left (ENABLE_IMMEDIATE_SPLATTING,
// gaussian_point_splatting.cu:272-287), and it is no survivor.
template <class Scene, bool kImmediate>
__device__ __forceinline__ bool preprocess_one(const PreprocessArgs& a, const Scene& scene, uint32_t gi, bool culled,
                                               const uint32_t* __restrict__ mask_prev, bool& loaded,
                                               uint32_t& out_points, uint32_t& out_bin) {
    const int idx = (int)gi;
    const FrameConst& fc = a.fc;
    bool splats = false;
    loaded = false;
    out_points = 0;
    out_bin = 0xFFFFFFFFu;
    do {
        if (idx >= (int)a.n) break;
        if (culled) break;
        if (a.only_previously_occluded && mask_bit(mask_prev, (uint32_t)idx)) break;
        loaded = true;
        u32x2 seed = make_seed((uint32_t)idx, (uint32_t)a.frame_seed);
        float opacity = scene.opacity((uint32_t)idx);
        if (opacity <= 0.0f) break;

        vec3 mean, scale;
        vec4 quat;
        scene.geometry((uint32_t)idx, mean, quat, scale);
        // loadAndTransformGaussian
        vec3 view_mean = transform_point4x3(mean, fc.view);
        float view_z = view_mean.z;
        if (-view_z <= 0.2f) break;
        vec4 proj_mean = fc.vp * make_v4(mean.x, mean.y, mean.z, 1.0f);
        proj_mean = proj_mean * (1.0f / proj_mean.w);
        if (proj_mean.z < -1.0f || proj_mean.z > 1.0f) break;
        mat3 cov = scale_rot_to_cov(scale, quat);
        vec3 cov2d = compute_cov2d(fc.view, cov, mean, fc.tan_fov, fc.focal);
        const float dil = 0.3f * (float)fc.ss * (float)fc.ss;
        cov2d = cov2d + make_v3(dil, 0.0f, dil);
        float det = cov2d.x * cov2d.z - cov2d.y * cov2d.y;
        double det64 = 0.0;
        bool precise = false;
        if constexpr (Scene::kFp64Conic) {
            if (det < 1.0e-3f * cov2d.x * cov2d.z) {  // a*c - b^2 cancels: recompute in FP64
                det64 = (double)cov2d.x * (double)cov2d.z - (double)cov2d.y * (double)cov2d.y;
                det = (float)det64;
                precise = true;
            }
        }
        if (det <= 0.0f) break;
        vec2 pixel_mean = make_v2((proj_mean.x * 0.5f + 0.5f) * (float)fc.up_width,
                                  (proj_mean.y * 0.5f + 0.5f) * (float)fc.up_height);
        ivec2 pmin, pmax;
        if (!gaussian_tile_bounds(pmin, pmax, {fc.up_width, fc.up_height}, cov2d, pixel_mean)) break;

        if (pmin.x >= fc.up_width || pmin.y >= fc.up_height || pmax.x < 0 || pmax.y < 0) break;
        if (fc.cull_small) {
            float trace = cov2d.x + cov2d.z;
            float half = 0.5f * trace;
            float term2 = __fsqrt_rn(fmaxf(0.1f, half * half - det));
            float e1 = half + term2;
            float e2 = half - term2;
            if (e1 < 0.02f || e2 < 0.02f) break;
        }
        constexpr float kTwoPi = 2.0f * 3.14159265358979323846f;
        float importance;
        float s_det = __fsqrt_rn(det);
        if (fc.use_unbiased) importance = kTwoPi * s_det * dilog(opacity);
        else importance = opacity * kTwoPi * s_det;

        if (fc.enable_occlusion) {
            ivec2 qmin = {pmin.x / fc.ss, pmin.y / fc.ss};
            ivec2 qmax = {pmax.x / fc.ss, pmax.y / fc.ss};
            if (hiz_occluded(a.hiz, proj_mean.z, qmin, qmax)) break;
        }
        const float kf = (float)fc.k_points;  // ss^2 x POINTS_PER_KERNEL, 1, or the K override
        uint32_t num_points;
        if (fc.use_unbiased) num_points = poisson(seed, importance);
        else num_points = (uint32_t)stochastic_round(importance, pcg2d(seed).x);
        if (kf > 1) num_points = (uint32_t)stochastic_round((float)num_points / kf, pcg2d(seed).x);
        if (num_points <= 0) break;
        uint32_t cap = (uint32_t)(fc.up_width * fc.up_height / (2 * kf));
        num_points = (cap < num_points) ? cap : num_points;

        vec3 campos = make_v3(fc.cam.c[3].x, fc.cam.c[3].y, fc.cam.c[3].z);
        vec3 color = scene.color((uint32_t)idx, mean, campos);

        // per-Gaussian prologue of splatGaussianPoint (gaussian_point_splatting.cu:88-96)
        const uint64_t view_depth_bits = depth_key(view_z, fc.near_plane, fc.far_plane) << kDepthShift;
        vec3 conic;
        if (precise) conic = make_v3((float)(cov2d.z / det64), (float)(-cov2d.y / det64), (float)(cov2d.x / det64));
        else conic = conic_of(cov2d, 1.0f / det);
        const float c0 = __fsqrt_rn(cov2d.x);
        const float c1 = cov2d.y / c0;
        const float c2 = __fsqrt_rn(cov2d.z - c1 * c1);
        uint32_t r12 = (uint32_t)(color.x * 255.0f) & 0xFFFu;
        uint32_t g12 = (uint32_t)(color.y * 255.0f) & 0xFFFu;
        uint32_t b12 = (uint32_t)(color.z * 255.0f) & 0xFFFu;
        uint64_t key = view_depth_bits | (uint64_t(r12) << 24) | (uint64_t(g12) << 12) | uint64_t(b12);

        SplatRecord rec;
        rec.a = make_float4(pixel_mean.x, pixel_mean.y, c0, c1);
        rec.b = make_float4(c2, conic.x, conic.y, conic.z);
        rec.c = make_float4(opacity, color.x, color.y, color.z);
        rec.d = make_uint4((uint32_t)pmin.x | ((uint32_t)pmin.y << 16), (uint32_t)pmax.x | ((uint32_t)pmax.y << 16),
                           (uint32_t)key, (uint32_t)(key >> 32));
        if constexpr (kImmediate) {
            if ((int)num_points <= a.immediate_threshold) {
                const int samples = fc.num_passes * fc.k_points;
                for (uint32_t pt = 0; pt < num_points; ++pt) {
                    if (fc.use_unbiased) splat_samples_unbiased(seed, rec, fc, a.buffer, nullptr, 0, samples);
                    else splat_samples_biased(seed, rec, fc, a.buffer, 0, samples);
                }
                a.counts[idx] = 0;
                break;
            }
        }
        a.records[idx] = rec;
        a.counts[idx] = num_points;
        out_points = num_points;
        if (a.bins)
            out_bin = screen_bin(pixel_mean.x, pixel_mean.y, fc.up_width, fc.up_height, a.bin_shift, a.bins_x, a.bins_y);
        splats = true;
    } while (false);
    return splats;
}

// Persistent over 32-Gaussian chunks (one mask word each): a warp takes chunk after chunk, so
// a pass over a mostly culled scene costs a bit test per Gaussian, not a thread-block launch
// per 256 Gaussians.  A frame's first pass without a cull launch ahead of it clears the splat buffer
// here, on the blocks after the first a.blocks_here.
//
// kCull: the block cull of a small scene (kSelfCullGaussians) inside, instead of a launch ahead: a warp
// has up to two chunks, half the scene apart so that a visible region's neighbours go to different
// warps, and its lanes test those chunks' nodes first.  Frames of the 60k town
// at 320x180 62.7 -> 56.3 us, 300k at 999x571 109.5 -> 106.0, with the clear here too a 20k cube 18.5 -> 17.7.
//
// kImmediate: the compiler takes 80 registers for the splat in it, three blocks per SM; held to 64 (and a few
// spills outside the sample loop), four: 150k town, compressed, 411x191, all Gaussians of up to 20 points
// splatted here, 8 spp: 917 -> 544 us (FP32 918 -> 544).
template <class Scene, bool kImmediate, bool kCull>
__global__ void __launch_bounds__(256, kImmediate ? 4 : 0) preprocess_kernel(PreprocessArgs a, Scene scene) {
    previous_kernel_done();
    if (blockIdx.x >= a.blocks_here) {
        clear_beside(a.clear, blockIdx.x - a.blocks_here, gridDim.x - a.blocks_here);
        return;
    }
    uint32_t* mask_cur = a.mask_cur;
    const uint32_t* mask_prev = a.mask_prev;
    if (a.mask_iter) {
        const bool odd = (*a.mask_iter & 1u) != 0u;
        mask_cur = odd ? a.mask_pair[1] : a.mask_pair[0];
        mask_prev = odd ? a.mask_pair[0] : a.mask_pair[1];
    }
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = a.blocks_here * (blockDim.x >> 5);
    const uint32_t first = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    uint32_t loaded_tally = 0;  // this warp's Gaussians whose attributes were read
    // this warp's running survivor / point totals of one scan tile, flushed on a tile change
    uint32_t tile = 0xFFFFFFFFu, tile_s = 0, tile_p = 0;
    auto flush_tile = [&]() {
        if (lane == 0 && tile != 0xFFFFFFFFu && tile_s) {
            // two 32-bit halves: the point total wraps mod 2^32 without carrying into the count
            uint32_t* w = reinterpret_cast<uint32_t*>(a.tile_totals + tile);
            atomicAdd(w, tile_p);
            atomicAdd(w + 1, tile_s);
        }
    };
    auto chunk = [&](uint32_t c, bool culled) {
        bool loaded;
        uint32_t pts, bin;
        const bool splats = preprocess_one<Scene, kImmediate>(a, scene, (c << 5) + lane, culled, mask_prev, loaded, pts, bin);
        const unsigned m = __ballot_sync(0xffffffffu, splats);
        loaded_tally += (uint32_t)__popc(__ballot_sync(0xffffffffu, loaded));
        if (lane == 0) mask_cur[c] = m;
        if (m) {
            const uint32_t t = (c << 5) >> a.tile_shift;
            if (t != tile) {
                flush_tile();
                tile = t;
                tile_s = tile_p = 0;
            }
            tile_s += (uint32_t)__popc(m);
            tile_p += __reduce_add_sync(0xffffffffu, pts);
        }
        if (a.bins && m) {  // one atomic per distinct bin cursor among the warp's survivors
            bin += (c & ((1u << a.bin_sub_log2) - 1u)) * a.bin_count;  // this chunk's cursor of each bin
            unsigned todo = m;
            while (todo) {
                const uint32_t key = __shfl_sync(0xffffffffu, bin, __ffs(todo) - 1);
                const unsigned members = __ballot_sync(0xffffffffu, ((todo >> lane) & 1u) && bin == key);
                const uint32_t sum = __reduce_add_sync(0xffffffffu, ((members >> lane) & 1u) ? pts : 0u);
                if (lane == 0) atomicAdd(a.bins + key, ((unsigned long long)__popc(members) << 32) | sum);
                todo &= ~members;
            }
        }
    };
    if constexpr (kCull) {
        const uint32_t chunks = (a.n + 31u) >> 5;
        // lane 8 q + k: node k of chunk first + q * warps (a chunk is eight nodes of four Gaussians)
        const uint32_t c = first + (lane >> 3) * warps, node = (c << 3) + (lane & 7u);
        bool outside, culled = false;
        if (lane < 8u * kSelfCullChunks && c < chunks && node < a.blocks.node_count)
            culled = node_culled(a.blocks, a.fc, a.hiz, node, true, outside);
        const uint32_t bits = __ballot_sync(0xffffffffu, culled);
        for (uint32_t q = 0; q < kSelfCullChunks; ++q) {
            const uint32_t at = first + q * warps;
            if (at >= chunks) break;
            const uint32_t byte = (bits >> (8u * q)) & 0xFFu;
            if (lane == 0) reinterpret_cast<uint8_t*>(a.blocks.culled)[at] = (uint8_t)byte;
            const bool mine = (byte >> (lane >> 2)) & 1u;
            if (__any_sync(0xffffffffu, !mine && (at << 5) + lane < a.n)) chunk(at, mine);
            else if (lane == 0) mask_cur[at] = 0u;
        }
    } else {
        // contiguous ranges of the list (or of all chunks), so that tile totals merge; the next listed
        // chunk's attributes are prefetched into L2 while this one is worked on (256M town: preprocess
        // 1.149 -> 1.130 ms/frame)
        const uint32_t chunks = (a.n + 31u) >> 5, count = a.chunk_list ? min(*a.chunk_count, chunks) : chunks;
        const uint32_t per = (count + warps - 1) / warps;
        const uint32_t b = first * per, e = min(count, b + per);
        uint32_t next = b < e && a.chunk_list ? __ldg(a.chunk_list + b) : b;
        for (uint32_t i = b; i < e; ++i) {
            const uint32_t c = next, g = (c << 5) + lane;
            ++next;
            if (a.chunk_list && i + 1 < e) {
                next = __ldg(a.chunk_list + i + 1);
                const uint32_t ahead = (next << 5) + lane;
                if (ahead < a.n) scene.prefetch(ahead);
            }
            chunk(c, a.fc.enable_hier && g < a.n && block_culled(a.blocks, g));
        }
    }
    flush_tile();
    if (a.loaded && lane == 0 && loaded_tally) atomicAdd(a.loaded, loaded_tally);
}

// ---------------------------------------------------------------------------------
// Scan over (survivor count, point count) pairs in up to three launches: per-tile totals (the
// render path's preprocess accumulates them instead), where needed a block scanning the tile
// totals and one scanning the bin cursors, a downsweep writing the compacted survivors
// (replaces workload_distributor.cu:62-145: 3 blocking D2H copies, an exclusive scan, a
// scatter and a P-long max-scan).  Tile word: [63:32] survivors, [31:0] points (mod 2^32 like
// the reference's u32 offsets).  No block waits on another, so there is no spin at all.
// ---------------------------------------------------------------------------------

// One round of a thread's Gaussians (16 consecutive): its mask bits and point counts.
__device__ __forceinline__ uint32_t scan_load(const ScanArgs& a, const uint32_t* __restrict__ mask, uint32_t base,
                                              uint32_t cnt[kScanItems]) {
    uint32_t bits = 0;
    if (base < a.n) {
        bits = (__ldg(&mask[base >> 5]) >> (base & 31)) & 0xFFFFu;
        if (a.n - base < (uint32_t)kScanItems) bits &= (1u << (a.n - base)) - 1u;
    }
#pragma unroll
    for (int q = 0; q < kScanItems / 4; ++q) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if ((bits >> (4 * q)) & 0xFu) v = __ldg(reinterpret_cast<const uint4*>(a.counts + base) + q);
        cnt[4 * q + 0] = ((bits >> (4 * q + 0)) & 1u) ? v.x : 0u;
        cnt[4 * q + 1] = ((bits >> (4 * q + 1)) & 1u) ? v.y : 0u;
        cnt[4 * q + 2] = ((bits >> (4 * q + 2)) & 1u) ? v.z : 0u;
        cnt[4 * q + 3] = ((bits >> (4 * q + 3)) & 1u) ? v.w : 0u;
    }
    return bits;
}

// Block-wide exclusive scan of (survivors, points) pairs; also returns the block totals.
template <int kThreads>
__device__ __forceinline__ void block_scan_pair(uint32_t s, uint32_t p, uint32_t& ex_s, uint32_t& ex_p,
                                                uint32_t& tot_s, uint32_t& tot_p) {
    __shared__ uint32_t w_s[kThreads / 32], w_p[kThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t is = s, ip = p;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t vs = __shfl_up_sync(0xffffffffu, is, o);
        const uint32_t vp = __shfl_up_sync(0xffffffffu, ip, o);
        if (lane >= o) {
            is += vs;
            ip += vp;
        }
    }
    if (lane == 31) {
        w_s[warp] = is;
        w_p[warp] = ip;
    }
    __syncthreads();
    uint32_t off_s = 0, off_p = 0, all_s = 0, all_p = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) {
        if (w < warp) {
            off_s += w_s[w];
            off_p += w_p[w];
        }
        all_s += w_s[w];
        all_p += w_p[w];
    }
    ex_s = off_s + is - s;
    ex_p = off_p + ip - p;
    tot_s = all_s;
    tot_p = all_p;
}

// Pass 1 of the scan: every tile's survivor and point totals, fully parallel.
template <int kScanRounds>
__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(ScanArgs a) {
    previous_kernel_done();
    const uint32_t* mask = a.mask;  // (a select, not a runtime index into the parameter array)
    if (a.mask_iter) mask = (*a.mask_iter & 1u) ? a.mask_pair[1] : a.mask_pair[0];
    const uint32_t tile = blockIdx.x;
    const uint32_t base = tile * (kScanThreads * kScanItems * kScanRounds) + threadIdx.x * (kScanItems * kScanRounds);
    uint32_t surv = 0, pts = 0;
#pragma unroll
    for (int q = 0; q < kScanRounds; ++q) {
        uint32_t cnt[kScanItems];
        surv += __popc(scan_load(a, mask, base + q * kScanItems, cnt));
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) pts += cnt[i];
    }
    uint32_t ex_s, ex_p, tot_s, tot_p;
    block_scan_pair<kScanThreads>(surv, pts, ex_s, ex_p, tot_s, tot_p);
    if (threadIdx.x == 0) a.tile_state[tile] = ((unsigned long long)tot_s << 32) | tot_p;
}

// Pass 2: one block turns the tile totals into exclusive tile prefixes (in place) and writes
// the pass counters (points mod 2^32, like the reference's u32 offsets).  The tile words go
// through shared memory in rounds of kTileScanThreads * 4 with coalesced loads and stores;
// each thread scans 4 consecutive words and a block scan plus a running carry joins them.
constexpr int kTileScanThreads = 1024;
constexpr int kTileScanPer = 4;

// One block: exclusive prefix of `count` packed (survivors << 32 | points) words in place,
// through shared memory in coalesced rounds; returns the totals.
__device__ __forceinline__ void scan_words_inplace(unsigned long long* words_g, uint32_t count, uint32_t& total_s,
                                                   uint32_t& total_p) {
    __shared__ unsigned long long words[kTileScanThreads * kTileScanPer];
    constexpr uint32_t kRound = kTileScanThreads * kTileScanPer;
    uint32_t carry_s = 0, carry_p = 0;
    for (uint32_t r0 = 0; r0 < count; r0 += kRound) {
        for (uint32_t i = threadIdx.x; i < kRound; i += kTileScanThreads)
            words[i] = r0 + i < count ? words_g[r0 + i] : 0ull;
        __syncthreads();
        uint32_t s = 0, p = 0;
#pragma unroll
        for (int k = 0; k < kTileScanPer; ++k) {
            const unsigned long long v = words[threadIdx.x * kTileScanPer + k];
            s += (uint32_t)(v >> 32);
            p += (uint32_t)v;
        }
        uint32_t ex_s, ex_p, tot_s, tot_p;
        block_scan_pair<kTileScanThreads>(s, p, ex_s, ex_p, tot_s, tot_p);
        ex_s += carry_s;
        ex_p += carry_p;
#pragma unroll
        for (int k = 0; k < kTileScanPer; ++k) {
            const unsigned long long v = words[threadIdx.x * kTileScanPer + k];
            words[threadIdx.x * kTileScanPer + k] = ((unsigned long long)ex_s << 32) | ex_p;
            ex_s += (uint32_t)(v >> 32);
            ex_p += (uint32_t)v;
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < kRound && r0 + i < count; i += kTileScanThreads) words_g[r0 + i] = words[i];
        carry_s += tot_s;
        carry_p += tot_p;
        __syncthreads();
    }
    total_s = carry_s;
    total_p = carry_p;
}

// One block of the downsweep: the bin cursors (cursor k of bin b at word k * bin_count + b) become
// exclusive prefixes in (b, k) order, in place; returns the largest bin's survivors.  2048 words at
// a time, eight per thread in registers, every load coalesced: it takes less than the downsweep beside it, where a launch of its own took 13.6 us
// (8160 words, 1080p) to 24 us (16320, 4K).
template <int kSubLog2>
__device__ __forceinline__ uint32_t scan_bins_inplace(unsigned long long* bins, uint32_t bin_count) {
    constexpr uint32_t kSubs = 1u << kSubLog2, kRounds = 8u >> kSubLog2, kWarps = kScanThreads / 32u;
    __shared__ uint32_t sum_s[kRounds][kWarps], sum_p[kRounds][kWarps], s_max;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned long long v[kRounds][kSubs];
    if (threadIdx.x == 0) s_max = 0;
    uint32_t carry_s = 0, carry_p = 0, most = 0;
    for (uint32_t b0 = 0; b0 < bin_count; b0 += kRounds * kScanThreads) {
        uint32_t es[kRounds], ep[kRounds];
#pragma unroll
        for (uint32_t r = 0; r < kRounds; ++r)
#pragma unroll
            for (uint32_t k = 0; k < kSubs; ++k) {
                const uint32_t b = b0 + r * kScanThreads + threadIdx.x;
                v[r][k] = b < bin_count ? __ldcg(bins + (size_t)k * bin_count + b) : 0ull;
            }
#pragma unroll
        for (uint32_t r = 0; r < kRounds; ++r) {
            uint32_t s = 0, p = 0;
#pragma unroll
            for (uint32_t k = 0; k < kSubs; ++k) {
                s += (uint32_t)(v[r][k] >> 32);
                p += (uint32_t)v[r][k];
            }
            most = max(most, s);
            es[r] = s;
            ep[r] = p;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t vs = __shfl_up_sync(0xffffffffu, es[r], o), vp = __shfl_up_sync(0xffffffffu, ep[r], o);
                if (lane >= (uint32_t)o) {
                    es[r] += vs;
                    ep[r] += vp;
                }
            }
            if (lane == 31u) {
                sum_s[r][warp] = es[r];
                sum_p[r][warp] = ep[r];
            }
            es[r] -= s;
            ep[r] -= p;
        }
        __syncthreads();
#pragma unroll
        for (uint32_t r = 0; r < kRounds; ++r) {
            uint32_t ps = 0, pp = 0, all_s = 0, all_p = 0;
#pragma unroll
            for (uint32_t w = 0; w < kWarps; ++w) {
                if (w == warp) {
                    ps = all_s;
                    pp = all_p;
                }
                all_s += sum_s[r][w];
                all_p += sum_p[r][w];
            }
            const uint32_t b = b0 + r * kScanThreads + threadIdx.x;
            uint32_t s = carry_s + ps + es[r], q = carry_p + pp + ep[r];
#pragma unroll
            for (uint32_t k = 0; k < kSubs; ++k) {
                if (b < bin_count) bins[(size_t)k * bin_count + b] = ((unsigned long long)s << 32) | q;
                s += (uint32_t)(v[r][k] >> 32);
                q += (uint32_t)v[r][k];
            }
            carry_s += all_s;
            carry_p += all_p;
        }
        __syncthreads();
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 0u) atomicMax(&s_max, most);
    __syncthreads();
    return s_max;
}

__device__ __forceinline__ void write_counters(const ScanArgs& a, uint32_t survivors, uint32_t points) {
    a.counters->survivors = survivors;
    a.counters->total_points = points;
    a.counters->points = points < a.max_points ? points : a.max_points;
    a.counters->truncated = points > a.max_points ? 1u : 0u;
    a.counters->scan_timeouts = 0u;
    a.counters->loaded = a.loaded ? *a.loaded : 0u;
    if (a.loaded) *a.loaded = 0u;  // the next pass's preprocess tallies from zero
    a.counters->work = 0u;
    if (!a.bins) a.counters->crowded = 0u;
}

// Pass 2, for more tiles than kDirectTiles: one block turns the tile totals into exclusive tile
// prefixes (in place) and writes the pass counters.
__global__ void __launch_bounds__(kTileScanThreads) scan_tiles_kernel(ScanArgs a, uint32_t num_tiles) {
    previous_kernel_done();
    uint32_t carry_s, carry_p;
    scan_words_inplace(a.tile_state, num_tiles, carry_s, carry_p);
    if (threadIdx.x == 0) write_counters(a, carry_s, carry_p);
}

// Records survivor `rank` as the owner of every 256-point splat tile that starts inside its points
// [first, first + count): one or none for most, but a Gaussian right in front of the camera owns
// thousands, which its whole warp then writes.  All lanes call it; count 0: nothing to do.
// (tiles starting at or past P are never walked, and the array holds max_points / 256 + 2)
template <bool kWide>
__device__ __forceinline__ void own_tiles(uint32_t* __restrict__ tile_first_rank, uint32_t first, uint32_t count,
                                          uint32_t rank, uint32_t P) {
    const uint64_t end = min((uint64_t)first + count, (uint64_t)P);
    const uint32_t t0 = (uint32_t)(((uint64_t)first + 255u) >> 8), t1 = count ? (uint32_t)((end + 255u) >> 8) : 0u;
    const uint32_t n = t1 > t0 ? t1 - t0 : 0u;
    if (n <= 4u)
        for (uint32_t i = 0; i < n; ++i) tile_first_rank[t0 + i] = rank;
    const uint32_t lane = threadIdx.x & 31u;
    for (unsigned big = __ballot_sync(0xffffffffu, n > 4u); big; big &= big - 1u) {
        const int src = __ffs(big) - 1;
        uint32_t t = __shfl_sync(0xffffffffu, t0, src), m = __shfl_sync(0xffffffffu, n, src);
        const uint32_t r = __shfl_sync(0xffffffffu, rank, src);
        // kWide: four at a time where there are many (a survivor of 100M points, in a scan of 2M counts, holds
        // up its warp for 26 us, one by one for 63).  A frame's Gaussians have at most half a point per
        // pixel, and the code for it costs its binning 5 us of 33.6M Gaussians.
        if (kWide && m > 128u) {
            const uint32_t head = (0u - (uint32_t)(reinterpret_cast<uintptr_t>(tile_first_rank + t) >> 2)) & 3u, quads = (m - head) / 4u;
            uint4* to = reinterpret_cast<uint4*>(tile_first_rank + t + head);
            if (lane < head) tile_first_rank[t + lane] = r;
#pragma unroll 4
            for (uint32_t i = lane; i < quads; i += 32u) to[i] = make_uint4(r, r, r, r);
            t += head + 4u * quads;
            m -= head + 4u * quads;
        }
        for (uint32_t i = lane; i < m; i += 32u) tile_first_rank[t + i] = r;
    }
}

// Pass 3, the downsweep: each tile of Gaussians writes its compacted survivors' ids and first
// points and, where the splat walks the Gaussian order, the owners of its 256-point tiles (points
// past P dropped as the reference drops them).  In a screen-binned pass the block before the first
// tile scans the bin cursors.  The survivors of 4096 Gaussians are gathered in shared memory, then
// taken one per thread: their writes are coalesced, and a thread whose own 16 Gaussians all
// survive doesn't hold up its block (60k town at 320x180: frame 73.4 -> 64.5 us,
// with the launch that scanned the tile totals gone).
//
// kDirect: the tile words are plain totals and every block adds up those before its own, which
// takes less time than a launch that scans them (up to kDirectTiles words, 32 KB from L2).
constexpr uint32_t kDirectTiles = 4096;

// A 16384-Gaussian tile whose warps need no more than kSparseSteps steps for their 2048 Gaussians is taken
// at once, not in four rounds with their barriers and lists.  200M counts, 1% of them marked: 273 -> 155 us
// (206 when a thread took its Gaussians twice and there were no lists), 64 neighbours in each
// tile 214 -> 99 (144); 70M, 10%, 12 steps (rounds) 162, 18 steps 182.  Not in the render path, where
// the survivors of a tile are many or none: 33.6M town 1167 -> 1177 us a frame with it.
constexpr uint32_t kSparseTile = 2560, kSparseSteps = 12;

template <int kScanRounds, bool kDirect, bool kBinned>
__global__ void __launch_bounds__(kScanThreads, kBinned ? 4 : 5) scan_write_kernel(ScanArgs a, uint32_t tiles) {
    previous_kernel_done();
    __shared__ uint16_t list_g[kScanTileSmall];
    __shared__ uint32_t list_p[kScanTileSmall + 1];
    __shared__ uint32_t sums[4][kScanThreads / 32];
    const uint32_t lane = threadIdx.x & 31u;
    if (kBinned && blockIdx.x == 0u) {
        const uint32_t most = a.bin_sub_log2 == 2   ? scan_bins_inplace<2>(a.bins, a.bin_count)
                              : a.bin_sub_log2 == 1 ? scan_bins_inplace<1>(a.bins, a.bin_count)
                                                    : scan_bins_inplace<0>(a.bins, a.bin_count);
        // a bin crowded past bin_crowded survivors would serialise the binning on its
        // cursors: the pass is then walked in Gaussian order
        if (threadIdx.x == 0) a.counters->crowded = most > a.bin_crowded ? 1u : 0u;
        return;
    }
    const uint32_t tile = blockIdx.x - (kBinned ? 1u : 0u);
    uint32_t r0, p0, P, in_tile;  // in_tile: its survivors
    if (kDirect) {
        // a tile without survivors has nothing to write (the first one writes the counters)
        in_tile = (uint32_t)(a.tile_state[tile] >> 32);
        if (tile != 0u && in_tile == 0u) return;
        uint32_t s_pre = 0, p_pre = 0, s_all = 0, p_all = 0;
        for (uint32_t i = threadIdx.x; i < tiles; i += kScanThreads) {
            const unsigned long long v = a.tile_state[i];
            s_all += (uint32_t)(v >> 32);
            p_all += (uint32_t)v;
            if (i < tile) {
                s_pre += (uint32_t)(v >> 32);
                p_pre += (uint32_t)v;
            }
        }
        s_pre = __reduce_add_sync(0xffffffffu, s_pre);
        p_pre = __reduce_add_sync(0xffffffffu, p_pre);
        s_all = __reduce_add_sync(0xffffffffu, s_all);
        p_all = __reduce_add_sync(0xffffffffu, p_all);
        if (lane == 0u) {
            sums[0][threadIdx.x >> 5] = s_pre;
            sums[1][threadIdx.x >> 5] = p_pre;
            sums[2][threadIdx.x >> 5] = s_all;
            sums[3][threadIdx.x >> 5] = p_all;
        }
        __syncthreads();
        r0 = p0 = s_all = p_all = 0u;
#pragma unroll
        for (int w = 0; w < kScanThreads / 32; ++w) {
            r0 += sums[0][w];
            p0 += sums[1][w];
            s_all += sums[2][w];
            p_all += sums[3][w];
        }
        if (tile == 0u && threadIdx.x == 0u) write_counters(a, s_all, p_all);
        P = min(p_all, a.max_points);
    } else {
        const unsigned long long pre = a.tile_state[tile];
        r0 = (uint32_t)(pre >> 32);
        p0 = (uint32_t)pre;
        // culled regions of the scene cost two loads, not a pass over their masks
        // (256M town: scan 0.586 -> 0.548 ms/frame)
        in_tile = (tile + 1u < tiles ? (uint32_t)(a.tile_state[tile + 1u] >> 32) : a.counters->survivors) - r0;
        if (in_tile == 0u) return;
        P = a.counters->points;
    }
    const uint32_t* mask = a.mask;  // (a select, not a runtime index into the parameter array)
    if (a.mask_iter) mask = (*a.mask_iter & 1u) ? a.mask_pair[1] : a.mask_pair[0];
    // The listed survivors of the Gaussians from `base` on, whose totals are tot_s and tot_p.
    auto write_out = [&](uint32_t base, uint32_t tot_s, uint32_t tot_p) {
        if (threadIdx.x == 0u) list_p[tot_s] = tot_p;
        __syncthreads();
        for (uint32_t k0 = threadIdx.x & ~31u; k0 < tot_s; k0 += kScanThreads) {
            const uint32_t k = k0 + lane;
            const bool live = k < tot_s;
            const uint32_t g = base + list_g[live ? k : 0u], pt = p0 + list_p[live ? k : 0u];
            const uint32_t cnt = live ? list_p[k + 1u] - list_p[k] : 0u;
            if (live) {
                a.surv_gid[r0 + k] = g;
                a.surv_start[r0 + k] = pt;
            }
            if (!kBinned) own_tiles<true>(a.tile_first_rank, pt, pt < P ? cnt : 0u, r0 + k, P);
        }
        r0 += tot_s;
        p0 += tot_p;
        __syncthreads();
    };
    // 16 Gaussians per thread from `base` on.
    auto take = [&](uint32_t base) {
        uint32_t cnt[kScanItems], pts = 0, at, pt, tot_s, tot_p;
        const uint32_t bits = scan_load(a, mask, base + threadIdx.x * kScanItems, cnt);
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) pts += cnt[i];
        block_scan_pair<kScanThreads>((uint32_t)__popc(bits), pts, at, pt, tot_s, tot_p);
#pragma unroll
        for (int i = 0; i < kScanItems; ++i)
            if ((bits >> i) & 1u) {
                list_g[at] = (uint16_t)(threadIdx.x * kScanItems + i);
                list_p[at++] = pt;
                pt += cnt[i];
            }
        write_out(base, tot_s, tot_p);
    };
    const uint32_t first = tile * (kScanRounds * kScanTileSmall);
    if constexpr (kScanRounds > 1 && !kBinned) {
        // few survivors: a warp has 64 mask words, a lane two of them.  The warp goes from bit to bit in every
        // lane's words together, or, where the survivors are neighbours, from word to word with a lane per
        // Gaussian, whichever takes fewer steps.
        static_assert(kScanRounds * kScanTileSmall == 64u * kScanThreads, "two mask words per thread");
        if (in_tile <= kSparseTile) {
            const uint32_t mine = first + 64u * threadIdx.x;
            const uint32_t lo = mine < a.n ? __ldg(&mask[mine >> 5]) : 0u, hi = mine + 32u < a.n ? __ldg(&mask[(mine >> 5) + 1u]) : 0u;
            uint64_t bits = ((uint64_t)hi << 32) | lo;
            if (mine < a.n && a.n - mine < 64u) bits &= (1ull << (a.n - mine)) - 1ull;
            const uint32_t words = __ballot_sync(0xffffffffu, bits != 0ull);  // (pairs of words)
            const uint32_t most = __reduce_max_sync(0xffffffffu, (uint32_t)__popcll(bits));
            const bool by_bit = most <= 2u * (uint32_t)__popc(words);
            if (!__syncthreads_or((by_bit ? most : 2u * (uint32_t)__popc(words)) > kSparseSteps)) {
                uint32_t pts = 0;
                const uint32_t warp = threadIdx.x >> 5, warp_first = first + 2048u * warp;
                if (by_bit) {
                    for (uint64_t m = bits; m; m &= m - 1ull) pts += __ldg(a.counts + mine + (uint32_t)(__ffsll((long long)m) - 1));
                } else {
                    for (uint32_t m = words; m; m &= m - 1u) {
                        const int src = __ffs(m) - 1;
                        const uint64_t both = __shfl_sync(0xffffffffu, bits, src);
                        const uint32_t* c = a.counts + warp_first + 64u * (uint32_t)src + lane;
                        if ((both >> lane) & 1ull) pts += __ldg(c);
                        if ((both >> (lane + 32u)) & 1ull) pts += __ldg(c + 32);
                    }
                }
                // the warps before this one and, going by bit, the lanes before this one
                const uint32_t survivors = (uint32_t)__popcll(bits);
                uint32_t s_in = survivors, p_in = pts;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t vs = __shfl_up_sync(0xffffffffu, s_in, o), vp = __shfl_up_sync(0xffffffffu, p_in, o);
                    if (lane >= (uint32_t)o) {
                        s_in += vs;
                        p_in += vp;
                    }
                }
                if (lane == 31u) {
                    sums[0][warp] = s_in;
                    sums[1][warp] = p_in;
                }
                __syncthreads();
                for (uint32_t v = 0; v < warp; ++v) {
                    r0 += sums[0][v];
                    p0 += sums[1][v];
                }
                if (by_bit) {
                    uint32_t r = r0 + s_in - survivors, pt = p0 + p_in - pts;
                    uint64_t m = bits;
                    for (uint32_t k = 0; k < most; ++k) {
                        const bool live = m != 0ull;
                        const uint32_t g = mine + (live ? (uint32_t)(__ffsll((long long)m) - 1) : 0u);
                        const uint32_t cnt = live ? __ldg(a.counts + g) : 0u;  // (again, from L1)
                        if (live) {
                            a.surv_gid[r] = g;
                            a.surv_start[r] = pt;
                        }
                        own_tiles<true>(a.tile_first_rank, pt, pt < P ? cnt : 0u, r, P);
                        r += live ? 1u : 0u;
                        pt += cnt;
                        m &= m - 1ull;
                    }
                } else {
                    for (uint32_t m = words; m; m &= m - 1u) {
                        const int src = __ffs(m) - 1;
                        const uint64_t both = __shfl_sync(0xffffffffu, bits, src);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t w = (uint32_t)(both >> (32 * h));
                            if (!w) continue;
                            const uint32_t g = warp_first + 64u * (uint32_t)src + 32u * (uint32_t)h + lane;
                            const uint32_t cnt = (w >> lane) & 1u ? __ldg(a.counts + g) : 0u;
                            uint32_t sum = cnt;
#pragma unroll
                            for (int o = 1; o < 32; o <<= 1) {
                                const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o);
                                if (lane >= (uint32_t)o) sum += v;
                            }
                            const uint32_t r = r0 + (uint32_t)__popc(w & ((1u << lane) - 1u)), pt = p0 + sum - cnt;
                            if ((w >> lane) & 1u) {
                                a.surv_gid[r] = g;
                                a.surv_start[r] = pt;
                            }
                            own_tiles<true>(a.tile_first_rank, pt, pt < P ? cnt : 0u, r, P);
                            r0 += (uint32_t)__popc(w);
                            p0 += __shfl_sync(0xffffffffu, sum, 31);
                        }
                    }
                }
                return;
            }
        }
    }
    for (int q = 0; q < kScanRounds; ++q) {
        const uint32_t base = first + (uint32_t)q * kScanTileSmall;
        if (base >= a.n) break;
        take(base);
    }
}

// The last step of a screen-binned pass: every survivor takes its slot and first walk position from
// one of its bin's cursors, with one 64-bit atomic per distinct cursor among a warp's 32 survivors, so
// that slot and position stay consistent and positions increase with the slot, and records itself
// as the owner of the 256-point tiles that start inside its points.  A pass that cannot be binned
// (truncated, or a crowded bin) records the owners of the Gaussian order here.
//
// The survivors are split evenly over the warps.  Inside the downsweep the chain record -> cursor
// -> stores (a DRAM access and a contended atomic with a result, 2 us) ran once per survivor of
// the fullest thread or tile: survivors are neighbours in the scene's order, so a few tiles hold
// most of them.  Scan stage, both passes: 107 -> 53 us (4M town, 1080p), 120 -> 59 (1M, 4K), 255 -> 91
// (33.6M, 2.6M survivors in pass 2).
__global__ void __launch_bounds__(256) bin_survivors_kernel(ScanArgs a) {
    previous_kernel_done();
    const uint32_t survivors = a.counters->survivors, P = a.counters->points;
    const bool binned = a.counters->truncated == 0u && a.counters->crowded == 0u;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t k0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; k0 < survivors; k0 += gridDim.x * blockDim.x) {
        const uint32_t k = k0 + lane;
        const bool live = k < survivors;
        uint32_t g = 0, pt = 0, cnt = 0, bin = 0xffffffffu;
        if (live) {
            g = a.surv_gid[k];
            pt = a.surv_start[k];
            cnt = a.counts[g];
        }
        if (!binned) {
            own_tiles<false>(a.tile_first_rank, pt, pt < P ? cnt : 0u, k, P);
            continue;
        }
        if (live) {
            const float2 pm = __ldg(reinterpret_cast<const float2*>(a.records + g));
            bin = screen_bin(pm.x, pm.y, a.up_width, a.up_height, a.bin_shift, a.bins_x, a.bins_y) +
                  ((g >> 5) & ((1u << a.bin_sub_log2) - 1u)) * a.bin_count;
        }
        // the lanes of each distinct cursor: their leader, place and points before them
        uint32_t leader = lane, rank = 0, before = 0;
        unsigned long long add = 0;
        for (unsigned todo = __ballot_sync(0xffffffffu, live); todo;) {
            const int src = __ffs(todo) - 1;
            const uint32_t key = __shfl_sync(0xffffffffu, bin, src);
            const bool mine = bin == key;
            const unsigned members = __ballot_sync(0xffffffffu, mine);
            if (members == (1u << src)) {
                if (mine) add = (1ull << 32) | cnt;
            } else {
                uint32_t sum = mine ? cnt : 0u;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= (uint32_t)o) sum += v;
                }
                const uint32_t total = __shfl_sync(0xffffffffu, sum, 31);
                if (mine) {
                    leader = (uint32_t)src;
                    rank = (uint32_t)__popc(members & ((1u << lane) - 1u));
                    before = sum - cnt;
                    if (lane == (uint32_t)src) add = ((unsigned long long)__popc(members) << 32) | total;
                }
            }
            todo &= ~members;
        }
        unsigned long long old = 0;
        if (live && leader == lane) old = atomicAdd(a.bins + bin, add);
        old = __shfl_sync(0xffffffffu, old, (int)leader);
        const uint32_t slot = (uint32_t)(old >> 32) + rank, first = (uint32_t)old + before;
        if (live) {
            a.sorted_gid[slot] = g;
            a.sorted_pstart[slot] = pt;
            a.sorted_qstart[slot] = first;
        }
        own_tiles<false>(a.tile_first_rank, first, cnt, slot, P);
    }
}

// ---------------------------------------------------------------------------------
// Splat (gaussian_point_splatting.cu:67-141 with num_points = 1, 383-432)
// ---------------------------------------------------------------------------------
constexpr int kSplatTile = 256;

// post_processing_kernels.cuh:13-42 with add_if_equal = true; `old` is a value the slot held
__device__ __forceinline__ void atomic_add_color(unsigned long long* address, unsigned long long old, uint64_t value) {
    const uint64_t target_depth = value & kDepthMask;
    unsigned long long assumed;
    do {
        assumed = old;
        uint64_t assumed_depth = assumed & kDepthMask;
        uint64_t new_value = value;
        if (target_depth > assumed_depth) return;
        if (target_depth == assumed_depth) {
            uint64_t new_lower = (assumed & kColorMask) + (value & kColorMask);
            new_value = (assumed & kDepthMask) | (new_lower & kColorMask);
        }
        old = atomicCAS(address, assumed, (unsigned long long)new_value);
    } while (assumed != old);
}

// Biased mode (use_unbiased_2d_splatting = false): one point's samples first..last - 1 (the seed
// advances, as splatGaussianPoint's does), in order: a slot's pre-test load, then the addition, which
// starts from the loaded value.  A load that missed an addition made since costs a second
// compare-and-swap, no more: a slot's depth only decreases.  What bounds it is those chains and the
// instructions around them, not the loads' latency, which the other warps cover: four samples at a time,
// with their loads together, took 340 us for 225 (700k town, 1280x720, 4 spp; with a load of its own for the
// addition 253), and no setting was faster that way.
__device__ __forceinline__ void splat_samples_biased(u32x2& seed, const SplatRecord& rec, const FrameConst& fc,
                                                     uint64_t* __restrict__ buffer, int first, int last) {
    const vec2 pixel_mean = make_v2(rec.a.x, rec.a.y);
    const float c0 = rec.a.z, c1 = rec.a.w, c2 = rec.b.x;
    const vec3 conic = make_v3(rec.b.y, rec.b.z, rec.b.w);
    const float opacity = rec.c.x;
    const int minx = (int)(rec.d.x & 0xFFFFu), miny = (int)(rec.d.x >> 16);
    const int maxx = (int)(rec.d.y & 0xFFFFu), maxy = (int)(rec.d.y >> 16);
    const uint64_t key = (uint64_t)rec.d.z | ((uint64_t)rec.d.w << 32);
    const uint64_t view_depth_bits = key & kDepthMask;
    const int k = fc.k_points;
    unsigned long long* buf = reinterpret_cast<unsigned long long*>(buffer);
    int pass = first / k, j = first - pass * k;  // sample s is draw j of spp pass `pass`
    for (int s = first; s < last; ++s) {
        vec2 u = pcg2d(seed);
        vec2 xy = box_muller(u.x, u.y);
        vec2 pixel = make_v2(pixel_mean.x + c0 * xy.x, pixel_mean.y + c1 * xy.x + c2 * xy.y);
        pixel = make_v2(floorf(pixel.x), floorf(pixel.y));
        int x = (int)pixel.x;
        int y = (int)pixel.y;
        vec2 delta = make_v2(pixel_mean.x - pixel.x, pixel_mean.y - pixel.y);
        if (x >= minx && x < maxx && y >= miny && y < maxy) {
            float gw = gaussian_value(conic, delta);
            float alpha = opacity * gw;
            if (!(alpha < 1.0f / 255.0f)) {
                unsigned long long* slot = buf + splat_index(x, y, pass, fc.num_passes, fc.up_width, fc.up_height);
                const unsigned long long seen = __ldcg(slot);
                if ((uint64_t)seen > view_depth_bits) atomic_add_color(slot, seen, key);
            }
        }
        if (++j == k) {
            j = 0;
            ++pass;
        }
    }
}

// Unbiased mode (the default).  A sample's slot is loaded before its atomicMin is issued (the
// pre-test), several loads in flight per thread.  Order does not matter for a min, and a slot is
// skipped only when it already holds a value <= this Gaussian's key, the exact condition under
// which atomicMin would leave it unchanged (the reference skips when the slot is <= the depth bits
// alone, a subset of these cases), so the buffer is identical.  Slot values only decrease during
// the kernel, so an L1-cached (possibly stale, hence larger) pre-test value can only cause an
// extra atomic, never a wrong skip.
// Pre-test before the atomic: 1 = L1-cached load, 2 = L2 load, 0 = none (every live sample
// issues its atomicMin; the buffer is the same in all three).  On the 16M-Gaussian town orbit
// (1080p, ss 2, 4 spp) the L1-cached pre-test measured fastest on B200 (splat 2.04 ms/frame vs
// 2.07 with the L2 load and 2.25 with none): it drops the atomics whose slot already holds a
// nearer or equal key, and an L1 hit costs less than the atomic it saves.
#ifndef GPS_SPLAT_PRETEST
#define GPS_SPLAT_PRETEST 1
#endif
// The draws of one step of a point: the K samples of an spp pass, or with K = 1 those of two passes
// (one, if that is the last), so that there is a pair to draw together.  Draw j belongs to
// pass + step_pass(j).
template <int K>
struct DrawStep {
    static_assert(K == 1 || K % 2 == 0, "samples are drawn in pairs");
    static constexpr int kPasses = K == 1 ? 2 : 1, kDraws = K == 1 ? 2 : K;
    uint32_t tile[kDraws], code[kDraws];
    bool live[kDraws];
    static __device__ __forceinline__ int step_pass(int j) { return K == 1 ? j : 0; }
    __device__ __forceinline__ void draw(u32x2& seed, const SampleConst& c, int pass) {
        if (K == 1 && pass + 1 >= c.passes) {
            live[0] = draw_one(seed, c, tile[0], code[0]);
            live[kDraws - 1] = false;
            tile[kDraws - 1] = code[kDraws - 1] = 0u;
            return;
        }
#pragma unroll
        for (int j = 0; j < kDraws; j += 2) draw_pair(seed, c, tile + j, code + j, live + j);
    }
};

// A point that draw_pair leaves out: one sample after the other, untested.  False for any other.
__device__ __forceinline__ bool splat_wide_point(u32x2& seed, const SampleConst& c, int k, int first, int last,
                                                 unsigned long long key, unsigned long long* buf) {
    if (!wide_sample(c)) return false;
    for (int i = first; i < last; ++i) {
        uint32_t tile, code;
        if (draw_sample(seed, c, tile, code)) atomicMin(buf + sample_slot(c, tile, code, i / k), key);
    }
    return true;
}

__device__ __forceinline__ unsigned long long pretest_load(const unsigned long long* at) {
    return GPS_SPLAT_PRETEST == 1 ? __ldca(at) : GPS_SPLAT_PRETEST == 2 ? __ldcg(at) : ~0ull;
}

// One point's samples first..last - 1 of its k * num_passes, any k (the seed advances from the first
// sample's to the one after the last, as splatGaussianPoint's does).
__device__ __forceinline__ void splat_samples_unbiased(u32x2& seed, const SplatRecord& rec, const FrameConst& fc,
                                                       uint64_t* __restrict__ buffer, const uint32_t* spread, int first, int last) {
    const SampleConst c = sample_const(rec, fc, spread);
    const unsigned long long key = (unsigned long long)rec.d.z | ((unsigned long long)rec.d.w << 32);
    unsigned long long* buf = reinterpret_cast<unsigned long long*>(buffer);
    const int k = fc.k_points;
    if (splat_wide_point(seed, c, k, first, last, key, buf)) return;
    int p = first / k, j = first - p * k;  // sample s0 + b is draw j of spp pass p
    for (int s0 = first; s0 < last; s0 += 4) {
        uint32_t tile[4], code[4], slot[4];
        bool live[4];
#pragma unroll
        for (int b = 0; b < 4; b += 2) {
            live[b] = live[b + 1] = false;
            tile[b] = tile[b + 1] = code[b] = code[b + 1] = 0u;
            if (s0 + b + 1 < last) draw_pair(seed, c, tile + b, code + b, live + b);
            else if (s0 + b < last) live[b] = draw_one(seed, c, tile[b], code[b]);
        }
        unsigned long long seen[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            slot[b] = sample_slot(c, tile[b], code[b], p);
            if (++j == k) {
                j = 0;
                ++p;
            }
            seen[b] = live[b] ? pretest_load(buf + slot[b]) : 0ull;
        }
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (live[b] && seen[b] > key) atomicMin(buf + slot[b], key);
    }
}

// The seed of a point's sample `first`: every sample is one step of the generator.
__device__ __forceinline__ u32x2 sample_seed(uint32_t point, int frame_seed, int first) {
    u32x2 seed = make_seed(point, (uint32_t)frame_seed);
    for (int i = 0; i < first; ++i) seed = pcg2d_step(seed);
    return seed;
}

// The same samples with K known at compile time.
template <int K>
__device__ __forceinline__ void splat_point_unbiased_k(uint32_t point, const SplatRecord& rec, const FrameConst& fc,
                                                       int frame_seed, uint64_t* __restrict__ buffer,
                                                       const uint32_t* spread) {
    using Step = DrawStep<K>;
    u32x2 seed = make_seed(point, (uint32_t)frame_seed);
    const SampleConst c = sample_const(rec, fc, spread);
    const unsigned long long key = (unsigned long long)rec.d.z | ((unsigned long long)rec.d.w << 32);
    unsigned long long* buf = reinterpret_cast<unsigned long long*>(buffer);
    if (splat_wide_point(seed, c, K, 0, c.passes * K, key, buf)) return;
    if (K == 1 && c.passes == 1) {  // nothing to pair or to pipeline
        uint32_t tile, code;
        const bool live = draw_one(seed, c, tile, code);
        unsigned long long* at = buf + sample_slot(c, tile, code, 0);
        if (live && pretest_load(at) > key) atomicMin(at, key);
        return;
    }
    // Software-pipelined over steps: the next step's samples are drawn and their pre-test loads
    // issued before this step's atomics consume its loads, so the load latency hides behind the
    // next step's arithmetic.  Samples are still drawn in stream order.
    uint32_t sa[Step::kDraws], sb[Step::kDraws];
    bool la[Step::kDraws], lb[Step::kDraws];
    unsigned long long va[Step::kDraws], vb[Step::kDraws];
    auto draw = [&](int p, uint32_t* sl, bool* lv, unsigned long long* vv) {
        Step step;
        step.draw(seed, c, p);
#pragma unroll
        for (int j = 0; j < Step::kDraws; ++j) {
            sl[j] = sample_slot(c, step.tile[j], step.code[j], p + Step::step_pass(j));
            lv[j] = step.live[j];
        }
#pragma unroll
        for (int j = 0; j < Step::kDraws; ++j) vv[j] = lv[j] ? pretest_load(buf + sl[j]) : 0ull;
    };
    auto commit = [&](const uint32_t* sl, const bool* lv, const unsigned long long* vv) {
#pragma unroll
        for (int j = 0; j < Step::kDraws; ++j)
            if (lv[j] && vv[j] > key) atomicMin(buf + sl[j], key);
    };
    constexpr int s = Step::kPasses;
    if (c.passes > 0) draw(0, sa, la, va);
    for (int p = 0; p < c.passes; p += 2 * s) {
        if (p + s < c.passes) draw(p + s, sb, lb, vb);
        commit(sa, la, va);
        if (p + s < c.passes) {
            if (p + 2 * s < c.passes) draw(p + 2 * s, sa, la, va);
            commit(sb, lb, vb);
        }
    }
}

// The same samples with the pre-test in shared memory: `nearest` holds the high words (the depth and
// the top colour bits) of one splat-buffer tile's smallest keys that this block knows of, a plane
// of kNearPlane words per spp pass.  A sample there whose high word is larger can't change its
// slot; one whose word is equal or smaller goes on to the buffer.  Samples of other tiles go to
// the buffer untested.
constexpr uint32_t kNearPlane = kTileSize * kTileSize + 8;

template <int K>
__device__ __forceinline__ void splat_point_in_tile(uint32_t point, const SplatRecord& rec, const FrameConst& fc,
                                                    int frame_seed, uint64_t* __restrict__ buffer, const uint32_t* spread,
                                                    uint32_t* nearest, uint32_t my_tile) {
    using Step = DrawStep<K>;
    u32x2 seed = make_seed(point, (uint32_t)frame_seed);
    const SampleConst c = sample_const(rec, fc, spread);
    const uint32_t key_high = rec.d.w;
    const unsigned long long key = (unsigned long long)rec.d.z | ((unsigned long long)rec.d.w << 32);
    unsigned long long* buf = reinterpret_cast<unsigned long long*>(buffer);
    if (splat_wide_point(seed, c, K, 0, c.passes * K, key, buf)) return;
    my_tile += c.tile_bias;
    for (int p = 0; p < c.passes; p += Step::kPasses, nearest += Step::kPasses * kNearPlane) {
        Step step;
        uint32_t seen[Step::kDraws];
        step.draw(seed, c, p);
#pragma unroll
        for (int j = 0; j < Step::kDraws; ++j)
            seen[j] = step.live[j] && step.tile[j] == my_tile ? nearest[step.code[j] + Step::step_pass(j) * kNearPlane] : 0xFFFFFFFFu;
#pragma unroll
        for (int j = 0; j < Step::kDraws; ++j)
            if (step.live[j] && key_high <= seen[j]) {
                atomicMin(buf + sample_slot(c, step.tile[j], step.code[j], p + Step::step_pass(j)), key);
                if (step.tile[j] == my_tile) atomicMin(nearest + step.code[j] + Step::step_pass(j) * kNearPlane, key_high);
            }
    }
}

// Points per thread between two block barriers: a block takes kSplatRounds consecutive 256-point
// tiles at once, with one survivor-start window of kSplatRounds * 256 entries (the survivors
// owning those points are the first tile's owner and at most that many more).  Fewer barriers
// mean less time waiting for a block's slowest warp: on the 16M-Gaussian town orbit (1080p,
// ss 2, 4 spp) the splat took 1.90 ms/frame with 1 round, 1.854 with 2 and 1.849 with 4.  With
// more than one round the kernel is held to 64 registers (4 blocks per SM) by its launch bounds.
#ifndef GPS_SPLAT_ROUNDS
#define GPS_SPLAT_ROUNDS 4
#endif
constexpr int kSplatRounds = GPS_SPLAT_ROUNDS;
constexpr int kSplatWindow = kSplatTile * kSplatRounds;

// The order in which a pass's points are walked.
struct PointOrder {
    uint32_t points, survivors;
    bool binned;
    const uint32_t *gids, *first_q, *point_base;
};

__device__ __forceinline__ PointOrder point_order(const SplatArgs& a) {
    PointOrder o;
    o.points = a.counters->points;
    o.survivors = a.counters->survivors;
    // the pass's work order: screen bins unless the scan had to truncate the pass or a bin was
    // too crowded to sort into
    o.binned = a.sorted_gid && a.counters->truncated == 0u && a.counters->crowded == 0u;
    o.gids = o.binned ? a.sorted_gid : a.surv_gid;
    o.first_q = o.binned ? a.sorted_qstart : a.surv_start;
    o.point_base = o.binned ? a.sorted_pstart : nullptr;
    return o;
}

// Whether this pass is splat_binned_kernel's: in screen-bin order, with enough points.
__device__ __forceinline__ bool takes_tile_test(const SplatArgs& a, const PointOrder& o) {
    return o.binned && o.points >= a.tile_test_from;
}

// What the next pass's kernels accumulate into is cleared here; nothing in the splat reads it.
__device__ __forceinline__ void clear_for_next_pass(const SplatArgs& a, uint32_t points) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.clear_a_words; i += gridDim.x * blockDim.x)
        a.clear_a[i] = 0ull;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.clear_b_words; i += gridDim.x * blockDim.x)
        a.clear_b[i] = 0ull;
    if (a.mask_iter && points > 0u && blockIdx.x == 0 && threadIdx.x == 0) *a.mask_iter += 1u;
    if (a.chunk_count && blockIdx.x == 0 && threadIdx.x == 0) *a.chunk_count = 0u;
}

// Group `group` of kThreads * kRounds consecutive walk positions: the starts of the survivors that
// may own them (the first position's owner and as many as there are positions) go to `starts`,
// then every thread takes kRounds positions and calls point(reference point index, record).
template <uint32_t kThreads, uint32_t kRounds, class Point>
__device__ __forceinline__ void splat_group(const SplatArgs& a, const PointOrder& o, uint32_t group, uint32_t* starts,
                                            Point&& point) {
    constexpr uint32_t group_points = kThreads * kRounds;
    static_assert(group_points % 256u == 0u && 256u % 32u == 0u, "groups are whole 256-point tiles");
    const uint32_t r0 = a.tile_first_rank[group * (group_points / 256u)];
#pragma unroll
    for (uint32_t q = 0; q < kRounds; ++q) {
        const uint32_t k = q * kThreads + threadIdx.x, r = r0 + k;
        starts[k] = (r0 < o.survivors && r < o.survivors) ? o.first_q[r] : 0xFFFFFFFFu;
    }
    __syncthreads();
    for (uint32_t q = 0; q < kRounds; ++q) {
        const uint32_t at = group * group_points + q * kThreads + threadIdx.x;
        if (at < o.points && starts[0] <= at) {
            // the position's owner is that of its 256-point tile's first point, of the next tile's,
            // or one between: the search starts from that range (splat 1.562 -> 1.545 ms/frame on
            // the 16M orbit)
            const uint32_t t = at >> 8;
            int hi = (int)group_points - 1;
            int lo = min((int)(__ldg(&a.tile_first_rank[t]) - r0), hi);
            if ((unsigned long long)(t + 1u) * 256u < o.points)
                hi = max(lo, min((int)(__ldg(&a.tile_first_rank[t + 1u]) - r0), hi));
            while (lo < hi) {  // largest k with starts[k] <= at
                const int mid = (lo + hi + 1) >> 1;
                if (starts[mid] <= at) lo = mid;
                else hi = mid - 1;
            }
            // the reference's point index (the seed): the walk position itself in Gaussian
            // order, the survivor's first point plus the offset in screen-bin order
            const uint32_t p = o.point_base ? __ldg(&o.point_base[r0 + lo]) + (at - starts[lo]) : at;
            const uint32_t g = __ldg(&o.gids[r0 + lo]);
            if (g < a.n) {  // always true unless the scan gave up (device_timeouts)
                const float4* rp = reinterpret_cast<const float4*>(a.records + g);
                SplatRecord rec;
                rec.a = __ldg(rp + 0);
                rec.b = __ldg(rp + 1);
                rec.c = __ldg(rp + 2);
                rec.d = __ldg(reinterpret_cast<const uint4*>(rp + 3));
                point(p, rec);
            }
        }
    }
    __syncthreads();
}

// Groups of kRounds positions per thread while there are at least two per block; a small pass keeps
// one position per thread and barrier so that its points still spread over every block, and one
// that would leave half the threads idle splits each point's samples into up to four shares: the
// pass then takes as long as a share's chain of draws (60k town at 320x180, 28k points of 16
// samples: frame 55.7 -> 53.5 us).  The code for it costs the other passes 1-2%, so only kernels for small
// views have it (kShares; see launch_splat).  point(p, record, first, last): samples first..last - 1.
template <uint32_t kThreads, uint32_t kRounds, bool kShares, class Point>
__device__ __forceinline__ void splat_walk(const SplatArgs& a, const PointOrder& o, uint32_t* starts, Point&& point) {
    const uint32_t samples = (uint32_t)(a.fc.num_passes * a.fc.k_points);
    auto walk = [&](auto rounds) {
        constexpr uint32_t r = decltype(rounds)::value;
        for (uint32_t group = blockIdx.x; (unsigned long long)group * (kThreads * r) < o.points; group += gridDim.x)
            splat_group<kThreads, r>(a, o, group, starts, [&](uint32_t p, const SplatRecord& rec) { point(p, rec, 0u, samples); });
    };
    const unsigned long long threads = (unsigned long long)gridDim.x * kThreads;
    if (o.points >= 2ull * threads * kRounds) {
        walk(std::integral_constant<uint32_t, kRounds>{});
    } else if (!kShares || o.points * 2ull > threads || samples < 4u) {
        walk(std::integral_constant<uint32_t, 1u>{});
    } else if constexpr (kShares) {
        const uint32_t shares = o.points * 4ull > threads || samples < 8u ? 2u : 4u;
        const uint32_t per = (samples / 2u + shares - 1u) / shares * 2u + (samples & 1u);  // pairs stay together
        for (uint32_t w = blockIdx.x; (unsigned long long)(w / shares) * kThreads < o.points; w += gridDim.x) {
            const uint32_t first = min(w % shares * per, samples), last = min(first + per, samples);
            splat_group<kThreads, 1>(a, o, w / shares, starts, [&](uint32_t p, const SplatRecord& rec) { point(p, rec, first, last); });
        }
    }
}

__device__ __forceinline__ void fill_spread(uint32_t* spread) {
    if (threadIdx.x < kTileSize) spread[threadIdx.x] = morton_spread(threadIdx.x);
}

// K > 0: unbiased splatting with K points per thread per pass; K = 0: any other setting.
// kShares: for views that may leave half the threads without a point (see splat_walk).
template <int K, bool kShares>
#ifndef GPS_SPLAT_MIN_BLOCKS
#define GPS_SPLAT_MIN_BLOCKS 4
#endif
// (K = 8 keeps two passes of eight samples in flight: more registers, fewer resident blocks)
__global__ void __launch_bounds__(kSplatTile, kSplatRounds > 1 ? (K >= 8 ? 2 : GPS_SPLAT_MIN_BLOCKS) : 1) splat_kernel(SplatArgs a) {
    previous_kernel_done();
    __shared__ uint32_t s_start[kSplatWindow];
    __shared__ uint32_t s_spread[kTileSize];
    const PointOrder o = point_order(a);
    if (takes_tile_test(a, o)) return;
    fill_spread(s_spread);
    clear_for_next_pass(a, o.points);
    splat_walk<kSplatTile, kSplatRounds, kShares>(a, o, s_start, [&](uint32_t p, const SplatRecord& rec, uint32_t first, uint32_t last) {
        if constexpr (K > 0) {
            if (!kShares || last - first == (uint32_t)(a.fc.num_passes * K)) {
                splat_point_unbiased_k<K>(p, rec, a.fc, a.frame_seed, a.buffer, s_spread);
                return;
            }
        }
        if constexpr (kShares) {
            u32x2 seed = sample_seed(p, a.frame_seed, (int)first);
            if (K > 0 || a.fc.use_unbiased) splat_samples_unbiased(seed, rec, a.fc, a.buffer, s_spread, (int)first, (int)last);
            else splat_samples_biased(seed, rec, a.fc, a.buffer, (int)first, (int)last);
        }
    });
}

// A frame's first pass in screen-bin order.  Its groups lie in one bin (a splat-buffer tile) each,
// but for the small bins and a bin's last group, so the block keeps that tile's nearest high words
// in shared memory, 16 KB per spp pass, and tests its samples there.
//
// Random 8-byte accesses bound this pass before its arithmetic did: every pre-test load and every
// atomic is an L1 set access of its own (4M town at 1080p, 4 spp: 106M of them for 68M samples, 72%
// of the cycles, warps waiting 8.7 cycles per issue for those loads, issue 50%), and an L1 line
// holds what the slot was when the line came in.  Tested in shared memory: 60M set accesses, issue
// 67%, and the pass 503 -> 373 us (33.6M town 232 -> 214, 1M town at 4K and 2 spp 448 -> 421).
//
// The buffer starts cleared, so a block starts a tile empty; what other blocks put there it does not
// know, which costs some atomics, and reading it (or giving every bin whole groups) cost more.
// The second pass would have to read its tiles, 128 KB each at 4 spp: 160 -> 209 us on the 4M town, so
// it keeps the test in L1.
//
// A block takes a.work's next run of consecutive groups, so that a tile serves several groups.
//
// Whether a pass is in screen-bin order, and how many points it has, is known on the device only: the
// plain kernel is launched too, and each of them returns at once where the other takes the pass (4M town
// at 1080p: 875 us a frame with and without the second launch).  The plain walk inside this kernel would run beside the planes' shared memory, with
// fewer blocks and next to no L1 for its pre-test: a crowded pass of the 1M town at 1080p, 4 spp, took
// 595 us that way against 331, a sparse one (60k town) 76 against 52.
//
// Up to 6 samples per pixel: blocks of 256 threads, four per SM as far as their shared memory allows.
// From 7 to 13 one block has the SM, with 1024 threads (16 views of a 1M town, five of them at 8 samples:
// 2625 -> 2441 us a batch; with one group per block enough instead of two, 2407).
constexpr uint32_t kBinnedGroup = 1024;
constexpr int binned_blocks(uint32_t threads) { return threads <= 256u ? 4 : 1; }

template <int K, uint32_t kBinnedThreads>
__global__ void __launch_bounds__(kBinnedThreads, binned_blocks(kBinnedThreads)) splat_binned_kernel(SplatArgs a) {
    constexpr uint32_t kBinnedRounds = kBinnedGroup / kBinnedThreads;
    previous_kernel_done();
    __shared__ uint32_t s_start[kBinnedGroup];
    __shared__ uint32_t s_spread[kTileSize];
    __shared__ uint32_t s_next;
    extern __shared__ __align__(16) uint32_t s_nearest[];  // num_passes planes of kNearPlane words
    const PointOrder o = point_order(a);
    if (!takes_tile_test(a, o)) return;
    fill_spread(s_spread);
    clear_for_next_pass(a, o.points);
    const uint32_t quads = (uint32_t)a.fc.num_passes * (kNearPlane / 4u);
    const uint32_t tiles_per_row = (uint32_t)(a.fc.up_width + kTileSize - 1) >> kTileBits;
    const uint32_t groups = (o.points + kBinnedGroup - 1u) / kBinnedGroup;
    const uint32_t run = min(max(groups / (gridDim.x * 8u), 1u), 8u);
    uint32_t my_tile = 0xFFFFFFFFu;
    for (;;) {
        if (threadIdx.x == 0u) s_next = atomicAdd(a.work, run);
        __syncthreads();
        const uint32_t first = s_next;
        if (first >= groups) break;
        for (uint32_t group = first; group < min(first + run, groups); ++group) {
            // the tile of the group's middle point
            const uint32_t mid = min(group * kBinnedGroup + kBinnedGroup / 2u, o.points - 1u);
            const uint32_t g = __ldg(&o.gids[__ldg(&a.tile_first_rank[mid >> 8])]);
            const float2 pm = __ldg(reinterpret_cast<const float2*>(a.records + g));
            const uint32_t tile = screen_bin(pm.x, pm.y, a.fc.up_width, a.fc.up_height, kTileBits, (int)tiles_per_row,
                                             (a.fc.up_height + kTileSize - 1) >> kTileBits);
            if (tile != my_tile) {  // (the last group's samples are done: splat_group ends in a barrier)
                my_tile = tile;
                for (uint32_t i = threadIdx.x; i < quads; i += kBinnedThreads)
                    reinterpret_cast<uint4*>(s_nearest)[i] = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
            }
            splat_group<kBinnedThreads, kBinnedRounds>(a, o, group, s_start, [&](uint32_t p, const SplatRecord& rec) {
                splat_point_in_tile<K>(p, rec, a.fc, a.frame_seed, a.buffer, s_spread, s_nearest, my_tile);
            });
        }
    }
}

// ---------------------------------------------------------------------------------
// Clear and resolve (gaussian_point_splatting.cu:484-548, 580-585)
// ---------------------------------------------------------------------------------
__global__ void clear_kernel(ulonglong2* __restrict__ buf, uint64_t pairs, unsigned long long value) {
    previous_kernel_done();
    const ulonglong2 v = make_ulonglong2(value, value);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < pairs; i += (uint64_t)gridDim.x * blockDim.x)
        buf[i] = v;
}

// One output pixel: the mean colour of its SS x SS x spp samples and their nearest NDC depth,
// in the reference's loop order, with the depth steps in the rounding that gps_math.cuh spells out.
template <bool kDepthOnly>
__device__ __forceinline__ float resolve_pixel(const ResolveArgs& a, int x, int y) {
    const uint32_t idx = (uint32_t)(y * a.width + x);
    const int bx = x * a.ss, by = y * a.ss;
    const int up_w = a.width * a.ss, up_h = a.height * a.ss;
    float depth = 1e9f;
    vec3 color = make_v3(0.0f, 0.0f, 0.0f);
    for (int dx = 0; dx < a.ss; dx++)
        for (int dy = 0; dy < a.ss; dy++)
            for (int p = 0; p < a.num_passes; ++p) {
                int i = splat_index(bx + dx, by + dy, p, a.num_passes, up_w, up_h);
                if ((uint64_t)(int64_t)i >= a.entries) continue;
                uint64_t val = __ldg(reinterpret_cast<const unsigned long long*>(a.buffer) + i);
                float view_depth = view_depth_from_key((val >> 36ull) & kDepthMax, a.near_plane, a.far_plane);
                float z_ndc = view_to_projected_depth(view_depth, a.near_plane, a.far_plane);
                depth = gmin(depth, z_ndc);
                if (kDepthOnly) continue;
                color.x += (float)((val >> 24) & 0xFFFu) / 255.0f;
                color.y += (float)((val >> 12) & 0xFFFu) / 255.0f;
                color.z += (float)((val >> 0) & 0xFFFu) / 255.0f;
            }
    float inv_passes = 1.0f / (float)(a.num_passes * a.ss * a.ss);
    if (!kDepthOnly) {
        a.color[3 * idx + 0] = color.x * inv_passes;
        a.color[3 * idx + 1] = color.y * inv_passes;
        a.color[3 * idx + 2] = color.z * inv_passes;
    }
    return depth;
}

// A 12-bit channel as a float by its bits under 2^23 (exact): no conversion instruction.
__device__ __forceinline__ float channel12(uint32_t c) { return __uint_as_float(0x4B000000u | (c & 0xFFFu)) - 8388608.0f; }

// Counts the keys whose depth is above the next key's.
constexpr uint32_t kSweepKeys = 256;  // consecutive keys of a thread

__global__ void __launch_bounds__(256) depth_monotone_kernel(float near_plane, float far_plane, uint32_t* falls) {
    const uint32_t first = (blockIdx.x * blockDim.x + threadIdx.x) * kSweepKeys;
    const uint32_t last = min(first + kSweepKeys, (uint32_t)kDepthMax);
    bool fell = false;
    float before = depth_of_key(first << 4, near_plane, far_plane);
    for (uint32_t k = first + 1u; k <= last; ++k) {
        const float depth = depth_of_key(k << 4, near_plane, far_plane);
        fell |= !(before <= depth);
        before = depth;
    }
    if (__any_sync(0xffffffffu, fell) && (threadIdx.x & 31u) == 0u) atomicAdd(falls, 1u);
}

// resolve_pixel with the factor known: the kSs x kSs samples of a pass are in flight together, and the
// nearest depth is that of the smallest key (see resolve_staged_kernel).  Sums in the reference's order.
template <bool kDepthOnly, int kSs>
__device__ __forceinline__ float resolve_pixel_ss(const ResolveArgs& a, int x, int y) {
    const uint32_t idx = (uint32_t)(y * a.width + x);
    vec3 color = make_v3(0.0f, 0.0f, 0.0f);
    uint32_t nearest = 0xFFFFFFFFu;
    const unsigned long long* buf = reinterpret_cast<const unsigned long long*>(a.buffer);
    auto add = [&](unsigned long long val) {
        const uint32_t lo = (uint32_t)val, hi = (uint32_t)(val >> 32);
        nearest = min(nearest, hi);
        color.x += channel12(__funnelshift_r(lo, hi, 24)) / 255.0f;
        color.y += channel12(lo >> 12) / 255.0f;
        color.z += channel12(lo) / 255.0f;
    };
    uint32_t at[kSs * kSs];
#pragma unroll
    for (int s = 0; s < kSs * kSs; ++s)
        at[s] = (uint32_t)splat_index(x * kSs + s / kSs, y * kSs + s % kSs, 0, a.num_passes, a.width * kSs, a.height * kSs);
    if (kDepthOnly || a.num_passes == 1) {  // the order of the samples makes no difference, or is this one
        for (int p = 0; p < a.num_passes; ++p) {
            unsigned long long v[kSs * kSs];
#pragma unroll
            for (int s = 0; s < kSs * kSs; ++s) v[s] = __ldg(buf + at[s] + p);
#pragma unroll
            for (int s = 0; s < kSs * kSs; ++s) {
                if (kDepthOnly) nearest = min(nearest, (uint32_t)(v[s] >> 32));
                else add(v[s]);
            }
        }
    } else {
#pragma unroll
        for (int s = 0; s < kSs * kSs; ++s)
#pragma unroll 4
            for (int p = 0; p < a.num_passes; ++p) add(__ldg(buf + at[s] + p));
    }
    if (!kDepthOnly) {
        const float inv_passes = 1.0f / (float)(a.num_passes * a.ss * a.ss);
        a.color[3 * idx + 0] = color.x * inv_passes;
        a.color[3 * idx + 1] = color.y * inv_passes;
        a.color[3 * idx + 2] = color.z * inv_passes;
    }
    return depth_of_key(nearest, a.near_plane, a.far_plane);
}

// The frame's counters written to pinned host memory by the first block of the final resolve: a
// copy in the stream after it would hold up the kernels behind it by some microseconds.
__device__ __forceinline__ void report_counters(const ResolveArgs& a) {
    constexpr uint32_t kWords = sizeof(PassCounters) / 4u;
    if (!a.report_to || (blockIdx.x | blockIdx.y) != 0u || threadIdx.x >= 2u * kWords) return;
    const bool ran = (int)(threadIdx.x / kWords) < a.report_passes;
    reinterpret_cast<volatile uint32_t*>(a.report_to)[threadIdx.x] =
        ran ? reinterpret_cast<const uint32_t*>(a.report_from)[threadIdx.x] : 0u;
}

__device__ __forceinline__ float hiz_op(bool use_min, float a, float b) { return use_min ? fminf(a, b) : fmaxf(a, b); }
__device__ __forceinline__ float hiz_identity(bool use_min) { return use_min ? INFINITY : -INFINITY; }

// The four finest Hi-Z levels (full size, 1/2, 1/4, 1/8), written by the resolve that has the
// depths in registers: thread m of a group of 64 holds the pixel with in-group Morton code m, so a
// texel's children are neighbouring lanes.  Level j from the finest reduces with min while
// j <= min_levels, else with max; texels past the image's edge don't exist and take no part.
// Called by all threads of the block (whole groups of 64); `exchange` holds a word per warp.
// Before, one launch read the depth image back and built the whole chain: with the minimum taken
// over keys below, two resolves and two builds went from 199 to 146 us a frame (4M town, 1080p,
// 4 spp) and from 441 to 306 (1M town, 4K, 2 spp); a frame of the 60k town at 320x180 89 -> 80.
__device__ __forceinline__ void hiz_fine_levels(const HizView& c, float depth, int x, int y, int min_levels,
                                                float* exchange) {
    const int L = c.levels - 1;  // the caller checked L >= 3
    const uint32_t m = threadIdx.x & 63u;
    bool exists = x < c.level_w[L] && y < c.level_h[L];
    // (32-bit indices: a view has fewer than 2^31 samples)
    if (exists) (c.mip + c.level_off[L])[(uint32_t)(y * c.level_w[L] + x)] = depth;
    float v = depth;
#pragma unroll
    for (int j = 1; j <= 3; ++j) {
        const bool use_min = j <= min_levels;
        const int l = L - j;
        if (!exists) v = hiz_identity(use_min);
        v = hiz_op(use_min, v, __shfl_xor_sync(0xffffffffu, v, 1 << (2 * j - 2)));
        if (j < 3) {
            v = hiz_op(use_min, v, __shfl_xor_sync(0xffffffffu, v, 2 << (2 * j - 2)));
        } else {  // the group's other half is the other warp
            if ((threadIdx.x & 31u) == 0u) exchange[threadIdx.x >> 5] = v;
            __syncthreads();
            v = hiz_op(use_min, v, exchange[(threadIdx.x >> 5) ^ 1u]);
        }
        x >>= 1;
        y >>= 1;
        exists = x < c.level_w[l] && y < c.level_h[l];
        if (exists && (m & ((1u << (2 * j)) - 1u)) == 0u) (c.mip + c.level_off[l])[(uint32_t)(y * c.level_w[l] + x)] = v;
    }
}

__device__ __forceinline__ uint32_t morton_compact(uint32_t a) {
    a &= 0x55555555u;
    a = (a | (a >> 1)) & 0x33333333u;
    a = (a | (a >> 2)) & 0x0F0F0F0Fu;
    a = (a | (a >> 4)) & 0x00FF00FFu;
    a = (a | (a >> 8)) & 0x0000FFFFu;
    return a;
}

// Any supersampling factor: 16 x 16 pixels per block, in Morton order so that groups of 64 threads
// are 8 x 8 pixels (hiz_fine_levels).  kSs: the factor at compile time, whose samples of a pass are then
// loaded together (0: any), for monotone planes (a.monotone).  kHiz: with the fine Hi-Z levels.
// Every thread reads runs of its own, so what bounds it is how many are resident and whether their
// lines stay in L1: the run-time factor is held to 32 registers (8 blocks per SM), the compiled one has
// up to 72 for its loads in flight.  With 40 and 48 instead, both resolves at 640x360 took 296 us for
// ss 5, 5 spp (now 260) and 512 for ss 3, 16 spp (now 296).
template <bool kDepthOnly, int kSs, bool kHiz>
__global__ void __launch_bounds__(256, kSs == 0 ? 8 : 1) resolve_kernel(ResolveArgs a, HizView hiz) {
    previous_kernel_done();
    report_counters(a);
    const int x = (int)(blockIdx.x * 16u + morton_compact(threadIdx.x)), y = (int)(blockIdx.y * 16u + morton_compact(threadIdx.x >> 1));
    const bool inside = x < a.width && y < a.height;
    float depth = 0.0f;
    if (inside) {
        if constexpr (kSs > 0) depth = resolve_pixel_ss<kDepthOnly, kSs>(a, x, y);
        else depth = resolve_pixel<kDepthOnly>(a, x, y);
        if (!(kDepthOnly && kHiz)) a.depth[y * a.width + x] = depth;
    }
    if constexpr (kHiz) {
        __shared__ float exchange[8];
        hiz_fine_levels(hiz, depth, x, y, a.hiz_min_levels, exchange);
    }
}

// Power-of-two supersampling: the pixels of each 64x64 splat tile in Morton order.  An
// output pixel's sub-pixels are then one contiguous Morton range, its samples one contiguous
// run of the buffer, and a warp reads 32 consecutive runs (4 KB at SS 2, 4 spp) instead of
// runs scattered over a tile.
// Pixel of thread g in Morton-tile order.
__device__ __forceinline__ void morton_pixel(const ResolveArgs& a, uint32_t g, int ss_log2, int& x, int& y) {
    const uint32_t tile_px = (uint32_t)kTileSize >> ss_log2;
    const uint32_t per_tile_log2 = 2u * (uint32_t)(kTileBits - ss_log2);
    const uint32_t tile = g >> per_tile_log2;
    const uint32_t m = g & ((1u << per_tile_log2) - 1u);
    const uint32_t tiles_per_row = (uint32_t)((a.width * a.ss + kTileSize - 1) >> kTileBits);
    x = (int)((tile % tiles_per_row) * tile_px + morton_compact(m));
    y = (int)((tile / tiles_per_row) * tile_px + morton_compact(m >> 1));
}

// kHiz: the fine Hi-Z levels come with it, and a depth-only launch then leaves the depth image itself
// to the final resolve.  Where the image fills the SMs (2048 threads each), the lines that its threads
// are reading are 256 KB an SM, all of L1, and the few bytes of shared memory and the wait for the block's
// other pixels cost more than the launch they save: 1080p, ss 2, 15 spp, both resolves and the chain
// 810 us with, 709 without, and 708 before there were fine levels here; ss 1, 24 spp 372 / 359 / 361, ss 1,
// 9 spp 119 / 123 / 130.  launch_resolve_any draws the line.
template <bool kDepthOnly, bool kHiz>
__global__ void __launch_bounds__(256, 8) resolve_morton_kernel(ResolveArgs a, HizView hiz, int ss_log2) {
    previous_kernel_done();
    report_counters(a);
    int x, y;
    morton_pixel(a, blockIdx.x * blockDim.x + threadIdx.x, ss_log2, x, y);
    const bool inside = x < a.width && y < a.height;
    float depth = 0.0f;
    if (inside) depth = resolve_pixel<kDepthOnly>(a, x, y);
    if (inside && !(kDepthOnly && kHiz)) a.depth[y * a.width + x] = depth;
    if constexpr (kHiz) {
        __shared__ float exchange[8];
        hiz_fine_levels(hiz, depth, x, y, a.hiz_min_levels, exchange);
    }
}

// Staged variant: a block's pixels are consecutive in Morton-tile order, so their samples are
// one contiguous run of the buffer (px_per_block x SS*SS*spp entries, at most 32 KB), which the
// block reads with coalesced 16-byte loads.  Used for SS 1, 2, 4, 8 with 1 to 8 or a power of two of
// samples per pixel and, in all, a power of two from 2 to 128 or any number below 64.
//   depth only: of every entry pair the smaller high word goes to shared memory; a pixel's depth
//     is that of its smallest key.  That is the smallest depth bit for bit where the conversion to NDC
//     does not fall anywhere as the key grows.  It ends in an approximate division, of which only an
//     error bound is promised, so a renderer sweeps all 2^28 keys of its planes once, when it is
//     created (a.monotone; under half a millisecond); for planes that fail (a near plane at or below zero: the
//     view depth passes through zero) every sample is converted, as in resolve_pixel.
//   final: the run itself goes to shared memory, two pad words after each pixel's samples to keep
//     a warp's 16-byte reads on different banks (an odd number of words per pixel where the run is no
//     power of two and read word by word); the 12-bit channels become floats by their bits
//     under 2^23 (exact), which keeps them off the conversion unit.
// The kernel was bound by instructions, not by the 8 bytes per sample: with run-time sizes, a
// division per pixel and 64-bit indices it took 40 (depth) and 63 (final) instructions per sample
// at 8 samples a pixel; sizes are now template parameters and the grid is tiles_x * blocks per
// tile by tiles_y:
// 28 and 44, and 1M town at 4K, 2 spp: 111 -> 88 us (depth; the 531 MB take 82 at the copy rate) and
// 175 -> 136 us, the frame 995 -> 943; 500k town at 720p, 1 spp: 139 -> 127.
constexpr int kResolveMaxRun = 128;
// 64 pixels per block (155 us for both resolves at 1080p; 32 196, 256 162), 32 above 64 samples each
__host__ __device__ constexpr uint32_t resolve_pixels(int run) { return run <= 64 ? 64u : 32u; }
__host__ __device__ constexpr int resolve_blocks_log2(int ss_log2, int run) {  // blocks per tile
    return 2 * (kTileBits - ss_log2) - (run <= 64 ? 6 : 5);
}

template <bool kDepthOnly, int kSsLog2, int kPasses>
__global__ void __launch_bounds__(resolve_pixels(kPasses << (2 * kSsLog2))) resolve_staged_kernel(ResolveArgs a, HizView hiz) {
    previous_kernel_done();
    report_counters(a);
    constexpr uint32_t kRun = (uint32_t)kPasses << (2 * kSsLog2), kHalf = kRun / 2u, kPx = resolve_pixels((int)kRun);
    constexpr int kBlocksLog2 = resolve_blocks_log2(kSsLog2, (int)kRun);
    constexpr uint32_t kTilePxLog2 = (uint32_t)(kTileBits - kSsLog2);
    constexpr bool kPow2 = (kRun & (kRun - 1u)) == 0u;
    // words per pixel.  A power of two: pairs of entries and a pad (depth only: 4 bytes a pair, final:
    // 16).  Otherwise entries, an odd number of places (4 or 8 bytes an entry)
    constexpr uint32_t kStride = kPow2 ? kHalf + 1u : kRun | 1u;
    __shared__ __align__(16) uint32_t stage[kPx * kStride * (kPow2 ? (kDepthOnly ? 1u : 4u) : (kDepthOnly ? 1u : 2u))];
    __shared__ float exchange[2];
    // blocks take the buffer from its end: the splat walks screen bins (buffer tiles) in
    // ascending order, so the tiles it touched last are the ones still in L2
    const uint32_t bx = gridDim.x - 1u - blockIdx.x, ty = gridDim.y - 1u - blockIdx.y;
    const uint32_t tx = bx >> kBlocksLog2, sub = bx & ((1u << kBlocksLog2) - 1u);
    const uint32_t tile = ty * (gridDim.x >> kBlocksLog2) + tx, t = threadIdx.x;
    const ulonglong2* src = reinterpret_cast<const ulonglong2*>(a.buffer) +
                            ((uint64_t)((tile << kBlocksLog2) + sub) * (kPx * kRun / 2u) + t);
    const int x = (int)((tx << kTilePxLog2) + morton_compact(sub * kPx) + morton_compact(t));
    const int y = (int)((ty << kTilePxLog2) + morton_compact((sub * kPx) >> 1) + morton_compact(t >> 1));
    const bool inside = x < a.width && y < a.height;
    uint32_t nearest = 0xFFFFFFFFu;
    constexpr uint32_t kLoads = kRun / 2u;  // 16-byte loads per thread (kRun entries each, kPx even)
    if constexpr (!kPow2) {
        // entry e of the block's run: place e % kRun of pixel e / kRun
        static_assert(kPx == 64u, "runs that are no power of two stay below 64 samples");
        uint64_t* words = reinterpret_cast<uint64_t*>(stage);
#pragma unroll 8
        for (uint32_t k = 0; k < (kRun + 1u) / 2u; ++k) {
            const uint32_t i = k * kPx + t;  // pair
            if (i >= kPx * kRun / 2u) break;
            const ulonglong2 q = __ldcs(src + k * kPx);
            const uint32_t e0 = 2u * i, e1 = e0 + 1u;
            const uint32_t d0 = e0 / kRun * kStride + e0 % kRun, d1 = e1 / kRun * kStride + e1 % kRun;
            if (kDepthOnly) {
                stage[d0] = (uint32_t)(q.x >> 32);
                stage[d1] = (uint32_t)(q.y >> 32);
            } else {
                words[d0] = q.x;
                words[d1] = q.y;
            }
        }
        __syncthreads();
        if (kDepthOnly) {
#pragma unroll
            for (uint32_t k = 0; k < kRun; ++k) nearest = min(nearest, stage[t * kStride + k]);
        }
    } else if (kDepthOnly) {
        uint32_t* put = stage + t + t / kHalf;
#pragma unroll 8
        for (uint32_t k = 0; k < kLoads; ++k) {
            const uint4 q = __ldcs(reinterpret_cast<const uint4*>(src + k * kPx));
            put[k * kPx + k * kPx / kHalf] = min(q.y, q.w);
        }
        __syncthreads();
        const uint32_t* mine = stage + t * (kHalf + 1u);
#pragma unroll
        for (uint32_t k = 0; k < kHalf; ++k) nearest = min(nearest, mine[k]);
    } else {
        ulonglong2* put = reinterpret_cast<ulonglong2*>(stage) + t + t / kHalf;
#pragma unroll 8
        for (uint32_t k = 0; k < kLoads; ++k) put[k * kPx + k * kPx / kHalf] = __ldcs(src + k * kPx);
        __syncthreads();
    }
    if (!kDepthOnly) {
        const uint64_t* mine = reinterpret_cast<const uint64_t*>(stage) + t * (kPow2 ? kRun + 2u : kStride);
        vec3 color = make_v3(0.0f, 0.0f, 0.0f);
        auto add = [&](uint64_t val) {
            const uint32_t lo = (uint32_t)val, hi = (uint32_t)(val >> 32);
            nearest = min(nearest, hi);
            color.x += channel12(__funnelshift_r(lo, hi, 24)) / 255.0f;
            color.y += channel12(lo >> 12) / 255.0f;
            color.z += channel12(lo) / 255.0f;
        };
#pragma unroll
        for (int dx = 0; dx < (1 << kSsLog2); ++dx)
#pragma unroll
            for (int dy = 0; dy < (1 << kSsLog2); ++dy) {
                const uint64_t* at = mine + morton_encode((uint32_t)dx, (uint32_t)dy) * (uint32_t)kPasses;
                if constexpr (!kPow2 || kPasses == 1) {
#pragma unroll 8
                    for (int p = 0; p < kPasses; ++p) add(at[p]);
                } else {
#pragma unroll 8
                    for (int p = 0; p < kPasses; p += 2) {
                        const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(at + p);
                        add(q.x);
                        add(q.y);
                    }
                }
            }
        if (inside) {
            const uint32_t idx = (uint32_t)(y * a.width + x);
            const float inv_passes = 1.0f / (float)(a.num_passes * a.ss * a.ss);
            a.color[3 * idx + 0] = color.x * inv_passes;
            a.color[3 * idx + 1] = color.y * inv_passes;
            a.color[3 * idx + 2] = color.z * inv_passes;
        }
    }
    const float depth = depth_of_key(nearest, a.near_plane, a.far_plane);
    if (inside && !(kDepthOnly && a.hiz_fused)) a.depth[(uint32_t)(y * a.width + x)] = depth;
    if constexpr (kPx == 64u) {
        if (a.hiz_fused) hiz_fine_levels(hiz, depth, x, y, a.hiz_min_levels, exchange);
    }
}

// ---------------------------------------------------------------------------------
// Hi-Z chain (depth_mip_chain.cu:7-67)
// ---------------------------------------------------------------------------------
// The whole chain in one launch, for views whose resolve does not write the fine levels (128 samples
// a pixel, images of up to four pixels).  A 16x16-thread block covers a 64x64 tile of the depth image:
// each thread copies its 4x4 texels into the finest level and reduces them in registers to
// the next two levels (2x2, then 1), the block reduces its 16x16 results through four more
// levels in shared memory, and the block that finishes last (a counter, no waiting) reduces
// the remaining coarse levels.  Every texel is the min/max of the same finest texels as with
// one launch per level, so the chain is identical.  Level j from the finest (j = 1, 2, ...)
// reduces with min while j <= min_levels, else with max.
constexpr int kHizThreads = 16;                  // threads per block edge
constexpr int kHizTile = 4 * kHizThreads;        // finest texels per block edge

// The levels above `have`, by the block that finishes last (a counter, no waiting), with 256
// threads: a level of up to 1024 texels is reduced in shared memory, so that the last levels cost
// a barrier each and not a round trip through L2 (1080p: five levels above 30 x 17).
__device__ __forceinline__ void hiz_coarse_levels(const HizView& c, int have, int min_levels) {
    constexpr int kIn = 1024;
    __shared__ float level[2][kIn];
    __shared__ int s_last;
    if (have <= 0) return;                                       // the chain is complete
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(c.done, 1u) == gridDim.x * gridDim.y - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int L = c.levels - 1;
    int cur = 0;
    bool staged = false;
    for (int l = have - 1; l >= 0; --l) {
        const bool use_min = (L - l) <= min_levels;
        const int wl = c.level_w[l], hl = c.level_h[l];
        const int wf = c.level_w[l + 1], hf = c.level_h[l + 1];
        const float* fine = c.mip + c.level_off[l + 1];
        if (!staged && wf * hf <= kIn) {
            for (int i = threadIdx.x; i < wf * hf; i += blockDim.x) level[cur][i] = __ldcg(fine + i);
            __syncthreads();
            staged = true;
        }
        for (int i = threadIdx.x; i < wl * hl; i += blockDim.x) {
            const int x = i % wl, y = i / wl;
            float acc = hiz_identity(use_min);
            for (int dy = 0; dy < 2; ++dy)
                for (int dx = 0; dx < 2; ++dx) {
                    const int fx = 2 * x + dx, fy = 2 * y + dy;
                    if (fx < wf && fy < hf)
                        acc = hiz_op(use_min, acc, staged ? level[cur][fy * wf + fx] : __ldcg(fine + (uint64_t)fy * wf + fx));
                }
            c.mip[c.level_off[l] + (uint64_t)y * wl + x] = acc;
            if (staged) level[cur ^ 1][i] = acc;
        }
        if (staged) cur ^= 1;
        else __threadfence_block();
        __syncthreads();
    }
    if (threadIdx.x == 0) *c.done = 0u;
}

__global__ void __launch_bounds__(kHizThreads * kHizThreads) hiz_build_kernel(HizView c, const float* __restrict__ src,
                                                                               int min_levels) {
    previous_kernel_done();
    __shared__ float sm[kHizThreads * kHizThreads];
    const int L = c.levels - 1;
    const int tx = threadIdx.x % kHizThreads, ty = threadIdx.x / kHizThreads;
    const int gx = blockIdx.x * kHizThreads + tx, gy = blockIdx.y * kHizThreads + ty;  // coords at level L-2
    const int W = c.level_w[L], H = c.level_h[L];
    float f[4][4];
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int x = 4 * gx + u, y = 4 * gy + v;
            f[v][u] = 0.0f;
            if (x < W && y < H) {
                f[v][u] = src[(uint64_t)y * W + x];
                c.mip[c.level_off[L] + (uint64_t)y * W + x] = f[v][u];
            }
        }
    float r = 0.0f;  // this thread's texel at the last level reduced so far
    bool have = false;
    if (L >= 1) {
        const int l = L - 1;
        const bool use_min = 0 < min_levels;
        const int wl = c.level_w[l], hl = c.level_h[l];
        float q[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                float acc = use_min ? INFINITY : -INFINITY;
#pragma unroll
                for (int dy = 0; dy < 2; ++dy)
#pragma unroll
                    for (int dx = 0; dx < 2; ++dx)
                        if (4 * gx + 2 * i + dx < W && 4 * gy + 2 * j + dy < H) acc = hiz_op(use_min, acc, f[2 * j + dy][2 * i + dx]);
                q[j][i] = acc;
                const int x = 2 * gx + i, y = 2 * gy + j;
                if (x < wl && y < hl) c.mip[c.level_off[l] + (uint64_t)y * wl + x] = acc;
            }
        if (L >= 2) {
            const int l2 = L - 2;
            const bool use_min2 = 1 < min_levels;
            float acc = use_min2 ? INFINITY : -INFINITY;
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    if (2 * gx + i < wl && 2 * gy + j < hl) acc = hiz_op(use_min2, acc, q[j][i]);
            r = acc;
            have = true;
            if (gx < c.level_w[l2] && gy < c.level_h[l2]) c.mip[c.level_off[l2] + (uint64_t)gy * c.level_w[l2] + gx] = acc;
        }
    }
    const int shared_levels = have ? min(4, L - 2) : 0;   // levels L-3 .. L-6 in shared memory
    if (have) sm[ty * kHizThreads + tx] = r;
    __syncthreads();
    for (int j = 1; j <= shared_levels; ++j) {
        const int l = L - 2 - j;
        const bool use_min = (j + 1) < min_levels;
        const int half = kHizThreads >> j;
        const int wf = c.level_w[l + 1], hf = c.level_h[l + 1];
        const bool act = tx < half && ty < half;
        const int bx = blockIdx.x * half + tx, by = blockIdx.y * half + ty;
        float acc = use_min ? INFINITY : -INFINITY;
        if (act) {
            for (int dy = 0; dy < 2; ++dy)
                for (int dx = 0; dx < 2; ++dx)
                    if (2 * bx + dx < wf && 2 * by + dy < hf) acc = hiz_op(use_min, acc, sm[(2 * ty + dy) * kHizThreads + 2 * tx + dx]);
        }
        __syncthreads();
        if (act) {
            sm[ty * kHizThreads + tx] = acc;
            if (bx < c.level_w[l] && by < c.level_h[l]) c.mip[c.level_off[l] + (uint64_t)by * c.level_w[l] + bx] = acc;
        }
        __syncthreads();
    }
    const int done_levels = (L >= 2 ? 2 : L) + shared_levels;   // levels below L written so far
    hiz_coarse_levels(c, L - done_levels, min_levels);
}

// The rest of the chain above the levels that the resolve wrote (hiz_fine_levels): a block reduces
// 16 x 16 texels of the 1/8-size level through four more levels, the last block does the others.
__global__ void __launch_bounds__(256) hiz_top_kernel(HizView c, int min_levels) {
    previous_kernel_done();
    __shared__ float sm[256];
    const int L = c.levels - 1, base = L - 3;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int gx = blockIdx.x * 16 + tx, gy = blockIdx.y * 16 + ty;
    if (gx < c.level_w[base] && gy < c.level_h[base])
        sm[threadIdx.x] = c.mip[c.level_off[base] + (uint64_t)gy * c.level_w[base] + gx];
    const int steps = min(4, base);
    for (int j = 1; j <= steps; ++j) {
        __syncthreads();
        const int l = base - j, half = 16 >> j;
        const bool use_min = (L - l) <= min_levels;
        const int bx = blockIdx.x * half + tx, by = blockIdx.y * half + ty;
        const bool act = tx < half && ty < half && bx < c.level_w[l] && by < c.level_h[l];
        float acc = hiz_identity(use_min);
        if (act) {
            for (int dy = 0; dy < 2; ++dy)
                for (int dx = 0; dx < 2; ++dx)
                    if (2 * bx + dx < c.level_w[l + 1] && 2 * by + dy < c.level_h[l + 1])
                        acc = hiz_op(use_min, acc, sm[(2 * ty + dy) * 16 + 2 * tx + dx]);
        }
        __syncthreads();
        if (act) {
            sm[ty * 16 + tx] = acc;
            c.mip[c.level_off[l] + (uint64_t)by * c.level_w[l] + bx] = acc;
        }
    }
    hiz_coarse_levels(c, base - steps, min_levels);
}

// ---------------------------------------------------------------------------------
// Half-precision scene: encode from the FP32 arrays, tile copies (load time)
// ---------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
    return (uint32_t)__half_as_ushort(__float2half_rn(lo)) | ((uint32_t)__half_as_ushort(__float2half_rn(hi)) << 16);
}

// origin of every kHalfOriginBlock Gaussians: the centre of their means' bounding box, and in w
// the step of the 16-bit fixed-point offsets from it (the largest half-extent / 32767)
__global__ void half_origins_kernel(const float4* __restrict__ pos_op, uint32_t n, float4* __restrict__ origin) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t begin = b * kHalfOriginBlock;
    if (begin >= n) return;
    const uint32_t end = min(begin + kHalfOriginBlock, n);
    float3 lo = make_float3(INFINITY, INFINITY, INFINITY), hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
    for (uint32_t g = begin; g < end; ++g) {
        const float4 p = pos_op[g];
        lo = make_float3(fminf(lo.x, p.x), fminf(lo.y, p.y), fminf(lo.z, p.z));
        hi = make_float3(fmaxf(hi.x, p.x), fmaxf(hi.y, p.y), fmaxf(hi.z, p.z));
    }
    const float3 o = make_float3(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z));
    const float h = fmaxf(fmaxf(fmaxf(hi.x - o.x, o.x - lo.x), fmaxf(hi.y - o.y, o.y - lo.y)),
                          fmaxf(hi.z - o.z, o.z - lo.z));
    const float k = __fdiv_rn(h, 32767.0f);
    origin[b] = make_float4(o.x, o.y, o.z, k >= 1.0e-30f ? k : 0.0f);
}

__device__ __forceinline__ uint32_t fixed16(float v, float o, float k) {
    const int q = k > 0.0f ? max(-32767, min(32767, __float2int_rn(__fdiv_rn(v - o, k)))) : 0;
    return (uint32_t)q & 0xFFFFu;
}

__global__ void encode_half_kernel(const float4* __restrict__ pos_op, const float4* __restrict__ rot,
                                   const float4* __restrict__ scale, const float4* __restrict__ sh,
                                   const float4* __restrict__ origin, uint32_t n, uint4* __restrict__ rec,
                                   uint4* __restrict__ scl, uint4* __restrict__ acq) {
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    const float4 p = pos_op[g], q = rot[g], c = scale[g], o = origin[g / kHalfOriginBlock];
    const uint32_t op16 = (uint32_t)__half_as_ushort(__float2half_rn(p.w));
    rec[g] = make_uint4(fixed16(p.x, o.x, o.w) | (fixed16(p.y, o.y, o.w) << 16), fixed16(p.z, o.z, o.w) | (op16 << 16),
                        pack_h2(q.x, q.y), pack_h2(q.z, q.w));
    float v[48];
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        const float4 t = sh[(size_t)g * 12 + i];
        v[4 * i] = t.x;
        v[4 * i + 1] = t.y;
        v[4 * i + 2] = t.z;
        v[4 * i + 3] = t.w;
    }
    // AC terms: 8-bit integers on a per-band scale (band 1: AC 0-8, band 2: 9-23, band 3: 24-44),
    // scale = the band's max |c| / 127 rounded up to bf16, so that every |c| / scale <= 127
    float mb[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int e = 0; e < 45; ++e) {
        const int b = e < 9 ? 0 : (e < 24 ? 1 : 2);
        mb[b] = fmaxf(mb[b], fabsf(v[3 + e]));
    }
    uint32_t sb[3];
    float sc[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        const uint32_t bits = __float_as_uint(mb[b] / 127.0f);
        sb[b] = (bits >> 16) + ((bits & 0xFFFFu) ? 1u : 0u);
        sc[b] = __uint_as_float(sb[b] << 16);
    }
    scl[g] = make_uint4(pack_h2(c.x, c.y), pack_h2(c.z, v[0]), pack_h2(v[1], v[2]), sb[0] | (sb[1] << 16));
    uint32_t w[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) w[i] = 0u;
#pragma unroll
    for (int e = 0; e < 45; ++e) {
        const float k = sc[e < 9 ? 0 : (e < 24 ? 1 : 2)];
        const int q = k > 0.0f ? max(-127, min(127, __float2int_rn(__fdiv_rn(v[3 + e], k)))) : 0;
        w[e >> 2] |= ((uint32_t)q & 0xFFu) << (8 * (e & 3));
    }
    w[11] |= sb[2] << 8;  // bytes 45-46: band 3's scale
#pragma unroll
    for (int i = 0; i < 3; ++i) acq[(size_t)g * 3 + i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
}

// copies of a half scene: origins of copy k = source origins + (dx[k], 0, dz[k])
__global__ void translate_origins_kernel(const float4* __restrict__ src, uint32_t count, float dx, float dz,
                                         float4* __restrict__ dst) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float4 o = src[i];
    dst[i] = make_float4(o.x + dx, o.y, o.z + dz, o.w);
}

// cull blocks of the tiled scene: node j covers Gaussians [j*pb, j*pb+pb) inside one copy and is
// the union of the source nodes it spans, translated with its copy
__global__ void tile_nodes_kernel(const float4* __restrict__ src, uint32_t src_pb, uint32_t src_n, uint32_t pb,
                                  uint32_t copies, const float2* __restrict__ offsets, uint64_t total,
                                  float4* __restrict__ dst, uint32_t nodes) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nodes) return;
    const uint64_t begin = (uint64_t)j * pb;
    const uint64_t end = min(begin + pb, total);
    const uint32_t k = (uint32_t)(begin / src_n);
    const uint32_t s0 = (uint32_t)((begin - (uint64_t)k * src_n) / src_pb);
    const uint32_t s1 = (uint32_t)((end - 1 - (uint64_t)k * src_n) / src_pb);
    float3 lo = make_float3(INFINITY, INFINITY, INFINITY), hi = make_float3(-INFINITY, -INFINITY, -INFINITY);
    for (uint32_t s = s0; s <= s1; ++s) {
        const float4 a = src[2 * s], b = src[2 * s + 1];
        lo = make_float3(fminf(lo.x, a.x), fminf(lo.y, a.y), fminf(lo.z, a.z));
        hi = make_float3(fmaxf(hi.x, b.x), fmaxf(hi.y, b.y), fmaxf(hi.z, b.z));
    }
    const float2 t = offsets[k];
    dst[2 * j] = make_float4(lo.x + t.x, lo.y, lo.z + t.y, __uint_as_float((uint32_t)begin));
    dst[2 * j + 1] = make_float4(hi.x + t.x, hi.y, hi.z + t.y, __uint_as_float((uint32_t)(end - begin)));
}

// ---------------------------------------------------------------------------------
// Block AABBs at load time (gaussian_bvh.cu:111-144).  The reference computes these on the
// host in IEEE single precision without fused multiply-adds; the _rn intrinsics below keep
// nvcc from contracting, so the boxes are bit-identical to the host computation.
// ---------------------------------------------------------------------------------
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float rsub(float a, float b) { return __fsub_rn(a, b); }

__device__ __forceinline__ void host_order_cov_diag(vec3 s, vec4 q, float out[3]) {
    const float w = q.x, x = q.y, y = q.z, z = q.w;
    float qxx = rmul(x, x), qyy = rmul(y, y), qzz = rmul(z, z);
    float qxz = rmul(x, z), qxy = rmul(x, y), qyz = rmul(y, z);
    float qwx = rmul(w, x), qwy = rmul(w, y), qwz = rmul(w, z);
    float r[3][3];
    r[0][0] = rsub(1.0f, rmul(2.0f, radd(qyy, qzz)));
    r[0][1] = rmul(2.0f, radd(qxy, qwz));
    r[0][2] = rmul(2.0f, rsub(qxz, qwy));
    r[1][0] = rmul(2.0f, rsub(qxy, qwz));
    r[1][1] = rsub(1.0f, rmul(2.0f, radd(qxx, qzz)));
    r[1][2] = rmul(2.0f, radd(qyz, qwx));
    r[2][0] = rmul(2.0f, radd(qxz, qwy));
    r[2][1] = rmul(2.0f, rsub(qyz, qwx));
    r[2][2] = rsub(1.0f, rmul(2.0f, radd(qxx, qyy)));
    // M = R * S, column j = (R0*S[j].x + R1*S[j].y) + R2*S[j].z with S diagonal
    float sd[3][3] = {{s.x, 0.0f, 0.0f}, {0.0f, s.y, 0.0f}, {0.0f, 0.0f, s.z}};
    float m[3][3];
    for (int j = 0; j < 3; ++j)
        for (int i = 0; i < 3; ++i)
            m[j][i] = radd(radd(rmul(r[0][i], sd[j][0]), rmul(r[1][i], sd[j][1])), rmul(r[2][i], sd[j][2]));
    // cov = M * M^T: cov[j][i] = (M0[i]*M[0][j] + M1[i]*M[1][j]) + M2[i]*M[2][j]; diagonal only
    for (int i = 0; i < 3; ++i)
        out[i] = radd(radd(rmul(m[0][i], m[0][i]), rmul(m[1][i], m[1][i])), rmul(m[2][i], m[2][i]));
}

__global__ void block_bounds_kernel(const float4* __restrict__ pos_op, const float4* __restrict__ rot,
                                    const float4* __restrict__ scale, uint32_t n, uint32_t per_block,
                                    float4* __restrict__ nodes, uint32_t node_count) {
    const uint32_t node = blockIdx.x * blockDim.x + threadIdx.x;
    if (node >= node_count) return;
    const uint32_t begin = node * per_block;
    const uint32_t end = min(begin + per_block, n);
    float bmin[3] = {3.402823466e+38f, 3.402823466e+38f, 3.402823466e+38f};
    float bmax[3] = {-3.402823466e+38f, -3.402823466e+38f, -3.402823466e+38f};
    for (uint32_t g = begin; g < end; ++g) {
        float4 p = pos_op[g], q = rot[g], s = scale[g];
        float d[3];
        host_order_cov_diag(make_v3(s.x, s.y, s.z), make_v4(q.x, q.y, q.z, q.w), d);
        float mean[3] = {p.x, p.y, p.z};
        for (int i = 0; i < 3; ++i) {
            float ext = rmul(kTruncationStd, __fsqrt_rn(d[i]));
            float lo = rsub(mean[i], ext), hi = radd(mean[i], ext);
            bmin[i] = (lo < bmin[i]) ? lo : bmin[i];
            bmax[i] = (bmax[i] < hi) ? hi : bmax[i];
        }
    }
    nodes[2 * node] = make_float4(bmin[0], bmin[1], bmin[2], __uint_as_float(begin));
    nodes[2 * node + 1] = make_float4(bmax[0], bmax[1], bmax[2], __uint_as_float(end - begin));
}

// ---------------------------------------------------------------------------------
// Post-processing (post_processing_kernels.cuh:108-285)
// ---------------------------------------------------------------------------------
__device__ __forceinline__ float mixf(float x, float y, float a) { return x * (1.0f - a) + y * a; }
__device__ __forceinline__ vec3 mix3s(vec3 x, vec3 y, float a) {
    return make_v3(mixf(x.x, y.x, a), mixf(x.y, y.y, a), mixf(x.z, y.z, a));
}
__device__ __forceinline__ vec3 ld3(const float* p, int i) { return make_v3(p[3 * i], p[3 * i + 1], p[3 * i + 2]); }

// temporalRender reads the 3x3 neighbourhood of the current colour buffer while other threads
// overwrite that same buffer with blended results, so its output depends on thread order.
// Here the blended colour goes to a separate buffer (out_color, never aliasing cur_color): the
// neighbourhood is always the unblended current frame and the result is deterministic.
//
// What bounded the kernel was L1 (40 four-byte loads a pixel, each three or four lines for a warp
// because pixels are 12 bytes apart) beside 395 instructions a pixel.  So a block's 32 x 16 pixels and
// a one-pixel rim go to shared memory with contiguous loads (a rim pixel outside the image is its
// nearest pixel inside, which every window that holds the rim pixel holds too), a warp slides down
// its two rows with the last rows' minima and maxima in registers, and colours and bytes leave
// through shared memory as contiguous words: 338 instructions, 4K 132.6 -> 123.5 us (the 357 MB take 55 at
// the copy rate; one row per warp 122, four 131).  What is left is mostly the history's 12 scattered
// loads and the arithmetic around them.
// (a NaN operand is passed over, as by the reference's selects from 1e9 and -1e9)
__device__ __forceinline__ float min3(float a, float b, float c) { return fminf(fminf(a, b), c); }
__device__ __forceinline__ float max3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }

constexpr int kTaaTile = 32, kTaaRows = 2, kTaaHeight = 8 * kTaaRows, kTaaSpan = (kTaaTile + 2) * 3;

__global__ void __launch_bounds__(256, 6) taa_kernel(uint8_t* __restrict__ image, float* __restrict__ out_color,
                           const float* __restrict__ cur_color,
                           const float* __restrict__ prev_color, const float* __restrict__ cur_depth,
                           const float* __restrict__ prev_depth, mat4 reproj, float blend, int width, int height) {
    previous_kernel_done();
    __shared__ float tile[(kTaaHeight + 2) * kTaaSpan];
    __shared__ float put[8][kTaaTile * 3];
    const int lane = (int)(threadIdx.x & 31u), warp = (int)(threadIdx.x >> 5);
    const int x0 = blockIdx.x * kTaaTile, y0 = blockIdx.y * kTaaHeight;
    float depths[kTaaRows];
#pragma unroll
    for (int r = 0; r < kTaaRows; ++r) {
        const int x = x0 + lane, y = y0 + warp * kTaaRows + r;
        depths[r] = x < width && y < height ? cur_depth[y * width + x] : 0.0f;
    }
    if (x0 > 0 && x0 + kTaaTile < width) {
        for (int r = warp; r < kTaaHeight + 2; r += 8) {
            const int yy = min(max(y0 - 1 + r, 0), height - 1);
            const float* row = cur_color + 3 * (yy * width + x0 - 1);
#pragma unroll
            for (int c = 0; c < kTaaSpan; c += 32)
                if (c + lane < kTaaSpan) tile[r * kTaaSpan + c + lane] = row[c + lane];
        }
    } else {
        for (int r = warp; r < kTaaHeight + 2; r += 8) {
            const int yy = min(max(y0 - 1 + r, 0), height - 1);
            for (int c = lane; c < kTaaSpan; c += 32) {
                const int xx = min(max(x0 - 1 + c / 3, 0), width - 1);
                tile[r * kTaaSpan + c] = cur_color[3 * (yy * width + xx) + c % 3];
            }
        }
    }
    __syncthreads();
    const int x = x0 + lane;
    // minima and maxima of a row's three pixels around x, and its middle pixel
    auto row_of = [&](int r, vec3& lo, vec3& hi, vec3& mid) {
        const float* p = tile + r * kTaaSpan + 3 * lane;
        mid = make_v3(p[3], p[4], p[5]);
        lo = make_v3(min3(p[0], mid.x, p[6]), min3(p[1], mid.y, p[7]), min3(p[2], mid.z, p[8]));
        hi = make_v3(max3(p[0], mid.x, p[6]), max3(p[1], mid.y, p[7]), max3(p[2], mid.z, p[8]));
    };
    vec3 lo0, hi0, lo1, hi1, lo2, hi2, mid1, mid2;
    row_of(warp * kTaaRows, lo0, hi0, mid1);
    row_of(warp * kTaaRows + 1, lo1, hi1, mid1);
#pragma unroll
    for (int r = 0; r < kTaaRows; ++r) {
        const int y = y0 + warp * kTaaRows + r;
        row_of(warp * kTaaRows + r + 2, lo2, hi2, mid2);
        vec3 color = mid1;
        const bool inside = x < width && y < height;
        const int idx = y * width + x;
        if (inside) {
            const float depth = depths[r];
            vec4 clip = make_v4((x + 0.5f) / width * 2.0f - 1.0f, (y + 0.5f) / height * 2.0f - 1.0f, depth, 1.0f);
            vec4 prev = reproj * clip;
            prev = make_v4(prev.x / prev.w, prev.y / prev.w, prev.z / prev.w, prev.w / prev.w);
            float px = (prev.x * 0.5f + 0.5f) * width - 0.5f;
            float py = (prev.y * 0.5f + 0.5f) * height - 0.5f;
            if (px >= 0 && px < width && py >= 0 && py < height) {
                // bilinearSampleCombined
                int x0 = (int)floorf(px), y0 = (int)floorf(py);
                int x1 = x0 + 1, y1 = y0 + 1;
                x0 = (x0 < 0) ? 0 : ((x0 >= width) ? width - 1 : x0);
                y0 = (y0 < 0) ? 0 : ((y0 >= height) ? height - 1 : y0);
                x1 = (x1 < 0) ? 0 : ((x1 >= width) ? width - 1 : x1);
                y1 = (y1 < 0) ? 0 : ((y1 >= height) ? height - 1 : y1);
                float tx = px - floorf(px);
                float ty = py - floorf(py);
                int i00 = y0 * width + x0, i10 = y0 * width + x1, i01 = y1 * width + x0, i11 = y1 * width + x1;
                (void)prev_depth;
                vec3 top = mix3s(ld3(prev_color, i00), ld3(prev_color, i10), tx);
                vec3 bottom = mix3s(ld3(prev_color, i01), ld3(prev_color, i11), tx);
                vec3 hist = mix3s(top, bottom, ty);
                // computeNeighborhoodMinMax
                const vec3 nmin = make_v3(fminf(1e9f, min3(lo0.x, lo1.x, lo2.x)), fminf(1e9f, min3(lo0.y, lo1.y, lo2.y)),
                                          fminf(1e9f, min3(lo0.z, lo1.z, lo2.z)));
                const vec3 nmax = make_v3(fmaxf(-1e9f, max3(hi0.x, hi1.x, hi2.x)), fmaxf(-1e9f, max3(hi0.y, hi1.y, hi2.y)),
                                          fmaxf(-1e9f, max3(hi0.z, hi1.z, hi2.z)));
                vec3 h = make_v3(gclamp(hist.x, nmin.x - 0.05f, nmax.x + 0.05f), gclamp(hist.y, nmin.y - 0.05f, nmax.y + 0.05f),
                                 gclamp(hist.z, nmin.z - 0.05f, nmax.z + 0.05f));
                color = mix3s(color, h, blend);
            }
        }
        vec3 o = make_v3(gclamp(color.x, 0.0f, 1.0f) * 255.0f, gclamp(color.y, 0.0f, 1.0f) * 255.0f,
                         gclamp(color.z, 0.0f, 1.0f) * 255.0f);
        const uint8_t b0 = (uint8_t)roundf(o.x), b1 = (uint8_t)roundf(o.y), b2 = (uint8_t)roundf(o.z);
        if (x0 + kTaaTile <= width && (width & 3) == 0) {  // whole rows of 32 pixels, their bytes on words
            if (y < height) {
                float* w = put[warp];
                w[3 * lane + 0] = color.x;
                w[3 * lane + 1] = color.y;
                w[3 * lane + 2] = color.z;
                __syncwarp();
                float* to = out_color + 3 * (y * width + x0);
                to[lane] = w[lane];
                to[lane + 32] = w[lane + 32];
                to[lane + 64] = w[lane + 64];
                __syncwarp();
                uint8_t* wb = reinterpret_cast<uint8_t*>(w);
                wb[3 * lane + 0] = b0;
                wb[3 * lane + 1] = b1;
                wb[3 * lane + 2] = b2;
                __syncwarp();
                uint8_t* bytes = image + 3 * (y * width + x0);
                if ((reinterpret_cast<uintptr_t>(image) & 3u) == 0u) {
                    if (lane < 24) reinterpret_cast<uint32_t*>(bytes)[lane] = reinterpret_cast<const uint32_t*>(w)[lane];
                } else {
                    for (int i = lane; i < 96; i += 32) bytes[i] = wb[i];
                }
                __syncwarp();
            }
        } else if (inside) {
            out_color[3 * idx + 0] = color.x;
            out_color[3 * idx + 1] = color.y;
            out_color[3 * idx + 2] = color.z;
            image[3 * idx + 0] = b0;
            image[3 * idx + 1] = b1;
            image[3 * idx + 2] = b2;
        }
        lo0 = lo1;
        hi0 = hi1;
        lo1 = lo2;
        hi1 = hi2;
        mid1 = mid2;
    }
}

// A frame without history: the colours as they are.  Four values per thread where the buffers are aligned
// for it; in taa_kernel, whose tile nobody needs then, 4K took 67.7 us (41.8 before it had one).
__global__ void __launch_bounds__(256) taa_first_kernel(uint8_t* __restrict__ image, float* __restrict__ out_color,
                                                        const float* __restrict__ cur_color, uint32_t values, int aligned) {
    previous_kernel_done();
    auto byte_of = [](float v) { return (uint8_t)roundf(gclamp(v, 0.0f, 1.0f) * 255.0f); };
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) * 4u;
    if (aligned && i + 4u <= values) {
        const float4 c = *reinterpret_cast<const float4*>(cur_color + i);
        *reinterpret_cast<float4*>(out_color + i) = c;
        *reinterpret_cast<uchar4*>(image + i) = make_uchar4(byte_of(c.x), byte_of(c.y), byte_of(c.z), byte_of(c.w));
        return;
    }
    for (uint32_t k = i; k < min(i + 4u, values); ++k) {
        out_color[k] = cur_color[k];
        image[k] = byte_of(cur_color[k]);
    }
}

__global__ void progressive_kernel(uint8_t* __restrict__ image, float* __restrict__ cur, float* __restrict__ accum,
                                   int width, int height, int frames) {
    previous_kernel_done();
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= width * height) return;
    vec3 color = ld3(cur, idx);
    if (frames > 1) color = color + ld3(accum, idx);
    cur[3 * idx + 0] = color.x;
    cur[3 * idx + 1] = color.y;
    cur[3 * idx + 2] = color.z;
    accum[3 * idx + 0] = 0.0f;
    accum[3 * idx + 1] = 0.0f;
    accum[3 * idx + 2] = 0.0f;
    color = color * (255.0f / (float)frames);
    color = make_v3(gclamp(color.x, 0.0f, 255.0f), gclamp(color.y, 0.0f, 255.0f), gclamp(color.z, 0.0f, 255.0f));
    image[3 * idx + 0] = (uint8_t)roundf(color.x);
    image[3 * idx + 1] = (uint8_t)roundf(color.y);
    image[3 * idx + 2] = (uint8_t)roundf(color.z);
}

int g_num_sms = 0;

}  // namespace

// ---------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------
namespace {
// Every frame kernel is launched as a programmatic dependent of the one before it in its stream:
// the launch is set up while that kernel runs, and its blocks start as soon as the last block of
// that kernel has left the GPU instead of after its completion has been reported back.  No kernel
// signals earlier (griddepcontrol.launch_dependents): blocks of the next kernel that wait beside
// a persistent grid's tail land unevenly on the SMs, and frames got slower (16M town: 2.79
// against 2.38 ms).  A frame is 4 to 18 launches, most of them a few microseconds long on small
// views.  Measured with the frame's counters handed over by the final resolve, against plain
// launches and a copy: 20k cube at 160x90 45.5 -> 22.0 us a frame, 60k town at 320x180 130 -> 89,
// 1M cube at 640x360 177 -> 154, 4M town at 1080p 1121 -> 1076.
template <typename... KArgs, typename... Args>
void launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchAttribute dependent{};
    dependent.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    dependent.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &dependent;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}
}  // namespace

uint32_t clear_blocks(const ClearArgs& c) {
    const uint64_t want = (c.pairs + 255u) / 256u;
    return want < 148u * 16u ? (uint32_t)want : 148u * 16u;
}

void launch_cull(const CullArgs& args, cudaStream_t stream) {
    CullArgs a = args;
    a.words_per_block = kCullWords;  // at least 4 blocks per SM where there is the work for it
    while (a.words_per_block > 8u && a.b.words < a.words_per_block * 592u) a.words_per_block >>= 1;
    a.cull_blocks = (a.b.words + a.words_per_block - 1u) / a.words_per_block;
    launch_k(cull_kernel, a.cull_blocks + clear_blocks(a.clear), 256, 0, stream, a);
}

void launch_super_bounds(const float4* nodes, uint32_t node_count, float4* supers, cudaStream_t stream) {
    const uint32_t words = (node_count + 31u) / 32u;
    if (words) super_bounds_kernel<<<(words + 255u) / 256u, 256, 0, stream>>>(nodes, node_count, supers, words);
}

// Resident blocks of the persistent preprocess on this device, capped by the work.
template <class Scene, bool kImmediate, bool kCull>
int preprocess_grid_size(uint32_t n) {
    static int per_sm = 0;
    if (per_sm == 0) {
        int blocks = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, preprocess_kernel<Scene, kImmediate, kCull>, 256, 0);
        per_sm = blocks < 1 ? 1 : blocks;
    }
    if (g_num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    }
    const uint64_t want = ((uint64_t)n + 255) / 256;
    const uint64_t cap = (uint64_t)g_num_sms * (uint64_t)per_sm;
    // a culling warp has one chunk where they all fit, else two
    if (kCull) return (int)(want <= cap ? want : (want + kSelfCullChunks - 1) / kSelfCullChunks);
    return (int)(want < cap ? want : cap);
}

template <class Scene, bool kImmediate, bool kCull>
void launch_preprocess_as(PreprocessArgs a, const Scene& s, cudaStream_t stream) {
    a.blocks_here = (uint32_t)preprocess_grid_size<Scene, kImmediate, kCull>(a.n);
    launch_k(preprocess_kernel<Scene, kImmediate, kCull>, a.blocks_here + clear_blocks(a.clear), 256, 0, stream, a, s);
}

template <class Scene>
void launch_preprocess(const PreprocessArgs& a, const Scene& s, cudaStream_t stream) {
    if (a.n == 0) return;
    if (a.immediate_threshold > 0) launch_preprocess_as<Scene, true, false>(a, s, stream);
    else if (a.cull_here) launch_preprocess_as<Scene, false, true>(a, s, stream);
    else launch_preprocess_as<Scene, false, false>(a, s, stream);
}

void launch_preprocess_fp32(const PreprocessArgs& a, const SceneFP32& s, cudaStream_t stream) {
    launch_preprocess(a, s, stream);
}

void launch_preprocess_half(const PreprocessArgs& a, const SceneHalf& s, cudaStream_t stream) {
    launch_preprocess(a, s, stream);
}

void launch_preprocess_compressed(const PreprocessArgs& a, const SceneCompressed& s, cudaStream_t stream) {
    launch_preprocess(a, s, stream);
}

static_assert(kScanTile == kScanTileGaussians, "scan tile size");
// tile words a scan of n Gaussians may use (the small-tile count, an upper bound)
uint32_t scan_tile_count(uint32_t n) { return (uint32_t)(((uint64_t)n + kScanTileSmall - 1) / kScanTileSmall); }

int scan_tile_shift(uint32_t n) { return n >= kScanBigScene ? 14 : 12; }

template <bool kBinned>
void launch_scan_write(const ScanArgs& a, uint32_t tiles, bool big, bool direct, cudaStream_t stream) {
    const uint32_t grid = tiles + (kBinned ? 1u : 0u);
    if (big && direct) launch_k(scan_write_kernel<kScanRoundsMax, true, kBinned>, grid, kScanThreads, 0, stream, a, tiles);
    else if (big) launch_k(scan_write_kernel<kScanRoundsMax, false, kBinned>, grid, kScanThreads, 0, stream, a, tiles);
    else if (direct) launch_k(scan_write_kernel<1, true, kBinned>, grid, kScanThreads, 0, stream, a, tiles);
    else launch_k(scan_write_kernel<1, false, kBinned>, grid, kScanThreads, 0, stream, a, tiles);
}

// The scan of the tile totals that many tiles need, the downsweep, the binning; returns the launches.
int launch_scan_passes(const ScanArgs& a, cudaStream_t stream) {
    const bool big = a.n >= kScanBigScene;  // fewer, larger tiles
    const uint32_t per = big ? kScanTile : kScanTileSmall;
    const uint32_t tiles = (uint32_t)(((uint64_t)a.n + per - 1) / per);
    const bool direct = tiles <= kDirectTiles;
    if (!direct) launch_k(scan_tiles_kernel, 1, kTileScanThreads, 0, stream, a, tiles);
    if (a.bins) launch_scan_write<true>(a, tiles, big, direct, stream);
    else launch_scan_write<false>(a, tiles, big, direct, stream);
    if (a.bins) {
        const uint32_t blocks = (a.n + 255u) / 256u;
        launch_k(bin_survivors_kernel, blocks < 148u * 8u ? blocks : 148u * 8u, 256, 0, stream, a);
    }
    return (direct ? 1 : 2) + (a.bins ? 1 : 0);
}

int launch_scan_fused(const ScanArgs& a, cudaStream_t stream) {
    if (a.n == 0) {
        cudaMemsetAsync(a.counters, 0, sizeof(PassCounters), stream);
        return 0;
    }
    return launch_scan_passes(a, stream);
}

void launch_scan(const ScanArgs& a, uint32_t scan_tiles, cudaStream_t stream) {
    if (scan_tiles == 0 || a.n == 0) {
        cudaMemsetAsync(a.counters, 0, sizeof(PassCounters), stream);
        return;
    }
    if (a.n >= kScanBigScene)
        launch_k(scan_reduce_kernel<kScanRoundsMax>, (unsigned)(((uint64_t)a.n + kScanTile - 1) / kScanTile), kScanThreads, 0, stream, a);
    else
        launch_k(scan_reduce_kernel<1>, (unsigned)(((uint64_t)a.n + kScanTileSmall - 1) / kScanTileSmall), kScanThreads, 0, stream, a);
    launch_scan_passes(a, stream);
}

template <int K, bool kShares>
int splat_blocks_per_sm() {
    static int per_sm = 0;
    if (per_sm == 0) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, splat_kernel<K, kShares>, kSplatTile, 0);
        if (per_sm < 1) per_sm = 1;
    }
    return per_sm;
}

int splat_grid_size(int block) {
    (void)block;
    if (g_num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    }
    return g_num_sms * splat_blocks_per_sm<0, true>();
}

// The shared-memory pre-test needs bins of one tile (up to 8192 x 8192 pixels), a buffer that starts
// cleared, and the planes in an SM's 227 KB beside the rest of a block's shared memory.
constexpr int kBinnedMaxPasses = 13, kBinnedSmallPasses = 6;
constexpr int kSmemPerSm = 227 * 1024;
constexpr int kBinnedStatic = (int)(kBinnedGroup + kTileSize + 4u) * 4 + 1024;  // starts, table, the system's 1 KB

// Groups per block from which the shared-memory test takes a pass.  In blocks of 256 threads, two: with
// one (777k points at 1080p, 4 spp) it takes 111 us against 105, with more it wins (3.4M points: 271 against 333).
// In blocks of 1024, one (182k points at 8 spp: 100 us either way, 773k: 199 against 229).
constexpr uint32_t tile_test_groups(uint32_t threads) { return threads <= 256u ? 2u : 1u; }

template <int K, uint32_t kThreads>
bool launch_splat_binned(SplatArgs& a, int max_passes, cudaStream_t stream) {
    const int smem = a.fc.num_passes * (int)kNearPlane * 4;
    // (the limit is the device context's, so it is not remembered here; one value for all callers)
    if (!allow_dynamic_smem(reinterpret_cast<const void*>(splat_binned_kernel<K, kThreads>), max_passes * (int)kNearPlane * 4))
        return false;
    const int blocks = std::min(kThreads <= 256u ? 4 : 1, kSmemPerSm / (smem + kBinnedStatic));
    a.tile_test_from = (uint32_t)(g_num_sms * blocks) * kBinnedGroup * tile_test_groups(kThreads);
    launch_k(splat_binned_kernel<K, kThreads>, g_num_sms * blocks, kThreads, (size_t)smem, stream, a);
    return true;
}

template <int K>
bool launch_splat_binned(SplatArgs& a, cudaStream_t stream) {
    return a.fc.num_passes <= kBinnedSmallPasses ? launch_splat_binned<K, 256u>(a, kBinnedSmallPasses, stream)
                                                 : launch_splat_binned<K, 1024u>(a, kBinnedMaxPasses, stream);
}

template <int K, bool kShares>
void launch_splat_plain(const SplatArgs& a, cudaStream_t stream) {
    launch_k(splat_kernel<K, kShares>, g_num_sms * splat_blocks_per_sm<K, kShares>(), kSplatTile, 0, stream, a);
}

int launch_splat(const SplatArgs& args, int grid, int block, cudaStream_t stream) {
    (void)block;
    SplatArgs a = args;
    a.tile_test_from = kNoTileTest;
    int launches = 1;
    if (g_num_sms == 0) splat_grid_size(kSplatTile);
    if (a.sorted_gid && a.bin_is_tile && a.fresh && a.fc.use_unbiased && a.fc.num_passes <= kBinnedMaxPasses) {
        const int k = a.fc.k_points;
        if (k == 4 ? launch_splat_binned<4>(a, stream) : k == 2 ? launch_splat_binned<2>(a, stream)
            : k == 1 ? launch_splat_binned<1>(a, stream) : false)
            ++launches;
    }
    // a persistent grid: as many blocks as fit on the device at once
    const int k = a.fc.use_unbiased ? a.fc.k_points : 0;
    // Views of up to 2M samples: at the one or two points per 16 of them that scenes have, fewer points
    // than half the threads (320x180, ss 2, 4 spp: 0.9M samples, 28k points, 152k threads).  60k town, split /
    // not: 320x180 at 8 spp (1.8M) 63.9 / 72.1 us a frame, 640x360 at 1 spp (0.9M, four samples a point) 54.4 /
    // 53.1; 1280x720 at 2 spp (7.4M) 82.0 / 80.3, 960x540 at 4 spp (8.3M) 84.5 / 85.1.
    const bool small = (uint64_t)a.fc.up_width * (uint64_t)a.fc.up_height * (uint64_t)a.fc.num_passes <= (2u << 20) &&
                       a.fc.num_passes * k >= 4;
    if (k == 4) small ? launch_splat_plain<4, true>(a, stream) : launch_splat_plain<4, false>(a, stream);
    else if (k == 2) small ? launch_splat_plain<2, true>(a, stream) : launch_splat_plain<2, false>(a, stream);
    else if (k == 1) small ? launch_splat_plain<1, true>(a, stream) : launch_splat_plain<1, false>(a, stream);
    else if (k == 8) launch_splat_plain<8, false>(a, stream);
    else launch_k(splat_kernel<0, true>, grid, kSplatTile, 0, stream, a);
    return launches;
}

void launch_clear(uint64_t* buf, uint64_t entries, uint64_t value, cudaStream_t stream) {
    uint64_t pairs = entries / 2;
    int grid = (int)((pairs + 255) / 256);
    if (grid > 148 * 16) grid = 148 * 16;
    if (grid < 1) grid = 1;
    launch_k(clear_kernel, grid, 256, 0, stream, reinterpret_cast<ulonglong2*>(buf), pairs, value);
    if (entries & 1) cudaMemcpyAsync(buf + entries - 1, &buf[0], 8, cudaMemcpyDeviceToDevice, stream);
}

// The staged kernel of these sizes, if there is one: kPasses runs through 1..8 and the powers of two.
template <bool kDepthOnly, int kSsLog2, int kPasses = 1>
bool launch_resolve_staged(const ResolveArgs& a, const HizView& hiz, dim3 tiles, int ss_log2, cudaStream_t stream) {
    constexpr int kRun = kPasses << (2 * kSsLog2);
    if constexpr (kSsLog2 > 3) {
        return false;
    } else if constexpr (kRun > kResolveMaxRun) {
        return launch_resolve_staged<kDepthOnly, kSsLog2 + 1>(a, hiz, tiles, ss_log2, stream);
    } else {
        constexpr bool kPow2 = (kRun & (kRun - 1)) == 0;
        if constexpr (kRun > 1 && (kPow2 || kRun < 64)) {
            if (ss_log2 == kSsLog2 && a.num_passes == kPasses) {
                launch_k(resolve_staged_kernel<kDepthOnly, kSsLog2, kPasses>,
                         dim3(tiles.x << resolve_blocks_log2(kSsLog2, kRun), tiles.y), resolve_pixels(kRun), 0, stream, a, hiz);
                return true;
            }
        }
        return launch_resolve_staged<kDepthOnly, kSsLog2, (kPasses < 8 ? kPasses + 1 : kPasses * 2)>(a, hiz, tiles, ss_log2, stream);
    }
}

template <bool kDepthOnly, bool kHiz>
void launch_resolve_plain(const ResolveArgs& a, const HizView& h, dim3 tiles, int ss_log2, cudaStream_t stream) {
    if (ss_log2 >= 0) {
        const uint64_t threads = ((uint64_t)tiles.x * tiles.y) << (2 * (kTileBits - ss_log2));
        launch_k(resolve_morton_kernel<kDepthOnly, kHiz>, (unsigned)((threads + 255) / 256), 256, 0, stream, a, h, ss_log2);
        return;
    }
    const dim3 grid((a.width + 15) / 16, (a.height + 15) / 16);
    if (a.monotone && a.ss == 3) launch_k(resolve_kernel<kDepthOnly, 3, kHiz>, grid, 256, 0, stream, a, h);
    else launch_k(resolve_kernel<kDepthOnly, 0, kHiz>, grid, 256, 0, stream, a, h);
}

void launch_depth_monotone(float near_plane, float far_plane, uint32_t* falls, cudaStream_t stream) {
    depth_monotone_kernel<<<(unsigned)((kDepthMax + 1u) / kSweepKeys / 256u), 256, 0, stream>>>(near_plane, far_plane, falls);
}

template <bool kDepthOnly>
int launch_resolve_any(ResolveArgs a, const HizView* hiz, cudaStream_t stream) {
    int ss_log2 = -1;
    for (int l = 0; l <= 3; ++l)
        if (a.ss == (1 << l)) ss_log2 = l;
    const dim3 tiles((unsigned)((a.width * a.ss + kTileSize - 1) >> kTileBits), (unsigned)((a.height * a.ss + kTileSize - 1) >> kTileBits));
    // the fine Hi-Z levels need a chain of four levels and groups of 64 pixels, which the staged blocks
    // of more than 64 samples a pixel are not
    const int run = a.ss * a.ss * a.num_passes;
    const bool chain = hiz && hiz->levels >= 4;
    a.hiz_fused = chain && run != kResolveMaxRun ? 1 : 0;
    if (ss_log2 >= 0 && a.monotone && launch_resolve_staged<kDepthOnly, 0>(a, a.hiz_fused ? *hiz : HizView{}, tiles, ss_log2, stream))
        return a.hiz_fused;
    // unstaged runs: see resolve_morton_kernel (ss 8: a group of 64 pixels is a tile; 640x360, 3 spp, 580 us
    // with the levels, 560 without)
    const bool morton_fused = a.ss < 8 && (run <= 16 || (uint64_t)a.width * (uint64_t)a.height <= 148u * 2048u);
    a.hiz_fused = chain && (ss_log2 < 0 || morton_fused) ? 1 : 0;
    if (a.hiz_fused) launch_resolve_plain<kDepthOnly, true>(a, *hiz, tiles, ss_log2, stream);
    else launch_resolve_plain<kDepthOnly, false>(a, HizView{}, tiles, ss_log2, stream);
    return a.hiz_fused;
}

int launch_resolve(const ResolveArgs& a, const HizView* hiz, bool depth_only, cudaStream_t stream) {
    return depth_only ? launch_resolve_any<true>(a, hiz, stream) : launch_resolve_any<false>(a, hiz, stream);
}

void launch_hiz_build(const HizView& h, const float* depth, int min_levels, bool fine_done, cudaStream_t stream) {
    const int L = h.levels - 1;
    if (fine_done) {
        if (L == 3) return;
        launch_k(hiz_top_kernel, dim3((h.level_w[L - 3] + 15) / 16, (h.level_h[L - 3] + 15) / 16), 256, 0, stream, h, min_levels);
        return;
    }
    dim3 grid((h.level_w[L] + kHizTile - 1) / kHizTile, (h.level_h[L] + kHizTile - 1) / kHizTile);
    launch_k(hiz_build_kernel, grid, kHizThreads * kHizThreads, 0, stream, h, depth, min_levels);
}

void launch_encode_half(const float4* pos_op, const float4* rot, const float4* scale, const float4* sh, uint32_t n,
                        float4* origin, uint4* rec, uint4* scl, uint4* acq, cudaStream_t stream) {
    if (n == 0) return;
    const uint32_t blocks = (n + kHalfOriginBlock - 1) / kHalfOriginBlock;
    half_origins_kernel<<<(blocks + 255) / 256, 256, 0, stream>>>(pos_op, n, origin);
    encode_half_kernel<<<(n + 255) / 256, 256, 0, stream>>>(pos_op, rot, scale, sh, origin, n, rec, scl, acq);
}

void launch_translate_origins(const float4* src, uint32_t count, float dx, float dz, float4* dst, cudaStream_t stream) {
    if (count) translate_origins_kernel<<<(count + 255) / 256, 256, 0, stream>>>(src, count, dx, dz, dst);
}

void launch_tile_nodes(const float4* src, uint32_t src_pb, uint32_t src_n, uint32_t pb, uint32_t copies,
                       const float2* offsets, uint64_t total, float4* dst, uint32_t nodes, cudaStream_t stream) {
    if (nodes) tile_nodes_kernel<<<(nodes + 255) / 256, 256, 0, stream>>>(src, src_pb, src_n, pb, copies, offsets, total, dst, nodes);
}

void launch_block_bounds(const float4* pos_op, const float4* rot, const float4* scale, uint32_t n,
                         uint32_t per_block, float4* nodes, cudaStream_t stream) {
    uint32_t node_count = (n + per_block - 1) / per_block;
    if (node_count == 0) return;
    block_bounds_kernel<<<(node_count + 255) / 256, 256, 0, stream>>>(pos_op, rot, scale, n, per_block, nodes,
                                                                       node_count);
}

void launch_taa(uint8_t* image, float* out_color, const float* cur_color, const float* prev_color,
                const float* cur_depth, const float* prev_depth, const mat4& reproj, float blend, int width, int height,
                int frame_number, cudaStream_t stream) {
    if (frame_number <= 0) {
        const uint32_t values = 3u * (uint32_t)width * (uint32_t)height;
        const uintptr_t at = reinterpret_cast<uintptr_t>(out_color) | reinterpret_cast<uintptr_t>(cur_color);
        const int aligned = (at & 15u) == 0 && (reinterpret_cast<uintptr_t>(image) & 3u) == 0;
        launch_k(taa_first_kernel, (values + 1023u) / 1024u, 256, 0, stream, image, out_color, cur_color, values, aligned);
        return;
    }
    const dim3 grid((unsigned)((width + kTaaTile - 1) / kTaaTile), (unsigned)((height + kTaaHeight - 1) / kTaaHeight));
    launch_k(taa_kernel, grid, 256, 0, stream, image, out_color, cur_color, prev_color, cur_depth, prev_depth, reproj,
             blend, width, height);
}

void launch_progressive(uint8_t* image, float* cur_color, float* accum, int width, int height, int frames,
                        cudaStream_t stream) {
    int n = width * height;
    launch_k(progressive_kernel, (n + 255) / 256, 256, 0, stream, image, cur_color, accum, width, height, frames);
}

// ---------------------------------------------------------------------------------
// Allocation-free point scan.
//
// Some callers cannot allocate device memory at the moment they need the scan: code running
// inside a CUDA-graph capture or a stream-ordered pipeline where cudaMalloc would synchronise
// the device, a host with a fixed device-memory pool or budget enforced by its own allocator,
// or a plugin host that owns every buffer and forbids its plugins from allocating. For them
// the scan's only scratch — the survivor and point totals of every scan tile — lives
// in this file-scope device array, and the caller passes all inputs and outputs. The array is
// shared by every call on a device and keeps the previous call's contents; each call rewrites
// every word it reads before reading it (tile totals, then prefixes); calls that overlap on the GPU
// (different streams, or host threads on the same device) race on it and must be serialised.
// ---------------------------------------------------------------------------------
constexpr uint32_t kNoAllocScanMaxTiles = 65536;  // 512 KiB of tile words
constexpr uint64_t kNoAllocScanMaxGaussians = 1ull << 28;  // the stated limit
static_assert(kNoAllocScanMaxGaussians / kScanTileSmall <= kNoAllocScanMaxTiles, "scratch too small");
static __device__ __align__(256) unsigned long long g_noalloc_scan_scratch[kNoAllocScanMaxTiles + 1];

namespace {
// The array's device address belongs to the module as loaded into one CUDA context: a driver
// API context other than the device's primary one, or the primary context re-created after
// cudaDeviceReset, loads the module again at another address.  So the cache is keyed on the
// current context's ID (cuCtxGetId: unique for the life of the process, never reused), fetched
// through the runtime's driver entry points so the library needs no libcuda link.
struct NoAllocScratchEntry {
    unsigned long long ctx_id;
    unsigned long long* ptr;
};
constexpr int kNoAllocCacheSlots = 64;
std::mutex g_noalloc_mutex;
NoAllocScratchEntry g_noalloc_cache[kNoAllocCacheSlots] = {};
int g_noalloc_cache_next = 0;
using CuCtxGetCurrentFn = int (*)(void**);
using CuCtxGetIdFn = int (*)(void*, unsigned long long*);

bool current_context_id(unsigned long long& id) {
    static CuCtxGetCurrentFn get_current = nullptr;
    static CuCtxGetIdFn get_id = nullptr;
    if (!get_current || !get_id) {
        void* f0 = nullptr;
        void* f1 = nullptr;
        cudaDriverEntryPointQueryResult q0, q1;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f0, cudaEnableDefault, &q0) != cudaSuccess ||
            q0 != cudaDriverEntryPointSuccess || !f0)
            return false;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f1, cudaEnableDefault, &q1) != cudaSuccess ||
            q1 != cudaDriverEntryPointSuccess || !f1)
            return false;
        get_current = reinterpret_cast<CuCtxGetCurrentFn>(f0);
        get_id = reinterpret_cast<CuCtxGetIdFn>(f1);
    }
    void* ctx = nullptr;
    if (get_current(&ctx) != 0 || !ctx) return false;
    return get_id(ctx, &id) == 0;
}
}  // namespace

}  // namespace gps

extern "C" gps_status gps_workload_scan_noalloc(const uint32_t* d_counts, const uint32_t* d_mask, uint32_t n,
                                                uint32_t max_points, uint32_t* d_surv_gid, uint32_t* d_surv_start,
                                                uint32_t* d_tile_first_rank, uint32_t* d_counters8, void* stream) {
    using namespace gps;
    const uint64_t tiles64 = ((uint64_t)n + kScanTile - 1) / kScanTile;
    if ((uint64_t)n > kNoAllocScanMaxGaussians) {
        set_last_error("gps_workload_scan_noalloc: " + std::to_string(n) + " Gaussians exceed the fixed scratch's limit of " +
                       std::to_string((unsigned long long)kNoAllocScanMaxGaussians) + " Gaussians");
        return GPS_ERR_SIZE;
    }
    const uint32_t tiles = (uint32_t)tiles64;
    if ((n && (!d_counts || !d_mask || !d_surv_gid || !d_surv_start)) || !d_tile_first_rank || !d_counters8) {
        set_last_error("gps_workload_scan_noalloc: null argument");
        return GPS_ERR_INVALID_ARGUMENT;
    }
    if ((reinterpret_cast<uintptr_t>(d_counts) & 15u) != 0 || (reinterpret_cast<uintptr_t>(d_counters8) & 3u) != 0) {
        set_last_error("gps_workload_scan_noalloc: d_counts must be 16-byte aligned, d_counters8 4-byte aligned");
        return GPS_ERR_INVALID_ARGUMENT;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        set_last_error(std::string("gps_workload_scan_noalloc: no usable current device: ") + cudaGetErrorString(e));
        return GPS_ERR_CUDA;
    }
    // An error left pending by earlier, unrelated work is reported as such and left in place
    // for the caller's own check; it is not taken for a failure of this scan.
    e = cudaPeekAtLastError();
    if (e != cudaSuccess) {
        set_last_error(std::string("gps_workload_scan_noalloc: a CUDA error from earlier work is pending: ") +
                       cudaGetErrorString(e));
        return GPS_ERR_CUDA;
    }
    unsigned long long* scratch = nullptr;
    {
        // Once per context, with it current: the host-side name of a __device__ array is not a
        // device address, the address must be looked up.
        unsigned long long ctx_id = 0;
        const bool have_id = current_context_id(ctx_id);
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (have_id)
            for (const NoAllocScratchEntry& en : g_noalloc_cache)
                if (en.ptr && en.ctx_id == ctx_id) scratch = en.ptr;
        if (!scratch) {
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_scan_scratch);
            if (e != cudaSuccess) {
                set_last_error(std::string("gps_workload_scan_noalloc: cudaGetSymbolAddress failed: ") + cudaGetErrorString(e));
                return GPS_ERR_CUDA;
            }
            scratch = static_cast<unsigned long long*>(p);
            if (have_id) {  // without a context ID the address is looked up on every call
                g_noalloc_cache[g_noalloc_cache_next] = {ctx_id, scratch};
                g_noalloc_cache_next = (g_noalloc_cache_next + 1) % kNoAllocCacheSlots;
            }
        }
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    ScanArgs a{};
    a.counts = d_counts;
    a.mask = d_mask;
    a.n = n;
    a.max_points = max_points;
    a.tile_points = 256;
    a.surv_gid = d_surv_gid;
    a.surv_start = d_surv_start;
    a.tile_first_rank = d_tile_first_rank;
    a.tile_state = scratch;
    a.counters = reinterpret_cast<PassCounters*>(d_counters8);
    launch_scan(a, tiles, st);  // writes every tile word and all eight counters
    e = cudaGetLastError();  // nothing was pending before the launches: this is theirs
    if (e != cudaSuccess) {
        set_last_error(std::string("gps_workload_scan_noalloc: ") + cudaGetErrorString(e));
        return GPS_ERR_CUDA;
    }
    return GPS_OK;
}

// ---------------------------------------------------------------------------------
// Scene order on the device: 3D Morton order of the Gaussian means, the same order as the host
// reorder (host_scene.cpp morton_sort: keys from the scene's bounding box, 21 bits per axis,
// a stable sort), computed with round-to-nearest arithmetic so that every key is the host's.
// ---------------------------------------------------------------------------------
#include <cub/device/device_radix_sort.cuh>

namespace gps {
namespace {

__device__ __forceinline__ uint32_t ordered_bits(float f) {  // monotone float -> uint32 map
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_ordered_bits(uint32_t b) {
    return __uint_as_float((b & 0x80000000u) ? (b & 0x7FFFFFFFu) : ~b);
}

__global__ void __launch_bounds__(256) mean_bounds_kernel(const float4* __restrict__ pos, uint32_t n,
                                                          uint32_t* __restrict__ bounds6) {
    uint32_t lo[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, hi[3] = {0u, 0u, 0u};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 p = __ldg(pos + i);
        const float f[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (f[c] != f[c]) continue;  // NaN never wins the host's comparisons
            const uint32_t v = ordered_bits(f[c]);
            lo[c] = min(lo[c], v);
            hi[c] = max(hi[c], v);
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[c] = min(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
            hi[c] = max(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
        }
        if ((threadIdx.x & 31u) == 0u) {
            atomicMin(bounds6 + c, lo[c]);
            atomicMax(bounds6 + 3 + c, hi[c]);
        }
    }
}

__device__ __forceinline__ uint64_t spread21(uint32_t v) {  // bit b -> bit 3b
    uint64_t x = v & 0x1FFFFFu;
    x = (x | (x << 32)) & 0x1F00000000FFFFull;
    x = (x | (x << 16)) & 0x1F0000FF0000FFull;
    x = (x | (x << 8)) & 0x100F00F00F00F00Full;
    x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

__global__ void __launch_bounds__(256) morton_keys_kernel(const float4* __restrict__ pos, uint32_t n,
                                                          const uint32_t* __restrict__ bounds6,
                                                          unsigned long long* __restrict__ keys,
                                                          uint32_t* __restrict__ index) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = __ldg(pos + i);
    const float v[3] = {p.x, p.y, p.z};
    uint32_t q[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float mn = from_ordered_bits(bounds6[c]), mx = from_ordered_bits(bounds6[3 + c]);
        const float den = __fsub_rn(mx, mn), num = __fsub_rn(v[c], mn);
        const float rel = den != 0.0f ? __fdiv_rn(num, den) : 0.0f;
        q[c] = (uint32_t)__float2int_rz(__fmul_rn(rel, (float)((1 << 21) - 1)));
    }
    keys[i] = spread21(q[0]) | (spread21(q[1]) << 1) | (spread21(q[2]) << 2);
    index[i] = i;
}

template <class T>
__global__ void __launch_bounds__(256) gather_kernel(const T* __restrict__ src, const uint32_t* __restrict__ order,
                                                     uint32_t n, uint32_t per, T* __restrict__ dst) {
    const uint64_t total = (uint64_t)n * per;
    for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < total; j += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = j / per, k = j - i * per;
        dst[j] = __ldg(src + (uint64_t)__ldg(order + i) * per + k);
    }
}

}  // namespace

cudaError_t morton_order_device(const float4* pos, uint32_t n, uint32_t* order, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    uint32_t* bounds6 = nullptr;
    unsigned long long *keys = nullptr, *keys_out = nullptr;
    uint32_t* index = nullptr;
    void* temp = nullptr;
    size_t temp_bytes = 0;
    const uint32_t init[6] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u, 0u};
    cudaError_t e = cudaMalloc(&bounds6, 6 * sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&keys, (size_t)n * 8);
    if (e == cudaSuccess) e = cudaMalloc(&keys_out, (size_t)n * 8);
    if (e == cudaSuccess) e = cudaMalloc(&index, (size_t)n * 4);
    if (e == cudaSuccess) e = cudaMemcpyAsync(bounds6, init, sizeof(init), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        mean_bounds_kernel<<<148 * 8, 256, 0, st>>>(pos, n, bounds6);
        morton_keys_kernel<<<(n + 255) / 256, 256, 0, st>>>(pos, n, bounds6, keys, index);
        e = cudaGetLastError();
    }
    // 63 key bits; the radix sort is stable, so equal keys keep their input order as the
    // host's std::stable_sort does
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(nullptr, temp_bytes, keys, keys_out, index, order, (int)n, 0, 63, st);
    if (e == cudaSuccess) e = cudaMalloc(&temp, temp_bytes);
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairs(temp, temp_bytes, keys, keys_out, index, order, (int)n, 0, 63, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(temp);
    cudaFree(index);
    cudaFree(keys_out);
    cudaFree(keys);
    cudaFree(bounds6);
    return e;
}

void launch_gather_rows(const float4* src, const uint32_t* order, uint32_t n, uint32_t per, float4* dst, cudaStream_t st) {
    if (n) gather_kernel<float4><<<148 * 8, 256, 0, st>>>(src, order, n, per, dst);
}

}  // namespace gps
