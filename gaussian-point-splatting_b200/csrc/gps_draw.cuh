// The unbiased splat's sample draw: one sample in the reference's form, and one or two at a time in
// the paired instructions of sm_100 (gaussian_point_splatting.cu:67-141, random.cuh:110-141).
#pragma once
#include "frame_kernels.h"
#include "gps_rng.cuh"

namespace gps {

// Samples are drawn without branches (bounds and alpha tests become predicates), so that the
// independent transcendental chains of several interleave, then the live ones are splatted.
struct SampleConst {
    vec2 pixel_mean;
    float c0, c1, c2, opacity, inv_alpha, li2_alpha;
    vec3 conic;
    int minx, miny, maxx, maxy;
    uint32_t span_x, span_y;  // max(maxx - minx, 0), max(maxy - miny, 0)
    int tiles_per_row, passes;
    uint32_t tile_bias;      // added to every tile index below, and taken off again with the slot
    uint32_t slot_bias;
    const uint32_t* spread;  // shared-memory Morton table (null: codes are computed)
};

// Adding 1.5 * 2^23 with rounding down leaves floor(v) in the low mantissa bits for |v| < 2^22:
// floor and conversion in one addition that pairs.  Outside that range the bits, less
// kFloorBits, are at least 200,000 as an unsigned number, so that no bounds test passes.
constexpr float kFloorMagic = 12582912.0f;
constexpr uint32_t kFloorBits = 0x4B400000u;

GPS_D float2 both(float v) { return make_float2(v, v); }

// floor(v) + kFloorBits, v below 2^22 in magnitude.
GPS_D float floor_bits(float v) { return __fadd_rd(v, kFloorMagic); }
GPS_D float2 floor_bits2(float2 v) { return __fadd2_rd(v, both(kFloorMagic)); }

// Minus the square root of -m, for m = 0 and m from -171 to -1e-7: the reciprocal root's product with
// one correction step in the residual m + g^2 (P. Markstein, Computation of elementary functions on the
// IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990), which is __fsqrt_rn's result for every
// float there; a root of zero comes out as -0, which changes no sum that it goes into.
GPS_D float neg_root(float m) {
    const float rs = rsqrtf(fmaxf(-m, 1.0e-30f)), ng = __fmul_rn(m, rs);
    return __fmaf_rn(__fmaf_rn(ng, ng, m), __fmul_rn(0.5f, rs), ng);
}
GPS_D float2 neg_root2(float2 m) {
    const float2 rs = make_float2(rsqrtf(fmaxf(-m.x, 1.0e-30f)), rsqrtf(fmaxf(-m.y, 1.0e-30f)));
    const float2 ng = __fmul2_rn(m, rs);
    return __ffma2_rn(__ffma2_rn(ng, ng, m), __fmul2_rn(both(0.5f), rs), ng);
}

// v / kLi2Max, v from 0 to 2, as inv_dilog divides it: the product with the reciprocal is equal.
GPS_D float2 by_li2_max2(float2 v) { return __fmul2_rn(v, both(1.0f / kLi2Max)); }

// The Morton code in its tile of a pixel: two loads from a 64-entry shared-memory table of spread
// 6-bit coordinates instead of two 4-step bit spreads (16M town, 1080p, ss 2, 4 spp: splat 1.90 vs 1.96
// ms/frame).  (The null test folds away where the kernel has a table.)
GPS_D uint32_t morton_code(const SampleConst& c, uint32_t x, uint32_t y) {
    x &= kTileSize - 1;
    y &= kTileSize - 1;
    return c.spread ? c.spread[x] | (c.spread[y] << 1) : morton_encode(x, y);
}

// One sample: whether it is live, its splat-buffer tile (plus c.tile_bias) and the Morton code of its
// place there.
GPS_D bool draw_sample(u32x2& seed, const SampleConst& c, uint32_t& tile, uint32_t& code) {
    const vec2 u = pcg2d(seed);
    float a = c.inv_alpha * inv_dilog((1.0f - u.x) * c.li2_alpha);
    a = gclamp(a, 1.e-37f, 1.0f);
    const float r = __fsqrt_rn(fmaxf(-2.0f * __logf(a), 0.0f));
    const float theta = 2.0f * kPiF * u.y;
    float sn, cs;
    __sincosf(theta, &sn, &cs);
    const vec2 xy = make_v2(r * cs, r * sn);
    vec2 pixel = make_v2(c.pixel_mean.x + c.c0 * xy.x, c.pixel_mean.y + c.c1 * xy.x + c.c2 * xy.y);
    pixel = make_v2(floorf(pixel.x), floorf(pixel.y));
    const int x = (int)pixel.x;
    const int y = (int)pixel.y;
    const vec2 delta = make_v2(c.pixel_mean.x - pixel.x, c.pixel_mean.y - pixel.y);
    // minx <= x < maxx as one unsigned compare (x - minx wraps to a large value below minx):
    // splat 1.572 -> 1.563 ms/frame on the 16M orbit
    const bool inside = ((uint32_t)x - (uint32_t)c.minx < c.span_x) & ((uint32_t)y - (uint32_t)c.miny < c.span_y);
    const float alpha = c.opacity * gaussian_value(c.conic, delta);
    code = morton_code(c, (uint32_t)x, (uint32_t)y);
    tile = (uint32_t)((y >> kTileBits) * c.tiles_per_row + (x >> kTileBits)) + c.tile_bias;
    return inside & !(alpha < 1.0f / 255.0f);
}

// Two samples drawn together: the random words come off the seed in stream order, and the
// floating-point steps the two share (the opacity-corrected inverse dilog polynomial, the square
// root, the Box-Muller products, the pixel position and its offset, the Gaussian weight) run as
// sm_100 paired FP32 instructions (FFMA2 / FMUL2 / FADD2), each lane rounded as the scalar
// instruction would.  The transcendental and per-lane steps stay scalar.  Same values as
// draw_sample, bit for bit, where wide_sample(c) is false:
//   - the square root is neg_root, whose radicand here is 0 or between 1e-7 and 171 (__logf is nowhere
//     positive from 1e-37 to 1), and the division by kLi2Max a product (the tests sweep all floats
//     of these ranges through both, through __logf and through floor_bits)
//   - the root, the offset and the mixed conic term are kept with the opposite sign where that
//     saves a negation: products of two of them, and sums, only change sign with it
// With the pairing alone the draw took 117 instructions a sample, floor and conversion on the
// conversion unit and the root through the compiler's sequence; now 104 (4M town, both passes: 385 ->
// 340 million warp instructions, pass 2 160 -> 152 us, frame 846 -> 827; 33.6M town 1180 -> 1143). The
// first pass is by now bound by its atomics: 61M random ones in 368 us, of the 185 G/s that L2 does.
GPS_D void draw_pair(u32x2& seed, const SampleConst& c, uint32_t* tile, uint32_t* code, bool* live) {
    const u32x2 s0 = pcg2d_step(seed);
    const u32x2 s1 = pcg2d_step(s0);
    seed = s1;
    const float2 nux = __fmul2_rn(make_float2((float)s0.x, (float)s1.x), both(-kRecip2e32));
    const float2 uy = __fmul2_rn(make_float2((float)s0.y, (float)s1.y), both(kRecip2e32));
    // inv_dilog((1 - u.x) * Li2(alpha)) (random.cuh:110-127, 132-141)
    const float2 x = by_li2_max2(__fmul2_rn(__fadd2_rn(both(1.0f), nux), both(c.li2_alpha)));
    const float2 t = make_float2(fminf(x.x, 1.0f), fminf(x.y, 1.0f));
    float2 y = both(-1.27463503e+01f);
    y = __ffma2_rn(y, t, both(5.88993459e+01f));
    y = __ffma2_rn(y, t, both(-1.16025780e+02f));
    y = __ffma2_rn(y, t, both(1.26945827e+02f));
    y = __ffma2_rn(y, t, both(-8.43108826e+01f));
    y = __ffma2_rn(y, t, both(3.48799862e+01f));
    y = __ffma2_rn(y, t, both(-8.89606235e+00f));
    y = __ffma2_rn(y, t, both(1.38640936e+00f));
    y = __ffma2_rn(y, t, both(-7.80640876e-01f));
    y = __ffma2_rn(y, t, both(1.64841888e+00f));
    y = __ffma2_rn(y, t, both(-2.82836687e-05f));
    const float2 a2 = __fmul2_rn(both(c.inv_alpha), y);
    // minus the radicand -2 log(a) (scaling by 2 is exact) and minus its root
    const float2 m = __fmul2_rn(both(2.0f), make_float2(__logf(gclamp(a2.x, 1.e-37f, 1.0f)), __logf(gclamp(a2.y, 1.e-37f, 1.0f))));
    const float2 nr = neg_root2(m);
    const float2 th = __fmul2_rn(both(2.0f * kPiF), uy);
    float sn[2], cs[2];
    __sincosf(th.x, &sn[0], &cs[0]);
    __sincosf(th.y, &sn[1], &cs[1]);
    const float2 nxyx = __fmul2_rn(nr, make_float2(cs[0], cs[1]));
    const float2 nxyy = __fmul2_rn(nr, make_float2(sn[0], sn[1]));
    const float2 px = __ffma2_rn(both(-c.c0), nxyx, both(c.pixel_mean.x));
    const float2 py = __ffma2_rn(both(-c.c2), nxyy, __ffma2_rn(both(-c.c1), nxyx, both(c.pixel_mean.y)));
    const float2 bx = floor_bits2(px), by = floor_bits2(py);
    // minus the offset pixel_mean - floor(pixel)
    const float2 ndx = __ffma2_rn(both(c.pixel_mean.x), both(-1.0f), __fadd2_rn(bx, both(-kFloorMagic)));
    const float2 ndy = __ffma2_rn(both(c.pixel_mean.y), both(-1.0f), __fadd2_rn(by, both(-kFloorMagic)));
    // gaussian_value (linalg.cuh:309-317) on both samples.  Its sums of two products are fused
    // as the compiler contracts them, the left product into the FMA: x*x-part first
    // (fma(cx dx, dx, (cz dy) dy)), then fma(-0.5, quad, -((cy dx) dy)).  The tests pin this:
    // fusing the right-hand products instead changed one entry of the 4K parity case.
    const float2 quad = __ffma2_rn(__fmul2_rn(both(c.conic.x), ndx), ndx, __fmul2_rn(__fmul2_rn(both(c.conic.z), ndy), ndy));
    const float2 nhh = __fmul2_rn(__fmul2_rn(both(-c.conic.y), ndx), ndy);
    const float2 sig = __ffma2_rn(both(-0.5f), quad, nhh);
    const float2 gv = make_float2(sig.x > 0.f ? 0.0f : __expf(sig.x), sig.y > 0.f ? 0.0f : __expf(sig.y));
    const float2 al = __fmul2_rn(both(c.opacity), gv);
#pragma unroll
    for (int l = 0; l < 2; ++l) {
        const uint32_t xb = __float_as_uint(l ? bx.y : bx.x), yb = __float_as_uint(l ? by.y : by.x);  // pixel + kFloorBits
        const bool inside = (xb - (kFloorBits + (uint32_t)c.minx) < c.span_x) & (yb - (kFloorBits + (uint32_t)c.miny) < c.span_y);
        code[l] = morton_code(c, xb, yb);
        tile[l] = (yb >> kTileBits) * (uint32_t)c.tiles_per_row + (xb >> kTileBits);  // plus c.tile_bias
        live[l] = inside & !((l ? al.y : al.x) < 1.0f / 255.0f);
    }
}

// One sample the same way (not where wide_sample(c)).
GPS_D bool draw_one(u32x2& seed, const SampleConst& c, uint32_t& tile, uint32_t& code) {
    const vec2 u = pcg2d(seed);
    const float a = c.inv_alpha * inv_dilog((1.0f - u.x) * c.li2_alpha);
    const float m = 2.0f * __logf(gclamp(a, 1.e-37f, 1.0f));
    const float nr = neg_root(m);
    float sn, cs;
    __sincosf(2.0f * kPiF * u.y, &sn, &cs);
    const float nx = __fmul_rn(nr, cs), ny = __fmul_rn(nr, sn);
    const float bx = floor_bits(__fmaf_rn(-c.c0, nx, c.pixel_mean.x));
    const float by = floor_bits(__fmaf_rn(-c.c2, ny, __fmaf_rn(-c.c1, nx, c.pixel_mean.y)));
    const float dx = __fsub_rn(c.pixel_mean.x, __fadd_rn(bx, -kFloorMagic)), dy = __fsub_rn(c.pixel_mean.y, __fadd_rn(by, -kFloorMagic));
    const float quad = __fmaf_rn(__fmul_rn(c.conic.x, dx), dx, __fmul_rn(__fmul_rn(c.conic.z, dy), dy));
    const float sig = __fmaf_rn(-0.5f, quad, -__fmul_rn(__fmul_rn(c.conic.y, dx), dy));
    const float alpha = c.opacity * (sig > 0.f ? 0.0f : __expf(sig));
    const uint32_t xb = __float_as_uint(bx), yb = __float_as_uint(by);
    code = morton_code(c, xb, yb);
    tile = (yb >> kTileBits) * (uint32_t)c.tiles_per_row + (xb >> kTileBits);
    return (xb - (kFloorBits + (uint32_t)c.minx) < c.span_x) & (yb - (kFloorBits + (uint32_t)c.miny) < c.span_y) &
           !(alpha < 1.0f / 255.0f);
}

GPS_D SampleConst sample_const(const SplatRecord& rec, const FrameConst& fc, const uint32_t* spread) {
    SampleConst c;
    c.spread = spread;
    c.pixel_mean = make_v2(rec.a.x, rec.a.y);
    c.c0 = rec.a.z;
    c.c1 = rec.a.w;
    c.c2 = rec.b.x;
    c.conic = make_v3(rec.b.y, rec.b.z, rec.b.w);
    c.opacity = rec.c.x;
    c.minx = (int)(rec.d.x & 0xFFFFu);
    c.miny = (int)(rec.d.x >> 16);
    c.maxx = (int)(rec.d.y & 0xFFFFu);
    c.maxy = (int)(rec.d.y >> 16);
    c.span_x = (uint32_t)max(c.maxx - c.minx, 0);
    c.span_y = (uint32_t)max(c.maxy - c.miny, 0);
    // the per-Gaussian factors of correctedBoxMuller (random.cuh:132-141), evaluated once
    c.inv_alpha = 1.0f / fmaxf(c.opacity, 1.e-37f);
    c.li2_alpha = dilog(c.opacity);
    c.passes = fc.num_passes;
    c.tiles_per_row = (fc.up_width + kTileSize - 1) >> kTileBits;
    c.tile_bias = (kFloorBits >> kTileBits) * ((uint32_t)c.tiles_per_row + 1u);
    c.slot_bias = 0u - c.tile_bias * (uint32_t)(kTileSize * kTileSize) * (uint32_t)c.passes;
    return c;
}

// Means or factors for which a pixel position may overflow or be no number: draw_pair leaves those
// to draw_sample, whose conversion takes a NaN to pixel 0.
GPS_D bool wide_sample(const SampleConst& c) {
    const float sum = fabsf(c.c0) + fabsf(c.c1) + fabsf(c.c2) + fabsf(c.pixel_mean.x) + fabsf(c.pixel_mean.y);
    return __float_as_uint(sum) >= __float_as_uint(1.0e30f);  // (by the bits: a NaN too)
}

GPS_D uint32_t sample_slot(const SampleConst& c, uint32_t tile, uint32_t code, int p) {
    return (tile * (uint32_t)(kTileSize * kTileSize) + code) * (uint32_t)c.passes + ((uint32_t)p + c.slot_bias);
}

}  // namespace gps
